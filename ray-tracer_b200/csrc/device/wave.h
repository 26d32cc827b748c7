#pragma once
// Host-visible launch interface of the sm_100a kernels (kernels.cu). Plain C++:
// no CUDA syntax, so the C++20 host code can include it.
#include <cstddef>
#include <cstdint>

#include <cuda_runtime_api.h>

#include "device/layout.h"

namespace rtg {

// Path slots resident per SM, at most: the paths left over by an iteration are no
// more than this times the SMs.
constexpr int kMaxPathsPerSm = 4096;

// Device buffers of one continuous wavefront (iterations of at most `capacity`
// paths) and the segment tables it draws new paths from.
struct WaveBuffers {
  // Paths left from one iteration to the next, by parity: min(capacity,
  // kMaxPathsPerSm * SMs) records.
  float4* st_a[2];
  float4* st_b[2];
  float4* st_c[2];
  uint4* st_d[2];
  float4* st_e[2];
  float4* radiance;            // one float4 per sample of every open segment
  WaveCounters* cnt;
  const RtgSceneDev* jobs;     // job descriptors, indexed by job slot
  const DevSegment* segs;      // indexed by segment slot
  SegmentProgress* seg_prog;   // indexed by segment slot
  const GenTable* gen;         // host-written generation order
  GenPlan* plan;               // this iteration's generation plan
  WaveSnapshot* ring;          // pinned, host-mapped snapshot ring
  std::uint32_t ring_size;
  std::uint32_t capacity;      // paths an iteration may hold
};

struct LaunchShape {
  int extend_blocks = 0;   // grid of the path kernel (0 = every resident block)
  int shade_blocks = 0, shadow_blocks = 0;  // kept for rtg_tuning; no kernel uses them
  int block = 128;         // threads per block of the path kernel: 64, 128 or 256
  bool chained = true;     // programmatic dependent launch between the wavefront kernels
  bool mis = false;        // a job with multiple importance sampling is open (kernel variant)
  bool general = false;    // counting, an eight-wide walk, or a brute-force job: the general variant
  int closest_tree = 2;    // closest-hit walk: 2 the binary tree, 8 the compressed eight-wide tree
  int shadow_tree = 4;     // any-hit walk: 4 the four-wide tree, 8 the compressed eight-wide tree
};

// The two launches of a wavefront iteration on `stream`, in this order; `parity`
// alternates 0/1 between iterations.
cudaError_t launch_plan(const WaveBuffers& wb, int parity, const LaunchShape& shape, cudaStream_t stream);
cudaError_t launch_paths(const WaveBuffers& wb, int parity, const LaunchShape& shape, cudaStream_t stream);

// Per-pixel reduction of finished passes into their job's framebuffer.
cudaError_t launch_accumulate(const RtgSceneDev* job_dev, std::uint64_t pixels, const PassList& passes,
                              const float4* radiance, cudaStream_t stream);

// Direct (Whitted) integrator over whole passes. Writes each sample's radiance slot.
// `by_warp` takes the kernel that schedules samples by warps, which is the faster one
// where direct_by_warp says so; else a thread traces a sample. The former's `pending`
// holds direct_pending_bytes(SMs, pending_depth) bytes for the samples' pending refraction
// branches, pending_depth of them a sample (direct_pending_depth of the job's maximum
// depth; 0 for a scene without dielectrics, whose samples have none).
// `general`: an eight-wide walk (tree 8) or brute force.
bool direct_by_warp(std::uint64_t samples);
int direct_pending_depth(int max_depth);
std::size_t direct_pending_bytes(int sms, int pending_depth);
cudaError_t launch_direct(const RtgSceneDev* job_dev, const PassList& passes, float4* radiance, WaveCounters* cnt,
                          bool by_warp, float4* pending, int pending_depth, bool general, int tree, cudaStream_t stream);

// Framebuffer means (mean_out, 3 doubles per pixel) and/or their tone-mapped
// sRGB encoding (rgb8, 3 bytes per pixel), each 16-byte aligned, in device or pinned
// host memory; either output may be null.
cudaError_t launch_resolve(const double* fb_sum, const std::uint32_t* fb_count, std::uint64_t pixels, int tone_map,
                           double exposure, std::uint8_t* rgb8, double* mean_out, cudaStream_t stream);

// Ray queries for parity tests and the ray API. rays: 2 float4 per ray
// (origin, tmin), (direction, tmax). Rays and results may be in pinned host memory.
// tree: 8 walks the eight-wide tree; otherwise the binary tree (closest hit) or
// the four-wide tree (any hit).
struct RayResults {
  float* t;
  std::int32_t* prim;
  std::int32_t* plane;
  float2* bary;
};
cudaError_t launch_ray_closest(const RtgSceneDev* job_dev, const float4* rays, std::uint32_t n, const RayResults& out,
                               int brute, int tree, cudaStream_t stream);
cudaError_t launch_ray_any(const RtgSceneDev* job_dev, const float4* rays, std::uint32_t n, std::uint8_t* out,
                           int brute, int tree, cudaStream_t stream);

}  // namespace rtg
