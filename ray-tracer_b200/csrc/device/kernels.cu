// Wavefront path tracer for sm_100a.
//
// One iteration over a list of at most `capacity` paths:
//   k_plan — one block: decides which open segments (passes of renders) the new
//            paths come from, in the host's priority order, and copies the
//            counters and segment progress to the pinned snapshot ring;
//   k_path — generates the camera paths (thin-lens generation,
//            src/rendering/renderer.cpp:33-37 + include/raytracer/core/camera.hpp:54-62)
//            and traces them: closest hits (Scene::intersect), emission, material
//            sampling, next-event estimation and Russian roulette
//            (src/rendering/integrator.cpp:97-139) and shadow rays
//            (Scene::occluded). Each warp is a small wavefront of its own (see
//            there); when the list is used up and more work is open, the paths
//            in flight are left for the next iteration.
// Every path owns one radiance slot addressed by (segment, pixel, sample-in-pass)
// and adds to its radiance in path order, so the result does not depend on
// scheduling, batch composition or timing. Paths that end count themselves done in
// their segment's progress record; once a segment is done, k_accumulate folds each
// pixel's samples into the double framebuffer in sample order (Framebuffer::add,
// include/raytracer/rendering/framebuffer.hpp:31), passes of one render in order.
#include <cfloat>
#include <map>
#include <mutex>

#include "device/shade.cuh"
#include "device/wave.h"

namespace rtg {

namespace {

constexpr float kRayTMin = 1e-6f;  // include/raytracer/math/ray.hpp:45
constexpr int kStackSmem = 8;  // stack entries per thread in shared memory (8 measured 1% faster than 16 or 24)
constexpr int kPathStack = 6;  // the same for the path kernel, whose path slots need the room (6 and 8 measure alike)
constexpr int kPathThreads = 896;  // threads per SM the path kernel is compiled for (72 registers)
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ std::uint64_t ld_u64(std::uint32_t lo, std::uint32_t hi) {
  return static_cast<std::uint64_t>(lo) | (static_cast<std::uint64_t>(hi) << 32);
}

__device__ __forceinline__ void warp_add_u64(std::uint64_t v, std::uint64_t* dst) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(kFull, v, off);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(reinterpret_cast<unsigned long long*>(dst), static_cast<unsigned long long>(v));
}

// Programmatic dependent launch: each wavefront kernel lets the next one be
// scheduled at once (its blocks take SM slots as this grid's blocks exit) and
// waits for the previous grid's completion and memory before touching any data.
__device__ __forceinline__ void chain_to_previous_grid() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct CameraSample {
  float3 o, d;
  Pcg rng;
  std::uint32_t sample;  // radiance slot
};

// Camera ray for local sample `local` of a segment, numbered pixel-major
// (local = pixel * pass_spp + (s - pass_s0)): a warp's new paths are samples of
// the same few pixels, which keeps their walks (and their later bounces) coherent;
// numbering sample-major measured 17% slower in the closest-hit stage.
// Jitter (2 draws), then the lens (2 draws). A segment holds fewer than 2^32 samples.
// The ray's rounding is pinned (explicit FMAs and unfused products), so every
// instance of the kernel generates the same bits.
__device__ __forceinline__ CameraSample camera_sample(const RtgSceneDev& J, const DevSegment& S, std::uint64_t local) {
  CameraSample cs;
  const std::uint32_t spp = S.pass_spp;
  const std::uint32_t l32 = static_cast<std::uint32_t>(local);
  const std::uint32_t pixel = l32 / spp;
  const std::uint32_t s = S.pass_s0 + (l32 - pixel * spp);
  const std::uint32_t px = static_cast<std::uint32_t>(pixel % static_cast<std::uint32_t>(J.width));
  const std::uint32_t py = static_cast<std::uint32_t>(pixel / static_cast<std::uint32_t>(J.width));
  cs.rng = Pcg::for_sample(J.seed, pixel, s);
  const float jx = cs.rng.uniform();
  const float jy = cs.rng.uniform();
  const float sx = __fadd_rn(static_cast<float>(px), jx), sy = __fadd_rn(static_cast<float>(py), jy);
  const float3 target = f3(fmaf(sy, J.cam_dv.x, fmaf(sx, J.cam_du.x, J.cam_corner.x)),
                           fmaf(sy, J.cam_dv.y, fmaf(sx, J.cam_du.y, J.cam_corner.y)),
                           fmaf(sy, J.cam_dv.z, fmaf(sx, J.cam_du.z, J.cam_corner.z)));
  cs.o = J.cam_origin;
  if (J.lens_radius > 0.f) {
    const float2 dk = unit_disk(cs.rng);
    const float lr = J.lens_radius;
    cs.o = f3(fmaf(lr, fmaf(dk.y, J.cam_v.x, __fmul_rn(dk.x, J.cam_u.x)), cs.o.x),
              fmaf(lr, fmaf(dk.y, J.cam_v.y, __fmul_rn(dk.x, J.cam_u.y)), cs.o.y),
              fmaf(lr, fmaf(dk.y, J.cam_v.z, __fmul_rn(dk.x, J.cam_u.z)), cs.o.z));
  }
  cs.d = unit_or(sub3p(target, cs.o), f3(0.f, 0.f, 0.f));
  cs.sample = static_cast<std::uint32_t>(S.sample_base + local);
  return cs;
}

// ---------------------------------------------------------------------------
// Inclusive scan over one block of kMaxGen threads (warp shuffles, then the warp
// totals); `tot` is a kMaxGen / 32 scratch array and receives the block total.
template <class T>
__device__ __forceinline__ T plan_scan(T v, T* tot, T& total) {
  constexpr int kWarps = kMaxGen / 32;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T y = __shfl_up_sync(kFull, v, off);
    if (lane >= off) v += y;
  }
  if (lane == 31) tot[w] = v;
  __syncthreads();
  if (w == 0) {
    T x = lane < kWarps ? tot[lane] : 0;
#pragma unroll
    for (int off = 1; off < kWarps; off <<= 1) {
      const T y = __shfl_up_sync(kFull, x, off);
      if (lane >= off) x += y;
    }
    if (lane < kWarps) tot[lane] = x;
  }
  __syncthreads();
  total = tot[kWarps - 1];
  return v + (w > 0 ? tot[w - 1] : 0);
}

// Generation plan: free slots go to the open segments greedily in the host's
// order. One block of kMaxGen threads, one table entry each.
__global__ void __launch_bounds__(kMaxGen) k_plan(WaveBuffers wb, int par) {
  __shared__ unsigned long long tot_rem[kMaxGen / 32];
  __shared__ std::uint32_t tot_flag[kMaxGen / 32];
  chain_to_previous_grid();
  WaveCounters* C = wb.cnt;
  const int t = threadIdx.x;
  const std::uint32_t live = C->live[par];
  const std::uint32_t room = wb.capacity - live;
  const std::uint32_t ng = min(wb.gen->n, static_cast<std::uint32_t>(kMaxGen));
  // Snapshot of the state the previous iteration left, before this plan changes it.
  const std::uint64_t iter = C->iteration;
  WaveSnapshot* snap = wb.ring + (iter % wb.ring_size);
  const std::uint32_t ns = min(wb.gen->snapshot_slots, static_cast<std::uint32_t>(kMaxSegments));
  for (std::uint32_t k = t; k < ns; k += kMaxGen) snap->seg[k] = wb.seg_prog[k];
  if (t == 0) snap->c = *C;
  std::uint32_t slot = 0, rem = 0;
  std::uint64_t gen0 = 0;
  if (t < static_cast<int>(ng)) {
    slot = wb.gen->slot[t];
    if (slot < static_cast<std::uint32_t>(kMaxSegments)) {
      gen0 = wb.seg_prog[slot].generated;
      const std::uint64_t count = wb.segs[slot].count;
      const std::uint64_t r = count > gen0 ? count - gen0 : 0;
      rem = r < room ? static_cast<std::uint32_t>(r) : room;
    } else {
      atomicExch(&C->error, 3u);
      C->error_info = slot;
    }
  }
  unsigned long long total = 0;
  std::uint32_t n_plan = 0;
  const unsigned long long before = plan_scan<unsigned long long>(rem, tot_rem, total) - rem;
  const std::uint32_t excl = before < room ? static_cast<std::uint32_t>(before) : room;
  const std::uint32_t take = min(rem, room - excl);
  const std::uint32_t flag = take > 0 ? 1u : 0u;
  const std::uint32_t fpos = plan_scan<std::uint32_t>(flag, tot_flag, n_plan);
  if (flag) {
    const std::uint32_t k = fpos - 1;
    wb.plan->end[k] = excl + take;
    wb.plan->seg[k] = slot;
    wb.plan->start[k] = gen0;
    wb.seg_prog[slot].generated = gen0 + take;
  }
  if (t == 0) {
    const std::uint32_t n_new = total < room ? static_cast<std::uint32_t>(total) : room;
    wb.plan->n = n_plan;
    wb.plan->n_new = n_new;
    C->n_items = live + n_new;
    // Fewer new paths than there is room for: nothing else is open, so this
    // iteration runs its paths to their end.
    C->finish = total < room ? 1u : 0u;
    C->live[par ^ 1] = 0;
    C->fetch = 0;
    C->generated += n_new;
    C->iteration = iter + 1;
  }
}

// ---------------------------------------------------------------------------
// The path kernel: a wavefront per warp.
//
// Every warp owns kWarpPaths path slots in shared memory and sorts them into three
// queues: `idle` (no path), `ready` (a ray to trace) and `lit` (a shadow ray to
// trace). A step takes up to 32 entries of one queue:
//   new     idle slots get the next items of the iteration's list (paths left by
//           the previous iteration, then new camera paths), and go on as
//   bounce  closest hit, emission, material sampling, next-event estimation and
//           Russian roulette of each path; its slot then moves to `lit`, `ready`
//           or `idle`;
//   shadow  any-hit test of each shadow ray, then on to `ready` or `idle`.
// The warp takes the first queue that can fill its lanes, so the walks and the
// shading run 29 to 31 of 32 lanes wide (one path per lane, refilled when it ends,
// leaves 40% of the lanes without a shadow ray and measured 1.4 to 1.6 times
// slower). There is no barrier, and path state stays on the SM. A path in `lit` is
// in no other queue, so the adds to its radiance keep their order.
//
// It replaces one kernel per stage over a pool of paths in HBM, where every bounce
// of every path moved some 300 bytes and every stage waited for its slowest warp
// (36 us of fixed cost an iteration on the sphere field, 160 us on the mesh). On
// B200, device time before and after, default pool: Cornell 256x256x64 2595 and
// 1940 us, sphere field 640x360x64 4446 and 2790 us; pool of 2^23: sphere field
// 512x512x128 8250 and 5970 us, mesh 1024x1024x64 52.9 and 50.2 ms, 16 scenes of the
// mix 123.2 and 110.7 ms.
//
// What bounds it: instruction issue (73% of the slots on Cornell) under divergence
// (11 to 16 of 32 lanes active in the walks), then the walks' dependent loads.
// - 56 slots a warp and 72 registers (7 blocks of 128 per SM) measured best: 48
//   slots fill 27 lanes (3 to 6% slower), 64 leave less L1 (1 to 2%), 96 only 16
//   warps an SM (18 to 25%); at 64 registers the shading spills (5 to 8%).
// - Instruction cache: closest-hit and shadow rays share one copy of the walk, and
//   what only some jobs need is in other instances. With a copy each (and the
//   four-wide walk for shadow rays), warps in different steps evict each other's
//   loops: 2.1 of 9.5 cycles per instruction went to fetching, now 0.5 to 0.9.
constexpr int kWarpPaths = 56;
// Least paths a warp takes at once where there are too few for full batches: 4 and 8
// measure alike, 16 loses half of the gain (mesh 64x64x1: 465 us with full batches only,
// 408 with 16, 313 with 8, 331 with 4; 32x32x1: 465, 355, 319, 260).
constexpr std::uint32_t kMinBatch = 4;

constexpr std::uint32_t kPathSpecular = 1u << 12;   // last bounce was specular (or the path is new)
constexpr std::uint32_t kPathContinues = 1u << 13;  // goes on after its shadow ray
constexpr int kPathSegShift = 16;                   // low 12 bits: depth; 16 and up: segment slot
static_assert(kMaxSegments <= 1 << 16, "the segment slot does not fit the path word");

// One warp's path slots, one 4-byte column per field.
template <bool kMis>
struct alignas(16) WarpPaths {
  float o[3][kWarpPaths];       // ray origin (and the shadow ray's, unless sh_tmax is negative)
  float d[3][kWarpPaths];
  float beta[3][kWarpPaths];    // throughput
  float light[3][kWarpPaths];   // radiance so far
  std::uint32_t rng[4][kWarpPaths];  // PCG32 state (lo, hi), increment (lo, hi)
  std::uint32_t sample[kWarpPaths];  // radiance slot
  std::uint32_t meta[kWarpPaths];
  float sh_d[3][kWarpPaths];    // shadow ray direction, length, contribution
  float sh_tmax[kWarpPaths];    // negative: the shadow ray's origin is in the radiance slot
  float sh_c[3][kWarpPaths];
  float pdf[kMis ? kWarpPaths : 1];  // pdf of the last diffuse bounce
  std::uint16_t job[kWarpPaths];
  std::uint8_t idle[kWarpPaths], ready[kWarpPaths], lit[kWarpPaths];
};

template <int kSlots>
__device__ __forceinline__ float3 get3(const float (&v)[3][kSlots], int p) { return f3(v[0][p], v[1][p], v[2][p]); }
template <int kSlots>
__device__ __forceinline__ void set3(float (&v)[3][kSlots], int p, float3 x) {
  v[0][p] = x.x;
  v[1][p] = x.y;
  v[2][p] = x.z;
}
// v[.][p] += x, and += a b, fused.
template <int kSlots>
__device__ __forceinline__ void add_to(float (&v)[3][kSlots], int p, float3 x) {
  set3(v, p, get3(v, p) + x);
}
template <int kSlots, class A>
__device__ __forceinline__ void mad_to(float (&v)[3][kSlots], int p, A a, float3 b) {
  set3(v, p, mad3(a, b, get3(v, p)));
}

// The walk of an instance. The common instance walks the binary tree; the general
// one also counts, walks the eight-wide tree and tests every primitive of jobs that
// ask for it. Kept out of the common instance, that code frees instruction cache: 3%
// (mesh) to 6% (Cornell).
template <bool kGeneral>
struct Walk;

template <>
struct Walk<false> {
  using Entry = int;
  __device__ __forceinline__ RayHit operator()(const RtgSceneDev& J, float3 o, float3 d, float tmax, bool any, Entry* stack,
                                               int, TraceCount& tc) {
    return walk_binary<kPathStack, 32, false>(J, o, d, kRayTMin, tmax, any, stack + (threadIdx.x & 31), tc);
  }
};

template <>
struct Walk<true> {
  using Entry = uint2;
  __device__ __forceinline__ RayHit operator()(const RtgSceneDev& J, float3 o, float3 d, float tmax, bool any, Entry* stack,
                                               int tree, TraceCount& tc) {
    // The columns of the two kinds of walk differ: their entries have different sizes.
    Entry* const column = stack + (threadIdx.x & 31);
    RayHit found{tmax, 0u, 0.f, 0.f};
    if (!J.use_bvh) {
      if (!any) return closest_brute<true>(J, o, d, kRayTMin, tmax, tc);
      if (!any_brute(J, o, d, kRayTMin, tmax)) found.word = kHitMiss;
      return found;
    }
    if (tree == 8) {
      if (!any) return closest_hit8<kPathStack, 32, true>(J, o, d, kRayTMin, tmax, column, tc);
      if (!any_hit8<kPathStack, 32, true>(J, o, d, kRayTMin, tmax, column, tc)) found.word = kHitMiss;
      return found;
    }
    return walk_binary<kPathStack, 32, true>(J, o, d, kRayTMin, tmax, any, reinterpret_cast<int*>(stack) + (threadIdx.x & 31),
                                       tc);
  }
};

template <bool kMis, bool kGeneral>
constexpr std::size_t kWarpSmem = sizeof(WarpPaths<kMis>) + sizeof(typename Walk<kGeneral>::Entry) * 32 * kPathStack;

// kMis: some open job uses multiple importance sampling. Without one, that code is
// compiled out. closest_tree and shadow_tree matter to the general instance only.
template <int kBlock, bool kMis, bool kGeneral>
__global__ void __launch_bounds__(kBlock, kPathThreads / kBlock)
k_path(WaveBuffers wb, int par, int closest_tree, int shadow_tree) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_total[3];
  using Entry = typename Walk<kGeneral>::Entry;
  const int lane = threadIdx.x & 31;
  unsigned char* const mine = smem + (threadIdx.x >> 5) * kWarpSmem<kMis, kGeneral>;
  WarpPaths<kMis>& S = *reinterpret_cast<WarpPaths<kMis>*>(mine);
  Entry* const stack = reinterpret_cast<Entry*>(mine + sizeof(WarpPaths<kMis>));  // of the warp
  if (threadIdx.x < 3) s_total[threadIdx.x] = 0;
#pragma unroll 1
  for (int k = lane; k < kWarpPaths; k += 32) S.idle[k] = static_cast<std::uint8_t>(k);
  __syncthreads();
  chain_to_previous_grid();
  WaveCounters* const C = wb.cnt;
  const std::uint32_t live = C->live[par], n = C->n_items;
  const bool finish = C->finish != 0;
  // New items come 32 at a time, or fewer when that gives every warp some: with few
  // paths the time is a warp's chain of steps, and a step is as long as its longest ray.
  const std::uint32_t warps = gridDim.x * (blockDim.x / 32);
  const int batch = static_cast<int>(min(32u, max(kMinBatch, (n + warps - 1) / warps)));
  const unsigned below = (1u << lane) - 1u;
  Walk<kGeneral> walk;
  TraceCount tc, sh_tc;
  std::uint32_t rays = 0, shadow_rays = 0, rr_killed = 0;     // of the warp
  std::uint32_t done_seg = 0xFFFFFFFFu, done_count = 0;       // finished paths not yet counted in their segment
  int n_idle = kWarpPaths, n_ready = 0, n_lit = 0;
  bool more = true;  // the iteration's list may have items left
  while (true) {
    const int n_new = more ? n_idle : 0;
    enum { kShadow, kBounce, kNew } step;
    if (!more && !finish) {
      // The list is used up and more will follow: leave the paths for the next
      // iteration, once no shadow ray is pending.
      if (n_lit == 0) break;
      step = kShadow;
    } else if (n_lit >= 32) {
      step = kShadow;
    } else if (n_ready >= 32) {
      step = kBounce;
    } else if (n_new >= 32) {
      step = kNew;
    } else {
      if ((n_lit | n_ready | n_new) == 0) break;
      step = n_lit >= n_ready && n_lit >= n_new ? kShadow : (n_ready >= n_new ? kBounce : kNew);
    }
    bool on = false, cont = false, shadow = false, killed = false;
    int p = 0;
    float3 o = f3(0.f, 0.f, 0.f), d = o;
    float tmax = FLT_MAX;
    std::uint32_t job = 0;
    if (step == kShadow) {
      const int take = min(n_lit, 32);
      n_lit -= take;
      shadow_rays += take;
      on = lane < take;
      if (on) {
        p = S.lit[n_lit + lane];
        o = get3(S.o, p);
        d = get3(S.sh_d, p);
        tmax = S.sh_tmax[p];
        if (tmax < 0.f) {
          o = f3(wb.radiance[S.sample[p]]);
          tmax = -tmax;
        }
        job = S.job[p];
      }
    } else if (step == kBounce) {
      const int take = min(n_ready, 32);
      n_ready -= take;
      rays += take;
      on = lane < take;
      if (on) {
        p = S.ready[n_ready + lane];
        o = get3(S.o, p);
        d = get3(S.d, p);
        job = S.job[p];
      }
    } else {
      int take = min(n_idle, batch);
      std::uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&C->fetch, static_cast<std::uint32_t>(take));
      base = __shfl_sync(kFull, base, 0);
      if (base >= n) {
        more = false;
        continue;
      }
      if (n - base < static_cast<std::uint32_t>(take)) {
        take = static_cast<int>(n - base);
        more = false;
      }
      n_idle -= take;
      rays += take;
      on = lane < take;
      if (on) {
        p = S.idle[n_idle + lane];
        const std::uint32_t i = base + lane;
        if (i < live) {
          // A path the previous iteration left.
          const float4 a = __ldcs(&wb.st_a[par][i]), b = __ldcs(&wb.st_b[par][i]), c = __ldcs(&wb.st_c[par][i]);
          const uint4 r = __ldcs(&wb.st_d[par][i]);
          const float4 l = __ldcs(&wb.st_e[par][i]);
          o = f3(a);
          d = f3(b);
          S.sample[p] = __float_as_uint(a.w);
          S.meta[p] = __float_as_uint(b.w);
          set3(S.beta, p, f3(c));
          job = __float_as_uint(c.w);
          S.rng[0][p] = r.x;
          S.rng[1][p] = r.y;
          S.rng[2][p] = r.z;
          S.rng[3][p] = r.w;
          set3(S.light, p, f3(l));
          if (kMis) S.pdf[p] = l.w;
        } else {
          const std::uint32_t j = i - live;
          // New path j: plan entry k is the first with end[k] > j.
          const GenPlan& P = *wb.plan;
          int lo = 0, hi = static_cast<int>(P.n) - 1;
#pragma unroll 1
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (P.end[mid] > j) hi = mid;
            else lo = mid + 1;
          }
          const std::uint32_t seg = P.seg[lo];
          const std::uint64_t local = P.start[lo] + (j - (lo > 0 ? P.end[lo - 1] : 0u));
          const DevSegment sg = wb.segs[seg];
          job = sg.job;
          const CameraSample cs = camera_sample(wb.jobs[job], sg, local);
          o = cs.o;
          d = cs.d;
          S.sample[p] = cs.sample;
          // Camera rays count as a specular bounce (no NEE double-count guard).
          S.meta[p] = kPathSpecular | (seg << kPathSegShift);
          set3(S.beta, p, f3(1.f, 1.f, 1.f));
          S.rng[0][p] = static_cast<std::uint32_t>(cs.rng.state);
          S.rng[1][p] = static_cast<std::uint32_t>(cs.rng.state >> 32);
          S.rng[2][p] = static_cast<std::uint32_t>(cs.rng.inc);
          S.rng[3][p] = static_cast<std::uint32_t>(cs.rng.inc >> 32);
          set3(S.light, p, f3(0.f, 0.f, 0.f));
        }
        S.job[p] = static_cast<std::uint16_t>(job);
      }
    }
    __syncwarp();
    if (on) {
      const RtgSceneDev& J = wb.jobs[job];
      // One copy of the walk serves both kinds of rays.
      const bool any = step == kShadow;
      const RayHit h = walk(J, o, d, tmax, any, stack, any ? shadow_tree : closest_tree, any ? sh_tc : tc);
      const std::uint32_t meta = S.meta[p];
      if (any) {
        if (h.word == kHitMiss) add_to(S.light, p, get3(S.sh_c, p));
        cont = (meta & kPathContinues) != 0;
      } else if (h.word == kHitMiss) {
        // The normals view shows misses black.
        if (J.integrator != 2) mad_to(S.light, p, get3(S.beta, p), background(J, d));
      } else {
        const Surface s = make_surface(J, o, d, h);
        if (J.integrator == 2) {
          // Normals view: outward shading normal mapped to [0, 1].
          const float3 nn = s.front ? s.n : -s.n;
          set3(S.light, p, (nn + f3(1.f, 1.f, 1.f)) * 0.5f);
        } else {
          const DevMaterial m = J.materials[s.material];
          const float3 le = emitted(m, s.front);
          // A light reached by a diffuse bounce was already counted by NEE. With
          // MIS both count, each weighted by the power heuristic against the other.
          if (!is_zero3(le)) {
            float w = 1.f;
            if (!(meta & kPathSpecular) && J.light_sampling && !s.is_plane)
              w = kMis && J.light_sampling == 2
                      ? power_heuristic(S.pdf[kMis ? p : 0],
                                        light_pdf_of_hit(J, o, d, h, s) / static_cast<float>(J.n_lights))
                      : 0.f;
            if (kMis && J.light_sampling == 2) {
              if (w > 0.f) mad_to(S.light, p, w, get3(S.beta, p) * le);
            } else if (w > 0.f) {
              mad_to(S.light, p, get3(S.beta, p), le);
            }
          }
          Pcg rng{ld_u64(S.rng[0][p], S.rng[1][p]), ld_u64(S.rng[2][p], S.rng[3][p])};
          Scatter sr;
          if (scatter(m, d, s, rng, sr)) {
            // The next ray goes to shared memory before the light sample, which
            // needs the registers.
            const bool outside = leaves_outside(s.gn, sr.dir);
            set3(S.o, p, spawn_point(s.p, outside ? s.gn : -s.gn));
            set3(S.d, p, sr.dir);
            if (J.light_sampling && !sr.specular && J.n_lights > 0) {
              const std::uint32_t nl = static_cast<std::uint32_t>(J.n_lights);
              const LightSample ls = sample_light(J.lights + rng.below(nl), s, rng);
              if (ls.valid) {
                // Only a Lambertian scatter is non-specular: its weight is the albedo.
                const float3 f = lambert_cos(sr.weight, s, ls.wi);
                if (!is_zero3(f) && !is_zero3(ls.li_over_pdf)) {
                  // Its origin is mostly the one stored above: a Lambertian scatter
                  // leaves, and lambert_cos is non-zero, on the side of s.gn. But
                  // leaves_outside rounds in another way than those tests: of a direction
                  // in the surface's plane it may find the other side. The origin then
                  // waits in the radiance slot, which is written when the path ends.
                  const ShadowRay sray = shadow_ray(s, ls);
                  S.sh_tmax[p] = sray.tmax;
                  if (leaves_outside(s.gn, ls.wi) != outside) {
                    S.sh_tmax[p] = -sray.tmax;
                    wb.radiance[S.sample[p]] = make_float4(sray.o.x, sray.o.y, sray.o.z, 0.f);
                  }
                  float w = 1.f;  // a point light (pdf 0) cannot be hit by BSDF sampling
                  if (kMis && J.light_sampling == 2 && ls.pdf > 0.f)
                    w = power_heuristic(ls.pdf / static_cast<float>(nl), __fmul_rn(dot3(s.n, ls.wi), kInvPiF));
                  set3(S.sh_d, p, sray.d);
                  set3(S.sh_c, p, get3(S.beta, p) * (f * ls.li_over_pdf) * __fmul_rn(static_cast<float>(nl), w));
                  shadow = true;
                }
              }
            }
            float3 beta = get3(S.beta, p) * sr.weight;
            const std::uint32_t depth = (meta & kMetaDepthMask) + 1;
            bool alive = !is_zero3(beta);
            if (alive && depth >= static_cast<std::uint32_t>(J.rr_min_depth)) {
              const float q = fminf(fmaxf(max3(beta), 0.05f), 0.95f);
              if (rng.uniform() >= q) {
                alive = false;
                killed = true;
              } else {
                beta = beta * (1.f / q);
              }
            }
            cont = alive && depth < static_cast<std::uint32_t>(J.max_depth);
            if (cont) {
              set3(S.beta, p, beta);
              S.rng[0][p] = static_cast<std::uint32_t>(rng.state);
              S.rng[1][p] = static_cast<std::uint32_t>(rng.state >> 32);
              // Cosine-hemisphere pdf of this bounce, for the MIS weight at the next hit.
              if (kMis && J.light_sampling == 2 && !sr.specular) S.pdf[kMis ? p : 0] = __fmul_rn(dot3p(s.n, sr.dir), kInvPiF);
            }
            S.meta[p] = (meta & ~0xFFFFu) | depth | (sr.specular ? kPathSpecular : 0u) | (cont ? kPathContinues : 0u);
          }
        }
      }
    }
    const bool ready = cont && !shadow, end = on && !cont && !shadow;
    const unsigned m_lit = __ballot_sync(kFull, shadow), m_ready = __ballot_sync(kFull, ready);
    const unsigned m_end = __ballot_sync(kFull, end);
    rr_killed += __popc(__ballot_sync(kFull, killed));
    if (shadow) S.lit[n_lit + __popc(m_lit & below)] = static_cast<std::uint8_t>(p);
    if (ready) S.ready[n_ready + __popc(m_ready & below)] = static_cast<std::uint8_t>(p);
    if (m_end) {
      std::uint32_t seg = 0;
      if (end) {
        S.idle[n_idle + __popc(m_end & below)] = static_cast<std::uint8_t>(p);
        const float3 l = get3(S.light, p);
        wb.radiance[S.sample[p]] = make_float4(l.x, l.y, l.z, 0.f);
        seg = S.meta[p] >> kPathSegShift;
      }
      // Finished paths are counted in their segment: the warp keeps a count while
      // they belong to one segment, as they mostly do.
      const std::uint32_t seg0 = __shfl_sync(kFull, seg, __ffs(m_end) - 1);
      if (__any_sync(kFull, end && seg != seg0)) {
        const unsigned same = __match_any_sync(kFull, end ? seg : 0xFFFFFFFFu);
        if (end && lane == __ffs(same) - 1) atomicAdd(&wb.seg_prog[seg].done, static_cast<std::uint32_t>(__popc(same)));
      } else {
        if (seg0 != done_seg) {
          if (lane == 0 && done_count) atomicAdd(&wb.seg_prog[done_seg].done, done_count);
          done_seg = seg0;
          done_count = 0;
        }
        done_count += __popc(m_end);
      }
    }
    n_lit += __popc(m_lit);
    n_ready += __popc(m_ready);
    n_idle += __popc(m_end);
    __syncwarp();
  }
  if (lane == 0 && done_count) atomicAdd(&wb.seg_prog[done_seg].done, done_count);
  if (n_ready) {
    std::uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&C->live[par ^ 1], static_cast<std::uint32_t>(n_ready));
    base = __shfl_sync(kFull, base, 0);
#pragma unroll 1
    for (int k = lane; k < n_ready; k += 32) {
      const int p = S.ready[k];
      const std::uint32_t i = base + k;
      const float3 o = get3(S.o, p), d = get3(S.d, p), b = get3(S.beta, p), l = get3(S.light, p);
      __stcs(&wb.st_a[par ^ 1][i], make_float4(o.x, o.y, o.z, __uint_as_float(S.sample[p])));
      __stcs(&wb.st_b[par ^ 1][i], make_float4(d.x, d.y, d.z, __uint_as_float(S.meta[p])));
      __stcs(&wb.st_c[par ^ 1][i], make_float4(b.x, b.y, b.z, __uint_as_float(S.job[p])));
      __stcs(&wb.st_d[par ^ 1][i], make_uint4(S.rng[0][p], S.rng[1][p], S.rng[2][p], S.rng[3][p]));
      __stcs(&wb.st_e[par ^ 1][i], make_float4(l.x, l.y, l.z, kMis ? S.pdf[kMis ? p : 0] : 0.f));
    }
  }
  // Counters: one atomic per block and counter.
  if (lane == 0) {
    atomicAdd(&s_total[0], static_cast<unsigned long long>(rays));
    atomicAdd(&s_total[1], static_cast<unsigned long long>(shadow_rays));
    atomicAdd(&s_total[2], static_cast<unsigned long long>(rr_killed));
  }
  __syncthreads();
  if (threadIdx.x < 3 && s_total[threadIdx.x]) {
    std::uint64_t* const to = threadIdx.x == 0 ? &C->rays : (threadIdx.x == 1 ? &C->shadow_rays : &C->rr_terminated);
    atomicAdd(reinterpret_cast<unsigned long long*>(to), s_total[threadIdx.x]);
  }
  if (kGeneral) {
    warp_add_u64(tc.nodes, &C->node_visits);
    warp_add_u64(tc.prims, &C->prim_tests);
    warp_add_u64(tc.spheres, &C->sphere_tests);
    warp_add_u64(sh_tc.nodes, &C->shadow_node_visits);
    warp_add_u64(sh_tc.prims, &C->shadow_prim_tests);
    warp_add_u64(sh_tc.spheres, &C->shadow_sphere_tests);
  }
}

// ---------------------------------------------------------------------------
// Sample i of a list of passes.
__device__ __forceinline__ CameraSample listed_sample(const RtgSceneDev& J, const PassList& passes, std::uint64_t i) {
  int k = 0;
  while (k + 1 < passes.n && i >= passes.seg[k].count) i -= passes.seg[k++].count;
  return camera_sample(J, passes.seg[k], i);
}

// Whitted-style direct integrator (src/rendering/integrator.cpp:141-174): every
// light at diffuse hits, recursion through metal, and a deterministic Fresnel
// split at dielectrics. The recursion becomes a depth-first walk of each sample's
// tree with a stack of pending refraction branches, which keeps the reference's RNG
// draw order.
//
// Two kernels. From kDirectWarpSamples samples a launch up, unless the branches below
// have no memory, k_direct schedules them like the path kernel: each warp holds kDirectPaths samples in shared memory; `ready` ones
// have a ray to trace, `lit` ones the next light of a diffuse hit to sample and test
// (its surface is made again from the hit for each light, which costs less than
// keeping it). Pending branches are in device memory: at most one per level, so
// min(max depth, kDirectStack) records a sample. Smaller launches take a thread a
// sample, k_direct_sample.
//
// What bounds both: the divergence between trees (k_direct's lanes are full, a warp of
// k_direct_sample waits for its longest tree), and the serial chain of the largest
// tree: on the mesh at depth 8 one sample a pixel takes 4.3 of the 7.2 ms that 640x360x16
// take. A vertex of that chain takes k_direct longer (its state goes through shared
// memory), so what wins is the number of samples. k_direct_sample's time over k_direct's
// on the mesh / the sphere field at depth 8: 16 ki samples 0.91 / 0.79, 256 ki 0.93 / 0.78,
// 1 Mi 1.11 to 1.28 / 0.95 to 0.98, 4 Mi 1.18 / 1.05, 12 Mi 1.26 / 1.04 (Cornell: 0.70 at 16
// ki, 1.0 at 1 Mi, 1.05 at 4 Mi). First in, first out queues, which advance the long
// samples sooner, cost 4%: they lose more coherence than tail.
constexpr std::uint64_t kDirectWarpSamples = std::uint64_t(1) << 20;
constexpr int kDirectStack = 48;
constexpr int kDirectPaths = 48;
constexpr int kPendingRows = 3;  // float4 rows of a pending branch: (o, d.x), (d.yz, w.xy), (w.z, depth)

struct alignas(16) DirectPaths {
  float o[3][kDirectPaths], d[3][kDirectPaths], w[3][kDirectPaths];  // ray and its weight
  float light[3][kDirectPaths];                                      // radiance so far
  float sum[3][kDirectPaths];                                        // of the lights at the current hit
  float f[3][kDirectPaths], li[3][kDirectPaths];                     // BRDF and light of the shadow ray in flight
  float hit[4][kDirectPaths];
  std::uint32_t rng[4][kDirectPaths];
  std::uint32_t sample[kDirectPaths];
  std::uint16_t depth[kDirectPaths];
  std::int32_t light_index[kDirectPaths];
  std::uint8_t pending[kDirectPaths];                                // refraction branches on the stack
  std::uint8_t idle[kDirectPaths], ready[kDirectPaths], lit[kDirectPaths];
};

template <bool kGeneral>
constexpr std::size_t kDirectWarpSmem = sizeof(DirectPaths) + sizeof(typename Walk<kGeneral>::Entry) * 32 * kPathStack;

template <int kBlock, bool kGeneral>
__global__ void __launch_bounds__(kBlock, kPathThreads / kBlock)
k_direct(const RtgSceneDev* __restrict__ job, const __grid_constant__ PassList passes, float4* radiance, WaveCounters* C,
         float4* stack_rows, int stack_depth, int tree) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Entry = typename Walk<kGeneral>::Entry;
  const int lane = threadIdx.x & 31;
  unsigned char* const mine = smem + (threadIdx.x >> 5) * kDirectWarpSmem<kGeneral>;
  DirectPaths& S = *reinterpret_cast<DirectPaths*>(mine);
  Entry* const stack = reinterpret_cast<Entry*>(mine + sizeof(DirectPaths));  // of the warp
  // Pending branches of this warp's slot p start at row (first_slot + p) * stack_depth * kPendingRows.
  const std::size_t first_slot =
      (static_cast<std::size_t>(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5)) * kDirectPaths;
#pragma unroll 1
  for (int k = lane; k < kDirectPaths; k += 32) S.idle[k] = static_cast<std::uint8_t>(k);
  __syncwarp();
  const RtgSceneDev& J = *job;
  const std::uint32_t count = static_cast<std::uint32_t>(passes.samples());  // under 2^32 (the radiance slots are)
  const unsigned below = (1u << lane) - 1u;
  Walk<kGeneral> walk;
  TraceCount tc;
  std::uint32_t rays = 0, shadow_rays = 0;  // of the warp
  bool overflow = false, more = true;
  int n_idle = kDirectPaths, n_ready = 0, n_lit = 0;
  while (true) {
    const int n_new = more ? n_idle : 0;
    // Full batches of one kind while there are any; else lights and rays together, so
    // that what is left of the long samples does not wait for each other's kind.
    int n_light = 0, n_trace = 0;
    if (n_lit >= 32) {
      n_light = 32;
    } else if (n_ready >= 32) {
      n_trace = 32;
    } else if (n_new < 32) {
      n_light = n_lit;
      n_trace = min(n_ready, 32 - n_lit);
    }
    bool on = false, ray = false;  // the lane has a sample; the sample has a ray to trace in this step
    bool light = false;            // that ray is a shadow ray
    int p = 0;
    float3 o = f3(0.f, 0.f, 0.f), d = o;
    float tmax = FLT_MAX;
    if (n_light + n_trace > 0) {
      n_lit -= n_light;
      n_ready -= n_trace;
      rays += n_trace;
      light = lane < n_light;
      on = lane < n_light + n_trace;
      if (light) {
        p = S.lit[n_lit + lane];
        const Surface s = make_surface(J, get3(S.o, p), get3(S.d, p),
                                       RayHit{S.hit[0][p], __float_as_uint(S.hit[1][p]), S.hit[2][p], S.hit[3][p]});
        Pcg rng{ld_u64(S.rng[0][p], S.rng[1][p]), ld_u64(S.rng[2][p], S.rng[3][p])};
        const LightSample ls = sample_light(J.lights + S.light_index[p], s, rng);
        S.rng[0][p] = static_cast<std::uint32_t>(rng.state);
        S.rng[1][p] = static_cast<std::uint32_t>(rng.state >> 32);
        if (ls.valid) {
          const float3 f = brdf_cos(J.materials[s.material], s, ls.wi);
          if (!is_zero3(f) && !is_zero3(ls.li_over_pdf)) {
            const ShadowRay sr = shadow_ray(s, ls);
            o = sr.o;
            d = sr.d;
            tmax = sr.tmax;
            set3(S.f, p, f);
            set3(S.li, p, ls.li_over_pdf);
            ray = true;
          }
        }
      } else if (on) {
        p = S.ready[n_ready + lane - n_light];
        o = get3(S.o, p);
        d = get3(S.d, p);
        ray = true;
      }
      shadow_rays += __popc(__ballot_sync(kFull, light && ray));
    } else if (n_new == 0) {
      break;
    } else {
      int take = min(n_idle, 32);
      std::uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&C->direct_fetch, static_cast<std::uint32_t>(take));
      base = __shfl_sync(kFull, base, 0);
      if (base >= count) {
        more = false;
        continue;
      }
      if (count - base < static_cast<std::uint32_t>(take)) {
        take = static_cast<int>(count - base);
        more = false;
      }
      n_idle -= take;
      on = ray = lane < take;
      rays += take;
      if (on) {
        p = S.idle[n_idle + lane];
        const CameraSample cs = listed_sample(J, passes, base + lane);
        o = cs.o;
        d = cs.d;
        set3(S.o, p, o);
        set3(S.d, p, d);
        set3(S.w, p, f3(1.f, 1.f, 1.f));
        set3(S.light, p, f3(0.f, 0.f, 0.f));
        S.rng[0][p] = static_cast<std::uint32_t>(cs.rng.state);
        S.rng[1][p] = static_cast<std::uint32_t>(cs.rng.state >> 32);
        S.rng[2][p] = static_cast<std::uint32_t>(cs.rng.inc);
        S.rng[3][p] = static_cast<std::uint32_t>(cs.rng.inc >> 32);
        S.sample[p] = cs.sample;
        S.depth[p] = 0;
        S.pending[p] = 0;
      }
    }
    __syncwarp();
    RayHit h{tmax, kHitMiss, 0.f, 0.f};
    if (ray) h = walk(J, o, d, tmax, light, stack, tree, tc);
    // What the sample does next: trace S.o, S.d; sample a light; or neither, and then
    // a pending branch is next, or the sample is done.
    bool go = false, lit = false;
    if (light) {
      if (ray && h.word == kHitMiss) mad_to(S.sum, p, get3(S.f, p), get3(S.li, p));
      const int next = S.light_index[p] + 1;
      S.light_index[p] = next;
      lit = next < J.n_lights;
      if (!lit) mad_to(S.light, p, get3(S.w, p), get3(S.sum, p));
    } else if (on) {
      const float3 w = get3(S.w, p);
      if (h.word == kHitMiss) {
        mad_to(S.light, p, w, background(J, d));
      } else {
        const Surface s = make_surface(J, o, d, h);
        const DevMaterial m = J.materials[s.material];
        mad_to(S.light, p, w, emitted(m, s.front));
        const int depth = S.depth[p];
        if (depth < J.max_depth) {
          const std::uint32_t kind = kind_of(m);
          if (kind == kLambertian) {
            if (J.n_lights > 0) {
              S.hit[0][p] = h.t;
              S.hit[1][p] = __uint_as_float(h.word);
              S.hit[2][p] = h.b1;
              S.hit[3][p] = h.b2;
              set3(S.sum, p, f3(0.f, 0.f, 0.f));
              S.light_index[p] = 0;
              lit = true;
            }
          } else if (kind == kMetal) {
            Pcg rng{ld_u64(S.rng[0][p], S.rng[1][p]), ld_u64(S.rng[2][p], S.rng[3][p])};
            Scatter sr;
            go = scatter(m, d, s, rng, sr);
            S.rng[0][p] = static_cast<std::uint32_t>(rng.state);
            S.rng[1][p] = static_cast<std::uint32_t>(rng.state >> 32);
            if (go) {
              set3(S.o, p, spawn_towards(s.p, s.gn, sr.dir));
              set3(S.d, p, sr.dir);
              set3(S.w, p, w * f3(m.colour_a));
            }
          } else if (kind == kDielectric) {
            const float ior = m.head.z;
            const float3 in = unit_or(d, f3(0.f, 0.f, 0.f));
            const float eta = s.front ? 1.f / ior : ior;
            const float cos_i = fminf(-dot3(in, s.n), 1.f);
            float3 refr;
            const bool can = refract3(in, s.n, eta, refr);
            const float F = can ? schlick(cos_i, eta) : 1.f;
            const float3 tint = f3(m.colour_a);
            if (can) {
              const int sp = S.pending[p];
              if (sp < stack_depth) {
                const float3 td = unit_or(refr, f3(0.f, 0.f, 0.f));
                const float3 to = spawn_towards(s.p, s.gn, td), tw = w * tint * __fsub_rn(1.f, F);
                float4* const row = stack_rows + ((first_slot + p) * stack_depth + sp) * kPendingRows;
                row[0] = make_float4(to.x, to.y, to.z, td.x);
                row[1] = make_float4(td.y, td.z, tw.x, tw.y);
                row[2] = make_float4(tw.z, __int_as_float(depth + 1), 0.f, 0.f);
                S.pending[p] = static_cast<std::uint8_t>(sp + 1);
              } else {
                overflow = true;
              }
            }
            const float3 rd = reflect3(in, s.n);
            set3(S.o, p, spawn_towards(s.p, s.gn, rd));
            set3(S.d, p, rd);
            set3(S.w, p, w * tint * F);
            go = true;
          }
          if (go) S.depth[p] = static_cast<std::uint16_t>(depth + 1);
        }
      }
    }
    if (on && !go && !lit && S.pending[p] > 0) {
      const int sp = S.pending[p] - 1;
      const float4* const row = stack_rows + ((first_slot + p) * stack_depth + sp) * kPendingRows;
      const float4 a = row[0], b = row[1], c = row[2];
      set3(S.o, p, f3(a.x, a.y, a.z));
      set3(S.d, p, f3(a.w, b.x, b.y));
      set3(S.w, p, f3(b.z, b.w, c.x));
      S.depth[p] = static_cast<std::uint16_t>(__float_as_int(c.y));
      S.pending[p] = static_cast<std::uint8_t>(sp);
      go = true;
    }
    const bool end = on && !go && !lit;
    if (end) {
      const float3 l = get3(S.light, p);
      radiance[S.sample[p]] = make_float4(l.x, l.y, l.z, 0.f);
    }
    const unsigned m_lit = __ballot_sync(kFull, lit), m_ready = __ballot_sync(kFull, go), m_end = __ballot_sync(kFull, end);
    if (lit) S.lit[n_lit + __popc(m_lit & below)] = static_cast<std::uint8_t>(p);
    if (go) S.ready[n_ready + __popc(m_ready & below)] = static_cast<std::uint8_t>(p);
    if (end) S.idle[n_idle + __popc(m_end & below)] = static_cast<std::uint8_t>(p);
    n_lit += __popc(m_lit);
    n_ready += __popc(m_ready);
    n_idle += __popc(m_end);
    __syncwarp();
  }
  if (overflow) atomicExch(&C->error, 2u);
  if (lane == 0) {
    atomicAdd(reinterpret_cast<unsigned long long*>(&C->rays), static_cast<unsigned long long>(rays));
    atomicAdd(reinterpret_cast<unsigned long long*>(&C->shadow_rays), static_cast<unsigned long long>(shadow_rays));
  }
}

struct Pending {
  float3 o, d, w;
  int depth;
};

// One sample a thread: the whole tree, with the pending branches in local memory.
template <int kBlock, bool kGeneral>
__global__ void __launch_bounds__(kBlock) k_direct_sample(const RtgSceneDev* __restrict__ job,
                                                          const __grid_constant__ PassList passes, float4* radiance,
                                                          WaveCounters* C, int tree) {
  __shared__ uint2 stack[kStackSmem * kBlock];
  int* const column = reinterpret_cast<int*>(stack) + threadIdx.x;
  TraceCount tc;
  std::uint64_t rays = 0, shadow_rays = 0;
  const RtgSceneDev& J = *job;
  const std::uint64_t count = passes.samples();
  auto closest = [&](float3 o, float3 d) {
    if (kGeneral) {
      if (!J.use_bvh) return closest_brute<false>(J, o, d, kRayTMin, FLT_MAX, tc);
      if (tree == 8) return closest_hit8<kStackSmem, kBlock, false>(J, o, d, kRayTMin, FLT_MAX, stack + threadIdx.x, tc);
    }
    return closest_hit<kStackSmem, kBlock, false>(J, o, d, kRayTMin, FLT_MAX, column, tc);
  };
  auto blocked = [&](const ShadowRay& r) {
    if (kGeneral) {
      if (!J.use_bvh) return any_brute(J, r.o, r.d, kRayTMin, r.tmax);
      if (tree == 8) return any_hit8<kStackSmem, kBlock, false>(J, r.o, r.d, kRayTMin, r.tmax, stack + threadIdx.x, tc);
    }
    return any_hit4<kStackSmem, kBlock, false>(J, r.o, r.d, kRayTMin, r.tmax, column, tc);
  };
  const std::uint64_t stride = static_cast<std::uint64_t>(gridDim.x) * kBlock;
  for (std::uint64_t w = static_cast<std::uint64_t>(blockIdx.x) * kBlock + threadIdx.x; w < count; w += stride) {
    CameraSample cs = listed_sample(J, passes, w);
    Pending todo[kDirectStack];
    int sp = 0;
    Pending cur{cs.o, cs.d, f3(1.f, 1.f, 1.f), 0};
    float3 L = f3(0.f, 0.f, 0.f);
    bool overflow = false;
    while (true) {
      ++rays;
      const RayHit h = closest(cur.o, cur.d);
      bool next = false;
      if (h.word == kHitMiss) {
        L = mad3(cur.w, background(J, cur.d), L);
      } else {
        const Surface s = make_surface(J, cur.o, cur.d, h);
        const DevMaterial m = J.materials[s.material];
        L = mad3(cur.w, emitted(m, s.front), L);
        if (cur.depth < J.max_depth) {
          const std::uint32_t kind = kind_of(m);
          if (kind == kLambertian) {
            // Every light, in order.
            float3 sum = f3(0.f, 0.f, 0.f);
            for (int li = 0; li < J.n_lights; ++li) {
              const LightSample ls = sample_light(J.lights + li, s, cs.rng);
              if (!ls.valid) continue;
              const float3 f = brdf_cos(m, s, ls.wi);
              if (is_zero3(f) || is_zero3(ls.li_over_pdf)) continue;
              ++shadow_rays;
              if (!blocked(shadow_ray(s, ls))) sum = mad3(f, ls.li_over_pdf, sum);
            }
            L = mad3(cur.w, sum, L);
          } else if (kind == kMetal) {
            Scatter sr;
            if (scatter(m, cur.d, s, cs.rng, sr)) {
              cur = Pending{spawn_towards(s.p, s.gn, sr.dir), sr.dir, cur.w * f3(m.colour_a), cur.depth + 1};
              next = true;
            }
          } else if (kind == kDielectric) {
            const float ior = m.head.z;
            const float3 in = unit_or(cur.d, f3(0.f, 0.f, 0.f));
            const float eta = s.front ? 1.f / ior : ior;
            const float cos_i = fminf(-dot3(in, s.n), 1.f);
            float3 refr;
            const bool can = refract3(in, s.n, eta, refr);
            const float F = can ? schlick(cos_i, eta) : 1.f;
            const float3 tint = f3(m.colour_a);
            if (can) {
              if (sp < kDirectStack) {
                const float3 td = unit_or(refr, f3(0.f, 0.f, 0.f));
                todo[sp++] = Pending{spawn_towards(s.p, s.gn, td), td, cur.w * tint * __fsub_rn(1.f, F), cur.depth + 1};
              } else {
                overflow = true;
              }
            }
            const float3 rd = reflect3(in, s.n);
            cur = Pending{spawn_towards(s.p, s.gn, rd), rd, cur.w * tint * F, cur.depth + 1};
            next = true;
          }
        }
      }
      if (next) continue;
      if (sp == 0) break;
      cur = todo[--sp];
    }
    if (overflow) atomicExch(&C->error, 2u);
    radiance[cs.sample] = make_float4(L.x, L.y, L.z, 0.f);
  }
  warp_add_u64(rays, &C->rays);
  warp_add_u64(shadow_rays, &C->shadow_rays);
}

// ---------------------------------------------------------------------------
// Folds finished passes of one job, in their order: each pixel's framebuffer entry is
// read and written once for all of them (136 bytes a pixel, as much as 8 samples).
__global__ void __launch_bounds__(256) k_accumulate(const RtgSceneDev* __restrict__ job,
                                                    const __grid_constant__ PassList passes,
                                                    const float4* __restrict__ radiance) {
  const RtgSceneDev& J = *job;
  const std::uint64_t pixels = static_cast<std::uint64_t>(J.width) * static_cast<std::uint64_t>(J.height);
  const std::uint64_t p = static_cast<std::uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  std::uint64_t bad = 0;
  if (p < pixels) {
    double s0 = J.fb_sum[4 * p], s1 = J.fb_sum[4 * p + 1], s2 = J.fb_sum[4 * p + 2];
    double q0 = J.fb_sumsq[4 * p], q1 = J.fb_sumsq[4 * p + 1], q2 = J.fb_sumsq[4 * p + 2];
    std::uint32_t n = 0;
    for (int i = 0; i < passes.n; ++i) {
      const std::uint32_t k = passes.seg[i].pass_spp;
      const float4* src = radiance + passes.seg[i].sample_base + p * k;
      n += k;
      for (std::uint32_t j = 0; j < k; ++j) {
        const float4 v = src[j];
        double r = v.x, g = v.y, b = v.z;
        // A non-finite or negative sample would poison the pixel: record it as black.
        if (!isfinite(r) || !isfinite(g) || !isfinite(b) || r < 0 || g < 0 || b < 0) {
          r = g = b = 0;
          ++bad;
        }
        s0 = __dadd_rn(s0, r); s1 = __dadd_rn(s1, g); s2 = __dadd_rn(s2, b);
        q0 = fma(r, r, q0); q1 = fma(g, g, q1); q2 = fma(b, b, q2);
      }
    }
    J.fb_sum[4 * p] = s0; J.fb_sum[4 * p + 1] = s1; J.fb_sum[4 * p + 2] = s2;
    J.fb_sumsq[4 * p] = q0; J.fb_sumsq[4 * p + 1] = q1; J.fb_sumsq[4 * p + 2] = q2;
    J.fb_count[p] += n;
  }
  warp_add_u64(bad, J.stats);
}

// Tone map (src/rendering/tonemap.cpp:15-53) in double: exposure, operator, exact
// sRGB transfer function, round half away from zero to 8 bits.
__device__ __forceinline__ double aces_curve(double x) {
  const double a = 2.51, b = 0.03, c = 2.43, d = 0.59, e = 0.14;
  const double v = (x * (a * x + b)) / (x * (c * x + d) + e);
  return v < 0 ? 0 : (v > 1 ? 1 : v);
}
__device__ __forceinline__ std::uint8_t srgb8(double v) {
  v = v < 0 ? 0 : (v > 1 ? 1 : v);
  double s = v <= 0.0031308 ? 12.92 * v : 1.055 * pow(v, 1.0 / 2.4) - 0.055;
  s = s < 0 ? 0 : (s > 1 ? 1 : s);
  return static_cast<std::uint8_t>(llround(s * 255.0));
}

// Means (mean_out) and/or their tone-mapped bytes (rgb8) of `pixels` pixels. A block's
// output is collected in shared memory and leaves in 16-byte (means) or 4-byte (image)
// pieces in order: the destination may be pinned host memory, where a pixel's own 8-
// and 1-byte stores would each cross the bus alone.
constexpr int kResolveBlock = 256;
__global__ void __launch_bounds__(kResolveBlock)
k_resolve(const double* __restrict__ fb_sum, const std::uint32_t* __restrict__ fb_count, std::uint64_t pixels, int op,
          double exposure, std::uint8_t* rgb8, double* mean_out) {
  __shared__ __align__(16) double s_mean[3 * kResolveBlock];
  __shared__ __align__(16) std::uint8_t s_rgb[3 * kResolveBlock];
  const std::uint64_t first = static_cast<std::uint64_t>(blockIdx.x) * kResolveBlock;
  const std::uint64_t p = first + threadIdx.x;
  const int here = static_cast<int>(pixels - first < kResolveBlock ? pixels - first : kResolveBlock);
  if (p < pixels) {
    const std::uint32_t n = fb_count[p];
    double c[3] = {0, 0, 0};
    if (n) {
      const double inv = 1.0 / static_cast<double>(n);
      for (int k = 0; k < 3; ++k) c[k] = fb_sum[4 * p + k] * inv;
    }
    if (mean_out)
      for (int k = 0; k < 3; ++k) s_mean[3 * threadIdx.x + k] = c[k];
    if (rgb8) {
      double t[3];
      bool finite = true;
      for (int k = 0; k < 3; ++k) {
        t[k] = c[k] * exposure;
        finite = finite && isfinite(t[k]);
      }
      for (int k = 0; k < 3; ++k) {
        double v = finite ? t[k] : 0.0;
        if (op == 0) v = v < 0 ? 0 : (v > 1 ? 1 : v);
        else if (op == 1) v = v / (1 + v);
        else v = aces_curve(v);
        s_rgb[3 * threadIdx.x + k] = srgb8(v);
      }
    }
  }
  __syncthreads();
  // Both outputs start 16-byte aligned and every block's part is a multiple of 16 bytes,
  // but for the last block's.
  if (mean_out) {
    double* const to = mean_out + 3 * first;
    const int n2 = 3 * here / 2;
    for (int k = threadIdx.x; k < n2; k += kResolveBlock)
      reinterpret_cast<double2*>(to)[k] = reinterpret_cast<const double2*>(s_mean)[k];
    if ((3 * here & 1) && threadIdx.x == 0) to[3 * here - 1] = s_mean[3 * here - 1];
  }
  if (rgb8) {
    std::uint8_t* const to = rgb8 + 3 * first;
    const int n4 = 3 * here / 4;
    for (int k = threadIdx.x; k < n4; k += kResolveBlock)
      reinterpret_cast<std::uint32_t*>(to)[k] = reinterpret_cast<const std::uint32_t*>(s_rgb)[k];
    for (int k = 4 * n4 + threadIdx.x; k < 3 * here; k += kResolveBlock) to[k] = s_rgb[k];
  }
}

// ---------------------------------------------------------------------------
// `tree` picks the walk: 8 the eight-wide tree; otherwise the binary tree
// (closest hit) or the four-wide tree (any hit).
// Results leave in the form the caller gets (t 0 and id -1 on a miss; the plane's
// index where `plane` is 1). Rays and results may be pinned host memory: each is read
// or written once, in order.
template <int kBlock>
__global__ void __launch_bounds__(kBlock) k_ray_closest(const RtgSceneDev* __restrict__ job, const float4* __restrict__ rays,
                                                        std::uint32_t n, RayResults out, int brute, int tree) {
  __shared__ uint2 stack[kStackSmem * kBlock];
  const std::uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  const float4 a = rays[2 * i], b = rays[2 * i + 1];
  TraceCount tc;
  RayHit h;
  if (brute) h = closest_brute<false>(*job, f3(a), f3(b), a.w, b.w, tc);
  else if (tree == 8) h = closest_hit8<kStackSmem, kBlock, false>(*job, f3(a), f3(b), a.w, b.w, stack + threadIdx.x, tc);
  else h = closest_hit<kStackSmem, kBlock, false>(*job, f3(a), f3(b), a.w, b.w, reinterpret_cast<int*>(stack) + threadIdx.x, tc);
  refine_hit(*job, f3(a), f3(b), h);
  const bool miss = h.word == kHitMiss, plane = !miss && (h.word & kHitPlaneBit);
  out.t[i] = miss ? 0.f : h.t;
  out.prim[i] = miss ? -1
                     : static_cast<std::int32_t>(plane ? h.word & ~kHitPlaneBit
                                                       : __float_as_uint(job->prims[3 * h.word].w) & kIdMask);
  out.plane[i] = plane ? 1 : 0;
  out.bary[i] = make_float2(h.b1, h.b2);
}

template <int kBlock>
__global__ void __launch_bounds__(kBlock) k_ray_any(const RtgSceneDev* __restrict__ job, const float4* __restrict__ rays,
                                                    std::uint32_t n, std::uint8_t* out, int brute, int tree) {
  __shared__ uint2 stack[kStackSmem * kBlock];
  const std::uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  const float4 a = rays[2 * i], b = rays[2 * i + 1];
  TraceCount tc;
  bool hit;
  if (brute) hit = any_brute(*job, f3(a), f3(b), a.w, b.w);
  else if (tree == 8) hit = any_hit8<kStackSmem, kBlock, false>(*job, f3(a), f3(b), a.w, b.w, stack + threadIdx.x, tc);
  else hit = any_hit4<kStackSmem, kBlock, false>(*job, f3(a), f3(b), a.w, b.w, reinterpret_cast<int*>(stack) + threadIdx.x, tc);
  out[i] = hit ? 1 : 0;
}

// Launch with programmatic stream serialization (when enabled) so the kernel's
// blocks are scheduled while the previous wavefront kernel drains.
template <class... KArgs, class... Args>
cudaError_t launch_chained(void (*kernel)(KArgs...), int grid, int block, std::size_t smem, bool pdl,
                           cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Persistent grid of a kernel on the current device: every resident block, at most
// `cap` an SM.
struct Grid {
  cudaError_t err = cudaSuccess;
  int sms = 0, per_sm = 0;
};

// A kernel's grids by device: the shared-memory limit is set on each device that the
// kernel runs on, and contexts of several devices launch from several threads. What
// fails is asked again at the next launch.
class GridTable {
 public:
  template <class K>
  Grid get(K kernel, int block, std::size_t smem, int cap) {
    Grid g;
    int dev = 0;
    g.err = cudaGetDevice(&dev);
    if (g.err != cudaSuccess) return g;
    std::lock_guard<std::mutex> hold(lock_);
    const auto known = by_device_.find(dev);
    if (known != by_device_.end()) return known->second;
    g.err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (g.err == cudaSuccess) g.err = cudaDeviceGetAttribute(&g.sms, cudaDevAttrMultiProcessorCount, dev);
    if (g.err == cudaSuccess) g.err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g.per_sm, kernel, block, smem);
    if (g.err != cudaSuccess) return g;
    g.per_sm = g.per_sm < 1 ? 1 : (g.per_sm > cap ? cap : g.per_sm);
    return by_device_.emplace(dev, g).first->second;
  }

 private:
  std::mutex lock_;
  std::map<int, Grid> by_device_;
};

// At most kMaxPathsPerSm path slots per SM, whatever extend_blocks asks for.
template <int kBlock, bool kMis, bool kGeneral>
cudaError_t launch_path(const WaveBuffers& wb, int par, const LaunchShape& shape, cudaStream_t stream) {
  constexpr std::size_t smem = kBlock / 32 * kWarpSmem<kMis, kGeneral>;
  constexpr int kMaxBlocksPerSm = kMaxPathsPerSm / kWarpPaths / (kBlock / 32);
  static GridTable grids;
  const Grid grid = grids.get(k_path<kBlock, kMis, kGeneral>, kBlock, smem, kMaxBlocksPerSm);
  if (grid.err != cudaSuccess) return grid.err;
  int blocks = shape.extend_blocks > 0 ? shape.extend_blocks : grid.sms * grid.per_sm;
  blocks = blocks < grid.sms * kMaxBlocksPerSm ? blocks : grid.sms * kMaxBlocksPerSm;
  return launch_chained(k_path<kBlock, kMis, kGeneral>, blocks, kBlock, smem, shape.chained, stream, wb, par,
                        shape.closest_tree, shape.shadow_tree);
}

template <int kBlock>
cudaError_t launch_path(const WaveBuffers& wb, int par, const LaunchShape& shape, cudaStream_t stream) {
  if (shape.general) return shape.mis ? launch_path<kBlock, true, true>(wb, par, shape, stream)
                                      : launch_path<kBlock, false, true>(wb, par, shape, stream);
  return shape.mis ? launch_path<kBlock, true, false>(wb, par, shape, stream)
                   : launch_path<kBlock, false, false>(wb, par, shape, stream);
}

}  // namespace

cudaError_t launch_plan(const WaveBuffers& wb, int parity, const LaunchShape& shape, cudaStream_t stream) {
  return launch_chained(k_plan, 1, kMaxGen, 0, shape.chained, stream, wb, parity);
}

cudaError_t launch_paths(const WaveBuffers& wb, int parity, const LaunchShape& shape, cudaStream_t stream) {
  switch (shape.block) {
    case 64: return launch_path<64>(wb, parity, shape, stream);
    case 256: return launch_path<256>(wb, parity, shape, stream);
    default: return launch_path<128>(wb, parity, shape, stream);
  }
}

cudaError_t launch_accumulate(const RtgSceneDev* job_dev, std::uint64_t pixels, const PassList& passes,
                              const float4* radiance, cudaStream_t stream) {
  const unsigned blocks = static_cast<unsigned>((pixels + 255) / 256);
  k_accumulate<<<blocks, 256, 0, stream>>>(job_dev, passes, radiance);
  return cudaGetLastError();
}

namespace {
constexpr int kDirectBlock = 128;
template <bool kGeneral>
cudaError_t launch_direct_instance(const RtgSceneDev* job_dev, const PassList& passes, float4* radiance,
                                   WaveCounters* cnt, bool by_warp, float4* pending, int pending_depth, int tree,
                                   cudaStream_t stream) {
  if (!by_warp) {
    constexpr int kMaxPerSm = 2048 / kDirectBlock;
    static GridTable grids;
    const Grid grid = grids.get(k_direct_sample<kDirectBlock, kGeneral>, kDirectBlock, 0, kMaxPerSm);
    if (grid.err != cudaSuccess) return grid.err;
    k_direct_sample<kDirectBlock, kGeneral><<<grid.sms * grid.per_sm, kDirectBlock, 0, stream>>>(job_dev, passes,
                                                                                               radiance, cnt, tree);
    return cudaGetLastError();
  }
  constexpr std::size_t smem = kDirectBlock / 32 * kDirectWarpSmem<kGeneral>;
  static GridTable grids;
  const Grid grid = grids.get(k_direct<kDirectBlock, kGeneral>, kDirectBlock, smem, kPathThreads / kDirectBlock);
  if (grid.err != cudaSuccess) return grid.err;
  const cudaError_t e = cudaMemsetAsync(&cnt->direct_fetch, 0, sizeof(cnt->direct_fetch), stream);
  if (e != cudaSuccess) return e;
  k_direct<kDirectBlock, kGeneral><<<grid.sms * grid.per_sm, kDirectBlock, smem, stream>>>(
      job_dev, passes, radiance, cnt, pending, pending_depth, tree);
  return cudaGetLastError();
}
}  // namespace

bool direct_by_warp(std::uint64_t samples) { return samples >= kDirectWarpSamples; }

int direct_pending_depth(int max_depth) { return max_depth < kDirectStack ? max_depth : kDirectStack; }

std::size_t direct_pending_bytes(int sms, int pending_depth) {
  return static_cast<std::size_t>(sms) * (kPathThreads / 32) * kDirectPaths * pending_depth * kPendingRows * sizeof(float4);
}

cudaError_t launch_direct(const RtgSceneDev* job_dev, const PassList& passes, float4* radiance, WaveCounters* cnt,
                          bool by_warp, float4* pending, int pending_depth, bool general, int tree, cudaStream_t stream) {
  return general ? launch_direct_instance<true>(job_dev, passes, radiance, cnt, by_warp, pending, pending_depth, tree, stream)
                 : launch_direct_instance<false>(job_dev, passes, radiance, cnt, by_warp, pending, pending_depth, tree, stream);
}

cudaError_t launch_resolve(const double* fb_sum, const std::uint32_t* fb_count, std::uint64_t pixels, int tone_map,
                           double exposure, std::uint8_t* rgb8, double* mean_out, cudaStream_t stream) {
  if (pixels == 0) return cudaSuccess;
  const unsigned blocks = static_cast<unsigned>((pixels + kResolveBlock - 1) / kResolveBlock);
  k_resolve<<<blocks, kResolveBlock, 0, stream>>>(fb_sum, fb_count, pixels, tone_map, exposure, rgb8, mean_out);
  return cudaGetLastError();
}

cudaError_t launch_ray_closest(const RtgSceneDev* job_dev, const float4* rays, std::uint32_t n, const RayResults& out,
                               int brute, int tree, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_ray_closest<128><<<(n + 127) / 128, 128, 0, stream>>>(job_dev, rays, n, out, brute, tree);
  return cudaGetLastError();
}

cudaError_t launch_ray_any(const RtgSceneDev* job_dev, const float4* rays, std::uint32_t n, std::uint8_t* out, int brute,
                           int tree, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_ray_any<128><<<(n + 127) / 128, 128, 0, stream>>>(job_dev, rays, n, out, brute, tree);
  return cudaGetLastError();
}

}  // namespace rtg
