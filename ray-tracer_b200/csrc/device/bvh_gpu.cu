// BVH build on the GPU (see bvh_gpu.h for the scheme).
//
// This file is compiled with --fmad=false: the SAH costs, box areas and bin
// indices must round exactly as the host's (and the reference's) double
// arithmetic does, and a fused multiply-add would round once where they round
// twice. The build follows src/geometry/bvh.cpp:28-163 of the reference: 16
// bins per axis, traversal cost 1, leaves of <= 4 primitives (<= 16 when no
// split is cheaper), depth cap 60, the middle split when every centroid
// coincides or a partition leaves one side empty, and std::partition.
#include "device/bvh_gpu.h"
#include "host/alloc_count.hpp"

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

namespace rtg {

namespace {

constexpr int kBins = 16;
constexpr int kDepthCap = 60;
constexpr int kSmallItems = 32;          // a warp builds a node this small, and its subtree, whole
constexpr int kMidItems = 1024;          // a block builds a node this small down to the small ones
constexpr int kMidWarps = 8;
constexpr int kChunk = 256;              // primitives per warp in the level passes (8 per lane)
constexpr int kBinWords = 3 * kBins * 7; // per large node: 3 axes x 16 bins x (6 box keys + count)
constexpr int kMaxLevels = 64;
constexpr int kWarpsPerBlock = 4;

#define BVH_CK(x)                                                                      \
  do {                                                                                 \
    cudaError_t e_ = (x);                                                              \
    if (e_ != cudaSuccess)                                                             \
      throw std::runtime_error(std::string("CUDA (bvh build): ") + cudaGetErrorString(e_)); \
  } while (0)

// Counters the build shares between kernels and with the host.
struct LevelCount {
  int tasks;   // large nodes of a level
  int chunks;  // their 256-primitive chunks
  int base;    // the first of them in the task list
};
struct Counters {
  int nodes;          // node ids handed out
  int mid_roots;      // nodes built by one block
  int small_roots;    // nodes built whole by one warp
  int error;          // 1: a leaf of more than 65535 primitives; 2: partition counts disagree
  int leaves, max_leaf, max_depth;
  int interior;       // interior nodes (root's interior subtree size)
  int wide_total;
  LevelCount lvl[kMaxLevels + 1];
  int wide_cnt[kMaxLevels + 2];
  int wide_off[kMaxLevels + 2];
};

// Doubles as integers whose signed order is the doubles' order, so atomicMin /
// atomicMax on the keys take box unions exactly.
__device__ __forceinline__ long long key_of(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (b ^ 0x7FFFFFFFFFFFFFFFLL);
}
__device__ __forceinline__ double value_of(long long k) {
  return __longlong_as_double(k >= 0 ? k : (k ^ 0x7FFFFFFFFFFFFFFFLL));
}
constexpr long long kKeyPosInf = 0x7FF0000000000000LL;   // key_of(+inf)
constexpr long long kKeyNegInf = -0x7FF0000000000001LL;  // key_of(-inf) = 0x800FFFFFFFFFFFFF

__device__ __forceinline__ double box_area(const double lo[3], const double hi[3]) {
  if (lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2]) return 0.0;
  const double ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
  return 2.0 * (ex * ey + ey * ez + ez * ex);
}

__device__ __forceinline__ int bin_of(double c, double lo, double inv_width) {
  const int b = static_cast<int>((c - lo) * inv_width);
  return min(max(b, 0), kBins - 1);
}

__device__ __forceinline__ int widest_axis(const double lo[3], const double hi[3]) {
  const double ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
  return (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
}

__device__ __forceinline__ void load_box(const double* boxes, unsigned id, double lo[3], double hi[3]) {
  const double2* b = reinterpret_cast<const double2*>(boxes + 6ull * id);
  const double2 a = __ldg(b), m = __ldg(b + 1), z = __ldg(b + 2);
  lo[0] = a.x; lo[1] = a.y; lo[2] = m.x;
  hi[0] = m.y; hi[1] = z.x; hi[2] = z.y;
}

// Smallest and largest double of a warp (no NaN), by the order of its key's words: four
// reductions in hardware in place of 30 shuffles and compares.
__device__ __forceinline__ double warp_min(double v) {
  const long long k = key_of(v);
  const int hi = static_cast<int>(k >> 32);
  const unsigned lo = static_cast<unsigned>(k);
  const int best = __reduce_min_sync(0xFFFFFFFFu, hi);
  const unsigned low = __reduce_min_sync(0xFFFFFFFFu, hi == best ? lo : 0xFFFFFFFFu);
  return value_of((static_cast<long long>(best) << 32) | low);
}
__device__ __forceinline__ double warp_max(double v) { return -warp_min(-v); }
// Of two doubles, no NaN (fmin and fmax spend most of their instructions on those).
__device__ __forceinline__ double less_of(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double more_of(double a, double b) { return b > a ? b : a; }

// One float step toward -inf / +inf by bits (std::nextafterf for finite f).
__device__ __forceinline__ float step_down(float f) {
  if (f == 0.f) return -__int_as_float(1);
  const unsigned u = __float_as_uint(f);
  return __uint_as_float(f > 0.f ? u - 1u : u + 1u);
}
__device__ __forceinline__ float step_up(float f) {
  if (f == 0.f) return __int_as_float(1);
  const unsigned u = __float_as_uint(f);
  return __uint_as_float(f > 0.f ? u + 1u : u - 1u);
}
// A node bound rounded outward to fp32 and widened, exactly as the host flattener
// does it (flatten.cpp down / up).
__device__ __forceinline__ float round_down(double v) {
  float f = __double2float_rn(v);
  if (static_cast<double>(f) > v) f = step_down(f);
  f -= fabsf(f) * 0x1p-22f;
  return step_down(f);
}
__device__ __forceinline__ float round_up(double v) {
  float f = __double2float_rn(v);
  if (static_cast<double>(f) < v) f = step_up(f);
  f += fabsf(f) * 0x1p-22f;
  return step_up(f);
}

}  // namespace

// Device pointers of one build's scratch memory.
struct GpuBvhBuilder::State {
  std::uint32_t n = 0, nn = 0, max_level_tasks = 0, max_chunks = 0;
  Counters* counters = nullptr;
  Counters* host_counters = nullptr;  // pinned copy
  std::uint32_t* items = nullptr;     // working order (becomes the leaf order)
  std::uint32_t* scratch = nullptr;   // partition partner positions
  // per node
  double* box = nullptr;              // 6 per node
  long long* key = nullptr;           // 12 per node: box lo, box hi, centroid lo, centroid hi (large nodes)
  int* left = nullptr;
  int* right = nullptr;
  std::uint32_t* first = nullptr;
  std::uint32_t* count = nullptr;
  int* depth = nullptr;
  int* axis = nullptr;
  int* size = nullptr;
  int* isize = nullptr;
  int* dfs = nullptr;
  int* idfs = nullptr;
  int* sub = nullptr;                 // small subtree root, or -1
  int* local = nullptr;               // preorder index inside the small subtree
  int* ilocal = nullptr;              // interior preorder index inside the small subtree
  int* tasks = nullptr;               // large nodes, level after level
  int* mid_roots = nullptr;
  int* mid_nodes = nullptr;           // nodes a block builds, level after level, from its root's first primitive on
  int* mid_ends = nullptr;            // ends of those levels, kMaxLevels per root
  int* small_roots = nullptr;
  // per level of large nodes, by parity
  long long* bins[2] = {};
  int* task_chunk0[2] = {};
  int* task_nchunks[2] = {};
  int* need_part[2] = {};
  int* part_t[2] = {};
  int* part_m[2] = {};
  int* part_axis[2] = {};
  int* part_bin[2] = {};
  double* part_lo[2] = {};
  double* part_inv[2] = {};
  int* chunk_task[2] = {};
  std::uint32_t* chunk_start[2] = {};
  int* cnt_lf[2] = {};
  int* cnt_rt[2] = {};
  int* base_lf[2] = {};
  int* base_rt[2] = {};
  unsigned* moves = nullptr;
  // four-wide collapse
  int* wide_list = nullptr;
  int* wide_kids = nullptr;           // 4 per binary node
  std::uint32_t* wflag = nullptr;     // by depth-first index
  std::uint32_t* wscan = nullptr;
  std::uint32_t* scan_sums = nullptr;
  std::uint8_t* last = nullptr;       // last slot of a leaf
};

namespace {

__device__ __forceinline__ double pos_inf() { return __longlong_as_double(0x7FF0000000000000LL); }

// Pointers the level kernels share; the *_next arrays belong to the level they create.
// Sizes come from the counters, so the host launches levels without waiting for them.
struct LevelArgs {
  const double* boxes;
  std::uint32_t* items;
  std::uint32_t* scratch;
  double* box;
  long long* key;
  int* left;
  int* right;
  std::uint32_t* first;
  std::uint32_t* count;
  int* depth;
  int* axis;
  int* sub;
  int* tasks;  // large nodes, level after level
  int* mid_roots;
  int* small_roots;
  Counters* counters;
  int level;
  long long* bins;
  int* need_part;
  int* part_t;
  int* part_m;
  int* part_axis;
  int* part_bin;
  double* part_lo;
  double* part_inv;
  int* task_chunk0;
  int* task_nchunks;
  int* chunk_task;
  std::uint32_t* chunk_start;
  int* cnt_lf;
  int* cnt_rt;
  int* base_lf;
  int* base_rt;
  unsigned* moves;  // 8 words a chunk
  long long* bins_next;
  int* task_chunk0_next;
  int* task_nchunks_next;
  int* chunk_task_next;
  std::uint32_t* chunk_start_next;
  __device__ int n_tasks() const { return counters->lvl[level].tasks; }
  __device__ int n_chunks() const { return counters->lvl[level].chunks; }
  __device__ int task(int i) const { return tasks[counters->lvl[level].base + i]; }
};

// One bin of one axis as a lane holds it.
struct BinData {
  double lo[3], hi[3];
  unsigned n;
};

__device__ __forceinline__ void bin_clear(BinData& e) {
  const double inf = pos_inf();
  for (int k = 0; k < 3; ++k) {
    e.lo[k] = inf;
    e.hi[k] = -inf;
  }
  e.n = 0;
}

__device__ __forceinline__ void note_leaf(Counters* c, std::uint32_t n, int d) {
  if (n > 0xFFFFu) atomicOr(&c->error, 1);
  atomicAdd(&c->leaves, 1);
  atomicMax(&c->max_leaf, static_cast<int>(n));
  atomicMax(&c->max_depth, d);
}

// Registers node c (primitives [first, first + n) of the working order, at
// `depth`) as a large node of level `next`, with its chunks, or as the root of a
// subtree that one block or one warp builds. Called by all 32 lanes of a warp.
__device__ void enqueue_node(const LevelArgs& a, int next, int next_base, int c, std::uint32_t first, std::uint32_t n,
                             int depth) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    a.first[c] = first;
    a.count[c] = n;
    a.depth[c] = depth;
    a.sub[c] = -1;
    a.left[c] = -1;
    a.right[c] = -1;
  }
  if (n > static_cast<std::uint32_t>(kMidItems)) {
    const int nch = static_cast<int>((n + kChunk - 1) / kChunk);
    int slot = 0, c0 = 0;
    if (lane == 0) {
      LevelCount& l = a.counters->lvl[next];
      slot = atomicAdd(&l.tasks, 1);
      c0 = atomicAdd(&l.chunks, nch);
      l.base = next_base;
      a.tasks[next_base + slot] = c;
      a.task_chunk0_next[slot] = c0;
      a.task_nchunks_next[slot] = nch;
    }
    slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
    c0 = __shfl_sync(0xFFFFFFFFu, c0, 0);
    // Empty bounds (lo +inf, hi -inf for the box and the centroids) and bins.
    if (lane < 12) a.key[12ll * c + lane] = (lane % 6) < 3 ? kKeyPosInf : kKeyNegInf;
    long long* g = a.bins_next + static_cast<long long>(slot) * kBinWords;
    for (int i = lane; i < kBinWords; i += 32) {
      const int f = i % 7;
      g[i] = f < 3 ? kKeyPosInf : (f < 6 ? kKeyNegInf : 0);
    }
    for (int j = lane; j < nch; j += 32) {
      a.chunk_task_next[c0 + j] = slot;
      a.chunk_start_next[c0 + j] = first + static_cast<std::uint32_t>(j) * kChunk;
    }
  } else if (lane == 0) {
    if (n > static_cast<std::uint32_t>(kSmallItems)) a.mid_roots[atomicAdd(&a.counters->mid_roots, 1)] = c;
    else a.small_roots[atomicAdd(&a.counters->small_roots, 1)] = c;
  }
}

// The root: node 0 over every primitive. Launched with one warp, with level 0's
// arrays as the next.
__global__ void k_init(LevelArgs a, std::uint32_t n, int* dfs, int* idfs) {
  if (blockIdx.x != 0) return;
  if (threadIdx.x == 0) {
    a.counters->nodes = 1;
    dfs[0] = 0;
    idfs[0] = 0;
  }
  enqueue_node(a, 0, 0, 0, 0, n, 0);
}

// Box and centroid bounds of each large node: one warp per 256-primitive chunk.
__global__ void __launch_bounds__(128) k_bounds(LevelArgs a) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= a.n_chunks()) return;
  const int t = a.task(a.chunk_task[w]);
  const std::uint32_t start = a.chunk_start[w];
  const std::uint32_t end = min(start + static_cast<std::uint32_t>(kChunk), a.first[t] + a.count[t]);
  const double inf = pos_inf();
  double lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
  double clo[3] = {inf, inf, inf}, chi[3] = {-inf, -inf, -inf};
  std::uint32_t id[kChunk / 32];
#pragma unroll
  for (int j = 0; j < kChunk / 32; ++j) {
    // Past the end, the chunk's first primitive once more: a union may take it twice.
    const std::uint32_t pos = start + static_cast<std::uint32_t>(j * 32 + lane);
    id[j] = a.items[pos < end ? pos : start];
  }
#pragma unroll 4
  for (int j = 0; j < kChunk / 32; ++j) {
    double bl[3], bh[3];
    load_box(a.boxes, id[j], bl, bh);
    for (int k = 0; k < 3; ++k) {
      lo[k] = less_of(lo[k], bl[k]);
      hi[k] = more_of(hi[k], bh[k]);
      const double c = 0.5 * (bl[k] + bh[k]);
      clo[k] = less_of(clo[k], c);
      chi[k] = more_of(chi[k], c);
    }
  }
  for (int k = 0; k < 3; ++k) {
    lo[k] = warp_min(lo[k]);
    hi[k] = warp_max(hi[k]);
    clo[k] = warp_min(clo[k]);
    chi[k] = warp_max(chi[k]);
  }
  if (lane == 0) {
    long long* key = a.key + 12ll * t;
    for (int k = 0; k < 3; ++k) {
      atomicMin(&key[k], key_of(lo[k]));
      atomicMax(&key[3 + k], key_of(hi[k]));
      atomicMin(&key[6 + k], key_of(clo[k]));
      atomicMax(&key[9 + k], key_of(chi[k]));
    }
  }
}

// Bin boxes and counts of each large node (16 bins per axis over the centroid
// bounds): warp-private bins in shared memory, then merged with atomics.
__global__ void __launch_bounds__(kWarpsPerBlock * 32) k_bins(LevelArgs a) {
  __shared__ long long s_bins[kWarpsPerBlock][kBinWords];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kWarpsPerBlock + wib;
  if (w >= a.n_chunks()) return;
  const int lt = a.chunk_task[w];
  const int t = a.task(lt);
  if (a.depth[t] >= kDepthCap) return;  // becomes a leaf
  const long long* key = a.key + 12ll * t;
  double clo[3], inv[3];
  bool use[3];
  for (int k = 0; k < 3; ++k) {
    clo[k] = value_of(key[6 + k]);
    const double chi = value_of(key[9 + k]);
    use[k] = chi > clo[k];
    inv[k] = use[k] ? kBins / (chi - clo[k]) : 0.0;
  }
  long long* s = s_bins[wib];
  for (int i = lane; i < kBinWords; i += 32) {
    const int f = i % 7;
    s[i] = f < 3 ? kKeyPosInf : (f < 6 ? kKeyNegInf : 0);
  }
  __syncwarp();
  // Each lane takes 8 consecutive primitives (neighbours in the working order
  // are usually neighbours in space) and merges a run of primitives that fall in
  // the same bin before it touches shared memory.
  const std::uint32_t start = a.chunk_start[w];
  const std::uint32_t end = min(start + static_cast<std::uint32_t>(kChunk), a.first[t] + a.count[t]);
  constexpr int kPerLane = kChunk / 32;
  int run_bin[3] = {-1, -1, -1};
  BinData run[3];
  auto flush = [&](int k) {
    if (run_bin[k] < 0) return;
    long long* e = s + 7 * (k * kBins + run_bin[k]);
    for (int m = 0; m < 3; ++m) {
      atomicMin(&e[m], key_of(run[k].lo[m]));
      atomicMax(&e[3 + m], key_of(run[k].hi[m]));
    }
    atomicAdd(reinterpret_cast<unsigned long long*>(&e[6]), static_cast<unsigned long long>(run[k].n));
  };
  for (int j = 0; j < kPerLane; ++j) {
    const std::uint32_t pos = start + static_cast<std::uint32_t>(lane * kPerLane + j);
    if (pos >= end) break;
    double bl[3], bh[3];
    load_box(a.boxes, a.items[pos], bl, bh);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (!use[k]) continue;
      const int b = bin_of(0.5 * (bl[k] + bh[k]), clo[k], inv[k]);
      if (b != run_bin[k]) {
        flush(k);
        run_bin[k] = b;
        bin_clear(run[k]);
      }
      for (int m = 0; m < 3; ++m) {
        run[k].lo[m] = less_of(run[k].lo[m], bl[m]);
        run[k].hi[m] = more_of(run[k].hi[m], bh[m]);
      }
      ++run[k].n;
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) flush(k);
  __syncwarp();
  long long* g = a.bins + static_cast<long long>(lt) * kBinWords;
  for (int q = lane; q < 3 * kBins; q += 32) {
    const long long* e = s + 7 * q;
    if (e[6] == 0) continue;
    long long* ge = g + 7 * q;
    atomicAdd(reinterpret_cast<unsigned long long*>(&ge[6]), static_cast<unsigned long long>(e[6]));
    for (int m = 0; m < 3; ++m) {
      atomicMin(&ge[m], e[m]);
      atomicMax(&ge[3 + m], e[3 + m]);
    }
  }
}

// A warp's bins during the sweep, 16 an axis: lower corners and negated upper ones, so
// that every union is a minimum, and counts.
struct Sweep {
  double box[3 * kBins][6];
  unsigned n[3 * kBins];
};

__device__ __forceinline__ void store_bins(Sweep& w, const BinData& r0, const BinData& r1) {
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < 3; ++k) {
    w.box[lane][k] = r0.lo[k];
    w.box[lane][3 + k] = -r0.hi[k];
  }
  w.n[lane] = r0.n;
  if (lane < kBins) {
    for (int k = 0; k < 3; ++k) {
      w.box[2 * kBins + lane][k] = r1.lo[k];
      w.box[2 * kBins + lane][3 + k] = -r1.hi[k];
    }
    w.n[2 * kBins + lane] = r1.n;
  }
}
__device__ __forceinline__ void merge_bins(const Sweep& w, BinData& r0, BinData& r1) {
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < 3; ++k) {
    r0.lo[k] = less_of(r0.lo[k], w.box[lane][k]);
    r0.hi[k] = more_of(r0.hi[k], -w.box[lane][3 + k]);
  }
  r0.n += w.n[lane];
  if (lane < kBins) {
    for (int k = 0; k < 3; ++k) {
      r1.lo[k] = less_of(r1.lo[k], w.box[2 * kBins + lane][k]);
      r1.hi[k] = more_of(r1.hi[k], -w.box[2 * kBins + lane][3 + k]);
    }
    r1.n += w.n[2 * kBins + lane];
  }
}

// The cheapest plane of each axis (src/geometry/bvh.cpp:62-88), as lane b of a
// 16-lane half holds the plane after bin b of that half's axis: the lowest bin on ties,
// which is the first strictly cheaper plane of the reference's loop.
__device__ __forceinline__ void half_best(double& cost, int& bin, unsigned& left_n) {
  const unsigned full = 0xFFFFFFFFu;
  for (int o = 8; o >= 1; o >>= 1) {
    const double oc = __shfl_xor_sync(full, cost, o, 16);
    const int ob = __shfl_xor_sync(full, bin, o, 16);
    const unsigned ol = __shfl_xor_sync(full, left_n, o, 16);
    if (oc < cost || (oc == cost && ob < bin)) {
      cost = oc;
      bin = ob;
      left_n = ol;
    }
  }
}

// The best split over the three axes, on every lane: r0 holds axis 0 (lanes
// 0-15) and axis 1 (lanes 16-31), r1 axis 2 (lanes 0-15). Axes in order, the
// first strictly cheaper wins; an axis whose centroids coincide is skipped.
//
// The unions left and right of each plane are running minima in shared memory, a lane
// for each axis and component: 2 x 16 short steps. Scans of 12 doubles by shuffles took
// some 1,500 instructions a node, and their unrolled code missed the instruction cache.
__device__ void warp_best_split(Sweep& w, const BinData& r0, const BinData& r1, const bool use[3], double parent_area,
                                double& best_cost, int& best_axis, int& best_bin, unsigned& best_left) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, b = lane & 15;
  const double area_floor = parent_area < 1e-30 ? 1e-30 : parent_area;
  // Of the planes after bin `lane` and bin 32 + lane: counts, and the left side's price.
  double price[2];
  unsigned ln[2], rn[2];
  double c0 = pos_inf(), c1 = pos_inf();
#pragma unroll 1
  for (int right = 0; right < 2; ++right) {
    store_bins(w, r0, r1);
    __syncwarp();
    if (lane < 18) {
      const int ax = lane / 6, c = lane - 6 * ax, step = right ? -1 : 1;
      int q = ax * kBins + (right ? kBins - 1 : 0);
      double v = w.box[q][c];
#pragma unroll 5
      for (int k = 1; k < kBins; ++k) {
        q += step;
        v = less_of(v, w.box[q][c]);
        w.box[q][c] = v;
      }
    } else if (lane < 21) {
      const int step = right ? -1 : 1;
      int q = (lane - 18) * kBins + (right ? kBins - 1 : 0);
      unsigned v = w.n[q];
#pragma unroll 5
      for (int k = 1; k < kBins; ++k) {
        q += step;
        v += w.n[q];
        w.n[q] = v;
      }
    }
    __syncwarp();
    auto side = [&](int q, unsigned& n) {
      const double* e = w.box[q];
      const double lo[3] = {e[0], e[1], e[2]}, hi[3] = {-e[3], -e[4], -e[5]};
      n = w.n[q];
      return box_area(lo, hi) * double(n);
    };
    // The right side of the plane after bin q starts at q + 1.
    for (int r = 0; r < 2; ++r) {
      if (r == 1 && lane >= kBins) break;
      const int q = 2 * kBins * r + lane;
      if (!right) {
        price[r] = side(q, ln[r]);
      } else if (b < kBins - 1) {
        const double p = side(q + 1, rn[r]);
        if (ln[r] != 0 && rn[r] != 0) (r ? c1 : c0) = 1.0 + (price[r] + p) / area_floor;
      }
    }
    __syncwarp();
  }
  int b0 = b, b1 = b;
  unsigned l0 = ln[0], l1 = lane < kBins ? ln[1] : 0u;
  half_best(c0, b0, l0);
  half_best(c1, b1, l1);
  const double cost[3] = {__shfl_sync(full, c0, 0), __shfl_sync(full, c0, 16), __shfl_sync(full, c1, 0)};
  const int bin[3] = {__shfl_sync(full, b0, 0), __shfl_sync(full, b0, 16), __shfl_sync(full, b1, 0)};
  const unsigned left[3] = {__shfl_sync(full, l0, 0), __shfl_sync(full, l0, 16), __shfl_sync(full, l1, 0)};
  best_cost = pos_inf();
  best_axis = -1;
  best_bin = -1;
  best_left = 0;
  for (int ax = 0; ax < 3; ++ax)
    if (use[ax] && cost[ax] < best_cost) {
      best_cost = cost[ax];
      best_axis = ax;
      best_bin = bin[ax];
      best_left = left[ax];
    }
}

// One warp per large node: box from the keys, SAH decision, children.
__global__ void __launch_bounds__(128) k_decide(LevelArgs a) {
  __shared__ Sweep s_sweep[4];
  const int i = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= a.n_tasks()) return;
  const int t = a.task(i);
  const long long* key = a.key + 12ll * t;
  double lo[3], hi[3], clo[3], chi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = value_of(key[k]);
    hi[k] = value_of(key[3 + k]);
    clo[k] = value_of(key[6 + k]);
    chi[k] = value_of(key[9 + k]);
  }
  if (lane == 0)
    for (int k = 0; k < 3; ++k) {
      a.box[6ll * t + k] = lo[k];
      a.box[6ll * t + 3 + k] = hi[k];
    }
  const std::uint32_t n = a.count[t], f0 = a.first[t];
  const int d = a.depth[t];
  bool leaf = n <= 4 || d >= kDepthCap;
  int split_axis = -1;
  std::uint32_t mid = 0;
  bool part = false;
  int best_bin = -1;
  if (!leaf) {
    bool use[3];
    for (int k = 0; k < 3; ++k) use[k] = chi[k] > clo[k];
    const long long* g = a.bins + static_cast<long long>(i) * kBinWords;
    BinData r[2];
    for (int round = 0; round < 2; ++round) {
      bin_clear(r[round]);
      if (round == 1 && lane >= 16) continue;
      const long long* e = g + 7 * ((round == 0 ? (lane >> 4) : 2) * kBins + (lane & 15));
      for (int k = 0; k < 3; ++k) {
        r[round].lo[k] = value_of(e[k]);
        r[round].hi[k] = value_of(e[3 + k]);
      }
      r[round].n = static_cast<unsigned>(e[6]);
    }
    double best_cost;
    unsigned left_n;
    warp_best_split(s_sweep[threadIdx.x >> 5], r[0], r[1], use, box_area(lo, hi), best_cost, split_axis, best_bin, left_n);
    if (split_axis < 0) {
      mid = n / 2;  // every centroid coincides
      split_axis = widest_axis(clo, chi);
    } else if (best_cost >= double(n) && n <= 16) {
      leaf = true;
    } else if (left_n == 0 || left_n == n) {
      mid = n / 2;  // rounding put everything on one side
    } else {
      mid = left_n;
      part = true;
    }
  }
  if (leaf) {
    if (lane == 0) {
      a.left[t] = -1;
      a.right[t] = -1;
      a.axis[t] = 0;
      a.need_part[i] = 0;
      note_leaf(a.counters, n, d);
    }
    return;
  }
  int c = 0;
  if (lane == 0) {
    a.axis[t] = split_axis;
    a.need_part[i] = part ? 1 : 0;
    if (part) {
      a.part_t[i] = static_cast<int>(mid);
      a.part_axis[i] = split_axis;
      a.part_bin[i] = best_bin;
      a.part_lo[i] = clo[split_axis];
      a.part_inv[i] = kBins / (chi[split_axis] - clo[split_axis]);
    }
    c = atomicAdd(&a.counters->nodes, 2);
    a.left[t] = c;
    a.right[t] = c + 1;
  }
  c = __shfl_sync(0xFFFFFFFFu, c, 0);
  const LevelCount& l = a.counters->lvl[a.level];
  const int next_base = l.base + l.tasks;
  enqueue_node(a, a.level + 1, next_base, c, f0, mid, d + 1);
  enqueue_node(a, a.level + 1, next_base, c + 1, f0 + mid, n - mid, d + 1);
}

// A warp's chunk in the partition passes.
struct PartChunk {
  int lt;                          // its node's task
  std::uint32_t f0, start, split, end, last;  // node's first, chunk's first, first of the right side, chunk's and node's end
  bool on;
  __device__ PartChunk(const LevelArgs& a, int w) : on(false) {
    if (w >= a.n_chunks()) return;
    lt = a.chunk_task[w];
    if (!a.need_part[lt]) return;
    on = true;
    const int t = a.task(lt);
    f0 = a.first[t];
    last = f0 + a.count[t];
    start = a.chunk_start[w];
    end = min(start + static_cast<std::uint32_t>(kChunk), last);
    split = f0 + static_cast<std::uint32_t>(a.part_t[lt]);
  }
  // Bits of 32 places from `pos` on that lie on the right side.
  __device__ unsigned right_side(std::uint32_t pos) const {
    return pos >= split ? 0xFFFFFFFFu : (split - pos >= 32 ? 0u : 0xFFFFFFFFu << (split - pos));
  }
};

// Partition, pass 1: per chunk, which primitives belong on the left (a word for 32
// places, which the next passes read in place of the primitives), and how many on the
// left belong on the right ("left-false") and the other way round.
__global__ void __launch_bounds__(128) k_pcount(LevelArgs a) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const PartChunk c(a, w);
  if (!c.on) return;
  const int ax = a.part_axis[c.lt], bin = a.part_bin[c.lt];
  const double lo = a.part_lo[c.lt], inv = a.part_inv[c.lt];
  std::uint32_t id[kChunk / 32];
#pragma unroll
  for (int j = 0; j < kChunk / 32; ++j) {
    const std::uint32_t pos = c.start + static_cast<std::uint32_t>(j * 32 + lane);
    id[j] = pos < c.end ? a.items[pos] : 0xFFFFFFFFu;
  }
  int lf = 0, rt = 0;
#pragma unroll
  for (int j = 0; j < kChunk / 32; ++j) {
    bool l = false;
    if (id[j] != 0xFFFFFFFFu) {
      const double* b = a.boxes + 6ull * id[j];
      l = bin_of(0.5 * (__ldg(b + ax) + __ldg(b + 3 + ax)), lo, inv) <= bin;
    }
    const unsigned bits = __ballot_sync(0xFFFFFFFFu, l);
    const std::uint32_t pos = c.start + static_cast<std::uint32_t>(j * 32);
    const unsigned there = pos >= c.end ? 0u : (c.end - pos >= 32 ? 0xFFFFFFFFu : (1u << (c.end - pos)) - 1u);
    const unsigned right = c.right_side(pos);
    lf += __popc(~bits & there & ~right);
    rt += __popc(bits & right);
    // Left-false and right-true places, the only ones that move.
    if (lane == 0) a.moves[w * (kChunk / 32) + j] = (~bits & there & ~right) | (bits & right);
  }
  if (lane == 0) {
    a.cnt_lf[w] = lf;
    a.cnt_rt[w] = rt;
  }
}

// Partition, pass 2: one warp per node scans its chunks' counts.
__global__ void __launch_bounds__(128) k_pscan(LevelArgs a) {
  const int i = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= a.n_tasks() || !a.need_part[i]) return;
  const int c0 = a.task_chunk0[i], nch = a.task_nchunks[i];
  int carry_lf = 0, carry_rt = 0;
  for (int b = 0; b < nch; b += 32) {
    const bool ok = b + lane < nch;
    const int c = c0 + b + lane;
    const int vl = ok ? a.cnt_lf[c] : 0, vr = ok ? a.cnt_rt[c] : 0;
    int il = vl, ir = vr;
    for (int o = 1; o < 32; o <<= 1) {
      const int xl = __shfl_up_sync(0xFFFFFFFFu, il, o), xr = __shfl_up_sync(0xFFFFFFFFu, ir, o);
      if (lane >= o) {
        il += xl;
        ir += xr;
      }
    }
    if (ok) {
      a.base_lf[c] = carry_lf + il - vl;
      a.base_rt[c] = carry_rt + ir - vr;
    }
    carry_lf += __shfl_sync(0xFFFFFFFFu, il, 31);
    carry_rt += __shfl_sync(0xFFFFFFFFu, ir, 31);
  }
  if (lane == 0) {
    a.part_m[i] = carry_lf;
    if (carry_lf != carry_rt) atomicOr(&a.counters->error, 2);
  }
}

// Partition, pass 3: the k-th right-side primitive that belongs on the left,
// counted from the right end, records its position at scratch[first + k].
__global__ void __launch_bounds__(128) k_pranks(LevelArgs a) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const PartChunk c(a, w);
  if (!c.on) return;
  const int m = a.part_m[c.lt];
  int run = a.base_rt[w];
#pragma unroll
  for (int j = 0; j < kChunk / 32; ++j) {
    const std::uint32_t pos = c.start + static_cast<std::uint32_t>(j * 32);
    const unsigned rt = a.moves[w * (kChunk / 32) + j] & c.right_side(pos);
    if ((rt >> lane) & 1u) {
      const int r = m - 1 - (run + __popc(rt & ((1u << lane) - 1u)));
      if (r >= 0 && r < m) a.scratch[c.f0 + static_cast<std::uint32_t>(r)] = pos + lane;
    }
    run += __popc(rt);
  }
}

// Partition, pass 4: the k-th left-side primitive that belongs on the right
// trades places with the position recorded at scratch[first + k] (Hoare's
// scheme, as std::partition runs it).
__global__ void __launch_bounds__(128) k_pswap(LevelArgs a) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const PartChunk c(a, w);
  if (!c.on) return;
  const int m = a.part_m[c.lt];
  int run = a.base_lf[w];
#pragma unroll
  for (int j = 0; j < kChunk / 32; ++j) {
    const std::uint32_t first = c.start + static_cast<std::uint32_t>(j * 32), pos = first + lane;
    const unsigned lf = a.moves[w * (kChunk / 32) + j] & ~c.right_side(first);
    if ((lf >> lane) & 1u) {
      const int k = run + __popc(lf & ((1u << lane) - 1u));
      if (k < m) {
        const std::uint32_t q = a.scratch[c.f0 + static_cast<std::uint32_t>(k)];
        if (q >= c.split && q < c.last) {  // always true; keeps the swap in the node's range
          const std::uint32_t mine = a.items[pos];
          a.items[pos] = a.items[q];
          a.items[q] = mine;
        }
      }
    }
    run += __popc(lf);
  }
}

}  // namespace

namespace {

// Adds 32 primitives to a node's bins: bin[k] is the bin of this lane's primitive on
// axis k (-1: none), box(p) the box of lane p's. r[0] is axis 0 on lanes 0-15 and axis 1
// on lanes 16-31, r[1] axis 2: primitives 0-15 on lanes 0-15, the others on lanes 16-31,
// until fold_axis2 brings them together. Each lane then visits its own bin's primitives
// only, two at a time. Before, every lane scanned all 32, in 64 divergent steps; with this,
// the sweep and the reductions, k_small takes 240 us on 174k triangles (513). Neighbours
// that share a bin make it slow: k_bins, with 256 neighbours a warp, merges runs instead
// (35 us a level; 59 this way).
template <class Box>
__device__ __forceinline__ void bin_lanes(unsigned* mask, const int bin[3], BinData r[2], Box box) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  for (int q = lane; q < 3 * kBins; q += 32) mask[q] = 0;
  __syncwarp();
  for (int k = 0; k < 3; ++k) {
    const unsigned same = __match_any_sync(full, bin[k]);
    if (bin[k] >= 0 && lane == __ffs(same) - 1) mask[k * kBins + bin[k]] = same;
  }
  __syncwarp();
#pragma unroll
  for (int round = 0; round < 2; ++round) {
    BinData& e = r[round];
    unsigned m = round == 0 ? mask[lane] : (mask[2 * kBins + (lane & 15)] & (lane < 16 ? 0xFFFFu : 0xFFFF0000u));
    e.n += __popc(m);
    while (m) {
      const double* b = box(__ffs(m) - 1);
      const unsigned rest = m & (m - 1);
      const double* b2 = box(__ffs(rest ? rest : m) - 1);  // with none left, the same one again
      m = rest & (rest - 1);
      for (int k = 0; k < 3; ++k) {
        e.lo[k] = less_of(e.lo[k], less_of(b[k], b2[k]));
        e.hi[k] = more_of(e.hi[k], more_of(b[3 + k], b2[3 + k]));
      }
    }
  }
  __syncwarp();
}
__device__ __forceinline__ void fold_axis2(BinData& e) {
  for (int k = 0; k < 3; ++k) {
    e.lo[k] = less_of(e.lo[k], __shfl_xor_sync(0xFFFFFFFFu, e.lo[k], 16));
    e.hi[k] = more_of(e.hi[k], __shfl_xor_sync(0xFFFFFFFFu, e.hi[k], 16));
  }
  e.n += __shfl_xor_sync(0xFFFFFFFFu, e.n, 16);
}

struct MidArgs {
  const double* boxes;
  std::uint32_t* items;
  double* box;
  int* left;
  int* right;
  std::uint32_t* first;
  std::uint32_t* count;
  int* depth;
  int* axis;
  int* sub;
  const int* mid_roots;
  int* mid_nodes;
  int* mid_ends;
  int* small_roots;
  Counters* counters;
};

// A block's workspace: its root's primitives by the place they came in, and their order.
struct MidBlock {
  double box[kMidItems][6];
  std::uint32_t id[kMidItems];
  std::uint16_t order[kMidItems], partner[kMidItems];
  unsigned mask[kMidWarps][3 * kBins];
  Sweep sweep[kMidWarps];
  double bounds[kMidWarps][12];
  int listed;
};

// The last part of a node's split; one warp. Bounds, bins and the rest as split_mids has them.
__device__ void split_mid(const MidArgs& a, MidBlock& s, int* list, std::uint32_t b0, int t, int lo, int n, int d,
                          const double bl[3], const double bh[3], const double cl[3], const double ch[3],
                          const bool use[3], const double inv[3], const BinData r[2]) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, hi = lo + n;
  const unsigned below = (1u << lane) - 1u;
  if (lane == 0)
    for (int k = 0; k < 3; ++k) {
      a.box[6ll * t + k] = bl[k];
      a.box[6ll * t + 3 + k] = bh[k];
    }
  if (d >= kDepthCap) {
    if (lane == 0) {
      a.left[t] = -1;
      a.right[t] = -1;
      a.axis[t] = 0;
      note_leaf(a.counters, static_cast<std::uint32_t>(n), d);
    }
    return;
  }
  double best_cost;
  int axis, best_bin;
  unsigned left_n;
  warp_best_split(s.sweep[threadIdx.x >> 5], r[0], r[1], use, box_area(bl, bh), best_cost, axis, best_bin, left_n);
  int mid = n / 2;  // every centroid coincides, or rounding put everything on one side
  if (axis < 0) {
    axis = widest_axis(cl, ch);
  } else if (left_n != 0 && left_n != static_cast<unsigned>(n)) {
    mid = static_cast<int>(left_n);
    const double c0 = cl[axis], scale = inv[axis];
    auto goes_left = [&](int i) {
      const double* b = s.box[s.order[i]];
      return bin_of(0.5 * (b[axis] + b[3 + axis]), c0, scale) <= best_bin;
    };
    // The k-th primitive from the right end that belongs on the left ...
    int n_right = 0, n_left = 0;
    for (int i0 = hi - 1; i0 >= lo + mid; i0 -= 32) {
      const int i = i0 - lane;
      const bool moves = i >= lo + mid && goes_left(i);
      const unsigned m = __ballot_sync(full, moves);
      if (moves) s.partner[lo + n_right + __popc(m & below)] = static_cast<std::uint16_t>(i);
      n_right += __popc(m);
    }
    __syncwarp();
    // ... trades places with the k-th from the left that belongs on the right.
    for (int i0 = lo; i0 < lo + mid; i0 += 32) {
      const int i = i0 + lane;
      const bool moves = i < lo + mid && !goes_left(i);
      const unsigned m = __ballot_sync(full, moves);
      const int k = n_left + __popc(m & below);
      if (moves && k < n_right) {
        const int q = s.partner[lo + k];
        const std::uint16_t v = s.order[i];
        s.order[i] = s.order[q];
        s.order[q] = v;
      }
      n_left += __popc(m);
    }
    if (lane == 0 && n_left != n_right) atomicOr(&a.counters->error, 2);
    __syncwarp();
  }
  if (lane == 0) {
    const int c = atomicAdd(&a.counters->nodes, 2);
    a.left[t] = c;
    a.right[t] = c + 1;
    a.axis[t] = axis;
    for (int k = 0; k < 2; ++k) {
      const int cn = k ? n - mid : mid;
      a.first[c + k] = b0 + static_cast<std::uint32_t>(k ? lo + mid : lo);
      a.count[c + k] = static_cast<std::uint32_t>(cn);
      a.depth[c + k] = d + 1;
      a.sub[c + k] = -1;
      a.left[c + k] = -1;
      a.right[c + k] = -1;
      if (cn > kSmallItems) list[atomicAdd(&s.listed, 1)] = c + k;
      else a.small_roots[atomicAdd(&a.counters->small_roots, 1)] = c + k;
    }
  }
}

// Splits the block's nodes list[begin .. end). The decisions are k_decide's, the
// exchange the one of k_pcount to k_pswap. Where a level has fewer nodes than the block
// has warps, a team of warps takes each: they share its bounds and its bins, and the
// team's first warp does the rest.
__device__ void split_mids(const MidArgs& a, MidBlock& s, int* list, std::uint32_t b0, int begin, int end) {
  const int warp = static_cast<int>(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const double inf = pos_inf();
  const int team_warps = max(1, kMidWarps / (end - begin)), teams = kMidWarps / team_warps;
  const int team = warp / team_warps, member = warp % team_warps, leader = warp - member;
  for (int at = begin; at < end; at += teams) {
    const bool on = team < teams && at + team < end;
    int t = 0, lo = 0, n = 0, hi = 0, d = kDepthCap;
    if (on) {
      t = list[at + team];
      lo = static_cast<int>(a.first[t] - b0);
      n = static_cast<int>(a.count[t]);
      hi = lo + n;
      d = a.depth[t];
    }
    // Box and centroid bounds, upper ends negated.
    double v[12];
    for (int k = 0; k < 12; ++k) v[k] = inf;
    for (int i = lo + 32 * member + lane; i < hi; i += 32 * team_warps) {
      const double* b = s.box[s.order[i]];
      for (int k = 0; k < 3; ++k) {
        v[k] = less_of(v[k], b[k]);
        v[3 + k] = less_of(v[3 + k], -b[3 + k]);
        const double c = 0.5 * (b[k] + b[3 + k]);
        v[6 + k] = less_of(v[6 + k], c);
        v[9 + k] = less_of(v[9 + k], -c);
      }
    }
    for (int k = 0; k < 12; ++k) v[k] = warp_min(v[k]);
    if (team_warps > 1) {
      if (lane == 0)
        for (int k = 0; k < 12; ++k) s.bounds[warp][k] = v[k];
      __syncthreads();
      for (int k = 0; k < 12; ++k)
        for (int m = 0; on && m < team_warps; ++m) v[k] = less_of(v[k], s.bounds[leader + m][k]);
    }
    const double bl[3] = {v[0], v[1], v[2]}, bh[3] = {-v[3], -v[4], -v[5]};
    const double cl[3] = {v[6], v[7], v[8]}, ch[3] = {-v[9], -v[10], -v[11]};
    bool use[3];
    double inv[3];
    for (int k = 0; k < 3; ++k) {
      use[k] = ch[k] > cl[k];
      inv[k] = use[k] ? kBins / (ch[k] - cl[k]) : 0.0;
    }
    BinData r[2];
    bin_clear(r[0]);
    bin_clear(r[1]);
    if (d < kDepthCap) {
      for (int i0 = lo + 32 * member; i0 < hi; i0 += 32 * team_warps) {
        int bin[3] = {-1, -1, -1};
        if (i0 + lane < hi) {
          const double* b = s.box[s.order[i0 + lane]];
          for (int k = 0; k < 3; ++k)
            if (use[k]) bin[k] = bin_of(0.5 * (b[k] + b[3 + k]), cl[k], inv[k]);
        }
        bin_lanes(s.mask[warp], bin, r, [&](int p) { return s.box[s.order[i0 + p]]; });
      }
      fold_axis2(r[1]);
    }
    if (team_warps > 1) {
      if (member > 0) store_bins(s.sweep[warp], r[0], r[1]);
      __syncthreads();
      if (member == 0 && on)
        for (int m = 1; m < team_warps; ++m) merge_bins(s.sweep[warp + m], r[0], r[1]);
    }
    if (member == 0 && on) split_mid(a, s, list, b0, t, lo, n, d, bl, bh, cl, ch, use, inv, r);
    __syncthreads();
  }
}

// Builds the subtree under each node of 33 to kMidItems primitives down to its small
// nodes: one block per root, its boxes in shared memory, level by level. A level of the
// level kernels is 7 launches and, before, a look at its size from the host: some 100 us,
// however little it holds. On 174,085 triangles this kernel takes 195 us in place of 6 of
// 15 levels; 2,048 primitives a block would save one level more and measure the same on
// 2,000 primitives, but 0.1 ms worse on 174k. Latency bounds it: two roots take as long as
// 250. With the shorter passes, the build takes 0.54 ms for 2,053 triangles (1.01 before),
// 0.91 for 25,525 (1.57) and 1.40 for 174,085 (2.45).
// Every node of the list holds more than 32 primitives, so a list never outgrows its
// root's share of mid_nodes (one entry per primitive).
__global__ void __launch_bounds__(kMidWarps * 32) k_mid(MidArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  MidBlock& s = *reinterpret_cast<MidBlock*>(smem);
  if (static_cast<int>(blockIdx.x) >= a.counters->mid_roots) return;
  const int root = a.mid_roots[blockIdx.x];
  const std::uint32_t b0 = a.first[root];
  const int n = static_cast<int>(a.count[root]);
  for (int i = threadIdx.x; i < n; i += kMidWarps * 32) {
    const std::uint32_t id = a.items[b0 + i];
    double lo[3], hi[3];
    load_box(a.boxes, id, lo, hi);
    for (int k = 0; k < 3; ++k) {
      s.box[i][k] = lo[k];
      s.box[i][3 + k] = hi[k];
    }
    s.id[i] = id;
    s.order[i] = static_cast<std::uint16_t>(i);
  }
  int* const list = a.mid_nodes + b0;
  int* const ends = a.mid_ends + static_cast<long long>(blockIdx.x) * kMaxLevels;
  if (threadIdx.x == 0) {
    list[0] = root;
    s.listed = 1;
  }
  __syncthreads();
  int begin = 0, end = 1, level = 0;
  // At most kDepthCap + 1 levels: deeper nodes are leaves.
  while (begin < end) {
    if (threadIdx.x == 0) ends[level] = end;
    ++level;
    split_mids(a, s, list, b0, begin, end);
    begin = end;
    end = s.listed;
    __syncthreads();
  }
  if (threadIdx.x == 0 && level < kMaxLevels) ends[level] = 0;
  for (int i = threadIdx.x; i < n; i += kMidWarps * 32) a.items[b0 + i] = s.id[s.order[i]];
}

constexpr int kSmallNodes = 2 * kSmallItems - 1;

struct SmallArgs {
  const double* boxes;
  std::uint32_t* items;
  double* box;
  int* left;
  int* right;
  std::uint32_t* first;
  std::uint32_t* count;
  int* depth;
  int* axis;
  int* size;
  int* isize;
  int* sub;
  int* local;
  int* ilocal;
  const int* small_roots;
  Counters* counters;
};

// One warp's workspace: the subtree's primitives (position = lane), its nodes in
// preorder, and the stack of nodes still to build. Bins live in registers (one
// lane per axis and bin).
struct SmallWarp {
  double box[kSmallItems][6];
  double cen[kSmallItems][3];
  std::uint32_t id[kSmallItems];
  double nbox[kSmallNodes][6];
  int nl[kSmallNodes], nr[kSmallNodes], nfirst[kSmallNodes], ncount[kSmallNodes], naxis[kSmallNodes];
  int ndepth[kSmallNodes], nsize[kSmallNodes], nisize[kSmallNodes], nilocal[kSmallNodes];
  unsigned mask[3 * kBins];
  Sweep sweep;
  int stk_lo[kSmallItems], stk_hi[kSmallItems], stk_depth[kSmallItems], stk_parent[kSmallItems], stk_side[kSmallItems];
};

// Position of the k-th highest set bit of `mask` (k = 0: the highest).
__device__ __forceinline__ int kth_highest(unsigned mask, int k) {
  for (int j = 0; j < k; ++j) mask &= ~(1u << (31 - __clz(mask)));
  return 31 - __clz(mask);
}

// Builds the whole subtree under each node of at most kSmallItems primitives, one
// warp per node, exactly as the recursive build would: nodes are made in
// preorder (left subtree before right), each with the same bounds, SAH decision
// and partition as at the large levels.
__device__ void build_small(const SmallArgs& a, SmallWarp& s, int r) {
  const int lane = threadIdx.x & 31;
  const std::uint32_t b0 = a.first[r];
  const int n = static_cast<int>(a.count[r]);
  const double inf = pos_inf();
  if (lane < n) {
    const std::uint32_t id = a.items[b0 + lane];
    double bl[3], bh[3];
    load_box(a.boxes, id, bl, bh);
    s.id[lane] = id;
    for (int k = 0; k < 3; ++k) {
      s.box[lane][k] = bl[k];
      s.box[lane][3 + k] = bh[k];
      s.cen[lane][k] = 0.5 * (bl[k] + bh[k]);
    }
  }
  if (lane == 0) {
    s.stk_lo[0] = 0;
    s.stk_hi[0] = n;
    s.stk_depth[0] = a.depth[r];
    s.stk_parent[0] = -1;
    s.stk_side[0] = 0;
  }
  int top = 1, m = 0;
  bool overflow = false;
  __syncwarp();
  while (top > 0) {
    --top;
    const int lo = s.stk_lo[top], hi = s.stk_hi[top], d = s.stk_depth[top];
    const int parent = s.stk_parent[top], side = s.stk_side[top];
    __syncwarp();
    const int me = m++;
    if (lane == 0 && parent >= 0) {
      if (side == 0) s.nl[parent] = me;
      else s.nr[parent] = me;
    }
    const int cnt = hi - lo;
    const bool act = lane >= lo && lane < hi;
    double bl[3], bh[3], cl[3], ch[3];
    for (int k = 0; k < 3; ++k) {
      bl[k] = warp_min(act ? s.box[lane][k] : inf);
      bh[k] = warp_max(act ? s.box[lane][3 + k] : -inf);
      cl[k] = warp_min(act ? s.cen[lane][k] : inf);
      ch[k] = warp_max(act ? s.cen[lane][k] : -inf);
    }
    if (lane == 0) {
      for (int k = 0; k < 3; ++k) {
        s.nbox[me][k] = bl[k];
        s.nbox[me][3 + k] = bh[k];
      }
      s.ndepth[me] = d;
      s.nfirst[me] = lo;
      s.ncount[me] = cnt;
    }
    int kind = 0;  // 0 leaf, 1 middle split, 2 SAH partition
    int sp_axis = 0, sp_bin = -1, mid = lo;
    if (!(cnt <= 4 || d >= kDepthCap)) {
      bool use[3];
      double inv[3];
      for (int k = 0; k < 3; ++k) {
        use[k] = ch[k] > cl[k];
        inv[k] = use[k] ? kBins / (ch[k] - cl[k]) : 0.0;
      }
      BinData r[2];
      bin_clear(r[0]);
      bin_clear(r[1]);
      int bin[3];
      for (int k = 0; k < 3; ++k) bin[k] = act && use[k] ? bin_of(s.cen[lane][k], cl[k], inv[k]) : -1;
      bin_lanes(s.mask, bin, r, [&](int p) { return s.box[p]; });
      fold_axis2(r[1]);
      double best_cost;
      int best_axis, best_bin;
      unsigned left_n;
      warp_best_split(s.sweep, r[0], r[1], use, box_area(bl, bh), best_cost, best_axis, best_bin, left_n);
      if (best_axis < 0) {
        kind = 1;
        sp_axis = widest_axis(cl, ch);
        mid = lo + cnt / 2;
      } else if (!(best_cost >= double(cnt) && cnt <= 16)) {
        sp_axis = best_axis;
        sp_bin = best_bin;
        if (left_n == 0 || left_n == static_cast<unsigned>(cnt)) {
          kind = 1;
          mid = lo + cnt / 2;
        } else {
          kind = 2;
          mid = lo + static_cast<int>(left_n);
        }
      }
      // Two more stack entries always fit (at most 29 for 32 primitives); the
      // check only keeps shared memory safe.
      if (kind != 0 && top + 2 > kSmallItems) {
        kind = 0;
        overflow = true;
      }
    }
    if (kind == 0) {
      if (lane == 0) {
        s.nl[me] = -1;
        s.nr[me] = -1;
        s.naxis[me] = 0;
      }
      continue;
    }
    if (lane == 0) s.naxis[me] = sp_axis;
    if (kind == 2) {
      const double inv = kBins / (ch[sp_axis] - cl[sp_axis]);
      const bool goes_left = act && bin_of(s.cen[lane][sp_axis], cl[sp_axis], inv) <= sp_bin;
      const unsigned lf = __ballot_sync(0xFFFFFFFFu, act && lane < mid && !goes_left);
      const unsigned rt = __ballot_sync(0xFFFFFFFFu, act && lane >= mid && goes_left);
      const int q = (lf & (1u << lane)) ? kth_highest(rt, __popc(lf & ((1u << lane) - 1u))) : -1;
      if (q >= lo && q < hi) {
        const std::uint32_t id = s.id[lane];
        s.id[lane] = s.id[q];
        s.id[q] = id;
        for (int k = 0; k < 6; ++k) {
          const double v = s.box[lane][k];
          s.box[lane][k] = s.box[q][k];
          s.box[q][k] = v;
        }
        for (int k = 0; k < 3; ++k) {
          const double v = s.cen[lane][k];
          s.cen[lane][k] = s.cen[q][k];
          s.cen[q][k] = v;
        }
      }
    }
    if (lane == 0) {
      s.stk_lo[top] = mid;
      s.stk_hi[top] = hi;
      s.stk_depth[top] = d + 1;
      s.stk_parent[top] = me;
      s.stk_side[top] = 1;
      s.stk_lo[top + 1] = lo;
      s.stk_hi[top + 1] = mid;
      s.stk_depth[top + 1] = d + 1;
      s.stk_parent[top + 1] = me;
      s.stk_side[top + 1] = 0;
    }
    top += 2;
    __syncwarp();
  }
  __syncwarp();
  int base = 0;
  if (lane == 0) {
    // Children follow their parent in preorder, so a reverse sweep sees them first.
    int leaves = 0, max_leaf = 0, max_depth = 0;
    for (int i = m - 1; i >= 0; --i) {
      if (s.nl[i] < 0) {
        s.nsize[i] = 1;
        s.nisize[i] = 0;
        ++leaves;
        max_leaf = max(max_leaf, s.ncount[i]);
        max_depth = max(max_depth, s.ndepth[i]);
      } else {
        s.nsize[i] = 1 + s.nsize[s.nl[i]] + s.nsize[s.nr[i]];
        s.nisize[i] = 1 + s.nisize[s.nl[i]] + s.nisize[s.nr[i]];
      }
    }
    int c = 0;
    for (int i = 0; i < m; ++i) s.nilocal[i] = s.nl[i] >= 0 ? c++ : -1;
    atomicAdd(&a.counters->leaves, leaves);
    atomicMax(&a.counters->max_leaf, max_leaf);
    atomicMax(&a.counters->max_depth, max_depth);
    if (overflow) atomicOr(&a.counters->error, 4);
    if (m > 1) base = atomicAdd(&a.counters->nodes, m - 1);
  }
  base = __shfl_sync(0xFFFFFFFFu, base, 0);
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    const int g = i == 0 ? r : base + i - 1;
    for (int k = 0; k < 6; ++k) a.box[6ll * g + k] = s.nbox[i][k];
    a.left[g] = s.nl[i] < 0 ? -1 : (s.nl[i] == 0 ? r : base + s.nl[i] - 1);
    a.right[g] = s.nr[i] < 0 ? -1 : (s.nr[i] == 0 ? r : base + s.nr[i] - 1);
    a.first[g] = b0 + static_cast<std::uint32_t>(s.nfirst[i]);
    a.count[g] = static_cast<std::uint32_t>(s.ncount[i]);
    a.depth[g] = s.ndepth[i];
    a.axis[g] = s.naxis[i];
    a.size[g] = s.nsize[i];
    a.isize[g] = s.nisize[i];
    a.sub[g] = r;
    a.local[g] = i;
    a.ilocal[g] = s.nilocal[i];
  }
  if (lane < n) a.items[b0 + lane] = s.id[lane];
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32) k_small(SmallArgs a) {
  __shared__ SmallWarp s_all[kWarpsPerBlock];
  const int wib = threadIdx.x >> 5;
  const int n_small = a.counters->small_roots;
  for (int w = blockIdx.x * kWarpsPerBlock + wib; w < n_small; w += gridDim.x * kWarpsPerBlock) {
    build_small(a, s_all[wib], a.small_roots[w]);
    __syncwarp();
  }
}

}  // namespace

namespace {

struct TreeArgs {
  const double* box;
  const int* left;
  const int* right;
  const std::uint32_t* first;
  const std::uint32_t* count;
  const int* axis;
  int* size;
  int* isize;
  int* dfs;
  int* idfs;
  const int* sub;
  const int* local;
  const int* ilocal;
  Counters* counters;
};

// Subtree sizes of a node whose children have theirs.
__device__ __forceinline__ void node_sizes(const TreeArgs& a, int t) {
  const int l = a.left[t], r = a.right[t];
  if (l < 0) {
    a.size[t] = 1;
    a.isize[t] = 0;
  } else {
    a.size[t] = 1 + a.size[l] + a.size[r];
    a.isize[t] = 1 + a.isize[l] + a.isize[r];
  }
}

// Of all large nodes, level by level: one block, since a level has few of them.
__global__ void __launch_bounds__(512) k_sizes(TreeArgs a, const int* tasks, int levels) {
  for (int k = levels - 1; k >= 0; --k) {
    const LevelCount l = a.counters->lvl[k];
    for (int i = threadIdx.x; i < l.tasks; i += blockDim.x) node_sizes(a, tasks[l.base + i]);
    __syncthreads();
  }
}

// Depth-first indices (all nodes, and interior nodes only) of a node's children:
// left follows its parent, right follows the left subtree.
__device__ __forceinline__ void child_indices(const TreeArgs& a, int t) {
  const int l = a.left[t], r = a.right[t];
  if (l < 0) return;
  a.dfs[l] = a.dfs[t] + 1;
  a.dfs[r] = a.dfs[t] + 1 + a.size[l];
  a.idfs[l] = a.idfs[t] + 1;
  a.idfs[r] = a.idfs[t] + 1 + a.isize[l];
}

__global__ void __launch_bounds__(512) k_dfs(TreeArgs a, const int* tasks, int levels) {
  for (int k = 0; k < levels; ++k) {
    const LevelCount l = a.counters->lvl[k];
    for (int i = threadIdx.x; i < l.tasks; i += blockDim.x) child_indices(a, tasks[l.base + i]);
    __syncthreads();
  }
}

// The same for the nodes that blocks built, one warp per block's list: levels from
// the last up, then from the first down.
__global__ void __launch_bounds__(128) k_mid_sizes(TreeArgs a, const int* mid_roots, const int* nodes, const int* ends) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= a.counters->mid_roots) return;
  const int root = mid_roots[w];
  nodes += a.first[root];
  ends += static_cast<long long>(w) * kMaxLevels;
  int n = 0;
  while (n < kMaxLevels && ends[n] > 0) ++n;
  for (int k = n - 1; k >= 0; --k) {
    for (int i = (k ? ends[k - 1] : 0) + lane; i < ends[k]; i += 32) node_sizes(a, nodes[i]);
    __syncwarp();
  }
}
__global__ void __launch_bounds__(128) k_mid_dfs(TreeArgs a, const int* mid_roots, const int* nodes, const int* ends) {
  const int w = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= a.counters->mid_roots) return;
  const int root = mid_roots[w];
  nodes += a.first[root];
  ends += static_cast<long long>(w) * kMaxLevels;
  for (int k = 0; k < kMaxLevels && ends[k] > 0; ++k) {
    for (int i = (k ? ends[k - 1] : 0) + lane; i < ends[k]; i += 32) child_indices(a, nodes[i]);
    __syncwarp();
  }
}

// Nodes inside warp-built subtrees: offsets from their subtree root.
__global__ void k_small_dfs(TreeArgs a, int capacity) {
  const int id = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (id >= capacity || id >= a.counters->nodes) return;
  const int root = a.sub[id];
  if (root < 0 || a.local[id] == 0) return;
  a.dfs[id] = a.dfs[root] + a.local[id];
  if (a.ilocal[id] >= 0) a.idfs[id] = a.idfs[root] + a.ilocal[id];
}

__global__ void k_finish(TreeArgs a) {
  if (blockIdx.x == 0 && threadIdx.x == 0) a.counters->interior = a.left[0] >= 0 ? a.isize[0] : 0;
}

struct WideArgs {
  const double* box;
  const int* left;
  const int* right;
  const int* dfs;
  int* wide_list;
  int* wide_kids;
  std::uint32_t* wflag;
  Counters* counters;
};

__global__ void k_wide_init(WideArgs a) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  a.counters->wide_off[0] = 0;
  if (a.left[0] >= 0) {
    a.wide_list[0] = 0;
    a.counters->wide_cnt[0] = 1;
  }
}

// One level of the four-wide collapse: each node starting a four-wide node takes
// its two children and replaces the interior child of largest surface area by
// its own children until there are four (flatten.cpp build_wide); the interior
// children then start the next level's four-wide nodes.
__global__ void k_wide(WideArgs a, int level) {
  const int cnt = a.counters->wide_cnt[level], off = a.counters->wide_off[level];
  if (blockIdx.x == 0 && threadIdx.x == 0) a.counters->wide_off[level + 1] = off + cnt;
  for (int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); i < cnt;
       i += static_cast<int>(gridDim.x * blockDim.x)) {
    const int b = a.wide_list[off + i];
    int kid[4] = {a.left[b], a.right[b], -1, -1};
    int nk = 2;
    while (nk < 4) {
      int pick = -1;
      double pick_area = -1;
      for (int q = 0; q < nk; ++q) {
        const int c = kid[q];
        if (a.left[c] < 0) continue;
        const double* cb = a.box + 6ll * c;
        const double area = box_area(cb, cb + 3);
        if (area > pick_area) {
          pick_area = area;
          pick = q;
        }
      }
      if (pick < 0) break;
      const int c = kid[pick];
      kid[pick] = a.left[c];
      kid[nk++] = a.right[c];
    }
    for (int q = 0; q < 4; ++q) a.wide_kids[4ll * b + q] = q < nk ? kid[q] : -1;
    const int at = a.dfs[b];
    if (at >= 0 && at < a.counters->nodes) a.wflag[at] = 1;
    for (int q = 0; q < nk; ++q)
      if (a.left[kid[q]] >= 0) a.wide_list[off + cnt + atomicAdd(&a.counters->wide_cnt[level + 1], 1)] = kid[q];
  }
}

// Exclusive scan of n 32-bit flags: per-block scans, a scan of the block sums,
// then the block offsets added.
constexpr int kScanBlock = 1024;

__global__ void __launch_bounds__(kScanBlock) k_scan_block(const std::uint32_t* in, std::uint32_t* out,
                                                           std::uint32_t* sums, int n) {
  __shared__ std::uint32_t warp_sum[32];
  const int i = static_cast<int>(blockIdx.x) * kScanBlock + static_cast<int>(threadIdx.x);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const std::uint32_t v = i < n ? in[i] : 0u;
  std::uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const std::uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const std::uint32_t t = warp_sum[lane];
    std::uint32_t y = t;
    for (int o = 1; o < 32; o <<= 1) {
      const std::uint32_t z = __shfl_up_sync(0xFFFFFFFFu, y, o);
      if (lane >= o) y += z;
    }
    warp_sum[lane] = y - t;
    if (lane == 31) sums[blockIdx.x] = y;
  }
  __syncthreads();
  if (i < n) out[i] = warp_sum[wid] + x - v;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_sums(std::uint32_t* sums, int nb) {
  __shared__ std::uint32_t warp_sum[32];
  __shared__ std::uint32_t carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += kScanBlock) {
    const int i = base + static_cast<int>(threadIdx.x);
    const std::uint32_t v = i < nb ? sums[i] : 0u;
    std::uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const std::uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      const std::uint32_t t = warp_sum[lane];
      std::uint32_t y = t;
      for (int o = 1; o < 32; o <<= 1) {
        const std::uint32_t z = __shfl_up_sync(0xFFFFFFFFu, y, o);
        if (lane >= o) y += z;
      }
      warp_sum[lane] = y - t;
    }
    __syncthreads();
    const std::uint32_t c = carry;
    if (i < nb) sums[i] = c + warp_sum[wid] + x - v;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = c + warp_sum[wid] + x;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kScanBlock) k_scan_add(std::uint32_t* out, const std::uint32_t* sums, int n) {
  const int i = static_cast<int>(blockIdx.x) * kScanBlock + static_cast<int>(threadIdx.x);
  if (i < n) out[i] += sums[blockIdx.x];
}

struct EmitArgs {
  TreeArgs t;
  const std::uint32_t* items;
  const float4* rows;
  const float4* normals;
  const std::uint32_t* material;
  const int* wide_list;
  const int* wide_kids;
  const std::uint32_t* wscan;
  std::uint8_t* last;
  DevNode* nodes;
  DevNode4* nodes4;
  float4* prims;
  std::uint32_t* slot_material;
  float4* slot_normals;
  std::uint32_t* order;
  int capacity;
};

__device__ __forceinline__ std::int32_t binary_link(const TreeArgs& t, int c) {
  return t.left[c] >= 0 ? t.idfs[c] : ~static_cast<std::int32_t>(t.first[c]);
}

__global__ void k_mark_last(EmitArgs a) {
  const int id = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (id >= a.capacity || id >= a.t.counters->nodes || a.t.left[id] >= 0) return;
  a.last[a.t.first[id] + a.t.count[id] - 1] = 1;
}

// Binary nodes at their interior depth-first index: both children's boxes rounded
// outward to fp32, links, split axis.
__global__ void k_emit_nodes(EmitArgs a) {
  const int id = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (id >= a.capacity || id >= a.t.counters->nodes) return;
  const int l = a.t.left[id], r = a.t.right[id];
  if (l < 0) return;
  const double* L = a.t.box + 6ll * l;
  const double* R = a.t.box + 6ll * r;
  DevNode d;
  d.xy0 = make_float4(round_down(L[0]), round_up(L[3]), round_down(L[1]), round_up(L[4]));
  d.xy1 = make_float4(round_down(R[0]), round_up(R[3]), round_down(R[1]), round_up(R[4]));
  d.zz = make_float4(round_down(L[2]), round_up(L[5]), round_down(R[2]), round_up(R[5]));
  d.link = make_int4(binary_link(a.t, l), binary_link(a.t, r), a.t.axis[id] << 16, 0);
  const int at = a.t.idfs[id];
  if (at >= 0 && at < a.t.counters->interior) a.nodes[at] = d;
}

// BinaryBvh::build's cost terms (host/bvh_build.cpp), a node's at its depth-first index.
__global__ void k_node_costs(TreeArgs t, int n, double* out) {
  const int id = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (id >= n) return;
  const double root = box_area(t.box, t.box + 3), area = box_area(t.box + 6ll * id, t.box + 6ll * id + 3);
  const double term = area / (root < 1e-30 ? 1e-30 : root) * (t.left[id] < 0 ? double(t.count[id]) : 1.0);
  const int at = t.dfs[id];
  if (at >= 0 && at < n) out[at] = term;
}

// Slots in leaf order, gathered from the per-primitive records.
__global__ void k_emit_slots(EmitArgs a, std::uint32_t n) {
  const std::uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const std::uint32_t id = a.items[k];
  float4 r0 = a.rows[3ull * id];
  if (a.last[k]) r0.w = __uint_as_float(__float_as_uint(r0.w) | kLastInLeaf);
  a.prims[3ull * k] = r0;
  a.prims[3ull * k + 1] = a.rows[3ull * id + 1];
  a.prims[3ull * k + 2] = a.rows[3ull * id + 2];
  a.slot_normals[3ull * k] = a.normals[3ull * id];
  a.slot_normals[3ull * k + 1] = a.normals[3ull * id + 1];
  a.slot_normals[3ull * k + 2] = a.normals[3ull * id + 2];
  a.slot_material[k] = a.material[id];
  a.order[k] = id;
}

// Four-wide nodes at their index: the rank of their binary node in depth-first
// order among the binary nodes that start a four-wide node.
__global__ void k_emit_wide(EmitArgs a, int n_wide) {
  const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n_wide) return;
  const int b = a.wide_list[i];
  float lo[3][4], hi[3][4];
  std::int32_t link[4];
  for (int q = 0; q < 4; ++q) {
    const int c = a.wide_kids[4ll * b + q];
    if (c < 0) {
      for (int k = 0; k < 3; ++k) lo[k][q] = hi[k][q] = 0.f;
      link[q] = kNoChild;
      continue;
    }
    const double* cb = a.t.box + 6ll * c;
    for (int k = 0; k < 3; ++k) {
      lo[k][q] = round_down(cb[k]);
      hi[k][q] = round_up(cb[3 + k]);
    }
    const int at = a.t.dfs[c];
    link[q] = a.t.left[c] >= 0 ? (at >= 0 && at < a.t.counters->nodes ? static_cast<std::int32_t>(a.wscan[at]) : kNoChild)
                               : ~static_cast<std::int32_t>(a.t.first[c]);
  }
  DevNode4 d;
  d.lo_x = make_float4(lo[0][0], lo[0][1], lo[0][2], lo[0][3]);
  d.hi_x = make_float4(hi[0][0], hi[0][1], hi[0][2], hi[0][3]);
  d.lo_y = make_float4(lo[1][0], lo[1][1], lo[1][2], lo[1][3]);
  d.hi_y = make_float4(hi[1][0], hi[1][1], hi[1][2], hi[1][3]);
  d.lo_z = make_float4(lo[2][0], lo[2][1], lo[2][2], lo[2][3]);
  d.hi_z = make_float4(hi[2][0], hi[2][1], hi[2][2], hi[2][3]);
  d.link = make_int4(link[0], link[1], link[2], link[3]);
  d.pad = make_int4(0, 0, 0, 0);
  const int at = a.t.dfs[b];
  if (at < 0 || at >= a.t.counters->nodes) return;
  const std::uint32_t slot = a.wscan[at];
  if (slot < static_cast<std::uint32_t>(n_wide)) a.nodes4[slot] = d;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side

namespace {

int blocks_for(long long threads, int per_block) {
  return static_cast<int>(std::max<long long>(1, (threads + per_block - 1) / per_block));
}

}  // namespace

// Conversions on the host cores wrote 152 bytes a primitive into pinned memory: 2.4 ms for
// 174,085 triangles before the first byte crossed the bus, then 2 ms of copying. The host
// now writes 80 (116 with vertex normals), whose copies and this kernel overlap with it.
// The whole upload takes 3.56 ms (6.5 with the conversion on the host), 1.77 for 25,525
// triangles (2.5), 0.78 for 2,053 (the same).
namespace {
__global__ void __launch_bounds__(256) k_convert(const RawPrim* __restrict__ raw, const float* __restrict__ normals,
                                                 std::uint32_t first, std::uint32_t n, double* boxes, float4* rows,
                                                 float4* row_normals, std::uint32_t* material, std::uint32_t* items) {
  const std::uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RawPrim p = raw[i];
  const std::uint32_t id = first + i;
  const double* a = p.v;
  const double* b = p.v + 3;
  const double* c = p.v + 6;
  double* box = boxes + 6ull * id;
  double residual[3];  // what rounding the position to fp32 lost
  for (int k = 0; k < 3; ++k) residual[k] = a[k] - static_cast<double>(__double2float_rn(a[k]));
  float4 r[3], rn[3];
  for (int k = 0; k < 3; ++k) rn[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  const std::uint32_t word = id | (p.sphere ? kSphereBit : 0u);
  r[0] = make_float4(__double2float_rn(a[0]), __double2float_rn(a[1]), __double2float_rn(a[2]), __uint_as_float(word));
  if (p.sphere) {
    const double radius = fabs(b[0]);
    for (int k = 0; k < 3; ++k) {
      box[k] = a[k] - radius;
      box[3 + k] = a[k] + radius;
    }
    r[1] = make_float4(__double2float_rn(b[0]), __double2float_rn(b[0] * b[0]), 0.f, 0.f);
    r[2] = make_float4(__double2float_rn(residual[0]), __double2float_rn(residual[1]), __double2float_rn(residual[2]), 0.f);
  } else {
    float e1[3], e2[3];
    for (int k = 0; k < 3; ++k) {
      // Flat triangles get a little thickness so no slab is empty.
      box[k] = fmin(fmin(fmin(pos_inf(), a[k]), b[k]), c[k]) - 1e-9;
      box[3 + k] = fmax(fmax(fmax(-pos_inf(), a[k]), b[k]), c[k]) + 1e-9;
      e1[k] = __double2float_rn(b[k] - a[k]);
      e2[k] = __double2float_rn(c[k] - a[k]);
    }
    const double u[3] = {e1[0], e1[1], e1[2]}, v[3] = {e2[0], e2[1], e2[2]};
    const double nx = u[1] * v[2] - u[2] * v[1], ny = u[2] * v[0] - u[0] * v[2], nz = u[0] * v[1] - u[1] * v[0];
    r[1] = make_float4(e1[0], e1[1], e1[2],
                       __double2float_rn(residual[0] * nx + residual[1] * ny + residual[2] * nz));
    r[2] = make_float4(e2[0], e2[1], e2[2], 0.f);
    if (p.material & 0x80000000u)
      for (int k = 0; k < 3; ++k) {
        const float* m = normals + 9ull * i + 3 * k;
        rn[k] = make_float4(m[0], m[1], m[2], 0.f);
      }
  }
  for (int k = 0; k < 3; ++k) {
    rows[3ull * id + k] = r[k];
    row_normals[3ull * id + k] = rn[k];
  }
  material[id] = p.material;
  if (items) items[id] = id;
}
}  // namespace

cudaError_t convert_prims(const RawPrim* raw, const float* normals, std::uint32_t first, std::uint32_t n, double* boxes,
                          float4* rows, float4* row_normals, std::uint32_t* material, std::uint32_t* items,
                          cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_convert<<<(n + 255) / 256, 256, 0, stream>>>(raw, normals, first, n, boxes, rows, row_normals, material, items);
  return cudaGetLastError();
}

void gpu_bvh_preload() {
  cudaFuncAttributes a;
  const void* kernels[] = {
      reinterpret_cast<const void*>(k_convert),    reinterpret_cast<const void*>(k_init),
      reinterpret_cast<const void*>(k_node_costs),
      reinterpret_cast<const void*>(k_bounds),
      reinterpret_cast<const void*>(k_bins),       reinterpret_cast<const void*>(k_decide),
      reinterpret_cast<const void*>(k_pcount),     reinterpret_cast<const void*>(k_pscan),
      reinterpret_cast<const void*>(k_pranks),     reinterpret_cast<const void*>(k_pswap),
      reinterpret_cast<const void*>(k_small),      reinterpret_cast<const void*>(k_mid),
      reinterpret_cast<const void*>(k_mid_sizes),  reinterpret_cast<const void*>(k_mid_dfs),
      reinterpret_cast<const void*>(k_sizes),
      reinterpret_cast<const void*>(k_dfs),        reinterpret_cast<const void*>(k_small_dfs),
      reinterpret_cast<const void*>(k_finish),     reinterpret_cast<const void*>(k_wide_init),
      reinterpret_cast<const void*>(k_wide),       reinterpret_cast<const void*>(k_scan_block),
      reinterpret_cast<const void*>(k_scan_sums),  reinterpret_cast<const void*>(k_scan_add),
      reinterpret_cast<const void*>(k_mark_last),  reinterpret_cast<const void*>(k_emit_nodes),
      reinterpret_cast<const void*>(k_emit_slots), reinterpret_cast<const void*>(k_emit_wide)};
  for (const void* k : kernels) BVH_CK(cudaFuncGetAttributes(&a, k));
}

GpuBvhBuilder::~GpuBvhBuilder() { release(); }

void GpuBvhBuilder::release() {
  for (int i = 0; i < n_blocks_; ++i) cudaFreeAsync(blocks_[i], stream_);
  n_blocks_ = 0;
  delete st_;
  st_ = nullptr;
}

void* GpuBvhBuilder::alloc(std::size_t bytes) {
  if (n_blocks_ >= static_cast<int>(sizeof(blocks_) / sizeof(blocks_[0])))
    throw std::logic_error("bvh build: too many scratch blocks");
  void* p = nullptr;
  count_allocation();
  BVH_CK(cudaMallocFromPoolAsync(&p, std::max<std::size_t>(bytes, 256), pool_, stream_));
  blocks_[n_blocks_++] = p;
  return p;
}

GpuBvhCounts GpuBvhBuilder::build(const GpuBvhInput& in) {
  release();
  counts_ = GpuBvhCounts{};
  const std::uint32_t n = in.n_items;
  if (n == 0) return counts_;
  if (n > (1u << 30)) throw std::runtime_error("too many primitives for the device BVH build");
  st_ = new State;
  State& s = *st_;
  s.n = n;
  s.nn = 2 * n;
  s.max_level_tasks = n / (kMidItems + 1) + 2;
  s.max_chunks = n / kChunk + s.max_level_tasks + 8;

  // Carve every scratch array out of one pool allocation.
  std::vector<std::pair<void**, std::size_t>> parts;
  auto add = [&](auto*& p, std::size_t count) {
    parts.push_back({reinterpret_cast<void**>(&p), count * sizeof(*p)});
  };
  const std::size_t nn = s.nn, lt = s.max_level_tasks, mc = s.max_chunks;
  add(s.counters, 1);
  add(s.items, n);
  add(s.scratch, n);
  add(s.box, 6 * nn);
  add(s.key, 12 * nn);
  for (int** p : {&s.left, &s.right, &s.depth, &s.axis, &s.size, &s.isize, &s.dfs, &s.idfs, &s.sub, &s.local,
                  &s.ilocal, &s.tasks})
    add(*p, nn);
  add(s.first, nn);
  add(s.count, nn);
  add(s.small_roots, n);
  const std::size_t max_mids = n / (kSmallItems + 1) + 1;
  add(s.mid_roots, max_mids);
  add(s.mid_nodes, n);
  add(s.mid_ends, max_mids * kMaxLevels);
  for (int q = 0; q < 2; ++q) {
    add(s.bins[q], lt * kBinWords);
    for (int** p : {&s.task_chunk0[q], &s.task_nchunks[q], &s.need_part[q], &s.part_t[q], &s.part_m[q],
                    &s.part_axis[q], &s.part_bin[q]})
      add(*p, lt);
    add(s.part_lo[q], lt);
    add(s.part_inv[q], lt);
    for (int** p : {&s.chunk_task[q], &s.cnt_lf[q], &s.cnt_rt[q], &s.base_lf[q], &s.base_rt[q]}) add(*p, mc);
    add(s.chunk_start[q], mc);
  }
  add(s.moves, mc * (kChunk / 32));
  add(s.wide_list, n + 1);
  add(s.wide_kids, 4 * nn);
  add(s.wflag, nn);
  add(s.wscan, nn);
  add(s.scan_sums, nn / kScanBlock + 2);
  add(s.last, n);
  std::size_t total = 0;
  for (auto& p : parts) total += (p.second + 255) & ~std::size_t(255);
  auto* base = static_cast<unsigned char*>(alloc(total));
  std::size_t at = 0;
  for (auto& p : parts) {
    *p.first = base + at;
    at += (p.second + 255) & ~std::size_t(255);
  }

  cudaEvent_t ev[2];
  BVH_CK(cudaEventCreate(&ev[0]));
  BVH_CK(cudaEventCreate(&ev[1]));
  struct EventGuard {
    cudaEvent_t* e;
    ~EventGuard() {
      cudaEventDestroy(e[0]);
      cudaEventDestroy(e[1]);
    }
  } guard{ev};
  BVH_CK(cudaEventRecord(ev[0], stream_));
  BVH_CK(cudaMemsetAsync(s.counters, 0, sizeof(Counters), stream_));
  BVH_CK(cudaMemcpyAsync(s.items, in.items, n * sizeof(std::uint32_t), cudaMemcpyDeviceToDevice, stream_));

  Counters host{};
  auto read_counters = [&] {
    BVH_CK(cudaMemcpyAsync(&host, s.counters, sizeof(Counters), cudaMemcpyDeviceToHost, stream_));
    BVH_CK(cudaStreamSynchronize(stream_));
    if (host.error & 1) throw std::runtime_error("BVH leaf too large");
    if (host.error) throw std::runtime_error("device BVH build: inconsistent partition");
  };
  auto level_args = [&](int level) {
    LevelArgs a{};
    a.boxes = in.boxes;
    a.items = s.items;
    a.scratch = s.scratch;
    a.box = s.box;
    a.key = s.key;
    a.left = s.left;
    a.right = s.right;
    a.first = s.first;
    a.count = s.count;
    a.depth = s.depth;
    a.axis = s.axis;
    a.sub = s.sub;
    a.tasks = s.tasks;
    a.mid_roots = s.mid_roots;
    a.small_roots = s.small_roots;
    a.counters = s.counters;
    a.level = level;
    const int p = level & 1, q = p ^ 1;
    a.bins = s.bins[p];
    a.need_part = s.need_part[p];
    a.part_t = s.part_t[p];
    a.part_m = s.part_m[p];
    a.part_axis = s.part_axis[p];
    a.part_bin = s.part_bin[p];
    a.part_lo = s.part_lo[p];
    a.part_inv = s.part_inv[p];
    a.task_chunk0 = s.task_chunk0[p];
    a.task_nchunks = s.task_nchunks[p];
    a.chunk_task = s.chunk_task[p];
    a.chunk_start = s.chunk_start[p];
    a.cnt_lf = s.cnt_lf[p];
    a.cnt_rt = s.cnt_rt[p];
    a.base_lf = s.base_lf[p];
    a.base_rt = s.base_rt[p];
    a.moves = s.moves;
    a.bins_next = s.bins[q];
    a.task_chunk0_next = s.task_chunk0[q];
    a.task_nchunks_next = s.task_nchunks[q];
    a.chunk_task_next = s.chunk_task[q];
    a.chunk_start_next = s.chunk_start[q];
    return a;
  };

  // Most tasks that a level can have, and their chunks.
  auto level_tasks = [&](int level) {
    return level < 30 ? std::min(1 << level, static_cast<int>(s.max_level_tasks)) : static_cast<int>(s.max_level_tasks);
  };
  auto level_chunks = [&](int level) {
    return std::min(static_cast<int>(n / kChunk) + level_tasks(level), static_cast<int>(s.max_chunks));
  };
  // The root lands in level 0's arrays, which are an odd level's next.
  k_init<<<1, 32, 0, stream_>>>(level_args(1), n, s.dfs, s.idfs);
  BVH_CK(cudaGetLastError());
  // A level has its largest node from at least n / 2^level primitives, so the first
  // levels follow one another without a look at their sizes (a look costs 25 us).
  int levels = 0, tasks = n > kMidItems ? 1 : 0;
  while (tasks > 0) {
    if (levels >= kMaxLevels - 1) throw std::logic_error("device BVH build: too many levels");
    const LevelArgs a = level_args(levels);
    const int nt = level_tasks(levels), nc = level_chunks(levels);
    k_bounds<<<blocks_for(32ll * nc, 128), 128, 0, stream_>>>(a);
    k_bins<<<blocks_for(nc, kWarpsPerBlock), kWarpsPerBlock * 32, 0, stream_>>>(a);
    k_decide<<<blocks_for(32ll * nt, 128), 128, 0, stream_>>>(a);
    k_pcount<<<blocks_for(32ll * nc, 128), 128, 0, stream_>>>(a);
    k_pscan<<<blocks_for(32ll * nt, 128), 128, 0, stream_>>>(a);
    k_pranks<<<blocks_for(32ll * nc, 128), 128, 0, stream_>>>(a);
    k_pswap<<<blocks_for(32ll * nc, 128), 128, 0, stream_>>>(a);
    BVH_CK(cudaGetLastError());
    ++levels;
    if (levels < 30 && (n >> levels) > static_cast<std::uint32_t>(kMidItems)) continue;
    read_counters();
    tasks = host.lvl[levels].tasks;
    if (tasks > static_cast<int>(s.max_level_tasks) || host.lvl[levels].chunks > static_cast<int>(s.max_chunks))
      throw std::logic_error("device BVH build: level overflow");
  }
  const int mids = levels > 0 ? host.mid_roots : (n > kSmallItems ? 1 : 0);
  if (mids > 0) {
    MidArgs ma{};
    ma.boxes = in.boxes;
    ma.items = s.items;
    ma.box = s.box;
    ma.left = s.left;
    ma.right = s.right;
    ma.first = s.first;
    ma.count = s.count;
    ma.depth = s.depth;
    ma.axis = s.axis;
    ma.sub = s.sub;
    ma.mid_roots = s.mid_roots;
    ma.mid_nodes = s.mid_nodes;
    ma.mid_ends = s.mid_ends;
    ma.small_roots = s.small_roots;
    ma.counters = s.counters;
    // Set on every build: the attribute belongs to the device that is current.
    BVH_CK(cudaFuncSetAttribute(k_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(MidBlock))));
    k_mid<<<mids, kMidWarps * 32, sizeof(MidBlock), stream_>>>(ma);
    BVH_CK(cudaGetLastError());
  }

  SmallArgs sa{};
  sa.boxes = in.boxes;
  sa.items = s.items;
  sa.box = s.box;
  sa.left = s.left;
  sa.right = s.right;
  sa.first = s.first;
  sa.count = s.count;
  sa.depth = s.depth;
  sa.axis = s.axis;
  sa.size = s.size;
  sa.isize = s.isize;
  sa.sub = s.sub;
  sa.local = s.local;
  sa.ilocal = s.ilocal;
  sa.small_roots = s.small_roots;
  sa.counters = s.counters;
  k_small<<<std::min(blocks_for(n, kWarpsPerBlock), 148 * 6), kWarpsPerBlock * 32, 0, stream_>>>(sa);

  TreeArgs ta{};
  ta.box = s.box;
  ta.left = s.left;
  ta.right = s.right;
  ta.first = s.first;
  ta.count = s.count;
  ta.axis = s.axis;
  ta.size = s.size;
  ta.isize = s.isize;
  ta.dfs = s.dfs;
  ta.idfs = s.idfs;
  ta.sub = s.sub;
  ta.local = s.local;
  ta.ilocal = s.ilocal;
  ta.counters = s.counters;
  if (mids > 0) k_mid_sizes<<<blocks_for(32ll * mids, 128), 128, 0, stream_>>>(ta, s.mid_roots, s.mid_nodes, s.mid_ends);
  if (levels > 0) {
    k_sizes<<<1, 512, 0, stream_>>>(ta, s.tasks, levels);
    k_dfs<<<1, 512, 0, stream_>>>(ta, s.tasks, levels);
  }
  if (mids > 0) k_mid_dfs<<<blocks_for(32ll * mids, 128), 128, 0, stream_>>>(ta, s.mid_roots, s.mid_nodes, s.mid_ends);
  k_small_dfs<<<blocks_for(s.nn, 256), 256, 0, stream_>>>(ta, static_cast<int>(s.nn));
  k_finish<<<1, 32, 0, stream_>>>(ta);
  BVH_CK(cudaGetLastError());
  read_counters();
  if (host.nodes > static_cast<int>(s.nn)) throw std::logic_error("device BVH build: node overflow");

  // Four-wide collapse, one launch per level (at most one per binary level).
  BVH_CK(cudaMemsetAsync(s.wflag, 0, std::size_t(host.nodes) * sizeof(std::uint32_t), stream_));
  WideArgs wa{s.box, s.left, s.right, s.dfs, s.wide_list, s.wide_kids, s.wflag, s.counters};
  k_wide_init<<<1, 32, 0, stream_>>>(wa);
  const int wide_levels = std::min(host.max_depth + 1, kMaxLevels);
  const int wide_grid = std::min(blocks_for(host.interior, 256), 148 * 8);
  for (int w = 0; w < wide_levels; ++w) k_wide<<<wide_grid, 256, 0, stream_>>>(wa, w);
  const int nb = blocks_for(host.nodes, kScanBlock);
  k_scan_block<<<nb, kScanBlock, 0, stream_>>>(s.wflag, s.wscan, s.scan_sums, host.nodes);
  k_scan_sums<<<1, kScanBlock, 0, stream_>>>(s.scan_sums, nb);
  k_scan_add<<<nb, kScanBlock, 0, stream_>>>(s.wscan, s.scan_sums, host.nodes);
  BVH_CK(cudaGetLastError());
  BVH_CK(cudaEventRecord(ev[1], stream_));
  read_counters();
  BVH_CK(cudaEventElapsedTime(&counts_.build_ms, ev[0], ev[1]));

  counts_.nodes = host.nodes;
  counts_.interior = host.interior;
  counts_.leaves = host.leaves;
  counts_.max_leaf = host.max_leaf;
  counts_.max_depth = host.max_depth;
  counts_.levels = levels;
  int wide = 0, depth4 = 0;
  for (int w = 0; w < kMaxLevels; ++w) {
    wide += host.wide_cnt[w];
    if (host.wide_cnt[w] > 0) depth4 = w + 1;
  }
  if (host.wide_cnt[wide_levels] != 0) throw std::logic_error("device BVH build: four-wide levels left over");
  counts_.wide = wide;
  counts_.depth4 = depth4;
  counts_.root = host.interior > 0 ? 0 : ~0;
  counts_.root4 = host.interior > 0 ? 0 : ~0;
  if (3 * depth4 + 1 > kWideStackDepth) throw std::runtime_error("BVH deeper than the traversal stack allows");
  return counts_;
}

void GpuBvhBuilder::emit(const GpuBvhInput& in, DevNode* nodes, DevNode4* nodes4, float4* prims,
                         std::uint32_t* slot_material, float4* slot_normals, std::uint32_t* order) {
  if (in.n_items == 0 || !st_) return;
  State& s = *st_;
  EmitArgs e{};
  e.t.box = s.box;
  e.t.left = s.left;
  e.t.right = s.right;
  e.t.first = s.first;
  e.t.count = s.count;
  e.t.axis = s.axis;
  e.t.size = s.size;
  e.t.isize = s.isize;
  e.t.dfs = s.dfs;
  e.t.idfs = s.idfs;
  e.t.sub = s.sub;
  e.t.local = s.local;
  e.t.ilocal = s.ilocal;
  e.t.counters = s.counters;
  e.items = s.items;
  e.rows = in.rows;
  e.normals = in.normals;
  e.material = in.material;
  e.wide_list = s.wide_list;
  e.wide_kids = s.wide_kids;
  e.wscan = s.wscan;
  e.last = s.last;
  e.nodes = nodes;
  e.nodes4 = nodes4;
  e.prims = prims;
  e.slot_material = slot_material;
  e.slot_normals = slot_normals;
  e.order = order;
  e.capacity = static_cast<int>(s.nn);
  BVH_CK(cudaMemsetAsync(s.last, 0, s.n, stream_));
  k_mark_last<<<blocks_for(counts_.nodes, 256), 256, 0, stream_>>>(e);
  if (counts_.interior > 0) k_emit_nodes<<<blocks_for(counts_.nodes, 256), 256, 0, stream_>>>(e);
  k_emit_slots<<<blocks_for(s.n, 256), 256, 0, stream_>>>(e, s.n);
  if (counts_.wide > 0) k_emit_wide<<<blocks_for(counts_.wide, 256), 256, 0, stream_>>>(e, counts_.wide);
  BVH_CK(cudaGetLastError());
}

void GpuBvhBuilder::node_costs(double* out) {
  if (!st_ || counts_.nodes == 0) return;
  TreeArgs t{};
  t.box = st_->box;
  t.left = st_->left;
  t.count = st_->count;
  t.dfs = st_->dfs;
  k_node_costs<<<blocks_for(counts_.nodes, 256), 256, 0, stream_>>>(t, counts_.nodes, out);
  BVH_CK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Slot order of the eight-wide tree

namespace {

__device__ __forceinline__ std::int32_t remap_leaf(std::int32_t link, const std::uint32_t* new_of, std::uint32_t n) {
  if (link >= 0 || link == INT32_MIN) return link;
  const std::uint32_t old = static_cast<std::uint32_t>(~link);
  return old < n ? ~static_cast<std::int32_t>(new_of[old]) : link;
}

__global__ void k_gather_slots(const std::uint32_t* old_of, std::uint32_t n, const float4* prims_in,
                               const float4* normals_in, const std::uint32_t* material_in, float4* prims,
                               float4* normals, std::uint32_t* material) {
  const std::uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const std::uint32_t o = old_of[k];
  if (o >= n) return;
  for (int r = 0; r < 3; ++r) {
    prims[3 * k + r] = prims_in[3 * o + r];
    normals[3 * k + r] = normals_in[3 * o + r];
  }
  material[k] = material_in[o];
}

__global__ void k_remap_links(const std::uint32_t* new_of, std::uint32_t n, DevNode* nodes, std::int32_t n_nodes,
                              DevNode4* nodes4, std::int32_t n_wide) {
  const std::int32_t i = static_cast<std::int32_t>(blockIdx.x * blockDim.x + threadIdx.x);
  if (i < n_nodes) {
    int4 l = nodes[i].link;
    l.x = remap_leaf(l.x, new_of, n);
    l.y = remap_leaf(l.y, new_of, n);
    nodes[i].link = l;
  }
  if (i < n_wide) {
    int4 l = nodes4[i].link;
    l.x = remap_leaf(l.x, new_of, n);
    l.y = remap_leaf(l.y, new_of, n);
    l.z = remap_leaf(l.z, new_of, n);
    l.w = remap_leaf(l.w, new_of, n);
    nodes4[i].link = l;
  }
}

}  // namespace

cudaError_t apply_slot_order(const std::uint32_t* old_of, const std::uint32_t* new_of, std::uint32_t n_slots,
                             const float4* prims_in, const float4* normals_in, const std::uint32_t* material_in,
                             float4* prims, float4* normals, std::uint32_t* material, DevNode* nodes,
                             std::int32_t n_nodes, DevNode4* nodes4, std::int32_t n_wide, cudaStream_t stream) {
  if (n_slots) {
    k_gather_slots<<<(n_slots + 255) / 256, 256, 0, stream>>>(old_of, n_slots, prims_in, normals_in, material_in,
                                                              prims, normals, material);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  const std::int32_t n = n_nodes > n_wide ? n_nodes : n_wide;
  if (n > 0) k_remap_links<<<(n + 255) / 256, 256, 0, stream>>>(new_of, n_slots, nodes, n_nodes, nodes4, n_wide);
  return cudaGetLastError();
}

}  // namespace rtg
