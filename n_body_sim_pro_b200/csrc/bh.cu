// GPU Barnes-Hut kernels for sm_100a.
//
// Reference (richie-rich90454/n_body_sim_pro, src/c/barnes_hut/barnes_hut.c):
//   root cube      :453-483   keys  :286-305   sort  :312-339
//   reorder        :402-440   COM   :214-253   walk  :549-636   scatter :692-704
//
// The Morton keys and the sort permutation are bit-exact with the reference:
// all FP64 arithmetic of the root cube and of morton_axis_code is done with
// explicitly rounded __d*_rn intrinsics (no contraction), and the 7 x 9-bit
// stable LSD sort yields the same permutation as the reference's stable
// 3 x 21-bit LSD sort (a stable sort by the full key, ties by original index).
//
// The tree differs from the reference's pointer octree by design: it is built
// in parallel from the sorted keys (a Karras binary radix tree, one thread per
// internal node), collapsed to a path-compressed octree whose leaves hold up to
// `leaf_capacity` Morton-contiguous particles, and stored in depth-first order
// with skip links so the walk needs no stack.  Parity is judged on forces
// against the FP64 all-pairs oracle, and the opening test is the reference's:
// accept a cell when (2h)^2 < theta^2 d^2, d to the cell centre of mass.  A
// bucket of >= 2 particles is the reference's cell of the same side and
// particles, so it takes the same test; where the reference would open it, its
// particles are summed exactly (a single particle is always exact).
#include "bh.h"
#include "mlp.cuh"
#include "mlp_umma.cuh"

#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

namespace {

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------
// bounds
// ---------------------------------------------------------------------------

constexpr int kBoundsThreads = 256;
constexpr int kBoundsBlocks = 4 * 148;  // one wave at 4 blocks of 256 per SM (58 registers)
constexpr int kBoundsVals = 11;  // min xyz, max xyz, m, mx, my, mz, |a|^2

// The combined values (from FIRST on) of the block's first kBoundsThreads threads
// in thread 0: each warp by shuffles, then the warps' results by the first warp.
template <int FIRST = 0>
__device__ __forceinline__ void bounds_block_reduce(double (&v)[kBoundsVals],
                                                    double (*sh)[kBoundsThreads / 32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < kBoundsThreads / 32) {
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int q = FIRST; q < kBoundsVals; ++q) {
        const double o = __shfl_xor_sync(0xffffffffu, v[q], off);
        v[q] = q < 3 ? fmin(v[q], o) : q < 6 ? fmax(v[q], o) : v[q] + o;
      }
    }
    if (lane == 0)
#pragma unroll
      for (int q = FIRST; q < kBoundsVals; ++q) sh[q][w] = v[q];
  }
  __syncthreads();
  if (w != 0) return;
#pragma unroll
  for (int q = FIRST; q < kBoundsVals; ++q)
    v[q] = lane < kBoundsThreads / 32 ? sh[q][lane]
           : q < 3                    ? INFINITY
           : q < 6                    ? -INFINITY
                                      : 0.0;
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int q = FIRST; q < kBoundsVals; ++q) {
      const double o = __shfl_xor_sync(0xffffffffu, v[q], off);
      v[q] = q < 3 ? fmin(v[q], o) : q < 6 ? fmax(v[q], o) : v[q] + o;
    }
  }
}

// Phase boundaries of an evaluation are read from the GPU's clock by the first
// thread of each phase's first kernel, or, where a memset comes before that, at the
// end of the kernel before (stamp NULL: not timed).  A timing event
// between two kernels held the second one back by about 3.5 us.
__device__ __forceinline__ unsigned long long gpu_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void stamp_start(unsigned long long* stamp) {
  if (stamp != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *stamp = gpu_clock();
}

// |a|^2, contracted the same way wherever it is summed.
__device__ __forceinline__ double square_sum(double x, double y, double z) {
  return fma(z, z, fma(y, y, x * x));
}

// KICK: the opening kick and drift of a device-resident leapfrog step first
// (kick_drift_kernel's arithmetic), the reductions then of the drifted state.
template <bool KICK>
__global__ void __launch_bounds__(kBoundsThreads) bounds_kernel(
    double* __restrict__ x, double* __restrict__ y, double* __restrict__ z,
    const double* __restrict__ m, size_t n, double* __restrict__ partial, int* status,
    const double* __restrict__ ax, const double* __restrict__ ay,
    const double* __restrict__ az, bool rms_of_a, double* __restrict__ vx,
    double* __restrict__ vy, double* __restrict__ vz, double h, double dt,
    unsigned long long* stamp) {
  stamp_start(stamp);
  __shared__ double sh[kBoundsVals][kBoundsThreads / 32];
  double v[kBoundsVals] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY,
                           0.0,      0.0,      0.0,      0.0,       0.0};
  bool bad = false;
#pragma unroll 4
  for (size_t i = blockIdx.x * (size_t)kBoundsThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kBoundsThreads) {
    double px = x[i], py = y[i], pz = z[i];
    const double pm = m[i];
    if (KICK) {
      const double u = __dadd_rn(vx[i], __dmul_rn(ax[i], h));
      const double w = __dadd_rn(vy[i], __dmul_rn(ay[i], h));
      const double q = __dadd_rn(vz[i], __dmul_rn(az[i], h));
      vx[i] = u;
      vy[i] = w;
      vz[i] = q;
      px = __dadd_rn(px, __dmul_rn(u, dt));
      py = __dadd_rn(py, __dmul_rn(w, dt));
      pz = __dadd_rn(pz, __dmul_rn(q, dt));
      x[i] = px;
      y[i] = py;
      z[i] = pz;
    }
    bad |= !(isfinite(px) && isfinite(py) && isfinite(pz));
    v[0] = fmin(v[0], px);
    v[1] = fmin(v[1], py);
    v[2] = fmin(v[2], pz);
    v[3] = fmax(v[3], px);
    v[4] = fmax(v[4], py);
    v[5] = fmax(v[5], pz);
    v[6] += pm;
    v[7] += pm * px;
    v[8] += pm * py;
    v[9] += pm * pz;
    if (rms_of_a) v[10] += square_sum(ax[i], ay[i], az[i]);
  }
  if (bad) atomicOr(status, NBSP_DEVICE_ERROR_NONFINITE_POSITION);
  bounds_block_reduce(v, sh);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < kBoundsVals; ++q) partial[blockIdx.x * kBoundsVals + q] = v[q];
}

// The blocks' partial results combined by a block's first kBoundsThreads threads
// (the others only join the barrier), and in thread 0 the root cube with the
// exact FP64 operation sequence of barnes_hut.c:471-483.
__device__ __forceinline__ void root_geometry(const double* __restrict__ partial, int blocks,
                                              size_t n, double (*sh)[kBoundsThreads / 32],
                                              double* geometry) {
  double v[kBoundsVals] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY,
                           0.0,      0.0,      0.0,      0.0,       0.0};
  if (threadIdx.x < kBoundsThreads)
    for (int b = threadIdx.x; b < blocks; b += kBoundsThreads) {
      for (int q = 0; q < 3; ++q) v[q] = fmin(v[q], partial[b * kBoundsVals + q]);
      for (int q = 3; q < 6; ++q) v[q] = fmax(v[q], partial[b * kBoundsVals + q]);
      for (int q = 6; q < kBoundsVals; ++q) v[q] += partial[b * kBoundsVals + q];
    }
  bounds_block_reduce(v, sh);
  if (threadIdx.x == 0) {
    const double lo[3] = {v[0], v[1], v[2]};
    const double hi[3] = {v[3], v[4], v[5]};
    double half = __dmul_rn(0.5, __dsub_rn(hi[0], lo[0]));
    for (int k = 1; k < 3; ++k) {
      const double e = __dmul_rn(0.5, __dsub_rn(hi[k], lo[k]));
      if (e > half) half = e;
    }
    if (half == 0.0) half = 0.5;
    half = __dmul_rn(half, 1.0 + 1.0e-9);
    for (int k = 0; k < 3; ++k) geometry[k] = __dmul_rn(0.5, __dadd_rn(lo[k], hi[k]));
    geometry[3] = half;
    const double mt = v[6];
    for (int k = 0; k < 3; ++k) geometry[4 + k] = mt != 0.0 ? v[7 + k] / mt : 0.0;
    geometry[7] = n > 0 ? sqrt(v[10] / (double)n) : 0.0;  // rms |a| (when given)
  }
}

__global__ void __launch_bounds__(kBoundsThreads) bounds_final_kernel(
    const double* __restrict__ partial, int blocks, size_t n, double* __restrict__ geometry,
    unsigned long long* end) {
  __shared__ double sh[kBoundsVals][kBoundsThreads / 32];
  root_geometry(partial, blocks, n, sh, geometry);
  if (end != nullptr && threadIdx.x == 0) *end = gpu_clock();
}

// ---------------------------------------------------------------------------
// the tree's arrays
// ---------------------------------------------------------------------------

// Scratch layout of one tree; binary ids: internal node i -> i (0..n-2),
// particle leaf k -> (n-1) + k.
struct Tree {
  int n;
  int2* range;        // [n-1] first, last of internal nodes
  int2* child;        // [n-1] binary ids of the two children
  int* cell;          // [2n-1] octree level of a cell node, -1 otherwise; keep_kernel
                      // adds 32 times a kept cell's place among its siblings
  int* oparent;       // [2n-1] octree parent (binary id) of a kept cell, from keep_kernel
  int2* below;        // [n-1] splitting cells: walk id of the first child, children
  int* split;         // [n-1] the splitting cells' binary ids
  int* split_child;   // [8(n-1)] their octree children's binary ids, -1 behind the last
  uint32_t* mask;     // [n]   levels of kept nodes starting at particle k
  uint32_t* offset;   // [n+1] exclusive scan of popcounts; offset[n] = node count
  uint32_t* block_sums;  // scan scratch
  // Octree nodes carry two numberings, capacity 2n-1 each.  Depth-first (info,
  // dnode) with skip links: the stackless walk and the training pairs.  Walk
  // ids (everything else): the root is 0 and the children of every node are
  // consecutive, in Morton order, so a node's record names them by the first
  // one and a count, their records share cache lines, and neither the
  // interaction-list walk nor the moments pass reads a list of children.
  int4* info;         // depth-first: next, first particle, leaf count (0: internal), walk id
  float4* dnode;      // depth-first, 2 per node: wnode's first six words
  int4* link;         // parent, first child (or first particle), count as in wnode, depth-first id
  int* level;
  int* arrive;
  int* height;
  double4* mom;       // mass, com xyz (relative to the centre of mass)
  double* quad64;     // 6 per node: xx xy xz yy yz zz (trace-free)
  double* trace64;    // sum m |x - com|^2 per node (FP64)
  // what the interaction-list walk reads of a node, in one 32-byte record: (com
  // xyz, mass), (ropen2 = (2h / theta)^2, kmass = M (2h)^2 of the relative test,
  // first particle of a bucket or first child, count as int bits: the particles
  // of a bucket, minus the children of an internal node)
  float4* wnode;      // 2 per node
  // quadrupole walk and correction, 2 per node: (xx, xy, xz, yy), (yz, side =
  // 2h, spread = sum m |x - com|^2 / (M side^2), shift = distance from the
  // cell's geometric centre to its centre of mass)
  float4* wquad;
  unsigned long long* leaves;  // [2]: buckets; splitting cells << 32 | walk ids below the root
};

constexpr int kScanItems = 2048;

// Sub-buffers of the tree scratch, each 256-byte aligned, carved from an
// integer base address (tree_bytes() carves from 0 to measure the layout).
template <typename T>
__host__ __device__ inline T* carve(uintptr_t& p, size_t count) {
  T* out = reinterpret_cast<T*>(p);
  p += (count * sizeof(T) + 255) & ~(size_t)255;
  return out;
}

__host__ __device__ inline Tree tree_layout(uintptr_t p, size_t n_, uintptr_t* end) {
  Tree t;
  const size_t n = n_ < 2 ? 2 : n_;
  const size_t ni = n - 1, nb = 2 * n - 1;
  t.n = (int)n_;
  t.range = carve<int2>(p, ni);
  t.child = carve<int2>(p, ni);
  t.cell = carve<int>(p, nb);
  t.oparent = carve<int>(p, nb);
  t.below = carve<int2>(p, ni);
  t.split = carve<int>(p, ni);
  t.split_child = carve<int>(p, 8 * ni);
  t.mask = carve<uint32_t>(p, n);
  t.offset = carve<uint32_t>(p, n + 1);
  t.block_sums = carve<uint32_t>(p, (n + kScanItems - 1) / kScanItems + 1);
  t.info = carve<int4>(p, nb);
  t.dnode = carve<float4>(p, 2 * nb);
  t.link = carve<int4>(p, nb);
  t.level = carve<int>(p, nb);
  t.arrive = carve<int>(p, nb);
  t.height = carve<int>(p, nb);
  t.mom = carve<double4>(p, nb);
  t.quad64 = carve<double>(p, 6 * nb);
  t.trace64 = carve<double>(p, nb);
  t.wnode = carve<float4>(p, 2 * nb);
  t.wquad = carve<float4>(p, 2 * nb);
  t.leaves = carve<unsigned long long>(p, 2);
  if (end != nullptr) *end = p;
  return t;
}

inline Tree tree_view(void* base, size_t n) {
  return tree_layout(reinterpret_cast<uintptr_t>(base), n, nullptr);
}

size_t tree_bytes(size_t n) {
  uintptr_t end = 0;
  tree_layout(0, n, &end);
  return (size_t)end;
}

// ---------------------------------------------------------------------------
// Morton keys
// ---------------------------------------------------------------------------

// barnes_hut.c:286-294 with every FP64 operation explicitly rounded.
__device__ __forceinline__ uint64_t axis_code(double value, double centre, double half) {
  double t = __dadd_rn(__ddiv_rn(__dsub_rn(value, centre), __dmul_rn(2.0, half)), 0.5);
  if (t < 0.0) {
    t = 0.0;
  } else if (t >= 1.0) {
    t = 1.0 - 1.0e-15;
  }
  return (uint64_t)__double2ull_rz(__dmul_rn(t, 2097152.0));
}

// Spread the low 21 bits of v to every third bit (bit b -> bit 3b).
__device__ __forceinline__ uint64_t spread3(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 32)) & 0x001f00000000ffffull;
  v = (v | (v << 16)) & 0x001f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

// ---------------------------------------------------------------------------
// stable LSD radix sort, 9-bit digits, one kernel per pass
//
// The keys kernel also counts the 7 digit histograms (one read of the keys), which
// every tile scans for the digits' bases.  Every pass is a single kernel: tiles take
// tickets in launch order, rank their keys in shared memory, and find their global
// offsets with a decoupled look-back over the preceding tiles' published digit
// counts (flag A: this tile's count, flag P: inclusive prefix).  A tile only waits
// on tiles with earlier tickets, which are already resident; every wait is bounded
// and flags an error when it runs out.
// ---------------------------------------------------------------------------

// A tile is THREADS x ITEMS keys (the figures are of passes by 8-bit digits).
// Large systems: 512 threads of 8 keys (at 10M keys 0.92 ms for the 8 passes
// against 1.10 with 256 x 16, whose ranking chain per warp is twice as long, and
// 1.17 with 1024 x 4, one block per SM).  Below
// kSortWide keys those tiles leave SMs idle and a pass is one tile's chain of
// load, rank, look back and scatter: 512 threads of 4 keys take 78 us for the 8
// passes at 100k-150k and 91 at 262k (wide tiles: 97 and 109; 256 x 4: 79 and
// 95), the same as wide tiles at 500k and more beyond (1M: 185 against 154).
struct SortWide {
  static constexpr int kThreads = 512, kItems = 8, kBlocks = 2;
};
struct SortNarrow {
  static constexpr int kThreads = 512, kItems = 4, kBlocks = 2;
};
constexpr size_t kSortWide = 450000;
// Digits of nine bits: seven passes over the 63-bit keys, a digit a thread of the
// tile in its look-back.  Against eight passes of 256 digits: 70 and 76 us at 98k
// keys, 82 and 92 at 262k, 147 and 152 at 1M, 882 and 934 at 10M.
constexpr int kRadixBits = 9, kRadix = 1 << kRadixBits;
constexpr int kLookback = 8;  // predecessors' flags read at once in the look-back
template <class S>
constexpr int sort_tile() {
  static_assert(S::kThreads >= kRadix, "one thread per digit");
  return S::kThreads * S::kItems;
}
constexpr int kSortPasses = 63 / kRadixBits;
constexpr uint32_t kFlagA = 1u << 30, kFlagP = 2u << 30, kCountMask = (1u << 30) - 1u;
constexpr int kLookbackSpins = 1 << 22;  // ~ms per predecessor before the error flag
constexpr int kKeysBlocks = 5 * 148;  // 40 warps per SM (48 registers): enough loads in flight

// Sort scratch (32-bit words): hist[7][512] | ticket[7] | status[7][tiles][512]
struct SortScratch {
  uint32_t* hist;
  uint32_t* ticket;
  uint32_t* status;
};
__device__ __forceinline__ unsigned sort_digit(uint64_t key, int shift) {
  return (unsigned)(key >> shift) & (unsigned)(kRadix - 1);
}
inline size_t sort_tiles(size_t n) {
  const size_t tile = n < kSortWide ? sort_tile<SortNarrow>() : sort_tile<SortWide>();
  return (n + tile - 1) / tile;
}
inline SortScratch sort_scratch(uint32_t* w) {
  SortScratch s;
  s.hist = w;
  s.ticket = w + kSortPasses * kRadix;
  s.status = s.ticket + kSortPasses;
  return s;
}
inline size_t sort_scratch_words(size_t n) {
  return kSortPasses * kRadix + kSortPasses + kSortPasses * sort_tiles(n) * kRadix;
}

// What the build and the walk count into starts at zero (with every particle's
// mask, which the keys kernels clear beside its key; memsets took a place of
// their own on the stream).
constexpr int kCounters = NBSP_BH_COUNTERS;
__device__ __forceinline__ void start_tree(const Tree& t, unsigned long long* counters,
                                           unsigned long long* stamp) {
  stamp_start(stamp);
  if (blockIdx.x == 0 && threadIdx.x < kCounters) {
    counters[threadIdx.x] = 0;
    if (threadIdx.x == 0) counters[kCounters + NBSP_BH_END] = 0;
    if (threadIdx.x < 2) t.leaves[threadIdx.x] = 0;
  }
}

// The relative opening test's alpha max(|a_old|, rms) / G of particle i.
__device__ __forceinline__ float opening_tolerance(size_t i, const double* __restrict__ ax,
                                                   const double* __restrict__ ay,
                                                   const double* __restrict__ az, double rms,
                                                   double tol_scale) {
  const double a = fmax(sqrt(square_sum(ax[i], ay[i], az[i])), rms);
  return a > 0.0 && isfinite(a) ? (float)(tol_scale * a) : INFINITY;
}

// Particle i's Morton key under root cube `geometry`, and its record for the
// walk, still in input order: the float4 (relative to the centre of mass) and
// with `unsorted_tol` the relative opening test's tolerance.
__device__ __forceinline__ uint64_t particle_key(
    size_t i, const double* __restrict__ x, const double* __restrict__ y,
    const double* __restrict__ z, const double* __restrict__ m, const double (&geometry)[8],
    const double* __restrict__ ax, const double* __restrict__ ay, const double* __restrict__ az,
    double tol_scale, float4* __restrict__ unsorted, float* __restrict__ unsorted_tol) {
  const double xi = x[i], yi = y[i], zi = z[i];
  unsorted[i] = make_float4((float)__dsub_rn(xi, geometry[4]), (float)__dsub_rn(yi, geometry[5]),
                            (float)__dsub_rn(zi, geometry[6]), (float)m[i]);
  if (unsorted_tol != nullptr)
    unsorted_tol[i] = opening_tolerance(i, ax, ay, az, geometry[7], tol_scale);
  return spread3(axis_code(xi, geometry[0], geometry[3])) |
         (spread3(axis_code(yi, geometry[1], geometry[3])) << 1) |
         (spread3(axis_code(zi, geometry[2], geometry[3])) << 2);
}

__global__ void __launch_bounds__(256) keys_kernel(
    const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
    const double* __restrict__ m, size_t n, const double* __restrict__ geometry,
    uint64_t* __restrict__ keys, uint32_t* __restrict__ index, float4* __restrict__ unsorted,
    uint32_t* __restrict__ hist, const double* __restrict__ ax, const double* __restrict__ ay,
    const double* __restrict__ az, double tol_scale, float* __restrict__ unsorted_tol, Tree tree,
    unsigned long long* counters) {
  __shared__ uint32_t h[kSortPasses][kRadix];
  start_tree(tree, counters, nullptr);
  for (int k = threadIdx.x; k < kSortPasses * kRadix; k += blockDim.x) (&h[0][0])[k] = 0;
  __syncthreads();
  double geo[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) geo[k] = geometry[k];
  const unsigned lane = threadIdx.x & 31;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  // every lane runs the same number of iterations (match_any needs the whole warp)
  const size_t rounds = (n + stride - 1) / stride;
  for (size_t r = 0; r < rounds; ++r) {
    const size_t i = first + r * stride;
    const bool valid = i < n;
    uint64_t key = 0;
    if (valid) {
      key = particle_key(i, x, y, z, m, geo, ax, ay, az, tol_scale, unsorted, unsorted_tol);
      keys[i] = key;
      index[i] = (uint32_t)i;
      tree.mask[i] = 0;
    }
#pragma unroll
    // digit counts: the low digits of the keys of one warp are spread over many
    // values (plain shared atomics); the top two (the first six octree levels)
    // repeat, so they are aggregated per warp first
    for (int p = 0; p < kSortPasses; ++p) {
      if (p < kSortPasses - 2) {
        if (valid) atomicAdd(&h[p][sort_digit(key, kRadixBits * p)], 1u);
      } else {
        const unsigned d = valid ? sort_digit(key, kRadixBits * p) : kRadix;
        const unsigned peers = __match_any_sync(kFull, d);
        if (valid && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(&h[p][d], (uint32_t)__popc(peers));
      }
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kSortPasses * kRadix; k += blockDim.x) {
    const uint32_t v = (&h[0][0])[k];
    if (v != 0) atomicAdd(&hist[k], v);
  }
}

__device__ __forceinline__ uint32_t load_volatile(const uint32_t* p) {
  return *reinterpret_cast<const volatile uint32_t*>(p);
}

// hist: the pass's digit counts over all keys; every tile scans them for the
// digits' first places (a launch of its own took 6 us).
template <class S>
__global__ void __launch_bounds__(S::kThreads, S::kBlocks) sort_pass_kernel(
    const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, size_t n, int shift,
    const uint32_t* __restrict__ hist, uint32_t* ticket, uint32_t* status, int* err,
    unsigned long long* stamp) {
  stamp_start(stamp);
  constexpr int kSortThreads = S::kThreads, kSortItems = S::kItems;
  constexpr int kSortWarps = kSortThreads / 32, kSortTile = sort_tile<S>();
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* sk = reinterpret_cast<uint64_t*>(smem);                     // kSortTile
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + kSortTile);           // kSortTile
  uint32_t* wc = sv + kSortTile;                                        // kSortWarps * kRadix
  uint32_t* start = wc + kSortWarps * kRadix;                           // kRadix
  uint32_t* gofs = start + kRadix;                                      // kRadix
  __shared__ int s_tile;
  __shared__ uint32_t s_hsum[kRadix / 32];

  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  if (t == 0) s_tile = (int)atomicAdd(ticket, 1u);
  uint32_t digit_base = 0;  // threads t < kRadix: keys of smaller digits
  if (t < kRadix) {
    const uint32_t own = hist[t];
    uint32_t x = own;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_up_sync(kFull, x, off);
      if (lane >= off) x += u;
    }
    if (lane == 31) s_hsum[w] = x;
    digit_base = x - own;
  }
  for (int k = t; k < kSortWarps * kRadix; k += kSortThreads) wc[k] = 0;
  __syncthreads();
  const int tile = s_tile;

  const size_t base_i = (size_t)tile * kSortTile + (size_t)w * (kSortItems * 32);
  const unsigned lt = (1u << lane) - 1u;
  uint64_t key[kSortItems];
  uint32_t val[kSortItems];
  uint32_t rank[kSortItems];
#pragma unroll
  for (int it = 0; it < kSortItems; ++it) {  // every load of the tile in flight at once
    const size_t i = base_i + (size_t)it * 32 + lane;
    const bool valid = i < n;
    key[it] = valid ? keys_in[i] : 0ull;
    val[it] = valid ? vals_in[i] : 0u;
  }
#pragma unroll
  for (int it = 0; it < kSortItems; ++it) {
    const bool valid = base_i + (size_t)it * 32 + lane < n;
    const unsigned digit = valid ? sort_digit(key[it], shift) : kRadix;
    const unsigned peers = __match_any_sync(kFull, digit);
    uint32_t before = 0;
    if (valid) before = wc[w * kRadix + digit];
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) wc[w * kRadix + digit] = before + __popc(peers);
    __syncwarp();
    rank[it] = before + __popc(peers & lt);
  }
  __syncthreads();
  // threads t < kRadix: digit t — this tile's count, publish, look back, and the
  // exclusive scan of the tile's digit totals (warp shuffles, then warp sums)
  __shared__ uint32_t s_wsum[kRadix / 32];
  if (t < kRadix) {
    uint32_t run = 0;
    for (int ww = 0; ww < kSortWarps; ++ww) {
      const uint32_t c = wc[ww * kRadix + t];
      wc[ww * kRadix + t] = run;
      run += c;
    }
    const uint32_t count = run;  // this tile's keys with digit t
    uint32_t* st = status + (size_t)tile * kRadix + t;
    atomicExch(st, (tile == 0 ? kFlagP : kFlagA) | count);
    uint32_t prefix = 0;
    if (tile > 0) {
      // kLookback predecessors at a time, nearest first: counts are added up
      // to the first unpublished flag (read again) or the first inclusive one
      int j = tile - 1, spins = 0;
      for (;;) {
        uint32_t v[kLookback];
#pragma unroll
        for (int k = 0; k < kLookback; ++k)
          v[k] = j - k >= 0 ? load_volatile(status + (size_t)(j - k) * kRadix + t) : kFlagP;
        int used = 0;
        bool done = false;
#pragma unroll
        for (int k = 0; k < kLookback; ++k) {
          if (done || used < k) continue;
          const uint32_t flag = v[k] & ~kCountMask;
          if (flag == 0u) continue;
          prefix += v[k] & kCountMask;
          used = k + 1;
          if (flag == kFlagP) done = true;
        }
        if (done) break;
        if (used == 0 && ++spins > kLookbackSpins) {
          atomicOr(err, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
          break;
        }
        j -= used;
      }
      atomicExch(st, kFlagP | ((prefix + count) & kCountMask));
    }
    for (int k = 0; k < w; ++k) digit_base += s_hsum[k];
    gofs[t] = digit_base + prefix;
    uint32_t x = count;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_up_sync(kFull, x, off);
      if (lane >= off) x += u;
    }
    if (lane == 31) s_wsum[w] = x;
    start[t] = x - count;
  }
  __syncthreads();
  if (t < kRadix) {
    uint32_t before = 0;
    for (int k = 0; k < w; ++k) before += s_wsum[k];
    start[t] += before;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < kSortItems; ++it) {
    const size_t i = base_i + (size_t)it * 32 + lane;
    if (i < n) {
      const unsigned digit = sort_digit(key[it], shift);
      const uint32_t pos = start[digit] + wc[w * kRadix + digit] + rank[it];
      if (pos < (uint32_t)kSortTile) {
        sk[pos] = key[it];
        sv[pos] = val[it];
      } else {
        atomicOr(err, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      }
    }
  }
  __syncthreads();
  const size_t tile_base = (size_t)tile * kSortTile;
  const int count_all = (int)(n - tile_base < (size_t)kSortTile ? n - tile_base : (size_t)kSortTile);
  for (int q = t; q < count_all; q += kSortThreads) {
    const uint64_t k = sk[q];
    const unsigned digit = sort_digit(k, shift);
    const size_t dst = (size_t)gofs[digit] + (size_t)(q - (int)start[digit]);
    if (dst < n) {
      keys_out[dst] = k;
      vals_out[dst] = sv[q];
    } else {
      atomicOr(err, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    }
  }
}

template <class S>
constexpr size_t sort_pass_smem() {
  return (size_t)sort_tile<S>() * (sizeof(uint64_t) + sizeof(uint32_t)) +
         (size_t)(S::kThreads / 32 * kRadix + 2 * kRadix) * sizeof(uint32_t);
}

// ---------------------------------------------------------------------------
// the same sort for up to NBSP_BH_SMALL_SORT keys: two kernels
//
// Seven passes of the radix sort are seven chains of load, rank, look back and
// scatter on a few tiles, about 10 us each however few keys there are.  Here
// every CTA computes the keys of one tile of 1024 particles (and first, from the
// bounds' partial results, the root cube) and sorts them in a bitonic network,
// by (key, index), so that equal keys keep their order; then each key finds its
// place by its rank among every other tile's keys, and the walk's records are
// written there directly (no gather pass).  The ranks cost n / 1024 binary
// searches per key, the radix passes none.  Sort and gather, small against
// radix: 10 against 91 us at 10k, 11 against 88 at 20k, 35 against 95 at 65k, 70
// against 82 at 100k, 132 against 82 at 150k: the line is where the two meet.
// ---------------------------------------------------------------------------

constexpr int kSmallTile = 1024;

__global__ void __launch_bounds__(kSmallTile) small_keys_kernel(
    const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
    const double* __restrict__ m, size_t n, const double* __restrict__ partial, int blocks,
    double* __restrict__ geometry, uint64_t* __restrict__ keys, uint32_t* __restrict__ index,
    float4* __restrict__ unsorted, const double* __restrict__ ax, const double* __restrict__ ay,
    const double* __restrict__ az, double tol_scale, float* __restrict__ unsorted_tol, Tree tree,
    unsigned long long* counters, unsigned long long* stamp) {
  __shared__ double sh[kBoundsVals][kBoundsThreads / 32];
  __shared__ double s_geo[8];
  __shared__ uint64_t sk[kSmallTile];
  __shared__ uint32_t sv[kSmallTile];
  const int t = threadIdx.x;
  start_tree(tree, counters, stamp);
  root_geometry(partial, blocks, n, sh, s_geo);
  __syncthreads();
  double geo[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) geo[k] = s_geo[k];
  if (blockIdx.x == 0 && t < 8) geometry[t] = s_geo[t];
  const size_t i = (size_t)blockIdx.x * kSmallTile + t;
  uint64_t key = ~0ull;  // past the end: behind every 63-bit key
  if (i < n) {
    tree.mask[i] = 0;
    key = particle_key(i, x, y, z, m, geo, ax, ay, az, tol_scale, unsorted, unsorted_tol);
  }
  uint32_t val = (uint32_t)t;
  for (int k = 2; k <= kSmallTile; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      uint64_t pk;
      uint32_t pv;
      if (j >= 32) {
        __syncthreads();
        sk[t] = key;
        sv[t] = val;
        __syncthreads();
        pk = sk[t ^ j];
        pv = sv[t ^ j];
      } else {
        pk = __shfl_xor_sync(kFull, (unsigned long long)key, j);
        pv = __shfl_xor_sync(kFull, val, j);
      }
      const bool less = pk < key || (pk == key && pv < val);  // the partner belongs first
      const bool first = ((t & j) == 0) == ((t & k) == 0);    // this slot takes the smaller
      if (less == first) {
        key = pk;
        val = pv;
      }
    }
  }
  if (i < n) {
    keys[i] = key;
    index[i] = blockIdx.x * kSmallTile + val;
  }
}

// 32 consecutive keys of one sorted tile per block; warp w ranks them among
// tiles w, w + 8, ... (a warp's keys are neighbours, so its searches of a tile
// run through nearly the same words), two tiles at a time.
constexpr int kMergeWarps = 8;
__global__ void __launch_bounds__(32 * kMergeWarps) small_merge_kernel(
    const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, int n,
    uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
    const float4* __restrict__ unsorted, float4* __restrict__ pos,
    const float* __restrict__ unsorted_tol, float* __restrict__ tol, int* err,
    unsigned long long* stamp) {
  stamp_start(stamp);
  __shared__ int s_rank[kMergeWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int s = blockIdx.x * 32 + lane;
  const bool valid = s < n;
  const uint64_t key = keys_in[valid ? s : n - 1];
  const uint32_t i = w == 0 && valid ? vals_in[s] : 0u;
  float4 record = make_float4(0.f, 0.f, 0.f, 0.f);
  if (w == 0 && valid && i < (uint32_t)n) record = unsorted[i];
  const int tile = blockIdx.x * 32 / kSmallTile, tiles = (n + kSmallTile - 1) / kSmallTile;
  int rank = 0;
  for (int t0 = w; t0 < tiles; t0 += 2 * kMergeWarps) {
    // keys of an earlier tile go before this one when not greater, keys of a
    // later tile when smaller
    int count[2], len[2];
    uint64_t below[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = t0 + q * kMergeWarps;
      count[q] = 0;
      len[q] = u < tiles && u != tile ? min(kSmallTile, n - u * kSmallTile) : 0;
      below[q] = key + (u < tile ? 1u : 0u);
    }
    const uint64_t* k0 = keys_in + (size_t)t0 * kSmallTile - 1;
#pragma unroll
    for (int step = kSmallTile; step > 0; step >>= 1) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int p = count[q] + step;
        if (p <= len[q] && k0[q * kMergeWarps * kSmallTile + p] < below[q]) count[q] = p;
      }
    }
    rank += count[0] + count[1];
  }
  s_rank[w][lane] = rank;
  __syncthreads();
  if (w != 0 || !valid) return;
  rank = s % kSmallTile;
#pragma unroll
  for (int q = 0; q < kMergeWarps; ++q) rank += s_rank[q][lane];
  if (rank >= n || i >= (uint32_t)n) {
    atomicOr(err, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    return;
  }
  keys_out[rank] = key;
  vals_out[rank] = i;
  pos[rank] = record;
  if (tol != nullptr) tol[rank] = unsorted_tol[i];
}

// The reference's insertion build fails with OVERFLOW when two particles share
// a position (barnes_hut.c:149-153: more than 128 subdivisions).  Equal
// positions have equal keys, so after the sort they sit in one run of equal
// keys; each particle is compared with the next kDupWindow particles of its run
// (runs of equal 63-bit keys are otherwise rare: cells of 2^-21 of the root).
constexpr int kDupWindow = 32;
__device__ __forceinline__ void flag_duplicates(size_t s, const uint64_t* __restrict__ keys,
                                                const uint32_t* __restrict__ perm,
                                                const double* __restrict__ x,
                                                const double* __restrict__ y,
                                                const double* __restrict__ z, size_t n,
                                                int* status) {
  const uint64_t k = keys[s];
  const uint32_t i = perm[s];
  if (i >= n) return;
  const double px = x[i], py = y[i], pz = z[i];
  for (size_t t = s + 1; t < n && t <= s + kDupWindow && keys[t] == k; ++t) {
    const uint32_t j = perm[t];
    if (j < n && x[j] == px && y[j] == py && z[j] == pz) {
      atomicOr(status, NBSP_DEVICE_ERROR_DUPLICATE_POSITION);
      return;
    }
  }
}

// ---------------------------------------------------------------------------
// gather / scatter
// ---------------------------------------------------------------------------

// pos[s] = unsorted[perm[s]]; the relative opening test's tolerances the same
// way when present.
__global__ void gather_kernel(const float4* __restrict__ unsorted,
                              const uint32_t* __restrict__ perm, size_t n,
                              float4* __restrict__ pos, const float* __restrict__ unsorted_tol,
                              float* __restrict__ tol, int* status, unsigned long long* stamp) {
  stamp_start(stamp);
  for (size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x; s < n;
       s += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = perm[s];
    if (i >= n) {
      atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      pos[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    pos[s] = unsorted[i];
    if (tol != nullptr) tol[s] = unsorted_tol[i];
  }
}

// The relative test's tolerances of accelerations that were still on their way
// while the tree was built (pinned upload at 1M particles: 24 MB, 0.44 ms, beside
// 0.3 ms of bounds, sort and build).  First the blocks' sums of |a|^2 in
// bounds_kernel's places and order, then, in every block again, their total as
// root_geometry forms it, and each sorted particle's tolerance.
__global__ void __launch_bounds__(kBoundsThreads) late_squares_kernel(
    const double* __restrict__ ax, const double* __restrict__ ay, const double* __restrict__ az,
    size_t n, double* __restrict__ partial) {
  __shared__ double sh[kBoundsVals][kBoundsThreads / 32];
  double v[kBoundsVals];
  v[10] = 0.0;
#pragma unroll 4
  for (size_t i = blockIdx.x * (size_t)kBoundsThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kBoundsThreads)
    v[10] += square_sum(ax[i], ay[i], az[i]);
  bounds_block_reduce<10>(v, sh);
  if (threadIdx.x == 0) partial[blockIdx.x * kBoundsVals + 10] = v[10];
}

__global__ void __launch_bounds__(kBoundsThreads) late_tolerances_kernel(
    const double* __restrict__ ax, const double* __restrict__ ay, const double* __restrict__ az,
    const double* __restrict__ partial, int blocks, size_t n, double tol_scale,
    const uint32_t* __restrict__ perm, float* __restrict__ tol, double* __restrict__ geometry) {
  __shared__ double sh[kBoundsVals][kBoundsThreads / 32];
  __shared__ double s_rms;
  double v[kBoundsVals];
  v[10] = 0.0;
  for (int b = threadIdx.x; b < blocks; b += kBoundsThreads) v[10] += partial[b * kBoundsVals + 10];
  bounds_block_reduce<10>(v, sh);
  if (threadIdx.x == 0) {
    s_rms = sqrt(v[10] / (double)n);
    if (blockIdx.x == 0) geometry[7] = s_rms;
  }
  __syncthreads();
  const double rms = s_rms;
  for (size_t s = blockIdx.x * (size_t)kBoundsThreads + threadIdx.x; s < n;
       s += (size_t)gridDim.x * kBoundsThreads) {
    const uint32_t i = perm[s];  // (a bad one is the gather's to report)
    tol[s] = i < n ? opening_tolerance(i, ax, ay, az, rms, tol_scale) : INFINITY;
  }
}

// a[i] = G * acc[i]: the walk wrote each target's sum at its input index
// (one aligned 32-byte record), so this pass is coalesced both ways.  KICK:
// the closing kick of a device-resident leapfrog step, v += h a, with
// kick_drift_kernel's arithmetic on the accelerations just written.
// The first thread copies the tree's node count, leaf count and depth to
// counters[2..4].
template <bool KICK>
__global__ void unsort_kernel(const double4* __restrict__ acc, size_t n, double g,
                              double* __restrict__ ax, double* __restrict__ ay,
                              double* __restrict__ az, double* __restrict__ vx,
                              double* __restrict__ vy, double* __restrict__ vz, double h, Tree t,
                              unsigned long long* counters, unsigned long long* stamp) {
  stamp_start(stamp);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[2] = t.offset[t.n];
    counters[3] = t.leaves[0];
    counters[4] = (unsigned long long)t.height[0];
  }
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const double4 a = acc[i];
    const double gx = g * a.x, gy = g * a.y, gz = g * a.z;
    ax[i] = gx;
    ay[i] = gy;
    az[i] = gz;
    if (KICK) {
      vx[i] = __dadd_rn(vx[i], __dmul_rn(gx, h));
      vy[i] = __dadd_rn(vy[i], __dmul_rn(gy, h));
      vz[i] = __dadd_rn(vz[i], __dmul_rn(gz, h));
    }
  }
  if (stamp != nullptr && threadIdx.x == 0)  // the last block's end is the evaluation's
    atomicMax(stamp + (NBSP_BH_END - NBSP_BH_INTEGRATE), gpu_clock());
}

// ---------------------------------------------------------------------------
// tree
// ---------------------------------------------------------------------------

// Common prefix length of sorted keys i and j in bits (Karras 2012, with the
// index as tie breaker); -1 outside [0, n).
__device__ __forceinline__ int prefix(const uint64_t* __restrict__ keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const uint64_t a = keys[i], b = keys[j];
  if (a != b) return __clzll(a ^ b) - 1;  // keys use the low 63 bits
  return 63 + __clz((unsigned)(i ^ j));
}

__device__ __forceinline__ int level_of_delta(int delta) { return min(delta / 3, 21); }

// Karras's radix tree over the sorted keys, and which of its nodes are octree
// cells: an internal node whose octree level (prefix length / 3) is deeper
// than its parent's, the root, and a particle below a node above level 21.
// The parent's prefix length is that of the node's range extended by one key
// on the side with the longer common prefix, max(delta(first - 1, first),
// delta(last, last + 1)), so each thread decides its own node and its leaf
// children without reading another thread's results; on i's own side of the
// range that is the bound its search began with.  Thread i compares key i with
// key i + 1 in any case, so it also looks for shared positions.
// Bound by the searches' chains (about three binary searches over the node's
// size): a probe asks whether two keys share more than `bound` bits, which is one
// shift of their difference, not a count of leading zeros (build at 1M 110 -> 105
// us, at 10M 0.92 -> 0.88 ms).
__global__ void radix_tree_kernel(const uint64_t* __restrict__ keys,
                                  const uint32_t* __restrict__ perm, const double* __restrict__ x,
                                  const double* __restrict__ y, const double* __restrict__ z,
                                  Tree t, int* status, unsigned long long* stamp) {
  stamp_start(stamp);
  const int n = t.n;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  if (keys[i] == keys[i + 1]) flag_duplicates((size_t)i, keys, perm, x, y, z, (size_t)n, status);
  const uint64_t key = keys[i];
  // prefix(keys, n, i, j) > bound
  auto deeper = [&](int j, int bound) -> bool {
    if ((unsigned)j >= (unsigned)n) return false;
    if (bound > 62) return prefix(keys, n, i, j) > bound;  // equal keys, told apart by index
    return ((key ^ keys[j]) >> (62 - bound)) == 0;
  };
  const int after = prefix(keys, n, i, i + 1), before = prefix(keys, n, i, i - 1);
  const int d = after >= before ? 1 : -1;
  const int dmin = min(after, before);
  int lmax = 2;
  while (deeper(i + lmax * d, dmin)) lmax <<= 1;
  int l = 0;
  for (int step = lmax >> 1; step >= 1; step >>= 1)
    if (deeper(i + (l + step) * d, dmin)) l += step;
  const int j = i + l * d;
  const int dnode = prefix(keys, n, i, j);
  int s = 0;
  int div = 2;
  for (;;) {
    const int step = (l + div - 1) / div;
    if (deeper(i + (s + step) * d, dnode)) s += step;
    if (step <= 1) break;
    div <<= 1;
  }
  const int gamma = i + s * d + (d < 0 ? -1 : 0);
  const int first = min(i, j), last = max(i, j);
  if (first < 0 || last >= n || gamma < first || gamma >= last) {
    atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    return;
  }
  const int left = first == gamma ? (n - 1) + gamma : gamma;
  const int right = last == gamma + 1 ? (n - 1) + gamma + 1 : gamma + 1;
  t.range[i] = make_int2(first, last);
  t.child[i] = make_int2(left, right);
  const int lvl = level_of_delta(dnode);
  const int pdelta = max(dmin, prefix(keys, n, j, j + d));
  t.cell[i] = (i == 0 || level_of_delta(pdelta) < lvl) ? lvl : -1;
  if (left >= n - 1) t.cell[left] = lvl <= 20 ? 22 : -1;
  if (right >= n - 1) t.cell[right] = lvl <= 20 ? 22 : -1;
}


__device__ __forceinline__ int first_of(const Tree& t, int b) {
  return b < t.n - 1 ? t.range[b].x : b - (t.n - 1);
}
__device__ __forceinline__ int last_of(const Tree& t, int b) {
  return b < t.n - 1 ? t.range[b].y : b - (t.n - 1);
}

// A splitting cell: an octree cell (binary node b with cell level >= 0) of
// more than leaf_capacity particles above level 21 — an internal node of the
// bucketed octree, whose octree children are all kept.  (A cell is kept when
// its octree parent splits; the root always is.)
__device__ __forceinline__ bool splits(const Tree& t, int b, int leaf_capacity) {
  if (b >= t.n - 1) return false;  // a particle
  const int cell = t.cell[b];
  if (cell < 0 || (cell & 31) >= 21) return false;
  const int2 r = t.range[b];
  return r.y - r.x + 1 > leaf_capacity;
}

// The octree children of splitting cell b, in Morton order: the cells met
// first below b in the binary tree, at most three binary levels down.  The
// eight slots are the binary paths; a node that is no cell (it has b's own
// level) makes room for its two children.  Cell marks, children and ranges of
// a level's nodes are loaded together, so the descent waits for three loads.
// first[k] is the first particle of children[k]; returns how many there are.
__device__ __forceinline__ int octree_children(const Tree& t, int b, int (&children)[8],
                                               int (&first)[8], int* status) {
  const int n = t.n;
  int slot[8], begin[8];
  const int2 c0 = t.child[b];
#pragma unroll
  for (int q = 0; q < 8; ++q) slot[q] = q == 0 ? c0.x : q == 4 ? c0.y : -1;
  bool bad = false;
#pragma unroll
  for (int stride = 4; stride >= 1; stride >>= 1) {
    int mark[8];
    int2 below[8];
#pragma unroll
    for (int q = 0; q < 8; q += stride) {
      const int c = slot[q];
      const bool there = c >= 0 && c < 2 * n - 1, inner = there && c < n - 1;
      bad |= c >= 2 * n - 1;
      mark[q] = there ? t.cell[c] : 0;
      below[q] = inner && stride > 1 ? t.child[c] : make_int2(-1, -1);
      begin[q] = inner ? t.range[c].x : c - (n - 1);
    }
#pragma unroll
    for (int q = 0; q < 8; q += stride) {
      if (mark[q] >= 0) continue;
      // a particle that is no cell, or a descent deeper than one octree level
      bad |= below[q].x < 0;
      slot[q] = below[q].x;
      if (stride > 1) slot[q + stride / 2] = below[q].y;
    }
  }
  int kids = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (slot[q] < 0) continue;
    bad |= begin[q] < 0 || begin[q] >= n;
#pragma unroll
    for (int k = 0; k <= q; ++k)
      if (k == kids) {
        children[k] = slot[q];
        first[k] = begin[q];
      }
    ++kids;
  }
  if (bad) {
    atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    return 0;
  }
  return kids;
}

// Octree level of cell node b, and its place among its octree siblings.
__device__ __forceinline__ int level_of(const Tree& t, int b) { return t.cell[b] & 31; }
__device__ __forceinline__ int sibling_of(const Tree& t, int b) { return t.cell[b] >> 5; }

// The kept cells, marked in mask[first particle] at their level (the depth-
// first numbering counts them): the root, and the octree children of every
// splitting cell, found by one thread per splitting cell, which also records
// itself as their octree parent and takes consecutive walk ids for them.  A
// block looks at kKeepNodes internal binary nodes and gathers the splitting ones
// (~N / leaf capacity of them) in shared memory first, so that their descents —
// chains of dependent loads — run side by side in whole warps; a descent per
// thread where it was found left one or two lanes of each warp working.  One
// atomic per block takes its places in the list of splitting cells and its walk
// ids (the order of blocks decides where records lie, nothing else).
// (keep and place, which takes a thread per child: 81 -> 41 us at 1M, 29 -> 20 us at 20k.)
constexpr int kKeepThreads = 256;
constexpr int kKeepNodes = 1024;
__global__ void __launch_bounds__(kKeepThreads) keep_kernel(Tree t, int leaf_capacity, int* status) {
  __shared__ int s_b[kKeepNodes];
  __shared__ int s_child[kKeepNodes * 8];
  __shared__ int warp_kids[kKeepThreads / 32];
  __shared__ int s_count;
  __shared__ unsigned long long s_base;
  const int n = t.n;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) s_count = 0;
  __syncthreads();
  if (blockIdx.x == 0 && tid == 0) {
    t.oparent[0] = -1;
    if (t.cell[0] < 0) {
      atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    } else {
      atomicOr(&t.mask[0], 1u << t.cell[0]);
    }
  }
#pragma unroll
  for (int i = 0; i < kKeepNodes / kKeepThreads; ++i) {
    const int b = blockIdx.x * kKeepNodes + i * kKeepThreads + tid;
    const bool split = b < n - 1 && splits(t, b, leaf_capacity);
    const unsigned m = __ballot_sync(kFull, split);
    int at = 0;
    if (lane == 0 && m != 0u) at = atomicAdd(&s_count, __popc(m));
    at = __shfl_sync(kFull, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (split) s_b[at] = b;
  }
  __syncthreads();
  const int count = s_count;
  int own = 0;
  for (int e = tid; e < count; e += kKeepThreads) {
    const int b = s_b[e];
    int child[8], begin[8];
    const int kids = octree_children(t, b, child, begin, status);
    own += kids;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      s_child[8 * e + k] = k < kids ? child[k] : -1;
      if (k < kids) {
        const int lvl = level_of(t, child[k]);
        t.oparent[child[k]] = b;
        t.cell[child[k]] = lvl + 32 * k;
        atomicOr(&t.mask[begin[k]], 1u << lvl);
      }
    }
  }
  int incl = own;
  for (int off = 1; off < 32; off <<= 1) {
    const int u = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += u;
  }
  if (lane == 31) warp_kids[w] = incl;
  __syncthreads();
  if (tid == 0) {
    int total = 0;
#pragma unroll
    for (int q = 0; q < kKeepThreads / 32; ++q) {
      const int c = warp_kids[q];
      warp_kids[q] = total;
      total += c;
    }
    s_base = count > 0 ? atomicAdd(&t.leaves[1], (unsigned long long)count << 32 | (unsigned)total) : 0;
  }
  __syncthreads();
  int first = 1 + (int)(unsigned)s_base + warp_kids[w] + incl - own;
  const size_t slot = (size_t)(s_base >> 32);
  for (int e = tid; e < count; e += kKeepThreads) {
    int kids = 0;
    for (int k = 0; k < 8; ++k) kids += s_child[8 * e + k] >= 0;
    t.below[s_b[e]] = make_int2(first, kids);
    first += kids;
  }
  for (int e = tid; e < count; e += kKeepThreads) t.split[slot + e] = s_b[e];
  for (int e = tid; e < 8 * count; e += kKeepThreads) t.split_child[8 * slot + e] = s_child[e];
}
// Inclusive scan of v over a block of WARPS warps.
template <int WARPS>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t u = __shfl_up_sync(kFull, x, off);
    if (lane >= off) x += u;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    uint32_t y = lane < WARPS ? warp_sums[lane] : 0u;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_up_sync(kFull, y, off);
      if (lane >= off) y += u;
    }
    if (lane < WARPS) warp_sums[lane] = y;
  }
  __syncthreads();
  x += w > 0 ? warp_sums[w - 1] : 0u;
  __syncthreads();  // (warp_sums may be used again)
  return x;
}

// Exclusive scan of popc(mask[k]) into offset[0..n].  Up to NBSP_BH_SMALL_SORT
// particles in one kernel, whose blocks count what lies before them themselves
// (at most 24 sixteen-byte loads a thread); then block sums first, scanned by a
// kernel of their own only when they are many (at 1M 488).
__device__ __forceinline__ uint32_t popc4(uint4 m) {
  return __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
}

constexpr int kSmallScanThreads = 1024;
__global__ void __launch_bounds__(kSmallScanThreads) scan_small_kernel(Tree t) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t s_before;
  const int n = t.n, tid = threadIdx.x;
  const int base = blockIdx.x * kScanItems;
  const uint4* mask4 = reinterpret_cast<const uint4*>(t.mask);
  uint32_t before = 0;
#pragma unroll 8
  for (int q = tid; q < base / 4; q += kSmallScanThreads) before += popc4(mask4[q]);
  before = block_scan<32>(before, warp_sums);
  if (tid == kSmallScanThreads - 1) s_before = before;
  const int i0 = base + 2 * tid, i1 = i0 + 1;
  const uint32_t v0 = i0 < n ? __popc(t.mask[i0]) : 0u, v1 = i1 < n ? __popc(t.mask[i1]) : 0u;
  const uint32_t incl = block_scan<32>(v0 + v1, warp_sums) + s_before;
  if (i0 < n) t.offset[i0] = incl - v0 - v1;
  if (i1 < n) t.offset[i1] = incl - v1;
  if (base + kScanItems >= n && tid == kSmallScanThreads - 1) t.offset[n] = incl;
}

constexpr int kScanThreads = 256;
constexpr int kScanSums = 1024;  // block sums that every block adds up itself
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(Tree t) {
  __shared__ uint32_t warp_sums[32];
  const int n = t.n;
  const size_t base = (size_t)blockIdx.x * kScanItems;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems / kScanThreads; ++k) {
    const size_t i = base + k * kScanThreads + threadIdx.x;
    if (i < (size_t)n) s += __popc(t.mask[i]);
  }
  s = block_scan<kScanThreads / 32>(s, warp_sums);
  if (threadIdx.x == kScanThreads - 1) t.block_sums[blockIdx.x] = s;
}

// Exclusive scan of the block sums in place (one block of 1024 threads, in
// chunks of 1024).
__global__ void __launch_bounds__(1024) scan_blocks_kernel(Tree t, int blocks) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < blocks; base += 1024) {
    const int b = base + threadIdx.x;
    const uint32_t v = b < blocks ? t.block_sums[b] : 0u;
    const uint32_t incl = block_scan<32>(v, warp_sums);
    const uint32_t c = carry;
    if (b < blocks) t.block_sums[b] = c + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = c + incl;
    __syncthreads();
  }
}

// SCANNED: the block sums hold what lies before each block.
template <bool SCANNED>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(Tree t) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t s_before;
  const int n = t.n, tid = threadIdx.x;
  if (SCANNED) {
    if (tid == 0) s_before = t.block_sums[blockIdx.x];
  } else {
    uint32_t before = 0;
#pragma unroll
    for (int k = 0; k < kScanSums / kScanThreads; ++k) {
      const unsigned b = k * kScanThreads + tid;
      if (b < blockIdx.x) before += t.block_sums[b];
    }
    before = block_scan<kScanThreads / 32>(before, warp_sums);
    if (tid == kScanThreads - 1) s_before = before;
  }
  const size_t base = (size_t)blockIdx.x * kScanItems;
  constexpr int per = kScanItems / kScanThreads;  // 8 contiguous items per thread
  uint32_t v[per];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < per; ++k) {
    const size_t i = base + (size_t)tid * per + k;
    v[k] = i < (size_t)n ? __popc(t.mask[i]) : 0u;
    s += v[k];
  }
  const uint32_t incl = block_scan<kScanThreads / 32>(s, warp_sums) + s_before;
  uint32_t run = incl - s;
#pragma unroll
  for (int k = 0; k < per; ++k) {
    const size_t i = base + (size_t)tid * per + k;
    if (i < (size_t)n) t.offset[i] = run;
    run += v[k];
  }
  if (base + kScanItems >= (size_t)n && tid == kScanThreads - 1) t.offset[n] = incl;
}

__device__ __forceinline__ int dfs_index(const Tree& t, int begin, int lvl) {
  return (int)(t.offset[begin] + __popc(t.mask[begin] & ((1u << lvl) - 1u)));
}

// The records of kept cell b, walk id `w` under parent `pw` (-1: the root):
// skip link (the first node after its subtree), first particle and particle
// count; a bucket's count is its particles, an internal node's is minus its
// children.
__device__ __forceinline__ void write_node(const Tree& t, int b, int w, int pw, bool leaf,
                                           int total, int* status) {
  const int begin = first_of(t, b), end = last_of(t, b) + 1;
  const int lvl = level_of(t, b);
  const int node = dfs_index(t, begin, lvl);
  int2 below = make_int2(begin, end - begin);
  if (!leaf) {
    below = t.below[b];
    below.y = -below.y;
  }
  if (node < 0 || node >= total || w < 0 || w >= total) {
    atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    return;
  }
  const int next = end >= t.n ? total : (int)t.offset[end];
  t.info[node] = make_int4(next, begin, leaf ? end - begin : 0, w);
  t.link[w] = make_int4(pw, below.x, below.y, node);
  t.level[w] = lvl;
  t.arrive[w] = 0;
  t.height[w] = 1;
}

// Octree records: eight threads per splitting cell, each writing one child's
// (whose parent's walk id is its place among its own parent's children); the
// root's by the first thread.
constexpr int kPlaceBlocks = 8 * 148;
__global__ void __launch_bounds__(256) place_kernel(Tree t, int leaf_capacity, int* status) {
  const int n = t.n;
  const int total = (int)t.offset[n];
  const unsigned long long made = t.leaves[1];
  const int splitting = (int)(made >> 32);
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  if (total < 1 || total > 2 * n - 1 || total != 1 + (int)(unsigned)made || splitting > n - 1) {
    if (thread == 0) atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
    return;
  }
  int leaves = 0;
  if (thread == 0) {  // the root may be the only node: one bucket
    write_node(t, 0, 0, -1, splitting == 0, total, status);
    leaves = splitting == 0;
  }
  for (long long q = thread; q < 8ll * splitting; q += (long long)gridDim.x * blockDim.x) {
    const int b = t.split[q >> 3], c = t.split_child[q];
    if (c < 0) continue;
    if (b < 0 || b >= n - 1 || c >= 2 * n - 1) {
      atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      continue;
    }
    int w = 0;
    if (b != 0) {
      const int p = t.oparent[b];  // keep_kernel: the splitting cell that found b
      w = p >= 0 && p < n - 1 ? t.below[p].x + sibling_of(t, b) : -1;
      if (w < 1 || w >= total) {
        atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
        continue;
      }
    }
    const bool leaf = !splits(t, c, leaf_capacity);
    write_node(t, c, t.below[b].x + sibling_of(t, c), w, leaf, total, status);
    leaves += leaf;
  }
  leaves = (int)__reduce_add_sync(kFull, (unsigned)leaves);
  if ((threadIdx.x & 31) == 0 && leaves > 0) atomicAdd(t.leaves, (unsigned long long)leaves);
}

// Trace-free quadrupole accumulation helpers (FP64).
struct Moments {
  double m, cx, cy, cz;
  double q[6];  // xx xy xz yy yz zz
  double t2;    // sum m |x - com|^2
};

// Inverse of spread3: bits 0, 3, 6, ... of v gathered into the low 21 bits.
__device__ __forceinline__ uint32_t compact3(uint64_t v) {
  v &= 0x1249249249249249ull;
  v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
  v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
  v = (v ^ (v >> 8)) & 0x001f0000ff0000ffull;
  v = (v ^ (v >> 16)) & 0x001f00000000ffffull;
  v = (v ^ (v >> 32)) & 0x1fffffull;
  return (uint32_t)v;
}

// What the opening test of every node is built from.
struct Opening {
  const uint64_t* keys;  // sorted Morton keys (a node's first key names its cell)
  const double* geometry;
  double inv_theta, inv_theta2;
  // relative opening test on: a state without previous accelerations (rms
  // |a_old| in geometry[7] zero or not finite) is opened at the start angle
  double start_inv_theta, start_inv_theta2;
  int relative;
  int criterion;         // NBSP_BH_OPENING_*
};

// The same once a thread has read the geometry: the climb's acquires would have
// every node read it again.
struct OpeningTerms {
  double root_side;
  double it, it2;  // 1 / theta and its square, at the angle in force
};
__device__ __forceinline__ OpeningTerms opening_terms(const Opening& o) {
  // Without previous accelerations every target's relative test passes (its
  // tolerance is +inf), so the geometric test alone decides: at the start
  // angle, not at the loose bound the relative test runs under.
  const double a_rms = o.geometry[7];
  const bool start = o.relative && !(a_rms > 0.0 && a_rms < INFINITY);
  return {2.0 * o.geometry[3], start ? o.start_inv_theta : o.inv_theta,
          start ? o.start_inv_theta2 : o.inv_theta2};
}

// The records of node `w` from its moments; `first` and `count` as its link has
// them, `particle` its first particle.
template <bool QUAD>
__device__ __forceinline__ void finish_node(const Tree& t, int w, const Moments& mo, int first,
                                            int count, int dfs, int particle, int lvl,
                                            const Opening& o, const OpeningTerms& terms) {
  t.mom[w] = make_double4(mo.m, mo.cx, mo.cy, mo.cz);
  // cell side 2h = root side / 2^lvl
  const int l = min(lvl, 21);
  const double side = terms.root_side * __hiloint2double((1023 - l) << 20, 0);
  double shift = 0.0;
  if (o.criterion == NBSP_BH_OPENING_OFFSET) {
    const double half = o.geometry[3];
    // the cell's centre from the first key's top 3 lvl bits, in the particles'
    // frame (relative to the centre of mass)
    const uint64_t key = o.keys[particle];
    double shift2 = 0.0;
    for (int a = 0; a < 3; ++a) {
      const double lo = o.geometry[a] - half - o.geometry[4 + a];
      const double centre = lo + ((double)(compact3(key >> a) >> (21 - l)) + 0.5) * side;
      const double d = (a == 0 ? mo.cx : a == 1 ? mo.cy : mo.cz) - centre;
      shift2 += d * d;
    }
    shift = sqrt(shift2);
  }
  // reference: accept when (2h)^2 < theta^2 d^2; offset: when 2h / theta + shift < d
  const double r2 = o.criterion == NBSP_BH_OPENING_OFFSET
                        ? (side * terms.it + shift) * (side * terms.it + shift)
                        : side * side * terms.it2;
  const float4 a = make_float4((float)mo.cx, (float)mo.cy, (float)mo.cz, (float)mo.m);
  const float4 b = make_float4((float)r2, (float)(mo.m * side * side), __int_as_float(first),
                               __int_as_float(count));
  t.wnode[2 * w] = a;
  t.wnode[2 * w + 1] = b;
  t.dnode[2 * dfs] = a;
  t.dnode[2 * dfs + 1] = b;
  if (QUAD) {
    for (int k = 0; k < 6; ++k) t.quad64[6 * w + k] = mo.q[k];
    t.trace64[w] = mo.t2;
    t.wquad[2 * w] = make_float4((float)mo.q[0], (float)mo.q[1], (float)mo.q[2], (float)mo.q[3]);
    t.wquad[2 * w + 1] =
        make_float4((float)mo.q[4], (float)side,
                    mo.m > 0.0 ? (float)(mo.t2 / (mo.m * side * side)) : 0.f, (float)shift);
  }
}

constexpr size_t kMomentsWide = 1500000;  // particles from which occupancy counts

// L2-coherent load of a double4 written by another thread of this grid.
__device__ __forceinline__ double4 ldcg_d4(const double4* p) {
  const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// Arrival at a parent: a release (this thread's node records are visible
// before the increment) and an acquire (the last child to arrive sees every
// sibling's records) in one atomic, instead of two full fences around it.
__device__ __forceinline__ int arrive_acq_rel(int* p) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
  return old;
}

// Bottom-up moments: leaves sum their particles, the last child to finish
// combines its parent, whose children are consecutive and in Morton order, so
// the combine's sums run in a fixed order and the result is deterministic.
// QUAD: also the trace-free quadrupoles and the spread (the quadrupole walk,
// the correction's features); the monopole walk reads neither.
// Bound by the latency of the climb: per level one atomic, then the children's
// moments.  The parent's link does not depend on the arrival, so it is loaded
// beside the atomic (and the grandparent's beside the moments); with lists of
// children and per-node arrays the climb waited for two more loads a level.
// Every acquire makes what a thread reads afterwards come from L2 again, so the
// opening terms are read once before the climb and nothing is spilled in it:
// 37 -> 25 us at 10k particles, 49 -> 31 at 150k.  From kMomentsWide particles
// on the leaves' loads are the larger part and the monopole pass runs 6 blocks
// per SM (40 registers, a few spilled): 152 -> 123 us at 4M, but 55 -> 61 at 1M;
// the quadrupole pass would spill hundreds of bytes per thread at 40 or 64.
template <bool QUAD, int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS) moments_kernel(const float4* __restrict__ pos, Tree t,
                                                              Opening open, int* status,
                                                              unsigned long long* stamp) {
  stamp_start(stamp);
  const int total = (int)t.offset[t.n];
  const OpeningTerms terms = opening_terms(open);
  for (int node = blockIdx.x * blockDim.x + threadIdx.x; node < total;
       node += gridDim.x * blockDim.x) {
    const int4 info = t.link[node];
    if (info.z < 0) continue;  // internal nodes are finished by their last child
    if (info.z == 0 || info.y < 0 || info.y + info.z > t.n || info.w < 0 || info.w >= total) {
      atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      continue;
    }
    int parent = info.x;
    int4 up = parent >= 0 && parent < total ? t.link[parent] : make_int4(-1, 0, 0, 0);
    Moments mo;
    {
      double m = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
      // eight particles' loads in flight at once (padding adds exact zeros, so
      // the sums are those of the plain sequential loop)
      const int end = info.y + info.z;
      for (int j0 = info.y; j0 < end; j0 += 8) {
        float4 q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          q[k] = j0 + k < end ? pos[j0 + k] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          m += (double)q[k].w;
          sx += (double)q[k].w * (double)q[k].x;
          sy += (double)q[k].w * (double)q[k].y;
          sz += (double)q[k].w * (double)q[k].z;
        }
      }
      mo.m = m;
      mo.cx = m != 0.0 ? sx / m : (double)pos[info.y].x;
      mo.cy = m != 0.0 ? sy / m : (double)pos[info.y].y;
      mo.cz = m != 0.0 ? sz / m : (double)pos[info.y].z;
      for (int k = 0; k < 6; ++k) mo.q[k] = 0.0;
      mo.t2 = 0.0;
#pragma unroll 4
      for (int j = info.y; QUAD && j < info.y + info.z; ++j) {
        const float4 p = pos[j];
        const double dx = (double)p.x - mo.cx, dy = (double)p.y - mo.cy, dz = (double)p.z - mo.cz;
        const double r2 = dx * dx + dy * dy + dz * dz;
        const double w = (double)p.w;
        mo.t2 += w * r2;
        mo.q[0] += w * (3.0 * dx * dx - r2);
        mo.q[1] += w * (3.0 * dx * dy);
        mo.q[2] += w * (3.0 * dx * dz);
        mo.q[3] += w * (3.0 * dy * dy - r2);
        mo.q[4] += w * (3.0 * dy * dz);
        mo.q[5] += w * (3.0 * dz * dz - r2);
      }
    }
    const int particle = info.y;
    finish_node<QUAD>(t, node, mo, info.y, info.z, info.w, particle, t.level[node], open, terms);
    for (int climb = 0; parent >= 0; ++climb) {
      const int nc = -up.z, first = up.y;
      if (climb > 64 || parent >= total || nc < 1 || nc > 8 || first < 1 ||
          first + nc > total || up.w < 0 || up.w >= total) {  // octree depth <= 23 levels
        atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
        break;
      }
      const int level = t.level[parent];
      if (arrive_acq_rel(&t.arrive[parent]) != nc - 1) break;
      const int4 next = up.x >= 0 && up.x < total ? t.link[up.x] : make_int4(-1, 0, 0, 0);
      double4 cm[8];
      int hmax = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        cm[k] = make_double4(0.0, 0.0, 0.0, 0.0);
        if (k < nc) {
          cm[k] = ldcg_d4(&t.mom[first + k]);
          hmax = max(hmax, __ldcg(&t.height[first + k]));
        }
      }
      double m = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k < nc) {
          m += cm[k].x;
          sx += cm[k].x * cm[k].y;
          sy += cm[k].x * cm[k].z;
          sz += cm[k].x * cm[k].w;
        }
      }
      Moments pm;
      pm.m = m;
      pm.cx = m != 0.0 ? sx / m : 0.0;
      pm.cy = m != 0.0 ? sy / m : 0.0;
      pm.cz = m != 0.0 ? sz / m : 0.0;
      for (int k = 0; k < 6; ++k) pm.q[k] = 0.0;
      pm.t2 = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (QUAD && k < nc) {
          const int c = first + k;
          const double dx = cm[k].y - pm.cx, dy = cm[k].z - pm.cy, dz = cm[k].w - pm.cz;
          const double r2 = dx * dx + dy * dy + dz * dz;
          const double w = cm[k].x;
          pm.t2 += __ldcg(&t.trace64[c]) + w * r2;
          pm.q[0] += __ldcg(&t.quad64[6 * c + 0]) + w * (3.0 * dx * dx - r2);
          pm.q[1] += __ldcg(&t.quad64[6 * c + 1]) + w * (3.0 * dx * dy);
          pm.q[2] += __ldcg(&t.quad64[6 * c + 2]) + w * (3.0 * dx * dz);
          pm.q[3] += __ldcg(&t.quad64[6 * c + 3]) + w * (3.0 * dy * dy - r2);
          pm.q[4] += __ldcg(&t.quad64[6 * c + 4]) + w * (3.0 * dy * dz);
          pm.q[5] += __ldcg(&t.quad64[6 * c + 5]) + w * (3.0 * dz * dz - r2);
        }
      }
      t.height[parent] = hmax + 1;
      // (the particle that names the cell's corner: any of the node's will do,
      // its key's top bits are the cell's)
      finish_node<QUAD>(t, parent, pm, first, -nc, up.w, particle, level, open, terms);
      parent = up.x;
      up = next;
    }
  }
}

__device__ __forceinline__ float rsqrt_mufu(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void fold(float& hi, float& lo, float a) {
  const float s = __fadd_rn(hi, a);
  const float bp = __fsub_rn(s, hi);
  const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(a, bp));
  hi = s;
  lo = __fadd_rn(lo, err);
}

constexpr int kWalkThreads = 256;

// Warp-cooperative stackless walk: the 32 lanes own 32 Morton-consecutive
// targets and visit the same node sequence; a cell is opened when any lane's
// opening test fails (so every lane's own test holds for every cell it
// accepts), otherwise all lanes apply its multipole and skip its subtree.
// Buckets (leaves of up to leaf_capacity particles) take the same test and are
// summed particle by particle when it fails; single particles are always exact.
// Opening test of a (node, target) pair at squared distance d2 from the node's
// centre of mass: the geometric test (d2 > ro, ro = the node's opening radius
// squared) and, with REL, the relative test G M side^2 / d^4 <= alpha |a_old|,
// i.e. M side^2 <= tol d^4 with tol = alpha |a_old| / G per target (Springel
// 2001); tol = +inf (no previous acceleration) leaves the geometric test.
template <bool REL>
__device__ __forceinline__ bool opening_passes(float d2, float ro, float km, float tol) {
  return d2 > ro && (!REL || d2 * d2 * tol >= km);
}

struct WalkAcc {
  float hx, hy, hz, lx, ly, lz;  // compensated acceleration / G
  unsigned approx, exact;        // accepted cells, particle-particle terms
};

template <int ORDER, bool REL>
__device__ __forceinline__ void stackless_walk(const float4* __restrict__ pos, int n,
                                               const Tree& t, float eps2, int s, bool active,
                                               float4 p, float tol, int lane, int* status,
                                               WalkAcc& out) {
  const int total = (int)t.offset[n];
  const int limit = 2 * total + 64;

  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  float px = 0.f, py = 0.f, pz = 0.f;
  int pending = 0;
  unsigned approx = 0, exact = 0;
  int node = 0, steps = 0;
  while ((unsigned)node < (unsigned)total) {
    if (++steps > limit) {
      if (lane == 0) atomicOr(status, NBSP_DEVICE_ERROR_WALK_LIMIT);
      break;
    }
    const int4 info = t.info[node];
    if (info.z < 0 || info.y < 0 || info.y + info.z > n || info.x <= node || info.w < 0 ||
        info.w >= total) {
      if (lane == 0) atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      break;
    }
    // A bucket of >= 2 particles is a cell like any other: its multipole is
    // used when every lane's opening test passes (barnes_hut.c:596-599).
    bool direct = info.z == 1;
    if (info.z >= 2) {
      const float4 c = t.dnode[2 * node], o = t.dnode[2 * node + 1];
      const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      direct = __any_sync(kFull, active && !opening_passes<REL>(d2, o.x, o.y, tol));
    }
    if (direct) {
      const int j1 = info.y + info.z;
      for (int j = info.y; j < j1; ++j) {
        const float4 q = pos[j];
        const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
        const float rinv = j == s ? 0.f : rsqrt_mufu(r2);  // barnes_hut.c:572
        const float w = q.w * (rinv * rinv * rinv);
        px = fmaf(w, dx, px);
        py = fmaf(w, dy, py);
        pz = fmaf(w, dz, pz);
      }
      exact += active ? (unsigned)(info.z - ((s >= info.y && s < j1) ? 1 : 0)) : 0u;
      pending += info.z;
      node = info.x;
    } else {
      const float4 c = t.dnode[2 * node], o = t.dnode[2 * node + 1];
      const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const bool open = active && !opening_passes<REL>(d2, o.x, o.y, tol);
      if (__any_sync(kFull, open)) {
        node = node + 1;
        continue;
      }
      const float r2 = d2 + eps2;
      const float rinv = rsqrt_mufu(r2);
      const float rinv2 = rinv * rinv;
      const float rinv3 = rinv * rinv2;
      float w = c.w * rinv3;
      if (ORDER == 2) {
        const float4 qa = t.wquad[2 * info.w];
        const float qyz = t.wquad[2 * info.w + 1].x;
        const float qzz = -qa.x - qa.w;
        // Q d and d.Q.d, d = com - target
        const float qdx = fmaf(qa.x, dx, fmaf(qa.y, dy, qa.z * dz));
        const float qdy = fmaf(qa.y, dx, fmaf(qa.w, dy, qyz * dz));
        const float qdz = fmaf(qa.z, dx, fmaf(qyz, dy, qzz * dz));
        const float dqd = fmaf(dx, qdx, fmaf(dy, qdy, dz * qdz));
        const float rinv5 = rinv3 * rinv2;
        const float rinv7 = rinv5 * rinv2;
        // a = G [ M d / r^3 - Q d / r^5 + 5/2 (d.Q.d) d / r^7 ]
        w = fmaf(2.5f * dqd, rinv7, w);
        px = fmaf(-qdx, rinv5, px);
        py = fmaf(-qdy, rinv5, py);
        pz = fmaf(-qdz, rinv5, pz);
      }
      px = fmaf(w, dx, px);
      py = fmaf(w, dy, py);
      pz = fmaf(w, dz, pz);
      approx += active ? 1u : 0u;
      pending += 1;
      node = info.x;
    }
    if (pending >= 32) {
      fold(hx, lx, px);
      fold(hy, ly, py);
      fold(hz, lz, pz);
      px = py = pz = 0.f;
      pending = 0;
    }
  }
  fold(hx, lx, px);
  fold(hy, ly, py);
  fold(hz, lz, pz);
  out.hx = hx;
  out.hy = hy;
  out.hz = hz;
  out.lx = lx;
  out.ly = ly;
  out.lz = lz;
  out.approx = approx;
  out.exact = exact;
}

// The compensated (hi, lo) sums combined in FP64, stored at the target's input
// index perm[s]: one aligned 32-byte record per target, so the scattered store
// writes whole sectors and the pass that scales them into the state's arrays is
// coalesced.
__device__ __forceinline__ void store_walk(const WalkAcc& a, int s, bool active, int lane,
                                           const uint32_t* __restrict__ perm, int n,
                                           double4* __restrict__ acc,
                                           unsigned long long* __restrict__ counters) {
  if (active) {
    const uint32_t i = perm[s];
    if (i < (uint32_t)n)  // (a bad permutation is flagged by the gather)
      acc[i] = make_double4((double)a.hx + (double)a.lx, (double)a.hy + (double)a.ly,
                            (double)a.hz + (double)a.lz, 0.0);
  }
  unsigned long long ap = a.approx, ex = a.exact;
  for (int off = 16; off > 0; off >>= 1) {
    ap += __shfl_down_sync(kFull, ap, off);
    ex += __shfl_down_sync(kFull, ex, off);
  }
  if (lane == 0) {
    atomicAdd(&counters[0], ap);
    atomicAdd(&counters[1], ex);
  }
}

template <int ORDER, bool REL>
__global__ void __launch_bounds__(kWalkThreads) walk_kernel(
    const float4* __restrict__ pos, const float* __restrict__ tol, int n, Tree t, float eps2,
    const uint32_t* __restrict__ perm, double4* __restrict__ acc,
    unsigned long long* __restrict__ counters, int* status, unsigned long long* stamp) {
  stamp_start(stamp);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kWalkThreads + threadIdx.x) >> 5;
  if (warp * 32 >= n) return;
  const int s = warp * 32 + lane;
  const bool active = s < n;
  const float4 p = pos[active ? s : n - 1];
  const float tl = REL ? tol[active ? s : n - 1] : 0.f;
  WalkAcc a;
  stackless_walk<ORDER, REL>(pos, n, t, eps2, s, active, p, tl, lane, status, a);
  store_walk(a, s, active, lane, perm, n, acc, counters);
}

// Point sources (bucket particles and monopole cells) gathered per warp in
// shared memory, interleaved by pairs so that one 16-byte load yields the
// 64-bit operands {x_2i, x_2i+1} and {y_2i, y_2i+1} (resp. z and m) of the
// paired .f32x2 instructions.
constexpr int kStage = 64;              // sources per tile
constexpr float kFarAway = 1e30f;       // padding: r^2 overflows to inf, rsqrt(inf) = 0
struct SourceTile {
  ulonglong2 xy[kStage / 2];  // {x_2i, x_2i+1}, {y_2i, y_2i+1}
  ulonglong2 zm[kStage / 2];  // {z_2i, z_2i+1}, {m_2i, m_2i+1}
};

__device__ __forceinline__ void stage_source(SourceTile& s, int k, float4 q) {
  float* a = reinterpret_cast<float*>(&s.xy[k >> 1]) + (k & 1);
  float* b = reinterpret_cast<float*>(&s.zm[k >> 1]) + (k & 1);
  a[0] = q.x;
  a[2] = q.y;
  b[0] = q.z;
  b[2] = q.w;
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The kStage terms of a full tile on this lane's target, two sources per
// instruction (every lane reads the same words: shared-memory broadcasts),
// summed in FP32 and folded once.  The target's own entry, when staged, has
// d = 0 and r^2 = eps^2 exactly: it adds W * 0 = 0 while its weight W = m /
// eps^3 is finite (checked once per warp by self_term_is_finite); otherwise
// GUARD drops every term with r^2 <= eps^2 (barnes_hut.c:572 skips it).
template <bool GUARD>
__device__ __forceinline__ void source_terms(const SourceTile& s, float4 p, float eps2,
                                             unsigned long long& ax, unsigned long long& ay,
                                             unsigned long long& az) {
  const unsigned long long PX = pack2(p.x, p.x), PY = pack2(p.y, p.y), PZ = pack2(p.z, p.z);
  const unsigned long long E2 = pack2(eps2, eps2);
#pragma unroll
  for (int j = 0; j < kStage / 2; ++j) {
    const ulonglong2 a = s.xy[j], b = s.zm[j];
    const unsigned long long dx = sub2(a.x, PX), dy = sub2(a.y, PY), dz = sub2(b.x, PZ);
    const unsigned long long r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, E2)));
    float r2a, r2b;
    unpack2(r2, r2a, r2b);
    float ra = rsqrt_mufu(r2a), rb = rsqrt_mufu(r2b);
    if (GUARD) {
      ra = r2a > eps2 ? ra : 0.f;
      rb = r2b > eps2 ? rb : 0.f;
    }
    const unsigned long long R = pack2(ra, rb);
    const unsigned long long W = mul2(b.y, mul2(mul2(R, R), R));
    ax = fma2(W, dx, ax);
    ay = fma2(W, dy, ay);
    az = fma2(W, dz, az);
  }
}

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Accepted cells of the quadrupole walk, pair-interleaved like SourceTile:
// centre of mass, mass and the five independent trace-free components.
struct QuadTile {
  ulonglong2 xy[kStage / 2];         // {x}, {y}
  ulonglong2 zm[kStage / 2];         // {z}, {m}
  ulonglong2 qa[kStage / 2];         // {Qxx}, {Qxy}
  ulonglong2 qb[kStage / 2];         // {Qxz}, {Qyy}
  unsigned long long qc[kStage / 2];  // {Qyz}
};

// c = (com, mass); qa = (Qxx, Qxy, Qxz, Qyy); qyz = Qyz.
__device__ __forceinline__ void stage_cell(QuadTile& s, int k, float4 c, float4 qa, float qyz) {
  const int i = k >> 1, o = k & 1;
  float* a = reinterpret_cast<float*>(&s.xy[i]) + o;
  float* b = reinterpret_cast<float*>(&s.zm[i]) + o;
  float* e = reinterpret_cast<float*>(&s.qa[i]) + o;
  float* f = reinterpret_cast<float*>(&s.qb[i]) + o;
  a[0] = c.x;
  a[2] = c.y;
  b[0] = c.z;
  b[2] = c.w;
  e[0] = qa.x;
  e[2] = qa.y;
  f[0] = qa.z;
  f[2] = qa.w;
  reinterpret_cast<float*>(&s.qc[i])[o] = qyz;
}

// The kStage cell terms of a full QuadTile on this lane's target, two cells per
// instruction: a = G [ M d / r^3 - Q d / r^5 + 5/2 (d.Q.d) d / r^7 ],
// d = com - target, r^2 = d^2 + eps^2, Qzz = -Qxx - Qyy.  Padding cells
// (far away, massless, Q = 0) add exactly 0.
__device__ __forceinline__ void quad_tile(const QuadTile& s, float4 p, float eps2, float& hx,
                                          float& hy, float& hz, float& lx, float& ly, float& lz) {
  const unsigned long long PX = pack2(p.x, p.x), PY = pack2(p.y, p.y), PZ = pack2(p.z, p.z);
  const unsigned long long E2 = pack2(eps2, eps2), H = pack2(2.5f, 2.5f);
  const unsigned long long ZERO = 0ull;
  unsigned long long ax = 0ull, ay = 0ull, az = 0ull;
#pragma unroll 8
  for (int j = 0; j < kStage / 2; ++j) {
    const ulonglong2 a = s.xy[j], b = s.zm[j], qa = s.qa[j], qb = s.qb[j];
    const unsigned long long qyz = s.qc[j];
    const unsigned long long dx = sub2(a.x, PX), dy = sub2(a.y, PY), dz = sub2(b.x, PZ);
    const unsigned long long r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, E2)));
    float r2a, r2b;
    unpack2(r2, r2a, r2b);
    const unsigned long long R = pack2(rsqrt_mufu(r2a), rsqrt_mufu(r2b));
    const unsigned long long R2 = mul2(R, R);
    const unsigned long long R3 = mul2(R2, R);
    const unsigned long long R5 = mul2(R3, R2);
    const unsigned long long R7 = mul2(R5, R2);
    const unsigned long long qdx = fma2(qa.x, dx, fma2(qa.y, dy, mul2(qb.x, dz)));
    const unsigned long long qdy = fma2(qa.y, dx, fma2(qb.y, dy, mul2(qyz, dz)));
    const unsigned long long qdz =
        sub2(fma2(qb.x, dx, mul2(qyz, dy)), mul2(add2(qa.x, qb.y), dz));
    const unsigned long long dqd = fma2(dx, qdx, fma2(dy, qdy, mul2(dz, qdz)));
    const unsigned long long w = fma2(mul2(H, dqd), R7, mul2(b.y, R3));
    const unsigned long long nr5 = sub2(ZERO, R5);
    ax = fma2(qdx, nr5, fma2(w, dx, ax));
    ay = fma2(qdy, nr5, fma2(w, dy, ay));
    az = fma2(qdz, nr5, fma2(w, dz, az));
  }
  float u, v;
  unpack2(ax, u, v);
  fold(hx, lx, u);
  fold(hx, lx, v);
  unpack2(ay, u, v);
  fold(hy, ly, u);
  fold(hy, ly, v);
  unpack2(az, u, v);
  fold(hz, lz, u);
  fold(hz, lz, v);
}

// True when the target's own term in source_terms is W * 0 with W finite:
// eps^2 a normal number and m * rsqrt(eps^2)^3, in the same operation order,
// below overflow.
__device__ __forceinline__ bool self_term_is_finite(float m, float eps2) {
  if (!(eps2 >= 1.17549435e-38f)) return false;
  const float r = rsqrt_mufu(eps2);
  return isfinite(m * ((r * r) * r));
}

__device__ __forceinline__ void source_tile(const SourceTile& s, float4 p, float eps2, bool guard,
                                            float& hx, float& hy, float& hz, float& lx,
                                            float& ly, float& lz) {
  unsigned long long ax = 0ull, ay = 0ull, az = 0ull;  // {0.f, 0.f}
  if (guard) {
    source_terms<true>(s, p, eps2, ax, ay, az);
  } else {
    source_terms<false>(s, p, eps2, ax, ay, az);
  }
  float a, b;
  unpack2(ax, a, b);
  fold(hx, lx, a);
  fold(hx, lx, b);
  unpack2(ay, a, b);
  fold(hy, ly, a);
  fold(hy, ly, b);
  unpack2(az, a, b);
  fold(hz, lz, a);
  fold(hz, lz, b);
}

// ---------------------------------------------------------------------------
// learned far-field correction: features, training pairs, labels
// ---------------------------------------------------------------------------

// The 10 MLP inputs of cell `node` seen from point (tx, ty, tz) (coordinates
// relative to the system's centre of mass, like the node data):
//   f0..2 = (t - com) / side          f3 = side / |t - com|   (opening ratio)
//   f4..8 = trace-free Q / (M side^2): xx, xy, xz, yy, yz
//   f9    = sum m |x - com|^2 / (M side^2)
// false for a massless cell.
__device__ __forceinline__ bool features_of(float4 c, float s, float4 qa, float qyz,
                                            float spread, float tx, float ty, float tz,
                                            float* f) {
  if (!(c.w > 0.f) || !(s > 0.f)) return false;
  const float rx = tx - c.x, ry = ty - c.y, rz = tz - c.z;
  const float inv_s = 1.f / s;
  const float d = sqrtf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
  if (!(d > 0.f)) return false;
  f[0] = rx * inv_s;
  f[1] = ry * inv_s;
  f[2] = rz * inv_s;
  f[3] = s / d;
  const float qs = 1.f / (c.w * s * s);
  f[4] = qa.x * qs;
  f[5] = qa.y * qs;
  f[6] = qa.z * qs;
  f[7] = qa.w * qs;
  f[8] = qyz * qs;
  f[9] = spread;
  return true;
}

// the same for the node of walk id w
__device__ __forceinline__ bool cell_features(const Tree& t, int w, float4 c, float tx,
                                              float ty, float tz, float* f) {
  const float4 qb = t.wquad[2 * w + 1];
  return features_of(c, qb.y, t.wquad[2 * w], qb.x, qb.z, tx, ty, tz, f);
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// The corrected walk evaluates the network once per (cell, 32-target group) at
// the group centre, for cells whose distance from that centre exceeds the
// group radius / kCorrGroup.
constexpr float kCorrGroup = 0.3f;
// Training pairs are the accepted cells with side / distance >= kCorrNear x
// theta: the near cells, where the monopole's residual is largest.  The
// trained feature range then excludes the far cells, so the walk leaves them
// to the plain monopole (the fallback outside the training range); measured on
// the 1M collision at theta 1.0 this both cuts the network evaluations and
// lowers the rms error (7.7e-3 -> 5.6e-3 against 8.6e-3 uncorrected).
constexpr float kCorrNear = 0.7f;

// Training pairs: sample k picks a random target and, walking the tree with the
// opening criterion at theta_train, one of the cells that target accepts and
// its group would correct, uniformly (reservoir sampling).  Up to 8 targets
// are tried per sample.
__global__ void mlp_pairs_kernel(const float4* __restrict__ pos, int n, Tree t, float theta,
                                 int opening, unsigned long long seed, int samples, int* __restrict__ target,
                                 int* __restrict__ cell, int* status) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= samples) return;
  const int total = (int)t.offset[n];
  const float th2 = theta * theta;
  unsigned long long state = mix64(seed ^ (0x9E3779B97F4A7C15ull * (unsigned long long)(k + 1)));
  int chosen = -1, tgt = 0;
  for (int attempt = 0; attempt < 8 && chosen < 0; ++attempt) {
    state = mix64(state + 0x9E3779B97F4A7C15ull);
    tgt = (int)(state % (unsigned long long)n);
    const float4 p = pos[tgt];
    // the target's walk group (32 Morton-consecutive particles): only cells
    // the corrected walk would correct for this group are sampled
    const int g0 = tgt & ~31, g1 = min(g0 + 32, n);
    float bx0 = p.x, bx1 = p.x, by0 = p.y, by1 = p.y, bz0 = p.z, bz1 = p.z;
    for (int j = g0; j < g1; ++j) {
      const float4 q = pos[j];
      bx0 = fminf(bx0, q.x);
      bx1 = fmaxf(bx1, q.x);
      by0 = fminf(by0, q.y);
      by1 = fmaxf(by1, q.y);
      bz0 = fminf(bz0, q.z);
      bz1 = fmaxf(bz1, q.z);
    }
    const float gx = 0.5f * (bx0 + bx1), gy = 0.5f * (by0 + by1), gz = 0.5f * (bz0 + bz1);
    const float ex = 0.5f * (bx1 - bx0), ey = 0.5f * (by1 - by0), ez = 0.5f * (bz1 - bz0);
    const float rg2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
    unsigned count = 0;
    int node = 0, steps = 0;
    while ((unsigned)node < (unsigned)total) {
      if (++steps > total + 64) {
        atomicOr(status, NBSP_DEVICE_ERROR_WALK_LIMIT);
        break;
      }
      const int4 info = t.info[node];
      if (info.x <= node || info.z == 1) {  // single particles are always exact
        node = info.x > node ? info.x : total;
        continue;
      }
      const float4 c = t.dnode[2 * node];
      const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float4 qb = t.wquad[2 * info.w + 1];
      const float s = qb.y;
      const float ro = s / theta + qb.w;
      const bool pass = opening == NBSP_BH_OPENING_OFFSET ? d2 > ro * ro : s * s < th2 * d2;
      if (d2 > 0.f && pass && c.w > 0.f) {
        const float gdx = c.x - gx, gdy = c.y - gy, gdz = c.z - gz;
        const float near = kCorrNear * theta;
        if (kCorrGroup * kCorrGroup * fmaf(gdx, gdx, fmaf(gdy, gdy, gdz * gdz)) > rg2 &&
            s * s >= near * near * d2) {
          ++count;
          state = mix64(state + 0x9E3779B97F4A7C15ull);
          if (state % count == 0) chosen = node;
        }
        node = info.x;
      } else {
        node = info.z > 0 ? info.x : node + 1;  // a failing bucket is summed exactly
      }
    }
  }
  target[k] = tgt;
  cell[k] = chosen;
}

// Labels from exact cell sums (all-pairs arithmetic, gravity.c:46-61, FP32
// with compensated per-lane sums; target excluded): one warp per pair.
//   label = (a_exact - a_monopole) |d|^2 / M   (units of G; d = com - target)
__global__ void mlp_labels_kernel(const float4* __restrict__ pos, int n, Tree t,
                                  const int* __restrict__ target, const int* __restrict__ cell,
                                  int samples, float eps2, float* __restrict__ feat,
                                  float* __restrict__ lab, int* __restrict__ ok) {
  const int lane = threadIdx.x & 31;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= samples) return;
  const int node = cell[k], i = target[k];
  const int total = (int)t.offset[n];
  if (node < 0 || node >= total || i < 0 || i >= n) {
    if (lane == 0) ok[k] = 0;
    return;
  }
  const int4 info = t.info[node];
  const float4 p = pos[i];
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  // A node's particles: [its first particle, the first particle of the node
  // that follows its subtree) — or its own count for a leaf.
  const int first = info.y;
  const int end = info.z > 0 ? first + info.z : (info.x < total ? t.info[info.x].y : n);
  float px = 0.f, py = 0.f, pz = 0.f;
  int pending = 0;
  for (int j = first + lane; j < end; j += 32) {
    if (j == i) continue;
    const float4 q = pos[j];
    const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
    const float rinv = rsqrt_mufu(r2);
    const float w = q.w * (rinv * rinv * rinv);
    px = fmaf(w, dx, px);
    py = fmaf(w, dy, py);
    pz = fmaf(w, dz, pz);
    if (++pending == 32) {
      fold(hx, lx, px);
      fold(hy, ly, py);
      fold(hz, lz, pz);
      px = py = pz = 0.f;
      pending = 0;
    }
  }
  fold(hx, lx, px);
  fold(hy, ly, py);
  fold(hz, lz, pz);
  double ax = (double)hx + (double)lx, ay = (double)hy + (double)ly, az = (double)hz + (double)lz;
  for (int off = 16; off > 0; off >>= 1) {
    ax += __shfl_xor_sync(kFull, ax, off);
    ay += __shfl_xor_sync(kFull, ay, off);
    az += __shfl_xor_sync(kFull, az, off);
  }
  if (lane != 0) return;
  const float4 c = t.dnode[2 * node];
  float f[nbsp_mlp::kIn];
  if (!cell_features(t, info.w, c, p.x, p.y, p.z, f)) {
    ok[k] = 0;
    return;
  }
  const double dx = (double)c.x - p.x, dy = (double)c.y - p.y, dz = (double)c.z - p.z;
  const double d2 = dx * dx + dy * dy + dz * dz;
  const double r2 = d2 + (double)eps2;
  const double mono = (double)c.w / (r2 * sqrt(r2));
  const double scale = d2 / (double)c.w;
  for (int q = 0; q < nbsp_mlp::kIn; ++q) feat[(size_t)k * nbsp_mlp::kIn + q] = f[q];
  lab[(size_t)k * 3 + 0] = (float)((ax - mono * dx) * scale);
  lab[(size_t)k * 3 + 1] = (float)((ay - mono * dy) * scale);
  lab[(size_t)k * 3 + 2] = (float)((az - mono * dz) * scale);
  ok[k] = 1;
}

// Column statistics of the kept rows: mean, 1/std, min, max of the 10 features
// and mean, std of the 3 labels, into the network's scaling tables.
__global__ void mlp_stats_kernel(const float* __restrict__ feat, const float* __restrict__ lab,
                                 const int* __restrict__ ok, int rows, nbsp_mlp::Net* net) {
  __shared__ double sh[4][256];
  const int col = blockIdx.x;  // 0..9 features, 10..12 labels
  const float* src = col < nbsp_mlp::kIn ? feat : lab;
  const int stride = col < nbsp_mlp::kIn ? nbsp_mlp::kIn : 3;
  const int c = col < nbsp_mlp::kIn ? col : col - nbsp_mlp::kIn;
  double s = 0.0, s2 = 0.0, mn = 1e300, mx = -1e300, cnt = 0.0;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    if (ok != nullptr && !ok[r]) continue;
    const double v = src[(size_t)r * stride + c];
    s += v;
    s2 += v * v;
    mn = fmin(mn, v);
    mx = fmax(mx, v);
    cnt += 1.0;
  }
  sh[0][threadIdx.x] = s;
  sh[1][threadIdx.x] = s2;
  sh[2][threadIdx.x] = cnt;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st)
      for (int q = 0; q < 3; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + st];
    __syncthreads();
  }
  const double tot = sh[0][0], tot2 = sh[1][0], n = sh[2][0];
  __syncthreads();
  sh[0][threadIdx.x] = mn;
  sh[1][threadIdx.x] = mx;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      sh[0][threadIdx.x] = fmin(sh[0][threadIdx.x], sh[0][threadIdx.x + st]);
      sh[1][threadIdx.x] = fmax(sh[1][threadIdx.x], sh[1][threadIdx.x + st]);
    }
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  const double mean = n > 0 ? tot / n : 0.0;
  const double var = n > 1 ? fmax(tot2 / n - mean * mean, 0.0) : 1.0;
  const double sd = var > 1e-30 ? sqrt(var) : 1.0;
  if (col < nbsp_mlp::kIn) {
    net->x_mean[c] = (float)mean;
    net->x_inv_std[c] = (float)(1.0 / sd);
    net->x_min[c] = (float)sh[0][0];
    net->x_max[c] = (float)sh[1][0];
  } else {
    net->y_mean[c] = (float)mean;
    net->y_std[c] = (float)sd;
  }
}

constexpr int kListThreads = 128;  // 4 warps, one traversal group each
constexpr int kListCap = 64;       // cells / leaves gathered before a flush (>= 32 + 32)
constexpr int kListStack = 1024;   // node ids per warp (4 KiB); overflow -> stackless walk
// the relative-test walk's stack: 960 ids per warp, so that its block (with
// the tolerances' words, 24,064 B of shared memory) fits 9 times in an SM
constexpr int kListStackRel = 960;
// blocks per SM of the monopole list walks (at most 56 registers at 9): 9
// where shared memory allows (the plain and the corrected walk's block at
// 1024 ids is 24,576 B)
// LATENCY > 0: blocks per SM of the walk of small systems, whose warps have their
// schedulers nearly to themselves, so that what counts is the length of their own
// chains.  Four blocks while all fit at once (75,776 particles); then six
// (quadrupole four) up to kLatencyBlocks blocks, which is two (three) times what
// fits: walk at 113k 204 -> 180 us, 170k 284 -> 257, 200k 321 -> 293, the same at
// 300k; quadrupole at 76k 212 -> 191, 150k 363 -> 356, 300k 680 -> 684
constexpr unsigned kLatencyBlocks = 148 * 12;
template <int ORDER, int STACK, bool CORR, bool REL, bool SHARED, int LATENCY>
constexpr int list_walk_blocks() {
  return LATENCY > 0  ? LATENCY
         : ORDER != 1 ? 5
         : (!SHARED && (REL ? STACK == kListStackRel : true)) ? 9 : 8;
}
// LATENCY: pending nodes of a step beyond which each lane tests its own against
// the 32 targets, rather than the lanes their targets against one node after
// another: 32 independent tests take as long as four to eight of the others (turns
// of 3, 6, 10, 16: walk at 10k 59, 59, 64, 67 us; at 56 registers it spills)
constexpr int kProbeTurn = 4;
// SHARED walk: the block's top-of-tree traversal keeps its stack and frontier
// in the warps' stack space (it ends before any warp walks)
constexpr int kCtaStack = 2048;    // warps 0 and 1's stacks
constexpr int kFrontier = 384;     // the start of warp 2's stack
static_assert(kCtaStack + kFrontier <= 3 * kListStack, "frontier inside warp 2's stack");

// Interaction-list walk.  The 32 Morton-consecutive targets of a warp share a
// traversal.  Each step the lanes pop up to 32 nodes from the warp's
// shared-memory stack and test them IN PARALLEL: a node is accepted when every
// target's own reference test (2h)^2 < theta^2 d^2 holds (d to the cell's
// centre of mass) — first tried in one shot against the group's bounding box
// (if the box's nearest point passes, every target does), then against the
// lane's own target (fails: opened), else for each remaining node in turn by
// the 32 lanes testing their own targets at once — so the accepted cells are
// exactly those of the stackless walk.  An accepted monopole cell is written,
// from the registers of the lane that tested it, straight into a 64-source
// shared tile that every lane evaluates on its own target with paired f32x2
// arithmetic whenever it is full.  Buckets that must be summed exactly are
// listed (first particle, count); whenever 32 have gathered, their particles
// are gathered into the same tile, one slot per lane and all loads of a tile in
// flight together.
// A quadrupole cell goes into a QuadTile with its moments when it is accepted.
// A warp whose stack would overflow restarts with the stackless walk.
//
// CORR: the learned far-field correction, listed here and applied by the
// correction pipeline that runs after the walk (corr_rows_kernel on the
// tcgen05 tensor cores, then corr_apply_kernel).  An accepted monopole cell
// whose opening ratio side / |com - group centre| lies in the range the
// network saw in training, and that lies further than 1/kCorrGroup group radii
// from the group centre (so one evaluation there stands for all 32 targets),
// is appended to the group's list; the walk itself computes the plain
// monopole, exactly as without the correction.
// Register budgets: monopole walk 56 (9 blocks of 4 warps per SM; the shared-top
// walk and the corrected walk under the relative test 64, 8 blocks), quadrupole
// walk 96 (5 blocks); the latency forms 80 (6 blocks) and 119 to 125 (4 blocks).
//
// SHARED: the top of the tree is traversed once for the block's 4 groups.  The
// 128 threads test up to 128 nodes at a time against the 4 group boxes: a node
// every group's box test accepts is staged once for all four (into every
// warp's source tile); an internal node whose opening test fails for every
// target of every group (the box's farthest point fails) is opened once for
// all; any other node goes to a frontier that each warp then walks on its own
// exactly as above.  Every group accepts, opens and sums exactly the nodes it
// would alone (the same interactions; only the order of the FP32 sums moves).
// A block whose shared stack or frontier would overflow starts every group
// from the root instead.
//
// LATENCY (small systems): the same steps with registers to spare; the records of
// the next step's nodes are loaded before this step's tiles are evaluated, four
// nodes at a time take the per-target test, and when more are pending each lane
// tests its own node against all targets (groups on a system's outskirts have
// wide boxes that decide little, and their steps set the walk's time): walk 106
// -> 59 us at 10k, 107 -> 65 at 20k, 152 -> 115 at 65k.
template <int ORDER, int STACK, bool CORR, bool REL, bool SHARED = false, int LATENCY = 0>
__global__ void __launch_bounds__(kListThreads, (list_walk_blocks<ORDER, STACK, CORR, REL, SHARED, LATENCY>())) walk_lists_kernel(
    const float4* __restrict__ pos, const float* __restrict__ tol, int n, Tree t, float eps2,
    const uint32_t* __restrict__ perm, double4* __restrict__ acc,
    unsigned long long* __restrict__ counters, int* status,
    const nbsp_mlp::Net* __restrict__ net, NbspCorrectionLists lists,
    unsigned long long* stamp) {
  stamp_start(stamp);
  static_assert(!SHARED || (ORDER == 1 && !CORR && STACK == kListStack), "shared top: monopole walk");
  __shared__ int s_stack[kListThreads / 32][STACK];
  __shared__ float s_probe_k[kListThreads / 32][REL ? 32 : 1];  // their M side^2
  // nodes awaiting per-target tests during a step; the same words hold the
  // buckets' particle offsets during a bucket flush (the two phases of an
  // iteration never overlap: a __syncwarp ends each)
  __shared__ float4 s_probe[kListThreads / 32][32];
  static_assert(sizeof(s_probe[0]) >= kListCap * sizeof(int), "offsets fit the probe words");
  __shared__ int2 s_leaves[kListThreads / 32][kListCap];  // (first particle, count)
  // ORDER 1: accepted cells are point masses in the source tile; ORDER 2:
  // cells fill a QuadTile
  static_assert(!(CORR && ORDER == 2), "the network corrects the monopole");
  __shared__ __align__(16) SourceTile s_src[kListThreads / 32];
  __shared__ __align__(16) QuadTile s_quad[ORDER == 2 ? kListThreads / 32 : 1];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  SourceTile& src = s_src[wib];
  int staged = 0;   // sources waiting in src (warp-uniform)
  int listed = 0;   // corrected walk: cells listed for the network (warp-uniform)
  int qstaged = 0;  // cells waiting in the QuadTile (ORDER 2)
  const int warp = (blockIdx.x * kListThreads + threadIdx.x) >> 5;
  const bool live = warp * 32 < n;  // (a SHARED block's idle warps join its shared phase)
  if (!SHARED && !live) return;
  int* stack = s_stack[wib];
  int2* leaves = s_leaves[wib];
  const int s = warp * 32 + lane;
  const bool active = s < n;
  const float4 p = pos[active ? s : n - 1];
  const unsigned lt = (1u << lane) - 1u;
  const bool guard = !__all_sync(kFull, !active || self_term_is_finite(p.w, eps2));
  // relative test: this lane's tolerance and the group's smallest (the box
  // test stands for every target only with the least tolerant one)
  float tl = REL && active ? tol[s] : INFINITY, tmin = tl;
  if (REL)
    for (int off = 16; off > 0; off >>= 1) tmin = fminf(tmin, __shfl_xor_sync(kFull, tmin, off));

  // group bounding box
  float bx0 = p.x, bx1 = p.x, by0 = p.y, by1 = p.y, bz0 = p.z, bz1 = p.z;
  for (int off = 16; off > 0; off >>= 1) {
    bx0 = fminf(bx0, __shfl_xor_sync(kFull, bx0, off));
    bx1 = fmaxf(bx1, __shfl_xor_sync(kFull, bx1, off));
    by0 = fminf(by0, __shfl_xor_sync(kFull, by0, off));
    by1 = fmaxf(by1, __shfl_xor_sync(kFull, by1, off));
    bz0 = fminf(bz0, __shfl_xor_sync(kFull, bz0, off));
    bz1 = fmaxf(bz1, __shfl_xor_sync(kFull, bz1, off));
  }
  const float gx = 0.5f * (bx0 + bx1), gy = 0.5f * (by0 + by1), gz = 0.5f * (bz0 + bz1);
  const float ex = 0.5f * (bx1 - bx0), ey = 0.5f * (by1 - by0), ez = 0.5f * (bz1 - bz0);
  const float rg2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));  // group radius^2
  if (CORR && lane == 0) reinterpret_cast<float4*>(lists.centre)[warp] = make_float4(gx, gy, gz, rg2);

  const int total = (int)t.offset[n];
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  unsigned approx = 0, exact = 0;
  int top = 1, nleaf = 0, iters = 0;
  bool overflow = false;
  if (SHARED) {
    constexpr int kGroups = kListThreads / 32;
    __shared__ float s_box[kGroups][8];  // centre, half extents, least and most tolerant
    __shared__ int s_live[kGroups];
    __shared__ int s_sum[kGroups][3];    // per warp: accepted, children, frontier nodes
    __shared__ int s_ctop, s_nfront, s_abort;
    int* cstack = &s_stack[0][0];
    int* front = &s_stack[0][0] + kCtaStack;
    float tmax = REL && active ? tl : -INFINITY;
    if (REL)
      for (int off = 16; off > 0; off >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(kFull, tmax, off));
    if (lane == 0) {
      s_box[wib][0] = gx;
      s_box[wib][1] = gy;
      s_box[wib][2] = gz;
      s_box[wib][3] = ex;
      s_box[wib][4] = ey;
      s_box[wib][5] = ez;
      s_box[wib][6] = tmin;
      s_box[wib][7] = tmax;
      s_live[wib] = live;
    }
    if (threadIdx.x == 0) {
      s_ctop = 1;
      cstack[0] = 0;
      s_nfront = 0;
      s_abort = 0;
    }
    __syncthreads();
    for (int csteps = 0;; ++csteps) {
      const int ctop = s_ctop;  // block-uniform: read after a barrier
      if (ctop == 0 || s_abort) break;
      if (csteps > total + 64) {  // every node is popped at most once
        if (threadIdx.x == 0) atomicOr(status, NBSP_DEVICE_ERROR_WALK_LIMIT);
        break;
      }
      const int take = min(kListThreads, ctop);
      int node = (int)threadIdx.x < take ? cstack[ctop - 1 - threadIdx.x] : -1;
      if (node >= total) {
        atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
        node = -1;
      }
      const bool valid = node >= 0;
      const int at = valid ? node : 0;
      const float4 w0 = t.wnode[2 * at], w1 = t.wnode[2 * at + 1];
      const int4 info = make_int4(0, __float_as_int(w1.z), __float_as_int(w1.w), 0);
      const float4 c = w0;
      const float ro = w1.x;
      const float km = REL ? w1.y : 0.f;
      const bool bad = valid && info.z > 0 && (info.y < 0 || info.y + info.z > n);
      if (bad) atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
      const bool ok = valid && !bad;
      bool all_accept = ok && info.z != 1, all_open = ok && info.z < 0;
#pragma unroll
      for (int w = 0; w < kGroups; ++w) {
        if (!s_live[w]) continue;
        const float ax = fabsf(c.x - s_box[w][0]), ay = fabsf(c.y - s_box[w][1]),
                    az = fabsf(c.z - s_box[w][2]);
        const float qx = fmaxf(ax - s_box[w][3], 0.f), qy = fmaxf(ay - s_box[w][4], 0.f),
                    qz = fmaxf(az - s_box[w][5], 0.f);
        const float fx = ax + s_box[w][3], fy = ay + s_box[w][4], fz = az + s_box[w][5];
        const float dmin2 = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
        const float dmax2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
        all_accept = all_accept && opening_passes<REL>(dmin2, ro, km, s_box[w][6]);
        all_open = all_open && (dmax2 <= ro || (REL && dmax2 * dmax2 * s_box[w][7] < km));
      }
      const bool to_front = ok && !all_accept && !all_open;
      const int kids = all_open ? min(-info.z, 8) : 0;
      // block-wide exclusive prefixes of the three counts
      int ia = all_accept, ik = kids, ifr = to_front;
      for (int off = 1; off < 32; off <<= 1) {
        const int ua = __shfl_up_sync(kFull, ia, off), uk = __shfl_up_sync(kFull, ik, off),
                  uf = __shfl_up_sync(kFull, ifr, off);
        if (lane >= off) {
          ia += ua;
          ik += uk;
          ifr += uf;
        }
      }
      if (lane == 31) {
        s_sum[wib][0] = ia;
        s_sum[wib][1] = ik;
        s_sum[wib][2] = ifr;
      }
      __syncthreads();  // (every entry popped above has been read)
      int ba = 0, bk = 0, bf = 0, na = 0, nk = 0, nf = 0;
#pragma unroll
      for (int w = 0; w < kGroups; ++w) {
        if (w < wib) {
          ba += s_sum[w][0];
          bk += s_sum[w][1];
          bf += s_sum[w][2];
        }
        na += s_sum[w][0];
        nk += s_sum[w][1];
        nf += s_sum[w][2];
      }
      const int ra = ba + ia - (int)all_accept, rk = bk + ik - kids, rf = bf + ifr - (int)to_front;
      const int cbase = ctop - take, front0 = s_nfront;
      const bool abort = cbase + nk > kCtaStack || front0 + nf > kFrontier;  // block-uniform
      if (!abort) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < kids) cstack[cbase + rk + k] = info.y + k;
        if (to_front) front[front0 + rf] = node;
        // cells every group accepts: into every live warp's source tile, in
        // rounds of what fits before the tiles are evaluated
        approx += (unsigned)na;
        for (int done = 0; done < na;) {
          const int put = min(kStage - staged, na - done);
          const int r = ra - done;
          if (all_accept && r >= 0 && r < put)
#pragma unroll
            for (int w = 0; w < kGroups; ++w)
              if (s_live[w]) stage_source(s_src[w], staged + r, c);
          staged += put;
          done += put;
          __syncthreads();
          if (staged == kStage) {
            if (live) source_tile(src, p, eps2, guard, hx, hy, hz, lx, ly, lz);
            staged = 0;
            __syncthreads();
          }
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        if (abort) {
          s_abort = 1;
        } else {
          s_ctop = cbase + nk;
          s_nfront = front0 + nf;
        }
      }
      __syncthreads();
    }
    const int nfront = s_nfront;
    const bool restart = s_abort != 0;
    __syncthreads();  // the shared stack's last reads
    if (restart) {  // start every group from the root, discarding the shared phase
      hx = hy = hz = lx = ly = lz = 0.f;
      approx = 0;
      staged = 0;
      top = 1;
      if (lane == 0) stack[0] = 0;
    } else {
      for (int k = lane; k < nfront; k += 32) stack[k] = front[k];
      top = nfront;
    }
    __syncthreads();  // warp 2's copy is in place before any warp walks
    if (!live) return;
  } else if (lane == 0) {
    stack[0] = 0;
  }
  __syncwarp();
  // the next step's nodes (a lane without one: -1) and with LATENCY their
  // records; idle lanes load the root's, so that no branch diverges
  int next = lane < top ? stack[top - 1 - lane] : -1;
  float4 next0 = make_float4(0.f, 0.f, 0.f, 0.f), next1 = next0;
  auto load_next = [&]() {
    const int at = next >= 0 && next < total ? next : 0;
    next0 = __ldg(&t.wnode[2 * at]);
    next1 = __ldg(&t.wnode[2 * at + 1]);
  };
  if (LATENCY > 0) load_next();
  // (staged > 0 with nothing left to walk: cells the shared phase staged; the
  // draining iteration evaluates them)
  for (;;) {  // until the stack, the bucket list and the tiles are drained
    if (top > 0) {
      if (++iters > total + 64) {  // every node is popped at most once
        if (lane == 0) atomicOr(status, NBSP_DEVICE_ERROR_WALK_LIMIT);
        break;
      }
      int node = next;
      top -= min(32, top);
      bool is_leaf = false, accept = false, test = false;
      int kids = 0;
      int4 info = make_int4(0, 0, 0, 0);
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      float ro = 0.f, km = 0.f;
      if (node >= total) {
        atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
        node = -1;
      }
      {  // every lane loads a node (idle lanes the root) so no branch diverges
        const bool valid = node >= 0;
        const int at = valid ? node : 0;
        // one 32-byte record: the centre of mass and mass, the opening terms,
        // and a bucket's particles or an internal node's children
        const float4 w0 = LATENCY > 0 ? next0 : __ldg(&t.wnode[2 * at]);
        const float4 w1 = LATENCY > 0 ? next1 : __ldg(&t.wnode[2 * at + 1]);
        c = w0;
        ro = w1.x;
        if (REL) km = w1.y;
        info.y = __float_as_int(w1.z);
        info.z = __float_as_int(w1.w);
        const bool bad = valid && info.z > 0 && (info.y < 0 || info.y + info.z > n);
        if (bad) atomicOr(status, NBSP_DEVICE_ERROR_TREE_INCONSISTENT);
        const bool ok = valid && !bad;
        is_leaf = ok && info.z == 1;
        const float qx = fmaxf(fabsf(c.x - gx) - ex, 0.f);
        const float qy = fmaxf(fabsf(c.y - gy) - ey, 0.f);
        const float qz = fmaxf(fabsf(c.z - gz) - ez, 0.f);
        const float dmin2 = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
        const bool cellish = ok && info.z != 1;
        const bool box = opening_passes<REL>(dmin2, ro, km, tmin);
        accept = cellish && box;
        test = cellish && !box;
      }
      // Nodes the box could not accept: a node that fails this lane's own
      // target is opened at once; for the rest every target's own test
      // decides, one node at a time with the 32 targets tested in parallel.
      const float d2own = fmaf(c.x - p.x, c.x - p.x, fmaf(c.y - p.y, c.y - p.y, (c.z - p.z) * (c.z - p.z)));
      const bool opened = test && active && !opening_passes<REL>(d2own, ro, km, tl);
      test = test && !opened;
      float4* probe = s_probe[wib];
      unsigned pend = __ballot_sync(kFull, test);
      if (LATENCY > 0 && __popc(pend) > kProbeTurn) {
        // many: each lane its own node against every target (an idle lane of the
        // last group repeats the last particle and tolerates everything)
        probe[lane] = make_float4(p.x, p.y, p.z, tl);
        __syncwarp();
        bool all = test;
#pragma unroll 8
        for (int q = 0; q < 32; ++q) {
          const float4 u = probe[q];
          const float dx = c.x - u.x, dy = c.y - u.y, dz = c.z - u.z;
          all = opening_passes<REL>(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), ro, km, u.w) && all;
        }
        accept = accept || all;
        pend = 0u;
      } else if (test) {
        probe[lane] = make_float4(c.x, c.y, c.z, ro);
        if (REL) s_probe_k[wib][lane] = km;
      }
      __syncwarp();
      constexpr int kProbes = LATENCY > 0 ? 4 : 1;
      while (pend != 0u) {
        int from[kProbes];
        bool fail[kProbes];
#pragma unroll
        for (int k = 0; k < kProbes; ++k) {  // (none left: the first one again)
          from[k] = k == 0 || pend != 0u ? __ffs(pend) - 1 : from[0];
          pend &= pend - 1u;
        }
#pragma unroll
        for (int k = 0; k < kProbes; ++k) {
          const float4 q = probe[from[k]];
          const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
          fail[k] = active && !opening_passes<REL>(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), q.w,
                                                   REL ? s_probe_k[wib][from[k]] : 0.f, tl);
        }
#pragma unroll
        for (int k = 0; k < kProbes; ++k) {
          const bool any = __any_sync(kFull, fail[k]);
          if (lane == from[k]) accept = !any;
        }
      }
      const bool open = (test || opened) && !accept;
      is_leaf = is_leaf || (open && info.z > 0);  // a failing bucket is summed exactly
      if (open && info.z < 0) kids = min(-info.z, 8);  // an opened cell pushes its children
      unsigned m = __ballot_sync(kFull, is_leaf);
      if (is_leaf) leaves[nleaf + __popc(m & lt)] = make_int2(info.y, info.z);
      nleaf += __popc(m);
      // the children go onto the stack before the accepted cells are staged: the
      // next step's nodes are then known while tiles are evaluated
      int incl = kids;
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, off);
        if (lane >= off) incl += v;
      }
      const int pushed = __shfl_sync(kFull, incl, 31);
      if (top + pushed > STACK) {
        overflow = true;
        break;
      }
      const int base = top + incl - kids;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < kids) stack[base + k] = info.y + k;
      top += pushed;
      __syncwarp();
      next = lane < top ? stack[top - 1 - lane] : -1;
      if (LATENCY > 0) load_next();
      m = __ballot_sync(kFull, accept);
      if (ORDER == 1) {
        // A monopole cell is a point mass at its centre of mass, already in
        // this lane's registers from the opening test: it goes straight into
        // the source tile (evaluated whenever 64 sources have gathered).  The
        // corrected walk also lists the cell for its network evaluation.
        if (CORR) {
          bool listme = false;
          if (accept) {
            const float side = t.wquad[2 * node + 1].y;
            const float gdx = c.x - gx, gdy = c.y - gy, gdz = c.z - gz;
            const float dg2 = fmaf(gdx, gdx, fmaf(gdy, gdy, gdz * gdz));
            const float lo = __ldg(&net->x_min[3]), hi = __ldg(&net->x_max[3]);
            listme = kCorrGroup * kCorrGroup * dg2 > rg2 && side * side >= lo * lo * dg2 &&
                     side * side <= hi * hi * dg2;
          }
          const unsigned lm = __ballot_sync(kFull, listme);
          const int at = listed + __popc(lm & lt);
          if (listme && at < lists.capacity) lists.cells[(size_t)warp * lists.capacity + at] = node;
          listed += __popc(lm);
        }
        const int nacc = __popc(m), rank = __popc(m & lt), room = kStage - staged;
        if (accept && rank < room) stage_source(src, staged + rank, c);
        if (nacc >= room) {
          __syncwarp();
          source_tile(src, p, eps2, guard, hx, hy, hz, lx, ly, lz);
          __syncwarp();
          if (accept && rank >= room) stage_source(src, rank - room, c);
          staged = nacc - room;
        } else {
          staged += nacc;
        }
        approx += (unsigned)nacc;  // (warp-uniform; an idle lane's is dropped at the end)
      } else {  // a quadrupole cell goes into the QuadTile with its moments
        QuadTile& qt = s_quad[ORDER == 2 ? wib : 0];
        float4 qa = make_float4(0.f, 0.f, 0.f, 0.f);
        float qyz = 0.f;
        if (accept) {
          qa = t.wquad[2 * node];
          qyz = t.wquad[2 * node + 1].x;
        }
        const int nacc = __popc(m), rank = __popc(m & lt), room = kStage - qstaged;
        if (accept && rank < room) stage_cell(qt, qstaged + rank, c, qa, qyz);
        if (nacc >= room) {
          __syncwarp();
          quad_tile(qt, p, eps2, hx, hy, hz, lx, ly, lz);
          __syncwarp();
          if (accept && rank >= room) stage_cell(qt, rank - room, c, qa, qyz);
          qstaged = nacc - room;
        } else {
          qstaged += nacc;
        }
        approx += (unsigned)nacc;  // (warp-uniform; an idle lane's is dropped at the end)
      }
    }
    const bool drain = top == 0;
    if (nleaf >= 32 || (drain && nleaf > 0)) {
      // The buckets' particles, concatenated, fill the tile, all loads of a tile
      // in flight at once.  A slot's bucket is the number of buckets that start
      // at or before it: those before the tile's first slot, plus the bits up to
      // it in the mask of the starts inside the tile (two words, one OR-reduction
      // each; a binary search over the counts' prefix took three times the
      // instructions and six dependent shared-memory loads).  The target's own
      // particle adds exactly 0 (d = 0).
      int* shift = reinterpret_cast<int*>(s_probe[wib]);  // first particle - first slot
      const int2 l0 = lane < nleaf ? leaves[lane] : make_int2(0, 0);
      const int2 l1 = lane + 32 < nleaf ? leaves[lane + 32] : make_int2(0, 0);
      int i0 = l0.y, i1 = l1.y;
      for (int off = 1; off < 32; off <<= 1) {
        const int v0 = __shfl_up_sync(kFull, i0, off), v1 = __shfl_up_sync(kFull, i1, off);
        if (lane >= off) {
          i0 += v0;
          i1 += v1;
        }
      }
      i1 += __shfl_sync(kFull, i0, 31);
      const int total_src = __shfl_sync(kFull, i1, 31);
      // first slot of each of this lane's buckets (none: past every slot)
      const int b0 = lane < nleaf ? i0 - l0.y : INT_MAX, b1 = lane + 32 < nleaf ? i1 - l1.y : INT_MAX;
      if (lane < nleaf) shift[lane] = l0.x - b0;
      if (lane + 32 < nleaf) shift[lane + 32] = l1.x - b1;
      {  // targets whose own particle is in one of these buckets: one term fewer
        // (only the group's own buckets overlap its targets: a vote first)
        const int g0 = warp * 32;
        const int lo0 = max(l0.x - g0, 0), hi0 = min(l0.x + l0.y - g0, 32);
        const int lo1 = max(l1.x - g0, 0), hi1 = min(l1.x + l1.y - g0, 32);
        if (__any_sync(kFull, hi0 > lo0 || hi1 > lo1)) {
          unsigned own = 0u;
          if (hi0 > lo0) own |= (hi0 >= 32 ? kFull : (1u << hi0) - 1u) & ~((1u << lo0) - 1u);
          if (hi1 > lo1) own |= (hi1 >= 32 ? kFull : (1u << hi1) - 1u) & ~((1u << lo1) - 1u);
          own = __reduce_or_sync(kFull, own);
          if (active && ((own >> lane) & 1u)) exact -= 1u;
        }
      }
      __syncwarp();
      exact += active ? (unsigned)total_src : 0u;  // own particles were taken off above
      const unsigned le = 2u * lt + 1u;  // this lane's bit and those below
      for (int f0 = 0; f0 < total_src;) {
        const int take = min(total_src - f0, kStage - staged);
        const bool h0 = lane < take, h1 = lane + 32 < take;
        const unsigned r0 = (unsigned)(b0 - f0), r1 = (unsigned)(b1 - f0);
        const unsigned m0 = __reduce_or_sync(
            kFull, (r0 < 32u ? 1u << r0 : 0u) | (r1 < 32u ? 1u << r1 : 0u));
        const unsigned m1 = __reduce_or_sync(
            kFull, (r0 - 32u < 32u ? 1u << (r0 - 32u) : 0u) | (r1 - 32u < 32u ? 1u << (r1 - 32u) : 0u));
        const int before = __popc(__ballot_sync(kFull, b0 < f0)) + __popc(__ballot_sync(kFull, b1 < f0)) - 1;
        float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
        if (h0) q0 = pos[shift[before + __popc(m0 & le)] + f0 + lane];
        if (h1) q1 = pos[shift[before + __popc(m0) + __popc(m1 & le)] + f0 + lane + 32];
        if (h0) stage_source(src, staged + lane, q0);
        if (h1) stage_source(src, staged + lane + 32, q1);
        staged += take;
        f0 += take;
        if (staged == kStage) {
          __syncwarp();
          source_tile(src, p, eps2, guard, hx, hy, hz, lx, ly, lz);
          staged = 0;
          __syncwarp();
        }
      }
      nleaf = 0;
    }
    if (drain && staged > 0) {  // the last, partial tile: pad with massless far sources
      for (int k = staged + lane; k < kStage; k += 32)
        stage_source(src, k, make_float4(kFarAway, kFarAway, kFarAway, 0.f));
      __syncwarp();
      source_tile(src, p, eps2, guard, hx, hy, hz, lx, ly, lz);
      staged = 0;
    }
    if (ORDER == 2 && drain && qstaged > 0) {  // the same for the last cells
      QuadTile& qt = s_quad[ORDER == 2 ? wib : 0];
      for (int k = qstaged + lane; k < kStage; k += 32)
        stage_cell(qt, k, make_float4(kFarAway, kFarAway, kFarAway, 0.f),
                   make_float4(0.f, 0.f, 0.f, 0.f), 0.f);
      __syncwarp();
      quad_tile(qt, p, eps2, hx, hy, hz, lx, ly, lz);
      qstaged = 0;
    }
    __syncwarp();
    if (drain) break;
  }
  if (CORR && lane == 0) {  // a group walked again keeps the plain monopole
    lists.count[warp] = overflow ? 0 : min(listed, lists.capacity);
    if (!overflow && listed > lists.capacity)
      atomicAdd(&counters[7], (unsigned long long)(listed - lists.capacity));
  }
  WalkAcc a;
  if (overflow) {
    if (lane == 0) atomicAdd(&counters[5], 1ull);  // groups walked again
    stackless_walk<ORDER, REL>(pos, n, t, eps2, s, active, p, tl, lane, status, a);
  } else {
    a.hx = hx;
    a.hy = hy;
    a.hz = hz;
    a.lx = lx;
    a.ly = ly;
    a.lz = lz;
    a.approx = active ? approx : 0u;
    a.exact = exact;
  }
  store_walk(a, s, active, lane, perm, n, acc, counters);
}

// ---- the correction pipeline after a corrected walk ------------------------
//
// 1. corr_scan_kernel: exclusive prefix of the per-group list lengths (one
//    row per listed (cell, group) pair, groups in order);
// 2. corr_rows_kernel: every row's 10 features at its group centre, the
//    network on 128-row tiles on the tcgen05 tensor cores, the de-standardised
//    output (zero for features outside the training range: the plain
//    monopole, the fallback);
// 3. corr_apply_kernel: one warp per group adds (M / |d|^2) * y of its rows,
//    in list order, to each target's walk result (deterministic).

__global__ void __launch_bounds__(1024) corr_scan_kernel(NbspCorrectionLists lists, int groups,
                                                         unsigned long long* counters) {
  __shared__ int warp_sums[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < groups; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < groups ? lists.count[i] : 0;
    int x = v;
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(kFull, x, off);
      if (lane >= off) x += u;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int w = warp_sums[lane];
      for (int off = 1; off < 32; off <<= 1) {
        const int u = __shfl_up_sync(kFull, w, off);
        if (lane >= off) w += u;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const int incl = x + (wid > 0 ? warp_sums[wid - 1] : 0);
    const int c = carry;
    if (i < groups) lists.offset[i] = c + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = c + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    lists.offset[groups] = carry;
    atomicAdd(&counters[6], (unsigned long long)carry);  // network evaluations
  }
}

// Row r -> (its group, its cell), one warp per group: the rows kernel reads
// both with one 8-byte load and needs no search.
__global__ void __launch_bounds__(128) corr_rowmap_kernel(NbspCorrectionLists lists, int groups) {
  const int lane = threadIdx.x & 31;
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g >= groups) return;
  const int cnt = lists.count[g], off = lists.offset[g];
  int2* rows = reinterpret_cast<int2*>(lists.row);
  for (int k = lane; k < cnt; k += 32)
    rows[off + k] = make_int2(g, lists.cells[(size_t)g * lists.capacity + k]);
}

// What the features of one row are computed from, loaded one tile ahead so the
// loads are in flight while the tensor cores run the current tile.
struct RowData {
  float4 c;    // cell centre of mass, mass
  float4 g;    // group centre, radius^2
  float4 qa;   // quadrupole xx, xy, xz, yy
  float qyz, side, spread;
  bool valid;
};

__device__ __forceinline__ RowData load_row(const Tree& t, const float4* centre, int2 gn,
                                            bool valid) {
  RowData d;
  d.valid = valid;
  const int node = valid ? gn.y : 0, grp = valid ? gn.x : 0;
  d.c = t.wnode[2 * node];
  d.g = centre[grp];
  d.qa = t.wquad[2 * node];
  const float4 qb = t.wquad[2 * node + 1];
  d.qyz = qb.x;
  d.side = qb.y;
  d.spread = qb.z;
  return d;
}

__global__ void __launch_bounds__(nbsp_umma::kThreads) corr_rows_kernel(
    const nbsp_mlp::Net* __restrict__ net, Tree t, NbspCorrectionLists lists, int groups,
    int* status) {
  extern __shared__ __align__(128) unsigned char umma_smem[];
  nbsp_umma::Smem& sm = *reinterpret_cast<nbsp_umma::Smem*>(umma_smem);
  nbsp_umma::setup(sm, nbsp_umma::weights_of(net), net);
  const uint32_t tmem = sm.tmem;
  uint32_t phase = 0;
  const int rows = lists.offset[groups];
  const int tiles = (rows + nbsp_umma::kRows - 1) / nbsp_umma::kRows;
  const float4* centre = reinterpret_cast<const float4*>(lists.centre);
  const int2* rowmap = reinterpret_cast<const int2*>(lists.row);
  const int stride = gridDim.x * nbsp_umma::kRows;
  // pipeline: the row map two tiles ahead, the row data one tile ahead
  int r = blockIdx.x * nbsp_umma::kRows + threadIdx.x;
  RowData cur = load_row(t, centre, r < rows ? rowmap[r] : make_int2(0, 0), r < rows);
  int2 ahead = r + stride < rows ? rowmap[r + stride] : make_int2(0, 0);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, r += stride) {
    float v[nbsp_mlp::kIn];
    bool ok = false;
    if (cur.valid) {
      float f[nbsp_mlp::kIn];
      ok = features_of(cur.c, cur.side, cur.qa, cur.qyz, cur.spread, cur.g.x, cur.g.y, cur.g.z,
                       f);
#pragma unroll
      for (int q = 0; q < nbsp_mlp::kIn; ++q) {
        ok = ok && f[q] >= net->x_min[q] && f[q] <= net->x_max[q];
        v[q] = (f[q] - net->x_mean[q]) * net->x_inv_std[q];
      }
    }
    if (!ok)
#pragma unroll
      for (int q = 0; q < nbsp_mlp::kIn; ++q) v[q] = 0.f;
    nbsp_umma::put_inputs(sm, v);
    nbsp_umma::fence_async_smem();
    __syncthreads();
    const RowData next = load_row(t, centre, ahead, r + stride < rows);
    ahead = r + 2 * stride < rows ? rowmap[r + 2 * stride] : make_int2(0, 0);
    float y[3];
    if (!nbsp_umma::forward(sm, tmem, phase, y)) {
      if (threadIdx.x == 0) atomicOr(status, NBSP_DEVICE_ERROR_MMA_TIMEOUT);
      break;
    }
    if (r < rows)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        lists.y[(size_t)r * 3 + c] = ok ? fmaf(y[c], net->y_std[c], net->y_mean[c]) : 0.f;
    cur = next;
  }
  nbsp_umma::teardown(sm, tmem);
}

__global__ void __launch_bounds__(128) corr_apply_kernel(const float4* __restrict__ pos, int n,
                                                         Tree t, NbspCorrectionLists lists,
                                                         const uint32_t* __restrict__ perm,
                                                         double4* __restrict__ acc) {
  const int lane = threadIdx.x & 31;
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g * 32 >= n) return;
  const int s = g * 32 + lane;
  const bool active = s < n;
  const float4 p = pos[active ? s : n - 1];
  const int cnt = lists.count[g], off = lists.offset[g];
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  for (int i0 = 0; i0 < cnt; i0 += 32) {
    const int k = i0 + lane;
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    float yx = 0.f, yy = 0.f, yz = 0.f;
    if (k < cnt) {
      c = t.wnode[2 * lists.cells[(size_t)g * lists.capacity + k]];
      const float* y = &lists.y[(size_t)(off + k) * 3];
      yx = c.w * y[0];
      yy = c.w * y[1];
      yz = c.w * y[2];
    }
    float ax = 0.f, ay = 0.f, az = 0.f;
    const int take = min(32, cnt - i0);
    for (int j = 0; j < take; ++j) {
      const float cx = __shfl_sync(kFull, c.x, j), cy = __shfl_sync(kFull, c.y, j);
      const float cz = __shfl_sync(kFull, c.z, j);
      const float Yx = __shfl_sync(kFull, yx, j), Yy = __shfl_sync(kFull, yy, j);
      const float Yz = __shfl_sync(kFull, yz, j);
      const float dx = cx - p.x, dy = cy - p.y, dz = cz - p.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float r = d2 > 0.f ? rsqrt_mufu(d2) : 0.f;
      const float w = r * r;
      ax = fmaf(w, Yx, ax);
      ay = fmaf(w, Yy, ay);
      az = fmaf(w, Yz, az);
    }
    fold(hx, lx, ax);
    fold(hy, ly, ay);
    fold(hz, lz, az);
  }
  if (active && cnt > 0) {  // the walk stored the target at its input index
    const uint32_t i = perm[s];
    if (i < (uint32_t)n) {
      double4 a = acc[i];
      a.x += (double)hx + (double)lx;
      a.y += (double)hy + (double)ly;
      a.z += (double)hz + (double)lz;
      acc[i] = a;
    }
  }
}

int grid_for(size_t n, int threads) {
  size_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 64) b = 148 * 64;
  return (int)b;
}

int bounds_blocks(size_t n) {
  const size_t blocks = (n + kBoundsThreads - 1) / kBoundsThreads;
  return blocks < 1 ? 1 : blocks > (size_t)kBoundsBlocks ? kBoundsBlocks : (int)blocks;
}

template <bool REL>
void launch_walk(const float4* p, const float* tol, size_t n, Tree t, int order, int mode,
                 const nbsp_mlp::Net* net, const NbspCorrectionLists* lists, float eps2,
                 const uint32_t* perm, double4* out, unsigned long long* counters, int* status,
                 unsigned long long* stamp, cudaStream_t stream) {
  if (mode == NBSP_BH_WALK_LISTS || mode == NBSP_BH_WALK_SHARED || net != nullptr) {
    const unsigned blocks = (unsigned)((n + kListThreads - 1) / kListThreads);
    NbspCorrectionLists none{};
    if (net != nullptr && lists != nullptr) {  // the network corrects the monopole term
      NBSP_COUNT_LAUNCH(1), walk_lists_kernel<1, kListStack, true, REL><<<blocks, kListThreads, 0, stream>>>(
          p, tol, (int)n, t, eps2, perm, out, counters, status, net, *lists, stamp);
    } else if (order == 1 && mode == NBSP_BH_WALK_SHARED) {
      NBSP_COUNT_LAUNCH(1), walk_lists_kernel<1, kListStack, false, REL, true><<<blocks, kListThreads, 0, stream>>>(
          p, tol, (int)n, t, eps2, perm, out, counters, status, nullptr, none, stamp);
    } else if (order == 2) {
      NBSP_COUNT_LAUNCH(1), (blocks <= kLatencyBlocks ? walk_lists_kernel<2, kListStack, false, REL, false, 4>
                                               : walk_lists_kernel<2, kListStack, false, REL>)
          <<<blocks, kListThreads, 0, stream>>>(p, tol, (int)n, t, eps2, perm, out, counters,
                                                status, nullptr, none, stamp);
    } else {
      constexpr int kStack = REL ? kListStackRel : kListStack;
      NBSP_COUNT_LAUNCH(1), (blocks <= 148 * 4   ? walk_lists_kernel<1, kStack, false, REL, false, 4>
                             : blocks <= kLatencyBlocks ? walk_lists_kernel<1, kStack, false, REL, false, 6>
                                                 : walk_lists_kernel<1, kStack, false, REL>)
          <<<blocks, kListThreads, 0, stream>>>(p, tol, (int)n, t, eps2, perm, out, counters,
                                                status, nullptr, none, stamp);
    }
    return;
  }
  const unsigned blocks = (unsigned)((n + kWalkThreads - 1) / kWalkThreads);
  if (order == 2) {
    NBSP_COUNT_LAUNCH(1), walk_kernel<2, REL><<<blocks, kWalkThreads, 0, stream>>>(
        p, tol, (int)n, t, eps2, perm, out, counters, status, stamp);
  } else {
    NBSP_COUNT_LAUNCH(1), walk_kernel<1, REL><<<blocks, kWalkThreads, 0, stream>>>(
        p, tol, (int)n, t, eps2, perm, out, counters, status, stamp);
  }
}

}  // namespace

extern "C" {

void nbsp_bh_bounds(double* x, double* y, double* z, const double* m, size_t n, double* partial,
                    double* geometry, int* status, const double* ax, const double* ay,
                    const double* az, int rms_of_a, const NbspLeapfrogFusion* leapfrog,
                    unsigned long long* stamp, unsigned long long* end, cudaStream_t stream) {
  const int blocks = bounds_blocks(n);
  if (leapfrog != nullptr && leapfrog->vx != nullptr) {
    NBSP_COUNT_LAUNCH(1), bounds_kernel<true><<<blocks, kBoundsThreads, 0, stream>>>(
        x, y, z, m, n, partial, status, ax, ay, az, rms_of_a != 0, leapfrog->vx, leapfrog->vy,
        leapfrog->vz, leapfrog->half_dt, leapfrog->dt, stamp);
  } else {
    NBSP_COUNT_LAUNCH(1), bounds_kernel<false><<<blocks, kBoundsThreads, 0, stream>>>(
        x, y, z, m, n, partial, status, ax, ay, az, rms_of_a != 0, nullptr, nullptr, nullptr,
        0.0, 0.0, stamp);
  }
  if (geometry != nullptr)
    NBSP_COUNT_LAUNCH(1), bounds_final_kernel<<<1, kBoundsThreads, 0, stream>>>(
                              partial, blocks, n, geometry, end);
}

void nbsp_bh_small_keys(const double* x, const double* y, const double* z, const double* m,
                        size_t n, const double* partial, double* geometry, uint64_t* keys,
                        uint32_t* index, void* unsorted, const double* ax, const double* ay,
                        const double* az, double tol_scale, float* unsorted_tol, void* tree,
                        unsigned long long* counters, unsigned long long* stamp,
                        cudaStream_t stream) {
  const unsigned tiles = (unsigned)((n + kSmallTile - 1) / kSmallTile);
  NBSP_COUNT_LAUNCH(1), small_keys_kernel<<<tiles, kSmallTile, 0, stream>>>(
      x, y, z, m, n, partial, bounds_blocks(n), geometry, keys, index, (float4*)unsorted, ax, ay,
      az, tol_scale, unsorted_tol, tree_view(tree, n), counters, stamp);
}

void nbsp_bh_small_merge(const uint64_t* keys_in, const uint32_t* index_in, size_t n,
                         uint64_t* keys, uint32_t* index, const void* unsorted, void* pos4,
                         const float* unsorted_tol, float* tol, int* status,
                         unsigned long long* stamp, cudaStream_t stream) {
  NBSP_COUNT_LAUNCH(1), small_merge_kernel<<<(unsigned)((n + 31) / 32), 32 * kMergeWarps, 0, stream>>>(
      keys_in, index_in, (int)n, keys, index, (const float4*)unsorted, (float4*)pos4,
      unsorted_tol, tol, status, stamp);
}

// (buffers for n hold every smaller system too, whose narrow tiles may be more)
size_t nbsp_bh_sort_scratch_words(size_t n) {
  const size_t narrow = sort_scratch_words(n < kSortWide ? n : kSortWide - 1);
  const size_t own = sort_scratch_words(n);
  return own > narrow ? own : narrow;
}

void nbsp_bh_keys(const double* x, const double* y, const double* z, const double* m, size_t n,
                  const double* geometry, uint64_t* keys, uint32_t* index, void* unsorted,
                  uint32_t* scratch, const double* ax, const double* ay, const double* az,
                  double tol_scale, float* unsorted_tol, void* tree,
                  unsigned long long* counters, cudaStream_t stream) {
  cudaMemsetAsync(scratch, 0, sort_scratch_words(n) * sizeof(uint32_t), stream);
  const SortScratch sc = sort_scratch(scratch);
  size_t blocks = (n + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > (size_t)kKeysBlocks) blocks = kKeysBlocks;
  NBSP_COUNT_LAUNCH(1), keys_kernel<<<(unsigned)blocks, 256, 0, stream>>>(
      x, y, z, m, n, geometry, keys, index, (float4*)unsorted, sc.hist, ax, ay, az, tol_scale,
      unsorted_tol, tree_view(tree, n), counters);
}

void nbsp_bh_sort(uint64_t* keys, uint32_t* index, uint64_t* keys_alt, uint32_t* index_alt,
                  size_t n, uint32_t* scratch, int* status, unsigned long long* stamp,
                  cudaStream_t stream) {
  const bool narrow = n < kSortWide;
  const auto pass_kernel = narrow ? sort_pass_kernel<SortNarrow> : sort_pass_kernel<SortWide>;
  const int threads = narrow ? SortNarrow::kThreads : SortWide::kThreads;
  const size_t smem = narrow ? sort_pass_smem<SortNarrow>() : sort_pass_smem<SortWide>();
  cudaFuncSetAttribute(pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const SortScratch sc = sort_scratch(scratch);
  const size_t tiles = sort_tiles(n);
  static_assert(kSortPasses % 2 == 1, "from (keys_alt, index_alt) to (keys, index)");
  uint64_t* kin = keys_alt;
  uint32_t* vin = index_alt;
  uint64_t* kout = keys;
  uint32_t* vout = index;
  for (int pass = 0; pass < kSortPasses; ++pass) {
    NBSP_COUNT_LAUNCH(1), pass_kernel<<<(unsigned)tiles, threads, smem, stream>>>(
        kin, vin, kout, vout, n, kRadixBits * pass, sc.hist + pass * kRadix, sc.ticket + pass,
        sc.status + (size_t)pass * tiles * kRadix, status, pass == 0 ? stamp : nullptr);
    uint64_t* tk = kin;
    kin = kout;
    kout = tk;
    uint32_t* tv = vin;
    vin = vout;
    vout = tv;
  }
}

void nbsp_bh_gather(const void* unsorted, const uint32_t* perm, size_t n, void* pos4,
                    const float* unsorted_tol, float* tol, int* status, unsigned long long* stamp,
                    cudaStream_t stream) {
  NBSP_COUNT_LAUNCH(1), gather_kernel<<<grid_for(n, 256), 256, 0, stream>>>(
      (const float4*)unsorted, perm, n, (float4*)pos4, unsorted_tol, tol, status, stamp);
}

void nbsp_bh_late_tolerances(const double* ax, const double* ay, const double* az, size_t n,
                             double tol_scale, const uint32_t* perm, double* partial, float* tol,
                             double* geometry, cudaStream_t stream) {
  const int blocks = bounds_blocks(n);
  NBSP_COUNT_LAUNCH(1), late_squares_kernel<<<blocks, kBoundsThreads, 0, stream>>>(ax, ay, az, n,
                                                                                 partial);
  NBSP_COUNT_LAUNCH(1), late_tolerances_kernel<<<blocks, kBoundsThreads, 0, stream>>>(
      ax, ay, az, partial, blocks, n, tol_scale, perm, tol, geometry);
}

size_t nbsp_bh_tree_bytes(size_t n) { return tree_bytes(n); }

void nbsp_bh_build(const uint64_t* keys, const uint32_t* perm, const double* x, const double* y,
                   const double* z, size_t n, int leaf_capacity, void* tree, int* status,
                   unsigned long long* stamp, cudaStream_t stream) {
  Tree t = tree_view(tree, n);
  if (n >= 2)
    NBSP_COUNT_LAUNCH(1), radix_tree_kernel<<<(unsigned)((n - 1 + 255) / 256), 256, 0, stream>>>(
        keys, perm, x, y, z, t, status, stamp);
  // (n >= 2: the caller handles a lone particle without a tree)
  const unsigned keep_blocks = (unsigned)((n - 1 + kKeepNodes - 1) / kKeepNodes);
  if (keep_blocks > 0)
    NBSP_COUNT_LAUNCH(1), keep_kernel<<<keep_blocks, kKeepThreads, 0, stream>>>(t, leaf_capacity, status);
  const int blocks = (int)((n + kScanItems - 1) / kScanItems);
  if (n <= NBSP_BH_SMALL_SORT) {
    NBSP_COUNT_LAUNCH(1), scan_small_kernel<<<blocks, kSmallScanThreads, 0, stream>>>(t);
  } else {
    NBSP_COUNT_LAUNCH(1), scan_reduce_kernel<<<blocks, kScanThreads, 0, stream>>>(t);
    if (blocks <= kScanSums) {
      NBSP_COUNT_LAUNCH(1), scan_apply_kernel<false><<<blocks, kScanThreads, 0, stream>>>(t);
    } else {
      NBSP_COUNT_LAUNCH(1), scan_blocks_kernel<<<1, 1024, 0, stream>>>(t, blocks);
      NBSP_COUNT_LAUNCH(1), scan_apply_kernel<true><<<blocks, kScanThreads, 0, stream>>>(t);
    }
  }
  // (at most a splitting cell per two particles: eight threads each)
  const size_t place_blocks = (4 * n + 255) / 256;
  NBSP_COUNT_LAUNCH(1), place_kernel<<<(unsigned)(place_blocks < kPlaceBlocks ? place_blocks : kPlaceBlocks), 256, 0, stream>>>(
      t, leaf_capacity, status);
}

void nbsp_bh_moments(const void* pos4, const uint64_t* keys, size_t n, const double* geometry,
                     double theta, double start_theta, int opening, int quadrupoles, void* tree,
                     int* status, unsigned long long* stamp, cudaStream_t stream) {
  Tree t = tree_view(tree, n);
  const size_t nb = 2 * n - 1;
  Opening o;
  o.keys = keys;
  o.geometry = geometry;
  o.inv_theta = theta > 0.0 ? 1.0 / theta : INFINITY;
  o.inv_theta2 = theta > 0.0 ? 1.0 / (theta * theta) : INFINITY;
  o.relative = start_theta > 0.0;
  o.start_inv_theta = o.relative ? 1.0 / start_theta : o.inv_theta;
  o.start_inv_theta2 = o.relative ? 1.0 / (start_theta * start_theta) : o.inv_theta2;
  o.criterion = opening;
  size_t blocks = (nb + 255) / 256;  // grid-stride over the octree nodes (<= 2n - 1)
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (quadrupoles)
    NBSP_COUNT_LAUNCH(1), moments_kernel<true, 1><<<(unsigned)blocks, 256, 0, stream>>>(
                              (const float4*)pos4, t, o, status, stamp);
  else
    NBSP_COUNT_LAUNCH(1), (n < kMomentsWide ? moments_kernel<false, 1> : moments_kernel<false, 6>)
        <<<(unsigned)blocks, 256, 0, stream>>>((const float4*)pos4, t, o, status, stamp);
}

void nbsp_bh_walk(const void* pos4, const float* tol, size_t n, const void* tree, int order,
                  int mode, const void* correction, const NbspCorrectionLists* lists, float eps2,
                  const uint32_t* perm, void* acc, unsigned long long* counters, int* status,
                  unsigned long long* stamp, cudaStream_t stream) {
  Tree t = tree_view(const_cast<void*>(tree), n);
  const nbsp_mlp::Net* net = (const nbsp_mlp::Net*)correction;
  const float4* p = (const float4*)pos4;
  double4* out = (double4*)acc;
  if (tol != nullptr)
    launch_walk<true>(p, tol, n, t, order, mode, net, lists, eps2, perm, out, counters, status,
                      stamp, stream);
  else
    launch_walk<false>(p, nullptr, n, t, order, mode, net, lists, eps2, perm, out, counters,
                       status, stamp, stream);
}

void nbsp_bh_correct(const void* pos4, size_t n, const void* tree, const void* correction,
                     const NbspCorrectionLists* lists, const uint32_t* perm, void* acc,
                     unsigned long long* counters, int* status, cudaStream_t stream) {
  Tree t = tree_view(const_cast<void*>(tree), n);
  const nbsp_mlp::Net* net = (const nbsp_mlp::Net*)correction;
  const int groups = (int)((n + 31) / 32);
  NBSP_COUNT_LAUNCH(1), corr_scan_kernel<<<1, 1024, 0, stream>>>(*lists, groups, counters);
  NBSP_COUNT_LAUNCH(1), corr_rowmap_kernel<<<(unsigned)((groups + 3) / 4), 128, 0, stream>>>(
      *lists, groups);
  const int smem = (int)sizeof(nbsp_umma::Smem);
  cudaFuncSetAttribute(corr_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  // persistent: kCtasPerSm CTAs per SM, each holding 64 of the 512 TMEM columns
  NBSP_COUNT_LAUNCH(1), corr_rows_kernel<<<148 * nbsp_umma::kCtasPerSm, nbsp_umma::kThreads, smem, stream>>>(
      net, t, *lists, groups, status);
  NBSP_COUNT_LAUNCH(1), corr_apply_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(
      (const float4*)pos4, (int)n, t, *lists, perm, (double4*)acc);
}

void nbsp_bh_unsort(const void* acc, size_t n, double g, double* ax, double* ay, double* az,
                    const NbspLeapfrogFusion* leapfrog, const void* tree,
                    unsigned long long* counters, unsigned long long* stamp,
                    cudaStream_t stream) {
  const Tree t = tree_view(const_cast<void*>(tree), n);
  if (leapfrog != nullptr && leapfrog->vx != nullptr) {
    NBSP_COUNT_LAUNCH(1), unsort_kernel<true><<<grid_for(n, 256), 256, 0, stream>>>(
        (const double4*)acc, n, g, ax, ay, az, leapfrog->vx, leapfrog->vy, leapfrog->vz,
        leapfrog->half_dt, t, counters, stamp);
  } else {
    NBSP_COUNT_LAUNCH(1), unsort_kernel<false><<<grid_for(n, 256), 256, 0, stream>>>(
        (const double4*)acc, n, g, ax, ay, az, nullptr, nullptr, nullptr, 0.0, t, counters, stamp);
  }
}

void nbsp_bh_mlp_pairs(const void* pos4, size_t n, const void* tree, float theta, int opening,
                       unsigned long long seed, int samples, int* target, int* cell, int* status,
                       cudaStream_t stream) {
  Tree t = tree_view(const_cast<void*>(tree), n);
  NBSP_COUNT_LAUNCH(1), mlp_pairs_kernel<<<(samples + 127) / 128, 128, 0, stream>>>(
      (const float4*)pos4, (int)n, t, theta, opening, seed, samples, target, cell, status);
}

void nbsp_bh_mlp_labels(const void* pos4, size_t n, const void* tree, const int* target,
                        const int* cell, int samples, float eps2, float* feat, float* lab, int* ok,
                        cudaStream_t stream) {
  Tree t = tree_view(const_cast<void*>(tree), n);
  const long long threads = (long long)samples * 32;
  NBSP_COUNT_LAUNCH(1), mlp_labels_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(
      (const float4*)pos4, (int)n, t, target, cell, samples, eps2, feat, lab, ok);
}

void nbsp_bh_mlp_stats(const float* feat, const float* lab, const int* ok, int rows, void* net,
                       cudaStream_t stream) {
  NBSP_COUNT_LAUNCH(1), mlp_stats_kernel<<<nbsp_mlp::kIn + nbsp_mlp::kOut, 256, 0, stream>>>(
      feat, lab, ok, rows, (nbsp_mlp::Net*)net);
}

}  // extern "C"
