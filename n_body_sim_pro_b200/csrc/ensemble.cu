// Ensembles of many small, independent systems in one persistent launch.
//
// Each system evolves under its own softened all-pairs gravity
// (src/c/physics/gravity.c:37-67 arithmetic, FP32 with compensated sums on
// positions relative to the system's FP64 centre of mass) with leapfrog KDK
// (src/c/physics/integrator.c:47-85, FP64 state).
//
// Scheduling: the host bundles systems of about the same size into work items of
// at most kCap particle slots, gives each system of an item the same number of
// warps, and orders the items by their time, longest first.  The grid is one
// resident wave; each CTA takes the next item from an atomic counter and runs ALL
// the requested steps of its systems before it takes another, so no grid-wide
// synchronisation is ever needed.
//
// A step's pair sums are bound by the FP32 pipe, so what matters is that its four
// quarters have the same work.  A system of T tiles (64 particles) is T x T
// tile pairs, 64 targets by 64 sources each; its warps take equal runs of them in
// target order, so that a tile of targets is shared by two warps at most (no
// more warps than tiles).  The second one goes on with the first one's sums, which
// the first one makes before anything else, so the cut changes no bit and the
// wait costs nothing (68.4 ms a call either way; adding the parts after a barrier
// let a system's bits depend on its neighbours).  With whole targets per thread
// instead (four of them, the system's threads rounded up to warps) a system of
// 2,100 particles ran on 17 warps, five of them on one quarter of the SM.  Sums
// wait in shared memory for the update pass, so a lane holds two targets and no
// spills.  Measured on 4096 systems of 32 to 4096 particles (3.4M, 7.1e9 pairs a
// step), 21 evaluations: 70.4 -> 63.3 ms (2.1e12 -> 2.4e12 pairs / s, 63% of the FP32
// peak in 20-flop pairs, of which the 12 instructions per pair allow 83%).  The
// tile's loop fully unrolled: 16 sources at a time 64.2, 4 at a time 65.9.
#include "internal.h"

#include <cuda_runtime.h>
#include <stdint.h>

namespace {

__device__ __forceinline__ float rsqrt_mufu(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Paired FP32 (sm_100 .f32x2): two targets share every add / mul / fma.
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

__device__ __forceinline__ void fold(float& hi, float& lo, float a) {
  const float s = __fadd_rn(hi, a);
  const float bp = __fsub_rn(s, hi);
  const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(a, bp));
  hi = s;
  lo = __fadd_rn(lo, err);
}

struct EnsembleArgs {
  double *x, *y, *z, *vx, *vy, *vz, *ax, *ay, *az;
  const double* m;
  const long long* offset;  // [systems + 1]
  const double* centre;     // [systems * 3]
  const int* item_start;    // [items + 1] into item_systems
  const int* item_systems;
  const int* item_slot;     // first particle slot of the system, parallel to item_systems
  const int* item_warps;    // warps per system of the item
  int items;
  int* counter;
  int* status;
  double g, h, dt;
  float eps2;
  int steps;
};

constexpr int kTile = 64;         // sources per compensated fold
constexpr float kFarAway = 1e30f;  // padding sources: r^2 overflows to inf, rsqrt(inf) = 0

constexpr int kCap = 4096;         // particle slots of a CTA (a system's are whole tiles)
constexpr int kSmemBytes = kCap * (2 * (int)sizeof(float4) + 3 * (int)sizeof(double));

// A target tile whose sources two warps share: the first one leaves its (hi, lo)
// sums where the tile's FP64 sums will be, the second one folds its sources into
// them, so that every target has one chain of folds over all tiles in order and
// its bits do not depend on where the cut lies.
__device__ __forceinline__ double pack_sum(float hi, float lo) {
  return __hiloint2double(__float_as_int(hi), __float_as_int(lo));
}
__device__ __forceinline__ void unpack_sum(double v, float& hi, float& lo) {
  hi = __int_as_float(__double2hiint(v));
  lo = __int_as_float(__double2loint(v));
}
__device__ __forceinline__ void sums_begun(unsigned* begun, unsigned turn, int lane) {
  __syncwarp();  // the warp's sums, then the word
  if (lane == 0)
    asm volatile("st.release.cta.shared.u32 [%0], %1;"
                 :: "r"((unsigned)__cvta_generic_to_shared(begun)), "r"(turn)
                 : "memory");
}
// False when the other warp's word did not come within the polls (it is the first
// thing that warp does in a step and waits for nothing).
constexpr int kTurnPolls = 1 << 22;
__device__ __forceinline__ bool wait_for_sums(const unsigned* begun, unsigned turn, int lane) {
  bool there = true;
  if (lane == 0) {
    unsigned seen = 0;
    for (int polls = 0; polls < kTurnPolls && seen != turn; ++polls)
      asm volatile("ld.acquire.cta.shared.u32 %0, [%1];"
                   : "=r"(seen)
                   : "r"((unsigned)__cvta_generic_to_shared(begun))
                   : "memory");
    there = seen == turn;
  }
  __syncwarp();
  return there;
}

// GUARD: drop r^2 = 0 terms (eps = 0, or m / eps^3 could overflow); otherwise
// a target's own entry has d = 0 and adds W * 0 = 0.
template <int BLOCK, bool GUARD>
__global__ void __launch_bounds__(BLOCK, 1) ensemble_kernel(EnsembleArgs a) {
  // kCap particles, each as two float4 (x, x, y, y), (z, z, m, m): one 16-byte
  // load yields the broadcast operands of two paired instructions; then their
  // accelerations / G
  extern __shared__ float4 sp[];
  double* const acc = reinterpret_cast<double*>(sp + 2 * kCap);
  __shared__ int s_item;
  __shared__ unsigned s_begun[BLOCK / 32];  // the last step whose shared tile a warp has begun
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned turn = 0;  // steps of this CTA, of all its items
  if (tid < BLOCK / 32) s_begun[tid] = 0;
  for (int guard = 0;; ++guard) {
    if (guard > a.items) {  // each CTA takes each item at most once
      if (tid == 0) atomicOr(a.status, NBSP_DEVICE_ERROR_ENSEMBLE_LIMIT);
      break;
    }
    __syncthreads();
    if (tid == 0) s_item = atomicAdd(a.counter, 1);
    __syncthreads();
    const int w = s_item;
    if (w >= a.items) break;
    const int warps = max(a.item_warps[w], 1);
    const int first = a.item_start[w];
    const int count = a.item_start[w + 1] - first;
    const int sub = warp / warps, lw = warp % warps;
    const bool has = sub < count;
    const int sys = has ? a.item_systems[first + sub] : 0;
    const int slot = has ? a.item_slot[first + sub] : 0;
    const long long off = has ? a.offset[sys] : 0;
    int n = has ? (int)(a.offset[sys + 1] - off) : 0;
    int tiles = (n + kTile - 1) / kTile;
    if (slot < 0 || slot + tiles * kTile > kCap || warps > max(tiles, 1)) {
      if (has) {  // the host packs the slots so this cannot happen
        if (lane == 0) atomicOr(a.status, NBSP_DEVICE_ERROR_ENSEMBLE_LIMIT);
        n = tiles = 0;
      }
    }
    float4* const pos = sp + 2 * slot;  // particle i at pos[2 i], pos[2 i + 1]
    double *const sx = acc + slot, *const sy = sx + kCap, *const sz = sy + kCap;
    const double cx = has ? a.centre[3 * sys] : 0.0;
    const double cy = has ? a.centre[3 * sys + 1] : 0.0;
    const double cz = has ? a.centre[3 * sys + 2] : 0.0;
    // whole tiles: massless far sources behind the last particle
    for (int i = lw * 32 + lane; i < tiles * kTile; i += warps * 32) {
      float px = kFarAway, py = kFarAway, pz = kFarAway, pm = 0.f;
      if (i < n) {
        const long long p = off + i;
        px = (float)__dsub_rn(a.x[p], cx);
        py = (float)__dsub_rn(a.y[p], cy);
        pz = (float)__dsub_rn(a.z[p], cz);
        pm = (float)a.m[p];
      }
      pos[2 * i] = make_float4(px, px, py, py);
      pos[2 * i + 1] = make_float4(pz, pz, pm, pm);
    }
    __syncthreads();
    const unsigned long long E2 = pack2(a.eps2, a.eps2);
    // this warp's run of the system's tile pairs: the sources from tile j0 on of the
    // first target tile, whole target tiles, the sources before tile j1 of the last
    const int begin = tiles * tiles * lw / warps, end = tiles * tiles * (lw + 1) / warps;
    const int t0 = tiles > 0 ? begin / tiles : 0, j0 = begin - t0 * tiles;
    const int t1 = tiles > 0 ? end / tiles : 0, j1 = end - t1 * tiles;
    for (int step = 0; step <= a.steps; ++step) {
      ++turn;
      // the last first: the tile that the next warp goes on with is begun at once,
      // the one that the warp before began comes at the end
      for (int target = begin == end ? -1 : j1 > 0 ? t1 : t1 - 1; target >= t0; --target) {
        const bool whole = target < t1;  // to the last source
        const int i0 = target * kTile + lane;
        int j = 0;
        float hx[2], hy[2], hz[2], lx[2], ly[2], lz[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) hx[k] = hy[k] = hz[k] = lx[k] = ly[k] = lz[k] = 0.f;
        if (target == t0 && j0 > 0) {
          j = j0;
          if (!wait_for_sums(&s_begun[warp - 1], turn, lane) && lane == 0)
            atomicOr(a.status, NBSP_DEVICE_ERROR_ENSEMBLE_LIMIT);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            unpack_sum(sx[i0 + 32 * k], hx[k], lx[k]);
            unpack_sum(sy[i0 + 32 * k], hy[k], ly[k]);
            unpack_sum(sz[i0 + 32 * k], hz[k], lz[k]);
          }
        }
        const float4 u0 = pos[2 * i0], u1 = pos[2 * i0 + 1];
        const float4 v0 = pos[2 * (i0 + 32)], v1 = pos[2 * (i0 + 32) + 1];
        const unsigned long long X = pack2(u0.x, v0.x), Y = pack2(u0.z, v0.z), Z = pack2(u1.x, v1.x);
        const ulonglong2* src = reinterpret_cast<const ulonglong2*>(pos + 2 * j * kTile);
        for (const int stop = whole ? tiles : j1; j < stop; ++j) {
          unsigned long long AX = 0ull, AY = 0ull, AZ = 0ull;
#pragma unroll
          for (int k = 0; k < kTile; ++k) {
            const ulonglong2 s0 = src[2 * k], s1 = src[2 * k + 1];
            const unsigned long long dx = sub2(s0.x, X), dy = sub2(s0.y, Y), dz = sub2(s1.x, Z);
            const unsigned long long r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, E2)));
            float r2a, r2b;
            unpack2(r2, r2a, r2b);
            float ra = rsqrt_mufu(r2a), rb = rsqrt_mufu(r2b);
            if (GUARD) {  // the self pair (r^2 = 0 when eps = 0) contributes 0
              ra = r2a > 0.f ? ra : 0.f;
              rb = r2b > 0.f ? rb : 0.f;
            }
            const unsigned long long R = pack2(ra, rb);
            const unsigned long long W = mul2(s1.y, mul2(mul2(R, R), R));
            AX = fma2(W, dx, AX);
            AY = fma2(W, dy, AY);
            AZ = fma2(W, dz, AZ);
          }
          src += 2 * kTile;
          float u, v;
          unpack2(AX, u, v);
          fold(hx[0], lx[0], u);
          fold(hx[1], lx[1], v);
          unpack2(AY, u, v);
          fold(hy[0], ly[0], u);
          fold(hy[1], ly[1], v);
          unpack2(AZ, u, v);
          fold(hz[0], lz[0], u);
          fold(hz[1], lz[1], v);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          sx[i0 + 32 * k] = whole ? (double)hx[k] + (double)lx[k] : pack_sum(hx[k], lx[k]);
          sy[i0 + 32 * k] = whole ? (double)hy[k] + (double)ly[k] : pack_sum(hy[k], ly[k]);
          sz[i0 + 32 * k] = whole ? (double)hz[k] + (double)lz[k] : pack_sum(hz[k], lz[k]);
        }
        if (!whole) sums_begun(&s_begun[warp], turn, lane);
      }
      __syncthreads();
      for (int i = lw * 32 + lane; i < n; i += warps * 32) {
        const long long p = off + i;
        const double a0 = a.g * sx[i], a1 = a.g * sy[i], a2 = a.g * sz[i];
        a.ax[p] = a0;
        a.ay[p] = a1;
        a.az[p] = a2;
        double u = a.vx[p], v = a.vy[p], wv = a.vz[p];
        if (step > 0) {  // closing half kick of step `step`
          u = __dadd_rn(u, __dmul_rn(a0, a.h));
          v = __dadd_rn(v, __dmul_rn(a1, a.h));
          wv = __dadd_rn(wv, __dmul_rn(a2, a.h));
        }
        if (step < a.steps) {  // opening half kick + drift of step `step + 1`
          u = __dadd_rn(u, __dmul_rn(a0, a.h));
          v = __dadd_rn(v, __dmul_rn(a1, a.h));
          wv = __dadd_rn(wv, __dmul_rn(a2, a.h));
          const double nx = __dadd_rn(a.x[p], __dmul_rn(u, a.dt));
          const double ny = __dadd_rn(a.y[p], __dmul_rn(v, a.dt));
          const double nz = __dadd_rn(a.z[p], __dmul_rn(wv, a.dt));
          a.x[p] = nx;
          a.y[p] = ny;
          a.z[p] = nz;
          const float px = (float)__dsub_rn(nx, cx), py = (float)__dsub_rn(ny, cy);
          const float pz = (float)__dsub_rn(nz, cz);
          pos[2 * i] = make_float4(px, px, py, py);
          *reinterpret_cast<float2*>(&pos[2 * i + 1]) = make_float2(pz, pz);
        }
        a.vx[p] = u;
        a.vy[p] = v;
        a.vz[p] = wv;
      }
      __syncthreads();  // the positions are in place, the sums read
    }
  }
}

typedef void (*EnsembleKernel)(EnsembleArgs);

EnsembleKernel select(int block, bool guard) {
  if (block == 1024) return guard ? ensemble_kernel<1024, true> : ensemble_kernel<1024, false>;
  if (block == 768) return guard ? ensemble_kernel<768, true> : ensemble_kernel<768, false>;
  if (block == 512) return guard ? ensemble_kernel<512, true> : ensemble_kernel<512, false>;
  return nullptr;
}

}  // namespace

extern "C" {

int nbsp_ensemble_resident_ctas(int block) {
  EnsembleKernel k = select(block, true);
  if (k == nullptr) return 0;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  int ctas = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, k, block, kSmemBytes) != cudaSuccess)
    return 0;
  return ctas;
}

void nbsp_ensemble_advance(int block, int grid, double* x, double* y, double* z, double* vx,
                           double* vy, double* vz, double* ax, double* ay, double* az,
                           const double* m, const long long* offset, const double* centre,
                           const int* item_start, const int* item_systems, const int* item_slot,
                           const int* item_warps, int items, int* counter, int* status, double g,
                           float eps2, double dt, int steps, int guard, cudaStream_t stream) {
  EnsembleKernel k = select(block, guard != 0);
  if (k == nullptr) return;
  EnsembleArgs a;
  a.x = x;
  a.y = y;
  a.z = z;
  a.vx = vx;
  a.vy = vy;
  a.vz = vz;
  a.ax = ax;
  a.ay = ay;
  a.az = az;
  a.m = m;
  a.offset = offset;
  a.centre = centre;
  a.item_start = item_start;
  a.item_systems = item_systems;
  a.item_slot = item_slot;
  a.item_warps = item_warps;
  a.items = items;
  a.counter = counter;
  a.status = status;
  a.g = g;
  a.h = 0.5 * dt;
  a.dt = dt;
  a.eps2 = eps2;
  a.steps = steps;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  NBSP_COUNT_LAUNCH(1), k<<<grid, block, kSmemBytes, stream>>>(a);
}

}  // extern "C"
