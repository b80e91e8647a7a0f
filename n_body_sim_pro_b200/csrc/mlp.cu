// Training of the far-field correction MLP on BF16 tensor cores.
//
// Every CTA owns 128 rows of a minibatch (8 warps x 16 rows).  Forward and the
// activation gradients (dH2 = dY W3^T, dH1 = dZ2 W2^T) run on mma.sync m16n8k16
// straight from register fragments; the weight gradients (dW = dZ^T H, a
// contraction over the 128 rows) run on mma.sync as well, from BF16 copies of
// the activations staged in shared memory, read back as transposed fragments by
// ldmatrix.  Each CTA writes its gradient to its own slot; the slots are summed
// in a fixed order (deterministic) for the Adam update of the FP32 master
// weights and of the BF16 fragments.
//
// A step of a small minibatch is bound by latency (1024 rows: 8 CTAs, 3e7 flop),
// so an epoch is one launch instead of three a step: of one cluster up to 8 CTAs,
// a cooperative one up to 32 (4096 rows; beyond, three a step).  With it, the
// ldmatrix fragments and the forward-only losses an epoch of 245,760 rows in
// steps of 1024, its shuffle and losses included, takes 3.1 ms instead of 8.7
// (1.2 of them the shuffle, on the host).
//
// Loss: mean squared error over the 3 outputs of the standardised labels,
// L = 1 / (3 B) sum_r sum_c (y_rc - t_rc)^2.
#include "internal.h"
#include "mlp.cuh"
#include "mlp_umma.cuh"

#include <cuda_runtime.h>
#include <stdint.h>

using namespace nbsp_mlp;

namespace {

constexpr int kRows = 128;  // rows per CTA
constexpr int kWarps = kRows / 16;

struct TrainFrags {
  uint2 w1[kFragW1];
  uint2 w2[kFragW2];
  uint2 w3[kFragW3];
  uint2 w2t[kFragW2T];
  uint2 w3t[kFragW3T];
  float b1[kHidden], b2[kHidden], b3[kOutPad];
};

__device__ __forceinline__ unsigned short bf16_bits(float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  return *reinterpret_cast<const unsigned short*>(&b);
}

// Row strides of the staged BF16 matrices: odd multiples of 16 bytes, so that the
// eight rows of an ldmatrix tile (and store_c's words) lie in different banks.
constexpr int kStrideX = kInPad + 8, kStrideH = kHidden + 8, kStrideY = kOutPad;

__device__ __forceinline__ uint32_t smem_address(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// A fragment of the transpose of a staged row-major matrix m, A[i][k] =
// m[row0 + k][col0 + i] (16 x 16 tile).
__device__ __forceinline__ void load_at(const unsigned short* m, int stride, int row0, int col0,
                                        int lane, uint32_t* a) {
  // tiles in register order: (k 0-7, i 0-7), (k 0-7, i 8-15), (k 8-15, i 0-7), (k 8-15, i 8-15)
  const int row = row0 + (lane & 7) + ((lane >> 4) << 3), col = col0 + (lane & 8);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(smem_address(m + row * stride + col))
               : "memory");
}

// B fragment of a staged row-major matrix m: B[k][n] = m[row0 + k][col0 + n]; for
// an 8-column matrix also the nonzero half (i < 8) of its transpose's A fragment.
__device__ __forceinline__ uint2 load_b(const unsigned short* m, int stride, int row0, int col0,
                                        int lane) {
  uint2 b;
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(b.x), "=r"(b.y)
               : "r"(smem_address(m + (row0 + (lane & 15)) * stride + col0))
               : "memory");
  return b;
}

// Two of them, for columns col0.. and col0 + 8..
__device__ __forceinline__ void load_b2(const unsigned short* m, int stride, int row0, int col0,
                                        int lane, uint2* b) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(b[0].x), "=r"(b[0].y), "=r"(b[1].x), "=r"(b[1].y)
               : "r"(smem_address(m + (row0 + (lane & 15)) * stride + col0 + ((lane >> 4) << 3)))
               : "memory");
}

// Store a 16 x 8 C fragment (rows row0.., cols col0..) as BF16.
__device__ __forceinline__ void store_c(unsigned short* m, int stride, int row0, int col0,
                                        int lane, const float* c) {
  const int g = lane >> 2, t = lane & 3;
  *reinterpret_cast<uint32_t*>(&m[(row0 + g) * stride + col0 + 2 * t]) = pack_bf16(c[0], c[1]);
  *reinterpret_cast<uint32_t*>(&m[(row0 + g + 8) * stride + col0 + 2 * t]) = pack_bf16(c[2], c[3]);
}

struct __align__(16) Stage {
  TrainFrags f;
  unsigned short x[kRows * kStrideX];
  unsigned short h1[kRows * kStrideH];
  unsigned short h2[kRows * kStrideH];
  unsigned short dz1[kRows * kStrideH];
  unsigned short dz2[kRows * kStrideH];
  unsigned short dy[kRows * kStrideY];
  float loss[kWarps];
};

// Threads of a training CTA: warps 0..7 carry the rows through the network (166
// registers: four more warps leave them without spills, eight more do not) and
// share the weight gradients; the last four sum the bias gradients meanwhile.
constexpr int kTrainThreads = 384;
// Floats per gradient slot (whole float4s).
constexpr int kSlot = (kParams + 3) / 4 * 4;

// What a lane feeds the network of its two rows: features and the standardised
// labels of the outputs its C fragment holds.
struct RowInputs {
  uint32_t x[4];
  float label[4];
  bool v0, v1;
};

// order NULL: rows in place.
__device__ __forceinline__ RowInputs load_rows(const uint32_t* __restrict__ x_bf16,
                                               const float* __restrict__ y,
                                               const int* __restrict__ order, int r0,
                                               int rows_total, int lane) {
  const int t = lane & 3, r1 = r0 + 8;
  RowInputs in;
  in.v0 = r0 < rows_total;
  in.v1 = r1 < rows_total;
  const int s0 = in.v0 ? (order != nullptr ? order[r0] : r0) : 0;
  const int s1 = in.v1 ? (order != nullptr ? order[r1] : r1) : 0;
  in.x[0] = in.v0 ? x_bf16[s0 * 8 + t] : 0u;
  in.x[1] = in.v1 ? x_bf16[s1 * 8 + t] : 0u;
  in.x[2] = in.v0 ? x_bf16[s0 * 8 + t + 4] : 0u;
  in.x[3] = in.v1 ? x_bf16[s1 * 8 + t + 4] : 0u;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int col = 2 * t + (q & 1);
    in.label[q] = (q < 2 ? in.v0 : in.v1) && col < kOut ? y[(q < 2 ? s0 : s1) * 3 + col] : 0.f;
  }
  return in;
}

// The 16 rows of one warp through the network and, unless LOSS_ONLY, back: the
// activations and their gradients staged for the weight gradients.  lane 0
// leaves the rows' summed squared error in st.loss[warp].
template <bool LOSS_ONLY>
__device__ __forceinline__ void rows_pass(Stage& st, const RowInputs& in, int warp, int lane,
                                          float inv_batch3) {
  const TrainFrags& f = st.f;
  const int g = lane >> 2, t = lane & 3;
  const int lr = warp * 16;  // local row base
  if (!LOSS_ONLY) {  // stage X (BF16) for dW1
    unsigned int* xs = reinterpret_cast<unsigned int*>(st.x);
    xs[(lr + g) * (kStrideX / 2) + t] = in.x[0];
    xs[(lr + g + 8) * (kStrideX / 2) + t] = in.x[1];
    xs[(lr + g) * (kStrideX / 2) + t + 4] = in.x[2];
    xs[(lr + g + 8) * (kStrideX / 2) + t + 4] = in.x[3];
  }
  // forward, keeping the activations' derivatives
  float g1[8][4], g2[8][4];
  uint32_t h1[16], h2[16];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16(c, in.x, f.w1[nt * 32 + lane]);
    const float bb0 = f.b1[8 * nt + 2 * t], bb1 = f.b1[8 * nt + 2 * t + 1];
    float a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = gelu_with_grad(c[q] + (q & 1 ? bb1 : bb0), g1[nt][q]);
    if (!LOSS_ONLY) store_c(st.h1, kStrideH, lr, 8 * nt, lane, a);
    const int ks = nt >> 1, hi = (nt & 1) * 2;
    h1[4 * ks + hi] = pack_bf16(a[0], a[1]);
    h1[4 * ks + hi + 1] = pack_bf16(a[2], a[3]);
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_bf16(c, &h1[4 * ks], f.w2[(ks * 8 + nt) * 32 + lane]);
    const float bb0 = f.b2[8 * nt + 2 * t], bb1 = f.b2[8 * nt + 2 * t + 1];
    float a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = gelu_with_grad(c[q] + (q & 1 ? bb1 : bb0), g2[nt][q]);
    if (!LOSS_ONLY) store_c(st.h2, kStrideH, lr, 8 * nt, lane, a);
    const int ks = nt >> 1, hi = (nt & 1) * 2;
    h2[4 * ks + hi] = pack_bf16(a[0], a[1]);
    h2[4 * ks + hi + 1] = pack_bf16(a[2], a[3]);
  }
  float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) mma_bf16(out, &h2[4 * ks], f.w3[ks * 32 + lane]);
  // dY = 2 (y - t) / (3 B) on the 3 real outputs of valid rows
  float dy[4];
  float lsum = 0.f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int col = 2 * t + (q & 1);
    const bool row_ok = q < 2 ? in.v0 : in.v1;
    float d = 0.f;
    if (row_ok && col < kOut) {
      const float e = out[q] + f.b3[col] - in.label[q];
      lsum += e * e;
      d = 2.f * e * inv_batch3;
    }
    dy[q] = d;
  }
  for (int off = 16; off > 0; off >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
  if (lane == 0) st.loss[warp] = lsum;
  if (LOSS_ONLY) return;
  store_c(st.dy, kStrideY, lr, 0, lane, dy);
  // dH2 = dY W3^T  (K 16 with columns 8..15 zero)
  uint32_t dya[4] = {pack_bf16(dy[0], dy[1]), pack_bf16(dy[2], dy[3]), 0u, 0u};
  uint32_t dz2a[16];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16(c, dya, f.w3t[nt * 32 + lane]);
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) d[q] = c[q] * g2[nt][q];
    store_c(st.dz2, kStrideH, lr, 8 * nt, lane, d);
    const int ks = nt >> 1, hi = (nt & 1) * 2;
    dz2a[4 * ks + hi] = pack_bf16(d[0], d[1]);
    dz2a[4 * ks + hi + 1] = pack_bf16(d[2], d[3]);
  }
  // dH1 = dZ2 W2^T
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_bf16(c, &dz2a[4 * ks], f.w2t[(ks * 8 + nt) * 32 + lane]);
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) d[q] = c[q] * g1[nt][q];
    store_c(st.dz1, kStrideH, lr, 8 * nt, lane, d);
  }
}

__device__ __forceinline__ float bf16_value(unsigned short b) {
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(&b));
}

// After rows_pass of all 128 rows and a barrier: the CTA's gradient into its slot
// `grad`.  Weight gradients on tensor cores, dW = dZ^T H over the 128 rows (8
// k-steps), by the first eight warps: four of dW2's 4 x 8 output tiles (one row of
// them, so that they share dZ2's fragment), one of dW1's 4 x 2 and one of dW3's
// 1 x 8 each, all six sums side by side (one tile after the other the products
// waited for their own sums: 2.0 us of a step instead of 1.4).  The last four
// warps sum the bias columns meanwhile.
__device__ __forceinline__ void weight_gradients(const Stage& st, int warp, int lane, int tid,
                                                 float* __restrict__ grad) {
  const int g = lane >> 2, t = lane & 3;
  if (warp >= kWarps) {
    const int c = tid - kWarps * 32;  // 0..127: columns of dZ1, then of dZ2
    const unsigned short* m = (c < kHidden ? st.dz1 : st.dz2) + (c & (kHidden - 1));
    float s = 0.f;
#pragma unroll 16
    for (int r = 0; r < kRows; ++r) s += bf16_value(m[r * kStrideH]);
    grad[(c < kHidden ? kOffB1 : kOffB2) + (c & (kHidden - 1))] = s;
    if (c < kOut) {
      float sy = 0.f;
#pragma unroll 16
      for (int r = 0; r < kRows; ++r) sy += bf16_value(st.dy[r * kStrideY + c]);
      grad[kOffB3 + c] = sy;
    }
    return;
  }
  const int m2 = warp & 3, n2 = (warp >> 2) * 4;  // dW2[out][in] = sum_r dZ2[r][out] H1[r][in]
  const int m1 = warp >> 1, n1 = warp & 1;        // dW1[out][in] = sum_r dZ1[r][out] X[r][in], in < 10
  const int n3 = warp;                            // dW3[out][in] = sum_r dY[r][out] H2[r][in], out < 3
  float c2[4][4] = {}, c1[4] = {}, c3[4] = {};
#pragma unroll 2
  for (int r = 0; r < kRows; r += 16) {
    uint32_t a2[4], a1[4];
    uint2 b2[4];
    load_at(st.dz2, kStrideH, r, m2 * 16, lane, a2);
    load_b2(st.h1, kStrideH, r, n2 * 8, lane, b2);
    load_b2(st.h1, kStrideH, r, n2 * 8 + 16, lane, b2 + 2);
    load_at(st.dz1, kStrideH, r, m1 * 16, lane, a1);
    const uint2 b1 = load_b(st.x, kStrideX, r, n1 * 8, lane);
    const uint2 y = load_b(st.dy, kStrideY, r, 0, lane);
    const uint2 b3 = load_b(st.h2, kStrideH, r, n3 * 8, lane);
    const uint32_t a3[4] = {y.x, 0u, y.y, 0u};  // A[i][k] = dY[k][i], zero for i >= 8
#pragma unroll
    for (int j = 0; j < 4; ++j) mma_bf16(c2[j], a2, b2[j]);
    mma_bf16(c1, a1, b1);
    mma_bf16(c3, a3, b3);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float* gw = grad + kOffW2 + (m2 * 16 + g) * kHidden + (n2 + j) * 8 + 2 * t;
    *reinterpret_cast<float2*>(gw) = make_float2(c2[j][0], c2[j][1]);
    *reinterpret_cast<float2*>(gw + 8 * kHidden) = make_float2(c2[j][2], c2[j][3]);
  }
  {
    float* gw = grad + kOffW1;
    const int o0 = m1 * 16 + g, i0 = n1 * 8 + 2 * t;
    if (i0 < kIn) gw[o0 * kIn + i0] = c1[0], gw[(o0 + 8) * kIn + i0] = c1[2];
    if (i0 + 1 < kIn) gw[o0 * kIn + i0 + 1] = c1[1], gw[(o0 + 8) * kIn + i0 + 1] = c1[3];
  }
  if (g < kOut) {
    float* gw = grad + kOffW3 + g * kHidden + n3 * 8 + 2 * t;
    gw[0] = c3[0];
    gw[1] = c3[1];
  }
}

// (all of a thread's words in flight at once; another CTA may have written them in
// this launch)
template <int THREADS>
__device__ __forceinline__ void copy_frags(Stage& st, const TrainFrags* f) {
  static_assert(sizeof(TrainFrags) % 16 == 0, "copied as uint4");
  constexpr int kWords = (int)(sizeof(TrainFrags) / 16), kEach = (kWords + THREADS - 1) / THREADS;
  const uint4* src = reinterpret_cast<const uint4*>(f);
  uint4* dst = reinterpret_cast<uint4*>(&st.f);
  uint4 v[kEach];
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int k = (int)threadIdx.x + j * THREADS;
    if (k < kWords) v[j] = __ldcg(src + k);
  }
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int k = (int)threadIdx.x + j * THREADS;
    if (k < kWords) dst[k] = v[j];
  }
}

// One forward/backward: CTA c's rows first_row + 128 c .. of `order` (NULL: rows
// in place), its gradient into slot c of grad, its loss sum into loss_out[c].
__global__ void __launch_bounds__(kTrainThreads, 1) train_step_kernel(
    const uint32_t* __restrict__ x_bf16, const float* __restrict__ y, const int* __restrict__ order,
    int first_row, int rows_total, float inv_batch3, const TrainFrags* __restrict__ f,
    float* __restrict__ grad, float* __restrict__ loss_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Stage& st = *reinterpret_cast<Stage*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  copy_frags<kTrainThreads>(st, f);
  RowInputs in = {};
  if (warp < kWarps)
    in = load_rows(x_bf16, y, order, first_row + blockIdx.x * kRows + warp * 16 + (lane >> 2),
                   rows_total, lane);
  __syncthreads();
  if (warp < kWarps) rows_pass<false>(st, in, warp, lane, inv_batch3);
  __syncthreads();
  weight_gradients(st, warp, lane, tid, grad + (size_t)blockIdx.x * kSlot);
  if (tid == 0) {
    float s = 0.f;
    for (int w = 0; w < kWarps; ++w) s += st.loss[w];
    loss_out[blockIdx.x] = s;
  }
}

// Summed squared errors of 128-row tiles of rows first_row.. (in place), one value
// per tile: the forward half alone.
__global__ void __launch_bounds__(kRows * 2) loss_kernel(
    const uint32_t* __restrict__ x_bf16, const float* __restrict__ y, int first_row, int tiles,
    const TrainFrags* __restrict__ f, float* __restrict__ loss_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Stage& st = *reinterpret_cast<Stage*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  copy_frags<kRows * 2>(st, f);
  __syncthreads();
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const RowInputs in =
        load_rows(x_bf16, y, nullptr, first_row + tile * kRows + warp * 16 + (lane >> 2),
                  first_row + tiles * kRows, lane);
    rows_pass<true>(st, in, warp, lane, 0.f);
    __syncthreads();
    if (tid == 0) {
      float s = 0.f;
      for (int w = 0; w < kWarps; ++w) s += st.loss[w];
      loss_out[tile] = s;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void adam(float gsum, float& param, float& m, float& v, float lr,
                                     float beta1, float beta2, float eps, float bias1,
                                     float bias2) {
  // (the fused forms are written out, so that every kernel rounds alike)
  const float mm = __fmaf_rn(1.f - beta1, gsum, __fmul_rn(beta1, m));
  const float vv = __fmaf_rn(__fmul_rn(1.f - beta2, gsum), gsum, __fmul_rn(beta2, v));
  m = mm;
  v = vv;
  param -= lr * (mm / bias1) / (sqrtf(vv / bias2) + eps);
}

// Parameter p = value in the BF16 fragments (build_fwd and build_bwd place the
// same elements) or the FP32 biases.
__device__ __forceinline__ void put_fragment(uint2* frag, int ntiles, int n, int k,
                                             unsigned short bits) {
  const int kk = k & 15;
  const int e = ((k >> 4) * ntiles + (n >> 3)) * 32 + (n & 7) * 4 + ((kk & 7) >> 1);
  reinterpret_cast<unsigned short*>(&frag[e])[(kk >> 3) * 2 + (kk & 1)] = bits;
}
__device__ __forceinline__ void put_parameter(TrainFrags& f, int p, float value) {
  const unsigned short bits = bf16_bits(value);
  if (p < kOffB1) {
    put_fragment(f.w1, 8, p / kIn, p % kIn, bits);
  } else if (p < kOffW2) {
    f.b1[p - kOffB1] = value;
  } else if (p < kOffB2) {
    const int o = (p - kOffW2) / kHidden, i = (p - kOffW2) % kHidden;
    put_fragment(f.w2, 8, o, i, bits);
    put_fragment(f.w2t, 8, i, o, bits);
  } else if (p < kOffW3) {
    f.b2[p - kOffB2] = value;
  } else if (p < kOffB3) {
    const int o = (p - kOffW3) / kHidden, i = (p - kOffW3) % kHidden;
    put_fragment(f.w3, 1, o, i, bits);
    put_fragment(f.w3t, 8, i, o, bits);
  } else if (p < kParams) {
    f.b3[p - kOffB3] = value;
  }
}

// Wait until all CTAs of the launch have arrived `round` times (their writes
// before are visible after); false when the wait ran out of its polls, and from
// then on at once.
constexpr int kBarrierPolls = 1 << 22;
__device__ __forceinline__ bool grid_arrive_wait(int* arrivals, int* failed, int round, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int seen;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(seen) : "l"(arrivals) : "memory");
    const int target = round * (int)gridDim.x;
    int polls = 0;
    ++seen;
    while (seen < target && ++polls < kBarrierPolls)
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(arrivals) : "memory");
    if (seen < target) atomicExch(failed, 1);
    *s_ok = seen >= target;
  }
  __syncthreads();
  return *s_ok != 0;
}

// The same between the CTAs of one cluster by its hardware barrier (which cannot
// run out): 1.4 us a wait become 0.7 at 8 CTAs.
__device__ __forceinline__ bool epoch_wait(bool one_cluster, int* arrivals, int* failed, int round,
                                           int* s_ok) {
  if (!one_cluster) return grid_arrive_wait(arrivals, failed, round, s_ok);
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  return true;
}

// A step's rows on their way to the warps that carry them: 8 words of BF16
// features, 3 labels, 1 if the row exists.  Rows of 12 words: the eight rows of an
// A fragment's words lie in different banks.  The four warps without rows of their
// own fetch the next step's during a pass (three dependent loads, 1.2 us where
// the pass's warps made them).
constexpr int kRowWords = 12;
__device__ __forceinline__ void fetch_row(uint32_t* rows, int c, const uint32_t* __restrict__ x_bf16,
                                          const float* __restrict__ y,
                                          const int* __restrict__ order, int r, int rows_total) {
  uint32_t* to = rows + c * kRowWords;
  uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a, l = a;
  if (r < rows_total) {
    const int s = order[r];
    const uint4* x = reinterpret_cast<const uint4*>(x_bf16 + (size_t)s * 8);
    a = x[0];
    b = x[1];
    l = make_uint4(__float_as_uint(y[s * 3]), __float_as_uint(y[s * 3 + 1]),
                   __float_as_uint(y[s * 3 + 2]), 1u);
  }
  *reinterpret_cast<uint4*>(to) = a;
  *reinterpret_cast<uint4*>(to + 4) = b;
  *reinterpret_cast<uint4*>(to + 8) = l;
}
__device__ __forceinline__ RowInputs fetched_rows(const uint32_t* rows, int warp, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const uint32_t* r0 = rows + (warp * 16 + g) * kRowWords;
  const uint32_t* r1 = r0 + 8 * kRowWords;
  RowInputs in;
  in.x[0] = r0[t];
  in.x[1] = r1[t];
  in.x[2] = r0[t + 4];
  in.x[3] = r1[t + 4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int col = 2 * t + (q & 1);
    in.label[q] = col < kOut ? __uint_as_float((q < 2 ? r0 : r1)[8 + col]) : 0.f;
  }
  in.v0 = r0[11] != 0u;
  in.v1 = r1[11] != 0u;
  return in;
}

// All the steps of an epoch in one launch (one cluster, or a cooperative launch),
// a CTA per 128 rows of the minibatch.  A step: every CTA's gradient into its slot;
// then every CTA sums all slots for its share of the parameters, in the slots'
// order, updates them and their moments (its own, in shared memory until the end)
// and puts their new BF16 forms into the fragments in global memory; then every
// CTA takes those.
// (Each CTA updating all parameters for itself saves the second wait, but the
// update is division-bound: 6.3 us of a step at 8 CTAs against 2.4, the second wait
// and the copy included.)
// The results go to next_params, next_m and next_v, so that an epoch in which a
// wait ran out leaves what it began with.
// bias: the step's 1 - beta^t for both moments.
constexpr int kEpochCtas = 32;
constexpr int kEpochCluster = 8;  // the largest cluster that every GPU can place
__global__ void __launch_bounds__(kTrainThreads, 1) train_epoch_kernel(
    const uint32_t* __restrict__ x_bf16, const float* __restrict__ y, const int* __restrict__ order,
    int rows_total, int steps, float inv_batch3, TrainFrags* f, float* slots,
    const float* __restrict__ params, const float* __restrict__ m, const float* __restrict__ v,
    float* __restrict__ next_params, float* __restrict__ next_m, float* __restrict__ next_v,
    float lr, float beta1, float beta2, float eps, const float2* __restrict__ bias, int* arrivals,
    int* failed, int one_cluster) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Stage& st = *reinterpret_cast<Stage*>(smem_raw);
  __shared__ int s_ok;
  // this CTA's share of the parameters and moments
  float* own = reinterpret_cast<float*>(smem_raw + sizeof(Stage));
  float *pp = own, *mm = own + kSlot, *vv = own + 2 * kSlot;
  uint32_t* rows = reinterpret_cast<uint32_t*>(own + 3 * kSlot);  // two steps' by parity
  constexpr int kStepRows = kRows * kRowWords;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ctas = gridDim.x, batch = ctas * kRows;
  const int share = (kParams + ctas - 1) / ctas;
  const int first = blockIdx.x * share, last = min(first + share, kParams);
  copy_frags<kTrainThreads>(st, f);
  for (int p = first + tid; p < last; p += kTrainThreads) {
    pp[p] = params[p];
    mm[p] = m[p];
    vv[p] = v[p];
  }
  const int c = tid - kWarps * 32;  // the fetching threads' row
  const int row = blockIdx.x * kRows + c;
  if (c >= 0) fetch_row(rows, c, x_bf16, y, order, row, rows_total);
  __syncthreads();
  for (int step = 0; step < steps; ++step) {
    if (warp < kWarps)
      rows_pass<false>(st, fetched_rows(rows + (step & 1) * kStepRows, warp, lane), warp, lane,
                       inv_batch3);
    else if (step + 1 < steps)
      fetch_row(rows + ((step + 1) & 1) * kStepRows, c, x_bf16, y, order, (step + 1) * batch + row,
                rows_total);
    __syncthreads();
    weight_gradients(st, warp, lane, tid, slots + (size_t)blockIdx.x * kSlot);
    const float2 b = bias[step];
    if (!epoch_wait(one_cluster, arrivals, failed, 2 * step + 1, &s_ok)) return;
    for (int p0 = first + tid; p0 < last; p0 += 2 * kTrainThreads) {  // two at a time
      const int p1 = min(p0 + kTrainThreads, last - 1);
      float gsum[2] = {0.f, 0.f};
#pragma unroll 8
      for (int s = 0; s < ctas; ++s) {
        gsum[0] += __ldcg(slots + (size_t)s * kSlot + p0);
        gsum[1] += __ldcg(slots + (size_t)s * kSlot + p1);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int p = p0 + e * kTrainThreads;
        if (p >= last) break;
        float value = pp[p], mp = mm[p], vp = vv[p];
        adam(gsum[e], value, mp, vp, lr, beta1, beta2, eps, b.x, b.y);
        pp[p] = value;
        mm[p] = mp;
        vv[p] = vp;
        put_parameter(*f, p, value);
      }
    }
    if (!epoch_wait(one_cluster, arrivals, failed, 2 * step + 2, &s_ok)) return;
    copy_frags<kTrainThreads>(st, f);
    __syncthreads();
  }
  for (int p = first + tid; p < last; p += kTrainThreads) {
    next_params[p] = pp[p];
    next_m[p] = mm[p];
    next_v[p] = vv[p];
  }
}

// Sum the per-CTA gradient slots (fixed order) into grad_out; optional Adam.
__global__ void reduce_adam_kernel(const float* __restrict__ partial, int slots,
                                   float* __restrict__ grad_out, float* __restrict__ params,
                                   float* __restrict__ m, float* __restrict__ v, float lr,
                                   float beta1, float beta2, float eps, float bias1, float bias2,
                                   int apply) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kParams) return;
  float gsum = 0.f;
  for (int s = 0; s < slots; ++s) gsum += partial[(size_t)s * kSlot + p];
  if (grad_out != nullptr) grad_out[p] = gsum;
  if (!apply) return;
  adam(gsum, params[p], m[p], v[p], lr, beta1, beta2, eps, bias1, bias2);
}

__device__ __forceinline__ float w_at(const float* w, int out, int in, int outs, int ins) {
  return (out < outs && in < ins) ? w[out * ins + in] : 0.f;
}

// B fragments of B[k][n] = W[n][k]  (forward: K = inputs, N = outputs)
__device__ void build_fwd(uint2* frag, const float* w, int outs, int ins, int ksteps, int ntiles) {
  for (int e = threadIdx.x; e < ksteps * ntiles * 32; e += blockDim.x) {
    const int lane = e & 31, tile = e >> 5;
    const int ks = tile / ntiles, nt = tile % ntiles;
    const int g = lane >> 2, t = lane & 3;
    const int n = nt * 8 + g, k = ks * 16 + 2 * t;
    frag[e] = make_uint2(pack_bf16(w_at(w, n, k, outs, ins), w_at(w, n, k + 1, outs, ins)),
                         pack_bf16(w_at(w, n, k + 8, outs, ins), w_at(w, n, k + 9, outs, ins)));
  }
}

// B fragments of B[k][n] = W[k][n]  (backward: K = outputs of the layer, N = inputs)
__device__ void build_bwd(uint2* frag, const float* w, int outs, int ins, int ksteps, int ntiles) {
  for (int e = threadIdx.x; e < ksteps * ntiles * 32; e += blockDim.x) {
    const int lane = e & 31, tile = e >> 5;
    const int ks = tile / ntiles, nt = tile % ntiles;
    const int g = lane >> 2, t = lane & 3;
    const int n = nt * 8 + g, k = ks * 16 + 2 * t;
    frag[e] = make_uint2(pack_bf16(w_at(w, k, n, outs, ins), w_at(w, k + 1, n, outs, ins)),
                         pack_bf16(w_at(w, k + 8, n, outs, ins), w_at(w, k + 9, n, outs, ins)));
  }
}

__global__ void build_frags_kernel(const float* __restrict__ params, TrainFrags* f, Net* net) {
  build_fwd(f->w1, params + kOffW1, kHidden, kIn, 1, 8);
  build_fwd(f->w2, params + kOffW2, kHidden, kHidden, 4, 8);
  build_fwd(f->w3, params + kOffW3, kOut, kHidden, 4, 1);
  build_bwd(f->w2t, params + kOffW2, kHidden, kHidden, 4, 8);
  build_bwd(f->w3t, params + kOffW3, kOut, kHidden, 1, 8);
  for (int i = threadIdx.x; i < kHidden; i += blockDim.x) {
    f->b1[i] = params[kOffB1 + i];
    f->b2[i] = params[kOffB2 + i];
  }
  for (int i = threadIdx.x; i < kOutPad; i += blockDim.x) f->b3[i] = i < kOut ? params[kOffB3 + i] : 0.f;
  __syncthreads();
  if (net != nullptr) {
    for (int e = threadIdx.x; e < kFragW1; e += blockDim.x) net->w1[e] = f->w1[e];
    for (int e = threadIdx.x; e < kFragW2; e += blockDim.x) net->w2[e] = f->w2[e];
    for (int e = threadIdx.x; e < kFragW3; e += blockDim.x) net->w3[e] = f->w3[e];
    for (int i = threadIdx.x; i < kHidden; i += blockDim.x) {
      net->b1[i] = f->b1[i];
      net->b2[i] = f->b2[i];
    }
    for (int i = threadIdx.x; i < kOutPad; i += blockDim.x) net->b3[i] = f->b3[i];
    nbsp_umma::build_weights(params, reinterpret_cast<nbsp_umma::Weights*>(net->umma_w));
  }
}

// The network on raw feature rows (10 per row): standardised, through the
// three layers, de-standardised into out (3 per row).  tcgen05 path: one
// 128-row tile per iteration of a persistent CTA.
__global__ void __launch_bounds__(nbsp_umma::kThreads) evaluate_umma_kernel(
    const Net* __restrict__ net, const float* __restrict__ feat, int rows,
    float* __restrict__ out, int* status) {
  extern __shared__ __align__(128) unsigned char umma_smem[];
  nbsp_umma::Smem& s = *reinterpret_cast<nbsp_umma::Smem*>(umma_smem);
  nbsp_umma::setup(s, nbsp_umma::weights_of(net), net);
  const uint32_t tmem = s.tmem;
  uint32_t phase = 0;
  const int tiles = (rows + nbsp_umma::kRows - 1) / nbsp_umma::kRows;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int r = tile * nbsp_umma::kRows + threadIdx.x;
    float v[kIn];
#pragma unroll
    for (int q = 0; q < kIn; ++q)
      v[q] = r < rows ? (feat[(size_t)r * kIn + q] - net->x_mean[q]) * net->x_inv_std[q] : 0.f;
    nbsp_umma::put_inputs(s, v);
    nbsp_umma::fence_async_smem();
    __syncthreads();
    float y[3];
    if (!nbsp_umma::forward(s, tmem, phase, y)) {
      if (threadIdx.x == 0) atomicOr(status, NBSP_DEVICE_ERROR_MMA_TIMEOUT);
      break;
    }
    if (r < rows)
      for (int c = 0; c < kOut; ++c)
        out[(size_t)r * kOut + c] = fmaf(y[c], net->y_std[c], net->y_mean[c]);
  }
  nbsp_umma::teardown(s, tmem);
}

// The same with mma.sync: one warp per 16 rows (the corrected walk's former
// per-warp path, kept as the cross-check of the tcgen05 one).
__global__ void evaluate_sync_kernel(const Net* __restrict__ net, const float* __restrict__ feat,
                                     int rows, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (tile * 16 >= rows) return;
  const int g = lane >> 2, t = lane & 3;
  auto val = [&](int row, int q) -> float {
    const int r = tile * 16 + row;
    return (r < rows && q < kIn) ? (feat[(size_t)r * kIn + q] - net->x_mean[q]) * net->x_inv_std[q]
                                 : 0.f;
  };
  const uint32_t x[4] = {pack_bf16(val(g, 2 * t), val(g, 2 * t + 1)),
                         pack_bf16(val(g + 8, 2 * t), val(g + 8, 2 * t + 1)),
                         pack_bf16(val(g, 2 * t + 8), val(g, 2 * t + 9)),
                         pack_bf16(val(g + 8, 2 * t + 8), val(g + 8, 2 * t + 9))};
  float o[4];
  forward_tile(x, net->w1, net->b1, net->w2, net->b2, net->w3, net->b3, lane, o);
  // o: C[g][2t], C[g][2t+1], C[g+8][2t], C[g+8][2t+1]; outputs are columns 0..2
  for (int h = 0; h < 2; ++h) {
    const int r = tile * 16 + g + 8 * h;
    for (int k = 0; k < 2; ++k) {
      const int c = 2 * t + k;
      if (r < rows && c < kOut) out[(size_t)r * kOut + c] = fmaf(o[2 * h + k], net->y_std[c], net->y_mean[c]);
    }
  }
}

// Standardise raw features / labels into the training layout.
__global__ void standardise_kernel(const float* __restrict__ feat, const float* __restrict__ lab,
                                   int rows, const Net* __restrict__ net, uint32_t* __restrict__ x,
                                   float* __restrict__ y) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  float v[kInPad];
  for (int i = 0; i < kInPad; ++i)
    v[i] = i < kIn ? (feat[r * kIn + i] - net->x_mean[i]) * net->x_inv_std[i] : 0.f;
  for (int w = 0; w < 8; ++w) x[r * 8 + w] = pack_bf16(v[2 * w], v[2 * w + 1]);
  for (int c = 0; c < kOut; ++c) y[r * 3 + c] = (lab[r * 3 + c] - net->y_mean[c]) / net->y_std[c];
}

}  // namespace

extern "C" {

size_t nbsp_mlp_net_bytes(void) { return sizeof(Net); }

// Scaling table: x_mean[10], x_inv_std[10], x_min[10], x_max[10], y_mean[3], y_std[3],
// contiguous in Net from x_mean on.
static_assert(offsetof(Net, y_std) + sizeof(float) * kOut - offsetof(Net, x_mean) ==
                  sizeof(float) * 46, "scaling table layout");

void nbsp_mlp_set_scaling(void* net, const float* table, cudaStream_t stream) {
  cudaMemcpyAsync(static_cast<char*>(net) + offsetof(Net, x_mean), table, 46 * sizeof(float),
                  cudaMemcpyDeviceToDevice, stream);
}

void nbsp_mlp_get_scaling(const void* net, float* table, cudaStream_t stream) {
  cudaMemcpyAsync(table, static_cast<const char*>(net) + offsetof(Net, x_mean), 46 * sizeof(float),
                  cudaMemcpyDeviceToDevice, stream);
}
size_t nbsp_mlp_frags_bytes(void) { return sizeof(TrainFrags); }
int nbsp_mlp_param_count(void) { return kParams; }
int nbsp_mlp_rows_per_cta(void) { return kRows; }
int nbsp_mlp_slot_floats(void) { return kSlot; }
int nbsp_mlp_epoch_ctas(void) { return kEpochCtas; }

void nbsp_mlp_build_frags(const float* params, void* frags, void* net, cudaStream_t stream) {
  NBSP_COUNT_LAUNCH(1), build_frags_kernel<<<1, 256, 0, stream>>>(params, (TrainFrags*)frags,
                                                                   (Net*)net);
}

void nbsp_mlp_standardise(const float* feat, const float* lab, int rows, const void* net,
                          uint32_t* x, float* y, cudaStream_t stream) {
  NBSP_COUNT_LAUNCH(1), standardise_kernel<<<(rows + 255) / 256, 256, 0, stream>>>(
      feat, lab, rows, (const Net*)net, x, y);
}

// One forward/backward over rows [first_row, first_row + ctas * 128) of `order`
// (NULL: rows in place); per-CTA gradients into partial[ctas][slot floats],
// per-CTA loss sums into loss.
void nbsp_mlp_train_step(const uint32_t* x, const float* y, const int* order, int first_row,
                         int rows_total, int ctas, float inv_batch3, const void* frags,
                         float* partial, float* loss, cudaStream_t stream) {
  const int smem = (int)sizeof(Stage);
  cudaFuncSetAttribute(train_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  NBSP_COUNT_LAUNCH(1), train_step_kernel<<<ctas, kTrainThreads, smem, stream>>>(
      x, y, order, first_row, rows_total, inv_batch3, (const TrainFrags*)frags, partial, loss);
}

// The loss sums of `tiles` 128-row tiles from first_row on, in place.
void nbsp_mlp_loss(const uint32_t* x, const float* y, int first_row, int tiles, const void* frags,
                   float* loss, cudaStream_t stream) {
  const int smem = (int)sizeof(Stage);
  cudaFuncSetAttribute(loss_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int grid = tiles < 2 * 148 ? tiles : 2 * 148;  // two CTAs of ~105 KB per SM
  NBSP_COUNT_LAUNCH(1), loss_kernel<<<grid, kRows * 2, smem, stream>>>(
      x, y, first_row, tiles, (const TrainFrags*)frags, loss);
}

static const float kBeta1 = 0.9f, kBeta2 = 0.999f, kAdamEps = 1e-8f;

// 1 - beta^step of both moments.
void nbsp_mlp_adam_bias(int step, float* bias) {
  bias[0] = 1.f - powf(kBeta1, (float)step);
  bias[1] = 1.f - powf(kBeta2, (float)step);
}

// `steps` minibatches of ctas * 128 rows of `order` from its start, forward,
// backward and Adam, in one launch (ctas <= nbsp_mlp_epoch_ctas()); slots: ctas
// gradient slots; bias: steps pairs of nbsp_mlp_adam_bias on the device; sync: two
// zeroed ints, the second nonzero when a wait ran out (next_params, next_m and next_v
// are then in part).  The fragments in `frags` follow the parameters; the inference
// network is not touched.
int nbsp_mlp_train_epoch(const uint32_t* x, const float* y, const int* order, int rows_total,
                         int steps, int ctas, float inv_batch3, void* frags, float* slots,
                         const float* params, const float* m, const float* v, float* next_params,
                         float* next_m, float* next_v, float lr, const void* bias, int* sync,
                         cudaStream_t stream) {
  const int smem =
      (int)(sizeof(Stage) + 3 * kSlot * sizeof(float) + 2 * kRows * kRowWords * sizeof(uint32_t));
  cudaFuncSetAttribute(train_epoch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  TrainFrags* f = (TrainFrags*)frags;
  const float2* b = (const float2*)bias;
  float beta1 = kBeta1, beta2 = kBeta2, eps = kAdamEps;
  int* failed = sync + 1;
  int one_cluster = ctas <= kEpochCluster;
  void* args[] = {&x, &y, &order, &rows_total, &steps, &inv_batch3, &f, &slots, &params, &m, &v,
                  &next_params, &next_m, &next_v, &lr, &beta1, &beta2, &eps, &b, &sync, &failed,
                  &one_cluster};
  cudaLaunchAttribute how;
  if (one_cluster) {
    how.id = cudaLaunchAttributeClusterDimension;
    how.val.clusterDim.x = (unsigned)ctas;
    how.val.clusterDim.y = how.val.clusterDim.z = 1;
  } else {
    how.id = cudaLaunchAttributeCooperative;
    how.val.cooperative = 1;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)ctas);
  config.blockDim = dim3(kTrainThreads);
  config.dynamicSmemBytes = (size_t)smem;
  config.stream = stream;
  config.attrs = &how;
  config.numAttrs = 1;
  NBSP_COUNT_LAUNCH(1);
  return (int)cudaLaunchKernelExC(&config, (const void*)train_epoch_kernel, args);
}

void nbsp_mlp_evaluate(const void* net, const float* feat, int rows, float* out, int tcgen05,
                       int* status, cudaStream_t stream) {
  if (rows <= 0) return;
  if (tcgen05) {
    const int smem = (int)sizeof(nbsp_umma::Smem);
    cudaFuncSetAttribute(evaluate_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const int tiles = (rows + nbsp_umma::kRows - 1) / nbsp_umma::kRows;
    const int cap = 148 * nbsp_umma::kCtasPerSm;
    const int grid = tiles < cap ? tiles : cap;
    NBSP_COUNT_LAUNCH(1), evaluate_umma_kernel<<<grid, nbsp_umma::kThreads, smem, stream>>>(
        (const Net*)net, feat, rows, out, status);
  } else {
    const int warps = (rows + 15) / 16;
    NBSP_COUNT_LAUNCH(1), evaluate_sync_kernel<<<(warps + 3) / 4, 128, 0, stream>>>(
        (const Net*)net, feat, rows, out);
  }
}

void nbsp_mlp_reduce_adam(const float* partial, int slots, float* grad_out, float* params, float* m,
                          float* v, float lr, int step, int apply, cudaStream_t stream) {
  float bias[2];
  nbsp_mlp_adam_bias(step, bias);
  NBSP_COUNT_LAUNCH(1), reduce_adam_kernel<<<(kParams + 255) / 256, 256, 0, stream>>>(
      partial, slots, grad_out, params, m, v, lr, kBeta1, kBeta2, kAdamEps, bias[0], bias[1], apply);
}

}  // extern "C"
