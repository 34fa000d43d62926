// Training kernels of the spectrum surrogate.
//
// The members of an ensemble are independent, so a step runs a group of them
// at once: every kernel takes G members ("slots" 0..G-1 of the group, members
// m0..m0+G-1 of the ensemble), every activation buffer is [G][rows][256].
// One member alone fills neither the SMs (128 row tiles of a 16,384-row batch)
// nor hides the launches: 27 launches and 410 us a step and member at 16,384
// rows, now 21 launches and 125 us a member for a group of five (200,000 rows,
// 2 epochs: 49.2 -> 15.8 ms).
//
// All operands are row-major in HBM, written once:
//   forward   Z_l  = X_{l-1} W_l^T    A = X_{l-1} [rows x in]   (K-major)  B = W_l   [256 x in]
//   dX        dH_{l-1} = dH_l W_l * SiLU'(Z_{l-1})  A = dH_l    (K-major)  B = W_l^T [in x 256]
//   dW        dW_l = dH_l^T X_{l-1}   A = dH_l, B = X_{l-1}, both read MN-major (the
//             reduction runs over the rows), so no transposed copy is written
// Weight gradients are split over the batch into FP32 partials of 256 rows,
// added in their order; bias and head gradients are sums over the rows of one
// class modulo 256, added by a fixed tree: a gradient is deterministic and
// does not depend on the group it is computed in.
#pragma once
#include "mlp_kernels.cuh"

namespace gelio {
namespace mlp {

constexpr int kMaxMembers = 16;
constexpr int kClasses = 256;     // row classes of the bias and head gradients
constexpr int kSplitRows = 256;   // batch rows of one dW partial
constexpr int kHeadRows = 128;    // rows of one loss partial

enum TrainMode { FWD = 0, FWD_LAST = 1, DX = 2, DW = 3 };

struct TrainArgs {
  int rows;                 // batch rows (a multiple of 256)
  int G;                    // members in this launch
  int m0;                   // first member (weights, parameters)
  int N;                    // GEMM columns: 256, or 64 for the first layer's DW
  int K;                    // layer fan-in (FWD*: 64 or 256, DX: 256); DW: kSplitRows
  const float *P[kMaxMembers];   // FP32 parameters by slot
  int off_bias;
  __nv_bfloat16 *z_out;     // FWD*: pre-activations
  __nv_bfloat16 *x_out;     // FWD*: activations
  float *y_out;             // FWD_LAST: head outputs [G][rows], zeroed before
  const __nv_bfloat16 *z_prev;   // DX
  __nv_bfloat16 *dh_out;    // DX
  float *partial;           // DW: [G][rows / 256][N][256]
  unsigned *error;
  unsigned long long timeout_ns;
};

// Columns [32 c_begin, 32 c_end) of one accumulator row (row = row0 + lane of
// the slot's batch); returns this thread's part of the head's dot product.
template <int MODE>
__device__ __forceinline__ float train_epilogue(const TrainArgs &a, size_t row, uint32_t trow, float *part, int c_begin,
                                                int c_end, unsigned char *stage, int lane, const float *sbias,
                                                const float *sw5) {
  const size_t row0 = row - lane;
  float ysum = 0.0f;
  for (int c = c_begin; c < c_end; ++c) {
    const int n0 = c * 32;
    __align__(16) __nv_bfloat16 zp[32];
    if constexpr (MODE == DX) {
      const uint4 *src = reinterpret_cast<const uint4 *>(a.z_prev + row * kWidth + n0);
#pragma unroll
      for (int q = 0; q < 4; ++q) reinterpret_cast<uint4 *>(zp)[q] = src[q];
    }
    float v[32];
    tc::tmem_ld32(trow + (uint32_t)(c * 32), v);     // warp-wide: every lane executes it
    if constexpr (MODE == DW) {
      float *p = part + (size_t)n0 * kWidth;
#pragma unroll
      for (int j = 0; j < 32; ++j) p[(size_t)j * kWidth] = v[j];
      continue;
    }
    __align__(16) __nv_bfloat16 out[32];
    if constexpr (MODE == DX) {
#pragma unroll
      for (int j = 0; j < 32; ++j) out[j] = __float2bfloat16_rn(v[j] * silu_grad_f(__bfloat162float(zp[j])));
      store_rows(reinterpret_cast<const uint4(&)[4]>(out), a.dh_out, row0, n0, stage, lane);
    } else {
      __align__(16) __nv_bfloat16 zb[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float z = v[j] + sbias[n0 + j];
        zb[j] = __float2bfloat16_rn(z);
        out[j] = __float2bfloat16_rn(silu_f(z));
        if (MODE == FWD_LAST) ysum += __bfloat162float(out[j]) * sw5[n0 + j];
      }
      store_rows(reinterpret_cast<const uint4(&)[4]>(zb), a.z_out, row0, n0, stage, lane);
      store_rows(reinterpret_cast<const uint4(&)[4]>(out), a.x_out, row0, n0, stage, lane);
    }
  }
  return ysum;
}

// One CTA per SM, warp-specialised.  FWD*, DX: CTA c serves member slot
// c % G, whose weight operand stays in shared memory for the launch, and takes
// the slot's 128-row tiles round-robin.  DW: a tile is (slot, split of 256
// rows, 128 output features), both operands through the ring.
//   warp 0  (one lane)  TMA producer
//   warp 1  (one lane)  MMA issuer: tcgen05.mma into one of two TMEM
//           accumulators (2 x 256 columns)
//   warps 2-9           epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, two
//           warps a quarter, each half of the columns; it overlaps the MMAs of
//           the next tile
// Shared memory: region 1 (128 KiB) the resident weights or the B stages of
// DW, region 2 (64 KiB) the A stages.
template <int MODE>
__global__ void __launch_bounds__(kGemmThreads, 1)
    k_train_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TrainArgs a) {
  constexpr bool kResidentB = (MODE != DW);
  constexpr uint32_t kBox = kChunk * 128;            // DW: a {64 columns, 64 rows} box
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(16) unsigned char s_stage[kEpiWarps][32 * kStagePitch];
  __shared__ float s_bias[kWidth], s_w5[kWidth];
  const uint32_t s0 = tc::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024u - (s0 & 1023u)) & 1023u);
  unsigned char *r1 = base;
  unsigned char *r2 = base + kRegion1;
  uint64_t *full = reinterpret_cast<uint64_t *>(r2 + kRegion2);
  uint64_t *empty = full + kStages;
  uint64_t *bfull = empty + kStages;
  uint64_t *accf = bfull + 1;
  uint64_t *acce = accf + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bytesB = (uint32_t)a.N * kChunk * 2;
  // this CTA's tiles: first, first + step, ... < tiles
  const int my_slot = kResidentB ? (int)blockIdx.x % a.G : 0;
  const int first = kResidentB ? (int)blockIdx.x / a.G : (int)blockIdx.x;
  const int step = kResidentB ? (int)gridDim.x / a.G : (int)gridDim.x;
  const int per_slot = kResidentB ? a.rows / kTileM : (a.rows / kSplitRows) * 2;
  const int tiles = kResidentB ? per_slot : per_slot * a.G;
  const int nk = a.K / kChunk;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(bfull, 1);
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&accf[b], 1);
      tc::mbar_init(&acce[b], kEpiWarps);
    }
    tc::fence_mbar_init();
    tc::tma_prefetch(&tmA);
    tc::tma_prefetch(&tmB);
  }
  if (MODE == FWD || MODE == FWD_LAST) {
    const float *P = a.P[my_slot];
    for (int i = tid; i < kWidth; i += blockDim.x) {
      s_bias[i] = P[a.off_bias + i];
      if (MODE == FWD_LAST) s_w5[i] = P[kOffW5 + i];
    }
  }
  if (warp == 1) {
    tc::tmem_alloc(tslot, 2 * kTmemCols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const unsigned long long deadline = tc::now_ns() + a.timeout_ns;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      if (kResidentB && first < tiles) {
        tc::mbar_expect_tx(bfull, (uint32_t)nk * bytesB);
        for (int c = 0; c < nk; ++c) tc::tma_load_3d(r1 + c * kStageB, &tmB, c * kChunk, 0, a.m0 + my_slot, bfull);
      }
      for (int t = first; t < tiles && ok; t += step) {
        const int slot = kResidentB ? my_slot : t / per_slot;
        const int local = kResidentB ? t : t % per_slot;
        for (int kc = 0; kc < nk; ++kc) {
          const uint32_t st = it % kStages;
          if (it >= (uint32_t)kStages && !tc::mbar_wait(&empty[st], ((it / kStages) - 1) & 1, deadline)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full[st], kStageA + (kResidentB ? 0u : bytesB));
          if (kResidentB) {
            tc::tma_load_3d(r2 + st * kStageA, &tmA, kc * kChunk, local * kTileM, slot, &full[st]);
          } else {
            const int row = (local >> 1) * kSplitRows + kc * kChunk, col = (local & 1) * kTileM;
            for (int b = 0; b < kTileM / 64; ++b)
              tc::tma_load_3d(r2 + st * kStageA + b * kBox, &tmA, col + b * 64, row, slot, &full[st]);
            for (int b = 0; b < a.N / 64; ++b)
              tc::tma_load_3d(r1 + st * kStageB + b * kBox, &tmB, b * 64, row, slot, &full[st]);
          }
          ++it;
        }
      }
      if (!ok) {
        atomicExch(a.error, 1u);
        // copies in flight land before the shared memory is given back
        const unsigned long long d2 = tc::now_ns() + 1000000000ull;
        for (uint32_t j = (it > (uint32_t)kStages ? it - kStages : 0u); j < it; ++j)
          tc::mbar_wait(&full[j % kStages], (j / kStages) & 1, d2);
        if (kResidentB) tc::mbar_wait(bfull, 0, d2);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && first < tiles) {
      const uint32_t idesc = tc::idesc_bf16_f32(kTileM, a.N) | (kResidentB ? 0u : tc::kIdescMnMajorAB);
      uint32_t it = 0, local = 0;
      bool ok = !kResidentB || tc::mbar_wait(bfull, 0, deadline);
      for (int t = first; t < tiles && ok; t += step) {
        const uint32_t buf = local & 1u;
        if (local >= 2 && !tc::mbar_wait(&acce[buf], ((local >> 1) - 1) & 1, deadline)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t d = tmem + buf * kTmemCols;
        for (int kc = 0; kc < nk; ++kc) {
          const uint32_t st = it % kStages;
          if (!tc::mbar_wait(&full[st], (it / kStages) & 1, deadline)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint32_t aa = tc::smem_u32(r2 + st * kStageA);
          const uint32_t bb = tc::smem_u32(r1 + (kResidentB ? (uint32_t)kc : st) * kStageB);
#pragma unroll
          for (int k = 0; k < kChunk / 16; ++k) {
            const uint32_t acc = (kc > 0 || k > 0) ? 1u : 0u;
            if (kResidentB)
              tc::mma_bf16(d, tc::sdesc_sw128(aa + k * 32), tc::sdesc_sw128(bb + k * 32), idesc, acc);
            else                                     // 16 rows of 128 bytes further
              tc::mma_bf16(d, tc::sdesc_sw128_mn(aa + k * 2048, kBox), tc::sdesc_sw128_mn(bb + k * 2048, kBox), idesc,
                           acc);
          }
          tc::mma_commit(&empty[st]);
          ++it;
        }
        if (!ok) break;
        tc::mma_commit(&accf[buf]);
        ++local;
      }
      if (!ok) {
        atomicExch(a.error, 2u);
        // products in flight finish before TMEM is given back
        const unsigned long long d2 = tc::now_ns() + 1000000000ull;
        if (it > 0) tc::mbar_wait(&empty[(it - 1) % kStages], ((it - 1) / kStages) & 1, d2);
      }
    }
  } else {
    const int q = warp & 3;                       // TMEM lane quarter of this warp
    const int h = (warp - 2) / 4;                 // column half of this warp
    const int per = (a.N / 32) / 2;
    uint32_t count = 0;
    for (int t = first; t < tiles; t += step) {
      const int slot = kResidentB ? my_slot : t / per_slot;
      const int local = kResidentB ? t : t % per_slot;
      const uint32_t buf = count & 1u;
      const bool got = tc::mbar_wait(&accf[buf], (count >> 1) & 1, deadline);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) atomicExch(a.error, 3u);
        break;
      }
      tc::tc_fence_after();
      const int r = q * 32 + lane;
      const size_t row = (size_t)slot * a.rows + (size_t)local * kTileM + r;
      float *part = nullptr;
      if constexpr (MODE == DW)
        part = a.partial + ((size_t)slot * (per_slot / 2) + (local >> 1)) * a.N * kWidth + (local & 1) * kTileM + r;
      const float ys = train_epilogue<MODE>(a, row, tmem + ((uint32_t)(q * 32) << 16) + buf * kTmemCols, part, h * per,
                                            (h + 1) * per, s_stage[warp - 2], lane, s_bias, s_w5);
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[buf]);
      if constexpr (MODE == FWD_LAST) {
        // y_out is zeroed before the launch; the two halves' sums meet by
        // atomic addition, (0 + x) + y == (0 + y) + x, so the order does not
        // change the result
        atomicAdd(&a.y_out[row], h == 0 ? ys + __ldg(a.P[my_slot] + kOffB5) : ys);
      }
      ++count;
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 2 * kTmemCols);
  }
}

// ----------------------------------------------------------------------------
// CUDA-core kernels around the GEMMs; blockIdx.y (or .z) is the slot.
// ----------------------------------------------------------------------------

// Batch rows order[slot][offset .. offset + rows) of the training set (past
// n_order: padding rows of zeros) into X0 [rows][64] (features in columns
// 0..6; the other columns stay zero from allocation) and the targets; the
// head's outputs are zeroed.
__global__ void k_gather(const float *__restrict__ feats, const float *__restrict__ targ, const int *__restrict__ order,
                         long long n_order, long long offset, int rows, __nv_bfloat16 *__restrict__ x0,
                         float *__restrict__ y, float *__restrict__ yhat) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= rows) return;
  const long long k = offset + m;
  const int src = (k < n_order) ? order[(size_t)blockIdx.y * n_order + k] : -1;
  __align__(16) __nv_bfloat16 v[8];
#pragma unroll
  for (int f = 0; f < kFeatures; ++f)
    v[f] = __float2bfloat16_rn(src >= 0 ? feats[(size_t)src * kFeatures + f] : 0.0f);
  v[7] = __float2bfloat16_rn(0.0f);
  const size_t row = (size_t)blockIdx.y * rows + m;
  *reinterpret_cast<uint4 *>(x0 + row * kInPad) = *reinterpret_cast<const uint4 *>(v);
  y[row] = (src >= 0) ? targ[src] : 0.0f;
  yhat[row] = 0.0f;
}

// Loss and the head's backward pass: dy = 2 (yhat - y) / n for the first n
// rows (0 for padding), dH4 = dy w5 SiLU'(Z4), and one squared-error partial
// per 128 rows.  HBM-bound (Z4 read, dH4 written): after the block's dy, its
// threads sweep the 128 rows 16 bytes each, a warp one whole row; one thread a
// row with two strided 2-byte stores a column took 63 us for 16,384 rows.
__global__ void __launch_bounds__(256) k_head_backward(const float *__restrict__ yhat, const float *__restrict__ y, int n_valid, int rows,
                                const TrainArgs a, const __nv_bfloat16 *__restrict__ z4,
                                __nv_bfloat16 *__restrict__ dh4, float *__restrict__ dy,
                                float *__restrict__ loss_part) {
  __shared__ float red[kHeadRows], s_d[kHeadRows];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slot = blockIdx.y;
  const size_t row0 = (size_t)slot * rows + (size_t)blockIdx.x * kHeadRows;
  if (tid < kHeadRows) {
    const int m = blockIdx.x * kHeadRows + tid;
    const float e = (m < n_valid) ? (yhat[row0 + tid] - y[row0 + tid]) : 0.0f;
    const float d = 2.0f * e / (float)n_valid;
    dy[row0 + tid] = d;
    s_d[tid] = d;
    red[tid] = e * e;
  }
  __syncthreads();
  for (int s = kHeadRows / 2; s > 0; s >>= 1) {
    if (tid < s) red[tid] += red[tid + s];
    __syncthreads();
  }
  if (tid == 0) loss_part[(size_t)slot * gridDim.x + blockIdx.x] = red[0];
  const float *w5 = a.P[slot] + kOffW5 + lane * 8;
  float w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = __ldg(w5 + j);
#pragma unroll 4
  for (int r = warp; r < kHeadRows; r += 8) {
    const float d = s_d[r];
    const uint4 zz = *reinterpret_cast<const uint4 *>(z4 + (row0 + r) * kWidth + lane * 8);
    const __nv_bfloat16 *z = reinterpret_cast<const __nv_bfloat16 *>(&zz);
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = __float2bfloat16_rn(d * w[j] * silu_grad_f(__bfloat162float(z[j])));
    *reinterpret_cast<uint4 *>(dh4 + (row0 + r) * kWidth + lane * 8) = *reinterpret_cast<const uint4 *>(o);
  }
}

// Class sums of the bias and head gradients: out[slot][t][f] = sum over the
// rows c = t, t + 256, ... of src[c][f] (* w[c]), in that order.  A block takes
// 32 classes x 64 columns, a thread 8 columns of a class (16-byte loads, four
// rows of 128 bytes a warp).  HBM-bound; read from transposed copies by one
// block a column it took 32 us a layer and member.
__global__ void __launch_bounds__(256) k_class_sums(const __nv_bfloat16 *__restrict__ src, const float *__restrict__ w,
                                                    int rows, float *__restrict__ out) {
  const int f0 = blockIdx.y * 64 + (threadIdx.x & 7) * 8;
  const int t = blockIdx.x * 32 + (threadIdx.x >> 3);
  const size_t base = (size_t)blockIdx.z * rows;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
  for (int c = t; c < rows; c += kClasses) {
    const uint4 v = *reinterpret_cast<const uint4 *>(src + (base + c) * kWidth + f0);
    const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(&v);
    const float wc = w ? w[base + c] : 1.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = fmaf(__bfloat162float(x[j]), wc, s[j]);
  }
  float4 *o = reinterpret_cast<float4 *>(out + ((size_t)blockIdx.z * kClasses + t) * kWidth + f0);
  o[0] = make_float4(s[0], s[1], s[2], s[3]);
  o[1] = make_float4(s[4], s[5], s[6], s[7]);
}

struct UpdateArgs {
  float *P[kMaxMembers], *M1[kMaxMembers], *M2[kMaxMembers];
  float lr[kMaxMembers], c1[kMaxMembers], c2[kMaxMembers];   // Adam: rate and bias corrections by slot
  float b1, b2, eps;
  float *grad;              // non-null: write the gradient (slot 0) and leave the parameters
  int rows, splits, N, fan_in, off_w, off_b;
  const float *partial;     // [G][splits][N][256]
  const float *cls;         // class sums of dH_l [G][256][256]
  const float *cls5;        // top layer: of X4 dy (head weights), else null
  const float *dy;          // top layer: [G][rows] (head bias)
  const float *loss_part;   // top layer: [G][rows / 128]
  float *loss;              // top layer: loss[slot * loss_stride]
  long long loss_stride;
  int m0;
  __nv_bfloat16 *w;         // BF16 operand copies of the layer, by member: [E][256][w_ld]
  __nv_bfloat16 *wt;        // transposed [E][256][256], null for the first layer
  int w_ld;
  float *epi;               // FP32 epilogue operands of inference [E][5][256]
  int epi_layer;            // this layer's row of it
};

// Adam (bias-corrected) on one FP32 master parameter; returns its new value.
__device__ __forceinline__ float adam(const UpdateArgs &u, int slot, int i, float gi) {
  float *p = u.P[slot], *m1 = u.M1[slot], *m2 = u.M2[slot];
  const float a = fmaf(1.0f - u.b1, gi, __fmul_rn(u.b1, m1[i]));
  const float b = fmaf(__fmul_rn(1.0f - u.b2, gi), gi, __fmul_rn(u.b2, m2[i]));
  m1[i] = a;
  m2[i] = b;
  const float v = p[i] - u.lr[slot] * (a / u.c1[slot]) / (sqrtf(b / u.c2[slot]) + u.eps);
  p[i] = v;
  return v;
}

// red[0..255][0..31] -> red[0][c] by the fixed tree (t += t + s, s = 128 .. 1).
__device__ __forceinline__ void class_tree(float (*red)[33], int tid) {
  for (int s = kClasses / 2; s > 0; s >>= 1) {
    for (int i = tid; i < s * 32; i += 256) red[i >> 5][i & 31] += red[(i >> 5) + s][i & 31];
    __syncthreads();
  }
}

// The gradient of one layer from its partials, the optimiser's step and the
// BF16 operand copies, in one pass: the gradient is not stored, the
// parameters are read and written once.  Blocks [0, tiles): 32 x 32 tiles of
// dW (o the contiguous axis of the partials, i that of the parameters: the
// tile turns in shared memory); then 8 blocks of 32 biases; for the top layer 8
// of 32 head weights and one of the head bias and the loss.
__global__ void __launch_bounds__(256) k_update(const UpdateArgs u) {
  __shared__ float red[kClasses][33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slot = blockIdx.y;
  const int i_tiles = (u.fan_in + 31) / 32;
  const int tiles = 8 * i_tiles;
  int b = blockIdx.x;
  if (b < tiles) {
    const int o0 = (b / i_tiles) * 32, i0 = (b % i_tiles) * 32;
    const float *part = u.partial + (size_t)slot * u.splits * u.N * kWidth + o0 + lane;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < u.splits; ++k) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + warp + 8 * j;
        if (i < u.fan_in) s[j] += part[((size_t)k * u.N + i) * kWidth];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) red[warp + 8 * j][lane] = s[j];       // [i][o]
    __syncthreads();
    const int i = i0 + lane;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int o = warp + 8 * j;
      if (i < u.fan_in) {
        const int idx = u.off_w + (o0 + o) * u.fan_in + i;
        const float gi = red[lane][o];
        if (u.grad) {
          u.grad[idx] = gi;
        } else {
          const float v = adam(u, slot, idx, gi);
          u.w[((size_t)(u.m0 + slot) * kWidth + o0 + o) * u.w_ld + i] = __float2bfloat16_rn(v);
          red[lane][o] = v;
        }
      }
    }
    if (u.wt && !u.grad) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int ii = warp + 8 * j;
        u.wt[((size_t)(u.m0 + slot) * kWidth + i0 + ii) * kWidth + o0 + lane] = __float2bfloat16_rn(red[ii][lane]);
      }
    }
    return;
  }
  b -= tiles;
  if (b < 16) {
    const float *src = (b < 8) ? u.cls : u.cls5;
    const int f0 = (b & 7) * 32, off = (b < 8) ? u.off_b : kOffW5;
    for (int t = warp; t < kClasses; t += 8)
      red[t][lane] = src[((size_t)slot * kClasses + t) * kWidth + f0 + lane];
    __syncthreads();
    class_tree(red, tid);
    if (tid < 32) {
      if (u.grad) {
        u.grad[off + f0 + lane] = red[0][lane];
      } else {
        const float v = adam(u, slot, off + f0 + lane, red[0][lane]);
        float *epi = u.epi + (size_t)(u.m0 + slot) * kEpiFloats + f0 + lane;
        if (b < 8) epi[u.epi_layer * kWidth] = 0.5f * v;
        else epi[4 * kWidth] = v;
      }
    }
    return;
  }
  // head bias and loss: class sums of dy and of the loss partials, same tree
  float *s0 = &red[0][0], *s1 = s0 + kClasses;
  float a0 = 0.f, a1 = 0.f;
  const float *dy = u.dy + (size_t)slot * u.rows;
  const int parts = u.rows / kHeadRows;
  for (int c = tid; c < u.rows; c += kClasses) a0 += dy[c];
  for (int c = tid; c < parts; c += kClasses) a1 += u.loss_part[(size_t)slot * parts + c];
  s0[tid] = a0;
  s1[tid] = a1;
  __syncthreads();
  for (int s = kClasses / 2; s > 0; s >>= 1) {
    if (tid < s) {
      s0[tid] += s0[tid + s];
      s1[tid] += s1[tid + s];
    }
    __syncthreads();
  }
  if (tid == 0) {
    u.loss[(size_t)slot * u.loss_stride] = s1[0];
    if (u.grad) u.grad[kOffB5] = s0[0];
    else adam(u, slot, kOffB5, s0[0]);
  }
}

}  // namespace mlp
}  // namespace gelio
