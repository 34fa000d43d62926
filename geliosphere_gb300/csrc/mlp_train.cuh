// Training kernels of the spectrum surrogate.
//
// The members of an ensemble are independent, so a step runs a group of them
// at once: every kernel takes G members ("slots" 0..G-1 of the group, members
// m0..m0+G-1 of the ensemble), every activation buffer is [G][rows][256].
// One member alone fills neither the SMs (128 row tiles of a 16,384-row batch)
// nor hides the launches: 27 launches and 410 us a step and member at 16,384
// rows, now 15 launches (12 where the class sums go all at once) and 85 us a member
// for a group of five (200,000 rows, 2 epochs: 49.2 -> 10.2 ms).
//
// All operands are row-major in HBM, written once:
//   forward   Z_l  = X_{l-1} W_l^T    A = X_{l-1} [rows x in]   (K-major)  B = W_l   [256 x in]
//   dX        dH_{l-1} = dH_l W_l * SiLU'(Z_{l-1})  A = dH_l    (K-major)  B = W_l^T [in x 256]
//   dW        dW_l = dH_l^T X_{l-1}   A = dH_l, B = X_{l-1}, both read MN-major (the
//             reduction runs over the rows), so no transposed copy is written
// Weight gradients are sums of FP32 partials of 256 batch rows, added in their
// order; bias and head gradients are sums over the rows of one class modulo 256,
// added by a fixed tree: a gradient is deterministic and does not depend on the
// group it is computed in.
#pragma once
#include "mlp_kernels.cuh"

namespace gelio {
namespace mlp {

constexpr int kMaxMembers = 16;
constexpr int kClasses = 256;     // row classes of the bias and head gradients
constexpr int kSplitRows = 256;   // batch rows of one dW partial
constexpr int kHeadRows = 128;    // rows of one loss partial

enum TrainMode { FWD = 0, FWD_LAST = 1, DX = 2 };

constexpr int kTrainStages = 4;
constexpr int kEpiWarps = 8;
constexpr int kTrainThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kRegion1 = 4 * kStageB;              // 128 KiB: a layer's weights
constexpr uint32_t kRegion2 = kTrainStages * kStageA;   // 64 KiB: row tiles
constexpr size_t kTrainSmem = 1024 + (size_t)kRegion1 + kRegion2 + 128;

struct TrainArgs {
  int rows;                 // batch rows (a multiple of 256)
  int G;                    // members in this launch
  int m0;                   // first member (weights, parameters)
  int K;                    // layer fan-in (FWD*: 64 or 256, DX: 256)
  const float *P[kMaxMembers];   // FP32 parameters by slot
  int off_bias;
  __nv_bfloat16 *z_out;     // FWD*: pre-activations
  __nv_bfloat16 *x_out;     // FWD*: activations
  float *y_out;             // FWD_LAST: head outputs [G][rows], zeroed before
  const __nv_bfloat16 *z_prev;   // DX
  __nv_bfloat16 *dh_out;    // DX
  unsigned *error;
  unsigned long long timeout_ns;
};

// Columns [32 c_begin, 32 c_end) of one accumulator row (row = row0 + lane of
// the slot's batch); returns this thread's part of the head's dot product.
template <int MODE>
__device__ __forceinline__ float train_epilogue(const TrainArgs &a, size_t row, uint32_t trow, int c_begin, int c_end,
                                                unsigned char *stage, int lane, const float *sbias, const float *sw5) {
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

// A layer's products of the forward pass and of dX.  One CTA per SM,
// warp-specialised: CTA c serves member slot c % G, whose weight operand stays
// in shared memory for the launch, and takes the slot's 128-row tiles
// round-robin.  Bound by its HBM traffic (X or dH and Z read, Z and X or dH
// written: 126 MB for five members of 16,384 rows in 27-32 us; 16 epilogue warps
// instead of 8 changed nothing).
//   warp 0  (one lane)  TMA producer
//   warp 1  (one lane)  MMA issuer: tcgen05.mma into one of two TMEM
//           accumulators (2 x 256 columns)
//   warps 2-9           epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, two
//           warps a quarter, each half of the columns; it overlaps the MMAs of
//           the next tile
// Shared memory: region 1 (128 KiB) the resident weights, region 2 (64 KiB) the
// row tiles.
template <int MODE>
__global__ void __launch_bounds__(kTrainThreads, 1)
    k_train_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TrainArgs a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(16) unsigned char s_stage[kEpiWarps][32 * kStagePitch];
  __shared__ float s_bias[kWidth], s_w5[kWidth];
  const uint32_t s0 = tc::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024u - (s0 & 1023u)) & 1023u);
  unsigned char *r1 = base;
  unsigned char *r2 = base + kRegion1;
  uint64_t *full = reinterpret_cast<uint64_t *>(r2 + kRegion2);
  uint64_t *empty = full + kTrainStages;
  uint64_t *bfull = empty + kTrainStages;
  uint64_t *accf = bfull + 1;
  uint64_t *acce = accf + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // this CTA's tiles: first, first + step, ... < tiles
  const int slot = (int)blockIdx.x % a.G, first = (int)blockIdx.x / a.G, step = (int)gridDim.x / a.G;
  const int tiles = a.rows / kTileM;
  const int nk = a.K / kChunk;

  if (tid == 0) {
    for (int s = 0; s < kTrainStages; ++s) {
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
    const float *P = a.P[slot];
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
    if (lane == 0 && first < tiles) {
      uint32_t it = 0;
      bool ok = true;
      tc::mbar_expect_tx(bfull, (uint32_t)nk * kStageB);
      for (int c = 0; c < nk; ++c) tc::tma_load_3d(r1 + c * kStageB, &tmB, c * kChunk, 0, a.m0 + slot, bfull);
      for (int t = first; t < tiles && ok; t += step) {
        for (int kc = 0; kc < nk; ++kc) {
          const uint32_t st = it % kTrainStages;
          if (it >= (uint32_t)kTrainStages && !tc::mbar_wait(&empty[st], ((it / kTrainStages) - 1) & 1, deadline)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full[st], kStageA);
          tc::tma_load_3d(r2 + st * kStageA, &tmA, kc * kChunk, t * kTileM, slot, &full[st]);
          ++it;
        }
      }
      if (!ok) {
        atomicExch(a.error, 1u);
        // copies in flight land before the shared memory is given back
        const unsigned long long d2 = tc::now_ns() + 1000000000ull;
        for (uint32_t j = (it > (uint32_t)kTrainStages ? it - kTrainStages : 0u); j < it; ++j)
          tc::mbar_wait(&full[j % kTrainStages], (j / kTrainStages) & 1, d2);
        tc::mbar_wait(bfull, 0, d2);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && first < tiles) {
      const uint32_t idesc = tc::idesc_bf16_f32(kTileM, kWidth);
      uint32_t it = 0, local = 0;
      bool ok = tc::mbar_wait(bfull, 0, deadline);
      for (int t = first; t < tiles && ok; t += step) {
        const uint32_t buf = local & 1u;
        if (local >= 2 && !tc::mbar_wait(&acce[buf], ((local >> 1) - 1) & 1, deadline)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t d = tmem + buf * kTmemCols;
        for (int kc = 0; kc < nk; ++kc) {
          const uint32_t st = it % kTrainStages;
          if (!tc::mbar_wait(&full[st], (it / kTrainStages) & 1, deadline)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint32_t aa = tc::smem_u32(r2 + st * kStageA);
          const uint32_t bb = tc::smem_u32(r1 + kc * kStageB);
#pragma unroll
          for (int k = 0; k < kChunk / 16; ++k)
            tc::mma_bf16(d, tc::sdesc_sw128(aa + k * 32), tc::sdesc_sw128(bb + k * 32), idesc,
                         (kc > 0 || k > 0) ? 1u : 0u);
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
        if (it > 0) tc::mbar_wait(&empty[(it - 1) % kTrainStages], ((it - 1) / kTrainStages) & 1, d2);
      }
    }
  } else {
    const int q = warp & 3;                       // TMEM lane quarter of this warp
    const int h = (warp - 2) / 4;                 // column half of this warp
    constexpr int per = (kWidth / 32) / 2;
    uint32_t count = 0;
    for (int t = first; t < tiles; t += step) {
      const uint32_t buf = count & 1u;
      const bool got = tc::mbar_wait(&accf[buf], (count >> 1) & 1, deadline);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) atomicExch(a.error, 3u);
        break;
      }
      tc::tc_fence_after();
      const size_t row = (size_t)slot * a.rows + (size_t)t * kTileM + q * 32 + lane;
      const float ys = train_epilogue<MODE>(a, row, tmem + ((uint32_t)(q * 32) << 16) + buf * kTmemCols, h * per,
                                            (h + 1) * per, s_stage[warp - 2], lane, s_bias, s_w5);
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[buf]);
      if constexpr (MODE == FWD_LAST) {
        // y_out is zeroed before the launch; the two halves' sums meet by
        // atomic addition, (0 + x) + y == (0 + y) + x, so the order does not
        // change the result
        atomicAdd(&a.y_out[row], h == 0 ? ys + __ldg(a.P[slot] + kOffB5) : ys);
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

struct UpdateArgs {
  float *P[kMaxMembers], *M1[kMaxMembers], *M2[kMaxMembers];
  float lr[kMaxMembers], c1[kMaxMembers], c2[kMaxMembers];   // Adam: rate and bias corrections by slot
  float b1, b2, eps;
  float *grad;              // non-null: write the gradient (slot 0) and leave the parameters
  int rows, G, m0;
  __nv_bfloat16 *w[4];      // BF16 operand copies of the layers, by member: [E][256][64 or 256]
  __nv_bfloat16 *wt[4];     // transposed [E][256][256], null for the first layer
  float *epi;               // FP32 epilogue operands of inference [E][5][256]
  const float *cls;         // class sums [G][5][256][256]: dH_1 .. dH_4, X4 dy
  const float *dy;          // [G][rows]
  const float *loss_part;   // [G][rows / 128]
  float *loss;              // loss[slot * loss_stride]
  long long loss_stride;
  unsigned *error;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ int layer_weights(int li) {
  return li == 0 ? kOffW1 : li == 1 ? kOffW2 : li == 2 ? kOffW3 : kOffW4;
}
__device__ __forceinline__ int layer_bias(int li) {
  return li == 0 ? kOffB1 : li == 1 ? kOffB2 : li == 2 ? kOffB3 : kOffB4;
}

// Adam (bias-corrected) on one FP32 master parameter p and its moments;
// returns its new value.
__device__ __forceinline__ float adam_step(const UpdateArgs &u, int slot, float gi, float p, float &m1, float &m2) {
  m1 = fmaf(1.0f - u.b1, gi, __fmul_rn(u.b1, m1));
  m2 = fmaf(__fmul_rn(1.0f - u.b2, gi), gi, __fmul_rn(u.b2, m2));
  return p - u.lr[slot] * (m1 / u.c1[slot]) / (sqrtf(m2 / u.c2[slot]) + u.eps);
}

__device__ __forceinline__ float adam(const UpdateArgs &u, int slot, int i, float gi) {
  float *p = u.P[slot], *m1 = u.M1[slot], *m2 = u.M2[slot];
  float a = m1[i], b = m2[i];
  const float v = adam_step(u, slot, gi, p[i], a, b);
  m1[i] = a;
  m2[i] = b;
  p[i] = v;
  return v;
}

// ----------------------------------------------------------------------------
// Weight gradients of all four layers and the optimiser's step, one launch.
//
// A work item is a tile of one layer's dW: 128 output features x N inputs (N =
// 64 or 128; the first layer's 64 padded inputs are one tile), reduced over the
// whole batch: dH_l^T X_{l-1}, both operands row-major in HBM and read MN-major.
// The tensor core forms one partial per 256 rows in one of four TMEM
// accumulators, the epilogue adds each to its FP32 registers, in order, and
// at the end takes the parameters' step: no partial goes through HBM (they were
// 335 MB a step for five members, written and read back), and the gradient is
// stored only where it is asked for.
//   warp 0  (one lane)  TMA producer: per 64 batch rows the boxes of both operands
//   warp 1  (one lane)  MMA issuer
//   warps 2-9           epilogue: warp w TMEM lanes 32 (w % 4) .. +31 (output
//           features), half (w - 2) / 4 of the tile's columns
// The update goes through shared memory (a lane an input, 128-byte rows): with a
// feature a lane its scattered accesses were 57 of 135 us.  Now 78 us for five
// members of 16,384 rows: the products (390 cycles a chunk of 64 rows) and the
// operands' way from L2 (6 MB an item at N = 64, 130 items) take about as long
// and overlap.  Through partials in HBM and an update kernel it was 250 us.
// With many members N = 128 halves the items.
// ----------------------------------------------------------------------------
constexpr int kDwStages = 6;
constexpr uint32_t kDwBox = kChunk * 128;               // 8 KiB: 64 columns of 64 rows
constexpr uint32_t kDwStage = 4 * kDwBox;               // 128 features, up to 128 inputs
constexpr int kDwBuffers = 4;
constexpr int kDwCols = 128;
constexpr int kDwPitch = 33;                            // floats a row of a warp's 32 x 32 piece
constexpr size_t kDwSmem = 1024 + (size_t)kDwStages * kDwStage + 256 + (size_t)kEpiWarps * 32 * kDwPitch * 4;

struct DwMaps {
  CUtensorMap dh[4], x[4];          // boxes of {64 columns, 64 rows, 1 slot}
};

__global__ void __launch_bounds__(kTrainThreads, 1)
    k_train_dw(const __grid_constant__ DwMaps maps, const UpdateArgs u, const int n_tile) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t s0 = tc::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024u - (s0 & 1023u)) & 1023u);
  uint64_t *full = reinterpret_cast<uint64_t *>(base + kDwStages * kDwStage);
  uint64_t *empty = full + kDwStages;
  uint64_t *accf = empty + kDwStages;
  uint64_t *acce = accf + kDwBuffers;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + kDwBuffers);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tiles = kWidth / n_tile;                  // of layers 2 to 4
  const int big = u.G * 3 * 2 * n_tiles, items = big + u.G * 2;
  const int chunks = u.rows / kChunk, parts = u.rows / kSplitRows;
  constexpr int kPart = kSplitRows / kChunk;            // chunks of a partial

  if (tid == 0) {
    for (int s = 0; s < kDwStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kDwBuffers; ++b) {
      tc::mbar_init(&accf[b], 1);
      tc::mbar_init(&acce[b], kEpiWarps);
    }
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tslot, kDwBuffers * kDwCols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const unsigned long long deadline = tc::now_ns() + u.timeout_ns;
  // item -> layer, slot, features' half, first input, inputs
  struct Item {
    int li, slot, m, n0, N;
  };
  auto item = [&](int w) {
    Item t;
    if (w < big) {
      const int r = w / n_tiles;
      t.n0 = (w % n_tiles) * n_tile;
      t.N = n_tile;
      t.m = r & 1;
      t.li = 1 + (r >> 1) % 3;
      t.slot = (r >> 1) / 3;
    } else {
      t.n0 = 0;
      t.N = kInPad;
      t.m = (w - big) & 1;
      t.li = 0;
      t.slot = (w - big) >> 1;
    }
    return t;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Item t = item(w);
        const uint32_t bytes = 2 * kDwBox + (uint32_t)(t.N / 64) * kDwBox;
        for (int c = 0; c < chunks; ++c) {
          const uint32_t st = it % kDwStages;
          if (it >= (uint32_t)kDwStages && !tc::mbar_wait(&empty[st], ((it / kDwStages) - 1) & 1, deadline)) {
            ok = false;
            break;
          }
          unsigned char *d = base + st * kDwStage;
          tc::mbar_expect_tx(&full[st], bytes);
          for (int b = 0; b < 2; ++b)
            tc::tma_load_3d(d + b * kDwBox, &maps.dh[t.li], t.m * kTileM + b * 64, c * kChunk, t.slot, &full[st]);
          for (int b = 0; b < t.N / 64; ++b)
            tc::tma_load_3d(d + (2 + b) * kDwBox, &maps.x[t.li], t.n0 + b * 64, c * kChunk, t.slot, &full[st]);
          ++it;
        }
      }
      if (!ok) {
        atomicExch(u.error, 4u);
        // copies in flight land before the shared memory is given back
        const unsigned long long d2 = tc::now_ns() + 1000000000ull;
        for (uint32_t j = (it > (uint32_t)kDwStages ? it - kDwStages : 0u); j < it; ++j)
          tc::mbar_wait(&full[j % kDwStages], (j / kDwStages) & 1, d2);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0, count = 0;                       // chunks; partials
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Item t = item(w);
        const uint32_t idesc = tc::idesc_bf16_f32(kTileM, t.N) | tc::kIdescMnMajorAB;
        for (int p = 0; p < parts && ok; ++p, ++count) {
          const uint32_t buf = count % kDwBuffers;
          if (count >= (uint32_t)kDwBuffers && !tc::mbar_wait(&acce[buf], ((count / kDwBuffers) - 1) & 1, deadline)) {
            ok = false;
            break;
          }
          for (int kc = 0; kc < kPart; ++kc) {
            const uint32_t st = it % kDwStages;
            if (!tc::mbar_wait(&full[st], (it / kDwStages) & 1, deadline)) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint32_t aa = tc::smem_u32(base + st * kDwStage), bb = aa + 2 * kDwBox;
#pragma unroll
            for (int k = 0; k < kChunk / 16; ++k)        // 16 rows of 128 bytes further
              tc::mma_bf16(tmem + buf * kDwCols, tc::sdesc_sw128_mn(aa + k * 2048, kDwBox),
                           tc::sdesc_sw128_mn(bb + k * 2048, kDwBox), idesc, (kc > 0 || k > 0) ? 1u : 0u);
            tc::mma_commit(&empty[st]);
            ++it;
          }
          if (!ok) break;
          tc::mma_commit(&accf[buf]);
        }
      }
      if (!ok) {
        atomicExch(u.error, 5u);
        // products in flight finish before TMEM is given back
        if (it > 0) tc::mbar_wait(&empty[(it - 1) % kDwStages], ((it - 1) / kDwStages) & 1, tc::now_ns() + 1000000000ull);
      }
    }
  } else {
    const int q = warp & 3;                       // TMEM lane quarter of this warp
    const int h = (warp - 2) / 4;                 // column half of this warp
    float *tile = reinterpret_cast<float *>(base + kDwStages * kDwStage + 256) + (warp - 2) * 32 * kDwPitch;
    uint32_t count = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const Item t = item(w);
      const int mine = t.N / 2;                   // columns of this warp: 64 or 32
      const uint32_t tcol = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * mine);
      float s[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) s[j] = 0.0f;
      for (int p = 0; p < parts; ++p, ++count) {
        const uint32_t buf = count % kDwBuffers;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&accf[buf], (count / kDwBuffers) & 1, deadline));
        if (!ok) break;
        tc::tc_fence_after();
        float v[32];
        tc::tmem_ld32(tcol + buf * kDwCols, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] += v[j];
        if (mine == 64) {
          tc::tmem_ld32(tcol + buf * kDwCols + 32, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) s[32 + j] += v[j];
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acce[buf]);
      }
      if (!ok) {
        if (lane == 0) atomicExch(u.error, 6u);
        break;
      }
      // features o0 .. o0 + 31 of this warp, 32 inputs at a time through the
      // warp's piece of shared memory: a lane holds one feature's sums and
      // updates one input's parameters of every feature
      const int o0 = t.m * kTileM + q * 32;
      const int fan_in = t.li == 0 ? kFeatures : kWidth, ld = t.li == 0 ? kInPad : kWidth;
      float *P = u.P[t.slot], *M1 = u.M1[t.slot], *M2 = u.M2[t.slot];
      __nv_bfloat16 *wr = u.w[t.li] + (size_t)(u.m0 + t.slot) * kWidth * ld;
      __nv_bfloat16 *wc = u.wt[t.li] ? u.wt[t.li] + (size_t)(u.m0 + t.slot) * kWidth * kWidth : nullptr;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (part * 32 >= mine) break;
        const int i0 = t.n0 + h * mine + part * 32, i = i0 + lane;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) tile[lane * kDwPitch + j] = s[part * 32 + j];
        __syncwarp();
        if (i < fan_in) {
          const int off = layer_weights(t.li) + o0 * fan_in + i;
          if (u.grad) {
            for (int r = 0; r < 32; ++r) u.grad[off + r * fan_in] = tile[r * kDwPitch + lane];
          } else {
            for (int r0 = 0; r0 < 32; r0 += 8) {
              float v[8], m1[8], m2[8];
#pragma unroll
              for (int r = 0; r < 8; ++r) {
                const int k = off + (r0 + r) * fan_in;
                v[r] = P[k];
                m1[r] = M1[k];
                m2[r] = M2[k];
              }
#pragma unroll
              for (int r = 0; r < 8; ++r) {
                const int k = off + (r0 + r) * fan_in;
                float &g = tile[(r0 + r) * kDwPitch + lane];
                v[r] = adam_step(u, t.slot, g, v[r], m1[r], m2[r]);
                P[k] = v[r];
                M1[k] = m1[r];
                M2[k] = m2[r];
                wr[(size_t)(o0 + r0 + r) * ld + i] = __float2bfloat16_rn(v[r]);
                g = v[r];
              }
            }
          }
        }
        __syncwarp();
        if (wc && !u.grad)
          for (int j = 0; j < 32; ++j)
            wc[(size_t)(i0 + j) * kWidth + o0 + lane] = __float2bfloat16_rn(tile[lane * kDwPitch + j]);
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, kDwBuffers * kDwCols);
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

// Class sums of the bias and head gradients: source k of slot g, its sums over
// the rows c = t, t + 256, ..., in that order, to out[g][k][t][f]: k = 0..3 dH_1
// .. dH_4, k = 4 X4 weighted by dy.  A block takes 16 classes x 64 columns of one
// source, a thread 4 columns of a class (8-byte loads, two rows of 128 bytes a
// warp, 16 rows in flight).  HBM-bound.  It runs beside the backward products, a
// source as soon as it is there, or beside the weight gradients: the n sources
// from k0 on (all of five members 42 us alone, 135 us beside those).
constexpr int kClassBlock = 16;
struct ClassSources {
  const __nv_bfloat16 *src[5];
  const float *dy;
};
__global__ void __launch_bounds__(256) k_class_sums(const ClassSources a, int k0, int n, int rows, float *__restrict__ out) {
  const int k = k0 + blockIdx.z % n, slot = blockIdx.z / n;
  const int f0 = blockIdx.y * 64 + (threadIdx.x & 15) * 4;
  const int t = blockIdx.x * kClassBlock + (threadIdx.x >> 4);
  const size_t base = (size_t)slot * rows;
  const __nv_bfloat16 *src = a.src[k];
  const float *w = (k == 4) ? a.dy : nullptr;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
  for (int c = t; c < rows; c += kClasses) {
    const uint2 v = *reinterpret_cast<const uint2 *>(src + (base + c) * kWidth + f0);
    const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(&v);
    const float wc = w ? w[base + c] : 1.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = fmaf(__bfloat162float(x[j]), wc, s[j]);
  }
  *reinterpret_cast<float4 *>(out + (((size_t)slot * 5 + k) * kClasses + t) * kWidth + f0) =
      make_float4(s[0], s[1], s[2], s[3]);
}

// Biases, head weights, head bias and loss from their class sums, by a fixed
// tree (t += t + s, s = 128 .. 1), and the optimiser's step: blocks 0..39 take
// 32 columns of a source, block 40 the head bias and the loss.
__global__ void __launch_bounds__(256) k_update_biases(const UpdateArgs u) {
  __shared__ float red[kClasses][33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slot = blockIdx.y, b = blockIdx.x;
  if (b < 40) {
    const int k = b >> 3, f0 = (b & 7) * 32, off = (k < 4) ? layer_bias(k) : kOffW5;
    for (int t = warp; t < kClasses; t += 8)
      red[t][lane] = u.cls[(((size_t)slot * 5 + k) * kClasses + t) * kWidth + f0 + lane];
    __syncthreads();
    for (int s = kClasses / 2; s > 0; s >>= 1) {
      for (int i = tid; i < s * 32; i += 256) red[i >> 5][i & 31] += red[(i >> 5) + s][i & 31];
      __syncthreads();
    }
    if (tid < 32) {
      if (u.grad) {
        u.grad[off + f0 + lane] = red[0][lane];
      } else {
        const float v = adam(u, slot, off + f0 + lane, red[0][lane]);
        u.epi[(size_t)(u.m0 + slot) * kEpiFloats + k * kWidth + f0 + lane] = (k < 4) ? 0.5f * v : v;
      }
    }
    return;
  }
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
