// Inference kernel of the spectrum surrogate and what training shares with it:
// a 7 -> 256 -> 256 -> 256 -> 256 -> 1 MLP with SiLU, BF16 weights and
// activations, FP32 accumulation.
//
// Every layer product is a tcgen05 GEMM, X_l = SiLU(X_{l-1} W_l^T + b_l), of
// the form C[M x N] = A[M x K] * B[N x K]^T with both operands K-major
// (row-major, K contiguous).  Training is in mlp_train.cuh.
#pragma once
#include <cuda_bf16.h>

#include "gelio.h"
#include "tc_sm103.cuh"

namespace gelio {
namespace mlp {

constexpr int kWidth = 256;       // hidden width
constexpr int kFeatures = 7;      // (K0, V, tilt, polarity, r, theta, log T)
constexpr int kInPad = 64;        // first-layer K padded to one 128-byte row
constexpr int kTileM = 128;       // GEMM rows per tile (TMEM lanes)
constexpr int kChunk = 64;        // K per pipeline stage (128 B of BF16)
constexpr uint32_t kStageA = kTileM * kChunk * 2;   // 16 KiB
constexpr uint32_t kStageB = kWidth * kChunk * 2;   // 32 KiB (N = 256)
constexpr uint32_t kTmemCols = 256;

// Flat parameter layout (FP32 master copy and gradients).
constexpr int kOffW1 = 0;                                   // [256][7]
constexpr int kOffB1 = kOffW1 + kWidth * kFeatures;         // [256]
constexpr int kOffW2 = kOffB1 + kWidth;                     // [256][256]
constexpr int kOffB2 = kOffW2 + kWidth * kWidth;
constexpr int kOffW3 = kOffB2 + kWidth;
constexpr int kOffB3 = kOffW3 + kWidth * kWidth;
constexpr int kOffW4 = kOffB3 + kWidth;
constexpr int kOffB4 = kOffW4 + kWidth * kWidth;
constexpr int kOffW5 = kOffB4 + kWidth;                     // [256]
constexpr int kOffB5 = kOffW5 + kWidth;                     // [1]
constexpr int kParams = kOffB5 + 1;                         // 199,681

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + __expf(-z)); }

// Inference SiLU of 32 accumulator columns v with pre-halved biases hb:
// z / (1 + e^-z) = h + h tanh(h), h = z / 2 = fma(v, 1/2, b / 2) (exact
// halving), one tanh.approx.f32 per element (2^-11 relative) instead of an
// exponential and a reciprocal, the FP32 arithmetic in pairs (f32x2) and the
// BF16 rounding two at a time.  Training keeps silu_f, whose derivative the
// backward pass uses.
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void silu_infer32(const float (&v)[32], const float *hb, __nv_bfloat16 (&out)[32]) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    const float4 b = __ldg(reinterpret_cast<const float4 *>(hb + j));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 h = __ffma2_rn(make_float2(v[j + 2 * i], v[j + 2 * i + 1]), make_float2(0.5f, 0.5f),
                                  i == 0 ? make_float2(b.x, b.y) : make_float2(b.z, b.w));
      const float2 t = make_float2(tanh_approx(h.x), tanh_approx(h.y));
      *reinterpret_cast<__nv_bfloat162 *>(&out[j + 2 * i]) = __float22bfloat162_rn(__ffma2_rn(h, t, h));
    }
  }
}
__device__ __forceinline__ float silu_grad_f(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// Row-major store of a warp's 32 rows x 32 columns (BF16) through a shared
// staging tile: lane l then writes row 8 i + l / 4, 16-byte piece l % 4, so
// each store instruction covers 8 rows x 64 contiguous bytes (full sectors)
// instead of 32 rows x 16 bytes.  The 80-byte pitch keeps the lanes' 16-byte
// staging writes on distinct banks.
constexpr int kStagePitch = 80;

__device__ __forceinline__ void store_rows(const uint4 (&v)[4], __nv_bfloat16 *dst, size_t row0, int n0,
                                           unsigned char *stage, int lane) {
  uint4 *mine = reinterpret_cast<uint4 *>(stage + lane * kStagePitch);
#pragma unroll
  for (int q = 0; q < 4; ++q) mine[q] = v[q];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 8 + (lane >> 2), piece = lane & 3;
    const uint4 val = *reinterpret_cast<const uint4 *>(stage + r * kStagePitch + piece * 16);
    *reinterpret_cast<uint4 *>(dst + (row0 + r) * kWidth + n0 + piece * 8) = val;
  }
  __syncwarp();
}

// ----------------------------------------------------------------------------
// Whole-network inference, several ensemble members in one persistent launch.
//
// Work item = (member, 256 query rows): two 128-row tiles X, Y (the last item of
// a member may have X alone) run the four hidden layers and share every weight
// chunk.  The activations never leave the SM: each layer's epilogue writes
// bias + SiLU as BF16 straight into shared memory in the K-major
// 128-byte-swizzle layout that the next layer's tcgen05.mma reads (the layout
// TMA would write), and the last layer's epilogue forms the 256 -> 1 head.  Only
// the first layer's input (the query features, TMA) and the weights (32 KiB
// K-chunks of [256 N][64 K], TMA from L2, a ring of kFusedStages) are loaded.
//   warp 0 (one lane)  TMA: the first item's input tiles, then 13 weight chunks
//                      an item
//   warp 1 (one lane)  MMA: per layer and K-chunk one N = 256 product per tile
//                      into that tile's TMEM accumulator (2 x 256 columns)
//   warps 2-17         epilogue: warp w takes TMEM lane quarter w % 4 of
//                      tile ((w - 2) / 4) % 2, columns 128 ((w - 2) / 8) ..
//                      + 127 of its 32 rows; the tile's first warp also loads
//                      its input for the next item as soon as the last layer's
//                      products have read the tile's buffer
//
// What bounds it: shared memory.  A product reads 48 KiB of operands for 512
// cycles of tensor core (96 of the 128 bytes a cycle), and the epilogues'
// stores and the weights' arrival share the same port: a product takes ~930
// cycles, an epilogue 3,300-5,500 (2,048 of them tanh on the special-function
// unit), and X's run ahead of Y's only as far as the ring's three stages let
// it.  The order of the products hardly matters (measured: 556-596 us of device
// time for 200,000 rows and 5 members in five orders; two stages and one batch
// per 65,536 rows: 625).  Per SM 0.40 of the tensor core's measured BF16 rate.
// ----------------------------------------------------------------------------
constexpr int kFusedMaxMembers = 16;
constexpr int kFusedStages = 3;
constexpr int kFusedEpiWarps = 16;
constexpr int kFusedThreads = 64 + 32 * kFusedEpiWarps;
constexpr uint32_t kFusedA = kTileM * kWidth * 2;                 // 64 KiB: one tile's activations
constexpr size_t kFusedSmem = 1024 + 2 * (size_t)kFusedA + kFusedStages * (size_t)kStageB + 256;

struct FusedMaps {
  CUtensorMap q0;                                  // queries [rows][64], box {64, 128}
  CUtensorMap w[kFusedMaxMembers][4];              // W1 [256][64], W2-W4 [256][256], box {64, 256}
};

// FP32 operands of the epilogues, by member: halved biases of the four layers
// and the head weights.
constexpr int kEpiFloats = 5 * kWidth;

struct FusedArgs {
  int M;                        // query rows
  int n_pairs;                  // ceil(M / 256)
  int E;                        // members
  long long stride;             // y row stride per member
  const float *epi;             // [E][5][256]
  const float *P[kFusedMaxMembers];   // FP32 parameters of each member (head bias)
  float *y;                     // [E][stride] head outputs, zeroed before the launch
  unsigned *error;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Programmatic dependent launch: the network kernel's and the ensemble's CTAs
// start as the kernel before them ends (small predicts are a chain of three
// short kernels) and wait here until its results are written.  One simulation:
// 61 -> 53 us for the call.  No kernel lets the next one start before its own
// end: CTAs of the next one that wait on an SM cost 100 to 1000 simulations
// 20 us (300 simulations: 152 -> 177 us) and gave the smaller calls nothing.
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Order of a layer's eight products, bit i = tile of the i-th (0 X, 1 Y), each
// tile's K-chunks in order: X0 X1 Y0 X2 X3 Y1 Y2 Y3.
constexpr uint32_t kFusedOrder = 0xE4u;

__global__ void __launch_bounds__(kFusedThreads, 1)
    k_mlp_infer_fused(const __grid_constant__ FusedMaps maps, const FusedArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t s0 = tc::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024u - (s0 & 1023u)) & 1023u);
  unsigned char *ring = base + 2 * kFusedA;          // A of tile t: base + t * kFusedA
  uint64_t *full = reinterpret_cast<uint64_t *>(ring + kFusedStages * kStageB);
  uint64_t *empty = full + kFusedStages;
  uint64_t *a_full = empty + kFusedStages;      // [tile]: the item's input landed
  uint64_t *acc_full = a_full + 2;              // [tile]: a layer's products are in TMEM
  uint64_t *acc_empty = acc_full + 2;           // [tile]: a layer's epilogue read TMEM and wrote A
  uint64_t *drain = acc_empty + 2;              // products finished, after a wait ran out
  uint32_t *tslot = reinterpret_cast<uint32_t *>(drain + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int items = a.E * a.n_pairs;
  // tiles of item w: Y is there if any of its rows is
  auto tiles_of = [&](int w) { return ((w % a.n_pairs) * 2 + 1) * kTileM < a.M ? 2 : 1; };
  if (tid == 0) {
    for (int st = 0; st < kFusedStages; ++st) {
      tc::mbar_init(&full[st], 1);
      tc::mbar_init(&empty[st], 1);
    }
    for (int t = 0; t < 2; ++t) {
      tc::mbar_init(&a_full[t], 1);
      tc::mbar_init(&acc_full[t], 1);
      tc::mbar_init(&acc_empty[t], kFusedEpiWarps / 2);
    }
    tc::mbar_init(drain, 1);
    tc::fence_mbar_init();
    tc::tma_prefetch(&maps.q0);
    if ((int)blockIdx.x < items)
      for (int l = 0; l < 4; ++l) tc::tma_prefetch(&maps.w[blockIdx.x / a.n_pairs][l]);
  }
  if (warp == 1) {
    tc::tmem_alloc(tslot, 2 * kTmemCols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  wait_for_previous_kernel();
  const unsigned long long deadline = tc::now_ns() + a.timeout_ns;
  // the first item from w on (this CTA's step) that has tile t
  auto next_with = [&](int w, int t) {
    while (w < items && t >= tiles_of(w)) w += (int)gridDim.x;
    return w;
  };
  auto load_input = [&](int w, int t) {
    tc::mbar_expect_tx(&a_full[t], kStageA);
    tc::tma_load_2d(base + t * kFusedA, &maps.q0, 0, ((w % a.n_pairs) * 2 + t) * kTileM, &a_full[t]);
  };

  if (warp == 0) {
    if (lane == 0 && (int)blockIdx.x < items) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = 0; t < 2; ++t) {
        const int n = next_with(blockIdx.x, t);
        if (n < items) load_input(n, t);
      }
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int e = w / a.n_pairs;
        for (int l = 0; l < 4 && ok; ++l) {
          const int nk = (l == 0) ? 1 : kWidth / kChunk;
          for (int kc = 0; kc < nk; ++kc) {
            const uint32_t st = it % kFusedStages;
            if (it >= (uint32_t)kFusedStages &&
                !tc::mbar_wait(&empty[st], ((it / kFusedStages) - 1) & 1, deadline)) {
              ok = false;
              break;
            }
            tc::mbar_expect_tx(&full[st], kStageB);
            tc::tma_load_2d(ring + st * kStageB, &maps.w[e][l], kc * kChunk, 0, &full[st]);
            ++it;
          }
        }
      }
      if (!ok) {
        atomicExch(a.error, 11u);
        // copies in flight land before the shared memory is given back
        const unsigned long long d2 = tc::now_ns() + 1000000000ull;
        for (uint32_t j = (it > (uint32_t)kFusedStages ? it - kFusedStages : 0u); j < it; ++j)
          tc::mbar_wait(&full[j % kFusedStages], (j / kFusedStages) & 1, d2);
        for (int t = 0; t < 2; ++t)
          if (next_with(blockIdx.x, t) < items) tc::mbar_wait(&a_full[t], 0, d2);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_bf16_f32(kTileM, kWidth);
      uint32_t it = 0, layers[2] = {0, 0}, inputs[2] = {0, 0};
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int nt = tiles_of(w);
        for (int l = 0; l < 4 && ok; ++l) {
          const int nk = (l == 0) ? 1 : kWidth / kChunk;
          int ready = 0;                            // chunks of this layer known to have landed
          // one product of the layer: waits for its operands and, with a tile's
          // first, for the tile's previous epilogue; commits what it completes
          auto product = [&](int t, int k) -> bool {
            if (k == 0) {
              if (l == 0 && !tc::mbar_wait(&a_full[t], inputs[t]++ & 1, deadline)) return false;
              if (layers[t] > 0 && !tc::mbar_wait(&acc_empty[t], (layers[t] - 1) & 1, deadline)) return false;
            }
            const uint32_t st = (it + k) % kFusedStages;
            if (k >= ready) {
              if (!tc::mbar_wait(&full[st], ((it + k) / kFusedStages) & 1, deadline)) return false;
              ready = k + 1;
            }
            tc::tc_fence_after();
            const uint32_t aa = tc::smem_u32(base + t * kFusedA + k * kStageA);
            const uint32_t bb = tc::smem_u32(ring + st * kStageB);
#pragma unroll
            for (int j = 0; j < kChunk / 16; ++j)
              tc::mma_bf16(tmem + (uint32_t)t * kTmemCols, tc::sdesc_sw128(aa + j * 32), tc::sdesc_sw128(bb + j * 32),
                           idesc, (k > 0 || j > 0) ? 1u : 0u);
            if (t == nt - 1) tc::mma_commit(&empty[st]);      // Y follows X on every chunk
            if (k == nk - 1) {
              tc::mma_commit(&acc_full[t]);
              ++layers[t];
            }
            return true;
          };
          if (l == 0) {
            ok = product(0, 0) && (nt == 1 || product(1, 0));
          } else if (nt == 1) {
            ok = product(0, 0) && product(0, 1) && product(0, 2) && product(0, 3);
          } else {
            int next[2] = {0, 0};
#pragma unroll                                      // (every index below is a constant)
            for (int i = 0; i < 8; ++i) {
              const int t = (kFusedOrder >> i) & 1u;
              ok = ok && product(t, next[t]);
              ++next[t];
            }
          }
          it += nk;
        }
      }
      if (!ok) {
        atomicExch(a.error, 12u);
        // products in flight finish before TMEM is given back
        tc::mma_commit(drain);
        tc::mbar_wait(drain, 0, tc::now_ns() + 1000000000ull);
      }
    }
  } else {
    const int q = warp & 3;                        // TMEM lane quarter (a warp reaches lanes 32 (warp % 4) ..)
    const int t = ((warp - 2) >> 2) & 1;           // tile of the pair
    const int half = (warp - 2) >> 3;              // columns 128 half .. 128 half + 127
    const int r = q * 32 + lane;                   // row in the tile
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)t * kTmemCols + (uint32_t)(half * 128);
    unsigned char *arow = base + t * kFusedA + r * 128;
    const bool loader = warp == 2 + 4 * t && lane == 0;
    uint32_t layer = 0, loads = 1;                  // layers of this tile; inputs of this tile loaded
    bool ok = true;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      if (t >= tiles_of(w)) continue;
      const int e = w / a.n_pairs, pair = w % a.n_pairs;
      const float *epi = a.epi + (size_t)e * kEpiFloats;
      for (int l = 0; l < 4; ++l, ++layer) {
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_full[t], layer & 1, deadline));
        if (!ok) break;
        tc::tc_fence_after();
        if (l == 3) {                              // every product has read the tile's buffer
          const int n = next_with(w + (int)gridDim.x, t);
          if (n < items) {
            if (loader) load_input(n, t);
            ++loads;
          }
          __syncwarp();                            // the loads of TMEM below are warp-wide
        }
        float hs = 0.0f;                       // head: this warp's half of the columns
        // 32-column chunks of the accumulator, the next chunk's TMEM load in
        // flight while this one is evaluated
        constexpr int kChunks = kWidth / 64;   // chunks of 32 columns in a half
        uint32_t buf[2][32];
        tc::tmem_ld32_issue(trow, buf[0]);
        tc::tmem_wait_ld(buf[0]);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          if (c + 1 < kChunks) tc::tmem_ld32_issue(trow + (uint32_t)((c + 1) * 32), buf[(c + 1) & 1]);
          const int cc = half * kChunks + c;   // 32-column chunk of the layer
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(buf[c & 1][j]);
          __align__(16) __nv_bfloat16 out[32];
          silu_infer32(v, epi + l * kWidth + cc * 32, out);
          if (l == 3) {
            const float *w5 = epi + 4 * kWidth + cc * 32;
#pragma unroll
            for (int j = 0; j < 32; ++j) hs = fmaf(__bfloat162float(out[j]), __ldg(w5 + j), hs);
          }
          if (l < 3) {
            // columns 32cc .. 32cc+31 = K-chunk cc / 2, 16-byte pieces 4 (cc % 2) .. +3
            const uint4 *src = reinterpret_cast<const uint4 *>(out);
            unsigned char *chunk = arow + (cc >> 1) * kStageA;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int piece = ((cc & 1) * 4 + i) ^ (r & 7);
              *reinterpret_cast<uint4 *>(chunk + piece * 16) = src[i];
            }
          }
          if (c + 1 < kChunks) tc::tmem_wait_ld(buf[(c + 1) & 1]);
        }
        if (l < 3) fence_proxy_async_smem();     // A written for the tensor core
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acc_empty[t]);
        if (l == 3) {
          // y is zeroed before the launch: (columns 0-127 + b5) and columns
          // 128-255 meet by atomic addition, (0 + x) + y == (0 + y) + x
          const int row = pair * 2 * kTileM + t * kTileM + r;
          if (row < a.M) atomicAdd(&a.y[(size_t)e * a.stride + row], half == 0 ? hs + __ldg(a.P[e] + kOffB5) : hs);
        }
      }
    }
    if (!ok && lane == 0) {
      atomicExch(a.error, 13u);
      // an input in flight lands before the shared memory is given back
      if (loader && loads > 1) tc::mbar_wait(&a_full[t], (loads - 1) & 1, tc::now_ns() + 1000000000ull);
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 2 * kTmemCols);
  }
}

// ----------------------------------------------------------------------------
// CUDA-core kernels around the GEMMs
// ----------------------------------------------------------------------------

// Query rows x [n][7] into the BF16 first-layer operand x0 [rows][64]
// (features in columns 0..6; the padding columns stay zero from allocation);
// rows past n are zero.
__global__ void k_query_rows(const float *__restrict__ x, int n, int rows, __nv_bfloat16 *__restrict__ x0) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= rows) return;
#pragma unroll
  for (int f = 0; f < kFeatures; ++f)
    x0[(size_t)m * kInPad + f] = __float2bfloat16_rn(m < n ? x[(size_t)m * kFeatures + f] : 0.0f);
}

// Operand copies of one member's master parameters: BF16 W1 padded to [256][64],
// W2..W4 and their transposes; FP32 epilogue operands.
__global__ void k_pack(const float *__restrict__ p, __nv_bfloat16 *__restrict__ w1, __nv_bfloat16 *__restrict__ w2,
                       __nv_bfloat16 *__restrict__ w3, __nv_bfloat16 *__restrict__ w4, __nv_bfloat16 *__restrict__ w2t,
                       __nv_bfloat16 *__restrict__ w3t, __nv_bfloat16 *__restrict__ w4t, float *__restrict__ epi) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < kWidth) {
    epi[idx] = 0.5f * p[kOffB1 + idx];
    epi[kWidth + idx] = 0.5f * p[kOffB2 + idx];
    epi[2 * kWidth + idx] = 0.5f * p[kOffB3 + idx];
    epi[3 * kWidth + idx] = 0.5f * p[kOffB4 + idx];
    epi[4 * kWidth + idx] = p[kOffW5 + idx];
  }
  if (idx < kWidth * kInPad) {
    const int o = idx / kInPad, i = idx % kInPad;
    w1[idx] = __float2bfloat16_rn(i < kFeatures ? p[kOffW1 + o * kFeatures + i] : 0.0f);
  }
  if (idx < kWidth * kWidth) {
    const int o = idx / kWidth, i = idx % kWidth;
    const __nv_bfloat16 a = __float2bfloat16_rn(p[kOffW2 + idx]);
    const __nv_bfloat16 b = __float2bfloat16_rn(p[kOffW3 + idx]);
    const __nv_bfloat16 c = __float2bfloat16_rn(p[kOffW4 + idx]);
    w2[idx] = a;
    w3[idx] = b;
    w4[idx] = c;
    w2t[i * kWidth + o] = a;
    w3t[i * kWidth + o] = b;
    w4t[i * kWidth + o] = c;
  }
}

// ---------------------------------------------------------------------------
// Inference queries built on the device (gelio_surrogate_predict).
// ---------------------------------------------------------------------------

// Rows [off, off + c) of the query (row = first[i] + j: grid point j of
// simulation i) into the BF16 first-layer operand x0 [M][kInPad]; rows c..M-1
// of the tile padding are zero.  Zeroes the members' outputs of these rows.
//
// The inputs are those of gelio_surrogate_features, evaluated in FP64 and
// rounded to FP32 as the host function does: six depend on the simulation and
// are formed once per simulation of the block's rows, the
// seventh is the LOG_GRID energy as the SDE kernels build it (FP64 exp, rounded
// to FP32) and log10 of it / 2.  Bound by the FP64 pipe.
constexpr int kQueryBlock = 128;
__global__ void __launch_bounds__(kQueryBlock) k_query(const gelio_sim_params *__restrict__ sims,
                                                       const long long *__restrict__ first, int n_sims, long long off,
                                                       int c, int M, int E, long long stride,
                                                       __nv_bfloat16 *__restrict__ x0, float *__restrict__ y) {
  __shared__ float s_f[kQueryBlock][6];
  __shared__ double s_lmin[kQueryBlock], s_lmax[kQueryBlock];
  __shared__ int s_points[kQueryBlock];
  const int m0 = blockIdx.x * kQueryBlock, m = m0 + threadIdx.x;
  // last simulation with first[i] <= row
  auto find = [&](long long row) {
    int lo = 0, hi = n_sims - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first[mid] <= row) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  // simulations have one grid point or more: the block's rows belong to at
  // most kQueryBlock of them.  Each warp forms its part of every one, since
  // the logarithms one after another are a small call's longest chain.
  const int i0 = find(off + min(m0, c - 1)), i1 = find(off + min(m0 + kQueryBlock, c) - 1);
  const int part = threadIdx.x >> 5;
  for (int j = threadIdx.x & 31; j <= i1 - i0; j += 32) {
    const gelio_sim_params &s = sims[i0 + j];
    float *f = s_f[j];
    if (part == 0) {
      f[0] = (float)((log10((double)s.K0 / 4.4683705e-27) - 22.5) * 2.0);
      s_points[j] = s.inj_points;
    } else if (part == 1) {
      s_lmin[j] = log((double)s.inj_min);
      f[3] = (float)s.polarity;
    } else if (part == 2) {
      s_lmax[j] = log((double)s.inj_max);
    } else {
      const double rad = 180.0 / 3.14159265358979323846;
      f[1] = (float)(((double)s.V / 6.68458712e-9 - 550.0) / 200.0);
      f[2] = (float)(((double)s.tilt * rad - 40.0) / 35.0);
      f[4] = (float)(((double)s.r_injection - 40.5) / 39.5);
      f[5] = (float)(((double)s.theta_injection * rad - 90.0) / 80.0);
    }
  }
  __syncthreads();
  if (m >= M) return;
  __align__(16) __nv_bfloat16 v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = __float2bfloat16_rn(0.0f);
  if (m < c) {
    const long long row = off + m;
    const int i = find(row), q = i - i0, j = (int)(row - first[i]), points = s_points[q];
    const double fr = (points > 1) ? (double)j / (double)(points - 1) : 0.0;
    const float T = (float)exp(s_lmin[q] + fr * (s_lmax[q] - s_lmin[q]));
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = __float2bfloat16_rn(s_f[q][k]);
    v[6] = __float2bfloat16_rn((float)(log10((double)T) / 2.0));
    for (int e = 0; e < E; ++e) y[(size_t)e * stride + row] = 0.0f;
  }
  *reinterpret_cast<uint4 *>(x0 + (size_t)m * kInPad) = *reinterpret_cast<const uint4 *>(v);
}

// Ensemble mean and sample standard deviation (FP64) of E member outputs
// y[e * stride + row]; the error flag follows the results, so that one copy
// brings both.
__global__ void k_ensemble(const float *__restrict__ y, int E, long long rows, long long stride,
                           double *__restrict__ mean, double *__restrict__ sd, const unsigned *__restrict__ error,
                           unsigned *__restrict__ error_out) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  wait_for_previous_kernel();
  if (r == 0) *error_out = *error;
  if (r >= rows) return;
  double mu = 0.0;
  for (int e = 0; e < E; ++e) mu += (double)y[(size_t)e * stride + r];
  mu /= E;
  double m2 = 0.0;
  for (int e = 0; e < E; ++e) {
    const double d = (double)y[(size_t)e * stride + r] - mu;
    m2 += d * d;
  }
  mean[r] = mu;
  sd[r] = (E > 1) ? sqrt(m2 / (E - 1)) : 0.0;
}

}  // namespace mlp
}  // namespace gelio
