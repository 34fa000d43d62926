// Spectrum surrogate: an ensemble of small MLPs trained on the GPU, on
// spectra the Monte Carlo kernels produced, by the tcgen05 kernels of
// mlp_kernels.cuh.  The network maps a 2D Geliosphere simulation's
// (K0, V, tilt, polarity, r, theta) and a 1 AU kinetic energy T to
// ln(J_mod(T) / J_LIS(T)); the ensemble's spread decides when a query falls
// back to the Monte Carlo.  No reference counterpart (a learned addition on
// top of the reference's method).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include "gelio.h"
#include "alloc.cuh"
#include "mlp_kernels.cuh"
#include "mlp_train.cuh"

int gelio_internal_device(const gelio_ctx *c);

namespace gelio {
namespace mlp {
namespace {

using bf16 = __nv_bfloat16;

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// libcuda link dependency).
using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

// BF16 matrix [outer][inner] (inner contiguous), tiles of {64, box_outer}
// with the 128-byte swizzle; out-of-range rows read as zero.
bool make_map(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint32_t box_outer) {
  EncodeFn f = encode_fn();
  if (!f) return false;
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {inner * 2};
  const cuuint32_t box[2] = {64, box_outer};
  const cuuint32_t estr[2] = {1, 1};
  return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// BF16 tensor [members][outer][inner], boxes of {64, box_outer, 1}.
bool make_map3(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint64_t members, uint32_t box_outer) {
  EncodeFn f = encode_fn();
  if (!f) return false;
  const cuuint64_t dims[3] = {inner, outer, members};
  const cuuint64_t strides[2] = {inner * 2, inner * outer * 2};
  const cuuint32_t box[3] = {64, box_outer, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Local interstellar spectra of the evaluators (TwoDimensionBpResults.cpp:50-60),
// for the training targets.
double lis(int which, double T) {
  const double l = std::log(T);
  if (which == 0) {
    return 21.1 * std::exp(-2.8 * l) / (1.0 + 5.85 * std::exp(-1.22 * l) + 1.18 * std::exp(-2.54 * l));
  }
  if (which == 1) {
    const double tt = T + 0.938, t2 = tt + 0.938;
    const double beta = std::sqrt(T * t2) / tt;
    const double tem = std::exp(-3.93 * std::log((T + 0.67) / 1.67));
    return 2.7e3 * std::exp(1.12 * l) * tem / (beta * beta);
  }
  const double p = std::sqrt(T * T + 2.0 * T * 0.938);
  return 1.9e4 * std::exp(-2.78 * std::log(p)) / (1.0 + 0.4866 * std::exp(-2.51 * std::log(p)));
}

// LOG_GRID energies exactly as the kernels build them.
float grid_energy(const gelio_sim_params &s, int j) {
  const double lmin = std::log((double)s.inj_min), lmax = std::log((double)s.inj_max);
  const double f = (s.inj_points > 1) ? (double)j / (double)(s.inj_points - 1) : 0.0;
  return (float)std::exp(lmin + f * (lmax - lmin));
}

uint64_t splitmix(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

struct Member {
  float *P = nullptr, *M1 = nullptr, *M2 = nullptr;
  bf16 *W1 = nullptr, *W[3] = {}, *WT[3] = {};       // in the ensemble's arrays
  CUtensorMap mW1, mW[3];
  int adam_t = 0;
  bool trained = false;
};

// Activations and gradients of a group of G members training at once
// (mlp_train.cuh), allocated by the first training step or gradient.
struct TrainBuffers {
  int G = 0;
  bf16 *X0 = nullptr, *Z[4] = {}, *X[4] = {}, *dH[4] = {};
  float *yhat = nullptr, *y = nullptr, *dy = nullptr, *cls = nullptr;
  float *loss_part = nullptr;
  CUtensorMap aX0, aX[3], adH[4];        // row tiles of 128 (K-major operands)
  DwMaps dw;                             // boxes of 64 rows (MN-major operands of dW)
};

}  // namespace
}  // namespace mlp
}  // namespace gelio

using namespace gelio::mlp;

constexpr size_t kQueryBatch = 262144;   // rows of one inference launch (33.5 MB of first-layer operand)

struct gelio_surrogate {
  gelio_ctx *ctx = nullptr;
  gelio_surrogate_opts o{};
  int device = 0, sm_count = 0, rows = 0;   // rows = batch rows
  cudaStream_t stream = nullptr, side = nullptr;   // side: bias and head gradients of a training step
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  std::vector<Member> mem;
  // BF16 operand copies of every member's weights, [members][256][fan-in]
  bf16 *W1 = nullptr, *W[3] = {}, *WT[3] = {};
  CUtensorMap tW1, tW[3], tWT[3];
  float *epi = nullptr;      // FP32 epilogue operands of inference, [members][5][256]
  TrainBuffers tb;
  float *grad = nullptr;     // gelio_surrogate_gradient's result
  float *step_loss = nullptr;
  size_t step_loss_cap = 0;
  int *ident = nullptr;      // 0, 1, ..., rows - 1
  int *order = nullptr;      // this epoch's shuffled row orders, [group][rows of the set]
  size_t order_cap = 0;
  int *h_order = nullptr;    // staging of two epochs' orders
  bool h_order_pinned = false;
  size_t h_order_cap = 0;
  cudaEvent_t ev_copy[2] = {nullptr, nullptr};   // an epoch's orders have left the staging
  unsigned *error = nullptr;
  // training rows (host) and their device copy
  std::vector<float> feats, targ;
  float *d_feats = nullptr, *d_targ = nullptr;
  size_t d_rows_cap = 0, d_rows_used = 0;
  float *d_query = nullptr, *d_yq = nullptr;   // forward: inputs / outputs
  size_t query_cap = 0;
  // predict: simulations and their row offsets on the device, member outputs
  // [E][stride], ensemble mean / std [2][rows] and the error flag, pinned
  // staging of both ends
  unsigned char *d_pup = nullptr;     // [n] gelio_sim_params, then [n + 1] row offsets
  size_t pup_cap = 0;
  float *d_py = nullptr;
  double *d_pstat = nullptr;
  size_t prows_cap = 0;
  unsigned char *h_pstage = nullptr;
  size_t pstage_cap = 0;
  // first-layer operand of an inference batch [kQueryBatch][64]; the padding
  // columns stay zero
  bf16 *Q0 = nullptr;
  CUtensorMap mQ0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;    // device time of the last inference
  double last_ms = 0.0, last_flop = 0.0;
  bool dirty = true;
  std::mutex mu;
};

namespace {

int cuda_status_at(cudaError_t e, int line) {
  if (e == cudaSuccess) return GELIO_OK;
  gelio::note_cuda_error(e, "mlp.cu", line);
  if (e == cudaErrorMemoryAllocation) return GELIO_ERR_OUT_OF_MEMORY;
  return GELIO_ERR_CUDA;
}
#define cuda_status(e) cuda_status_at((e), __LINE__)
#define SUR_TRY(x)                            \
  do {                                        \
    cudaError_t e_ = (x);                     \
    if (e_ != cudaSuccess) return cuda_status(e_); \
  } while (0)

int set_smem_attrs() {
  static int rc = -1;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void *f) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
    };
    set((const void *)k_train_gemm<FWD>);
    set((const void *)k_train_gemm<FWD_LAST>);
    set((const void *)k_train_gemm<DX>);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute((const void *)k_train_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwSmem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute((const void *)k_mlp_infer_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kFusedSmem);
    rc = cuda_status(e);
  });
  return rc;
}

void free_train(TrainBuffers &t) {
  auto f = [](void *p) { if (p) cudaFree(p); };
  f(t.X0);
  for (int i = 0; i < 4; ++i) { f(t.Z[i]); f(t.X[i]); f(t.dH[i]); }
  f(t.yhat); f(t.y); f(t.dy); f(t.cls); f(t.loss_part);
  t = TrainBuffers();
}

void free_orders(gelio_surrogate *s) {
  if (s->h_order) s->h_order_pinned ? (void)cudaFreeHost(s->h_order) : std::free(s->h_order);
  s->h_order = nullptr;
  s->h_order_cap = 0;
}

void free_all(gelio_surrogate *s) {
  auto f = [](void *p) { if (p) cudaFree(p); };
  for (auto &m : s->mem) { f(m.P); f(m.M1); f(m.M2); }
  f(s->W1);
  for (int i = 0; i < 3; ++i) { f(s->W[i]); f(s->WT[i]); }
  free_train(s->tb);
  f(s->grad); f(s->step_loss);
  f(s->ident); f(s->order); f(s->error); f(s->d_feats); f(s->d_targ); f(s->d_query); f(s->d_yq);
  f(s->Q0); f(s->epi);
  f(s->d_pup); f(s->d_py); f(s->d_pstat);
  if (s->h_pstage) cudaFreeHost(s->h_pstage);
  free_orders(s);
  for (auto &e : s->ev_copy) if (e) cudaEventDestroy(e);
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  if (s->ev_fork) cudaEventDestroy(s->ev_fork);
  if (s->ev_join) cudaEventDestroy(s->ev_join);
  if (s->side) cudaStreamDestroy(s->side);
  if (s->stream) cudaStreamDestroy(s->stream);
}

int pack(gelio_surrogate *s, Member &m) {
  const int n = kWidth * kWidth;
  k_pack<<<(n + 255) / 256, 256, 0, s->stream>>>(m.P, m.W1, m.W[0], m.W[1], m.W[2], m.WT[0], m.WT[1], m.WT[2],
                                                 s->epi + (&m - s->mem.data()) * kEpiFloats);
  return cuda_status(cudaGetLastError());
}

int check_error(gelio_surrogate *s) {
  unsigned e = 0;
  SUR_TRY(cudaMemcpyAsync(&e, s->error, sizeof(e), cudaMemcpyDeviceToHost, s->stream));
  SUR_TRY(cudaStreamSynchronize(s->stream));
  if (e) {
    cudaMemsetAsync(s->error, 0, sizeof(unsigned), s->stream);
    cudaStreamSynchronize(s->stream);
    return GELIO_ERR_TIMEOUT;
  }
  return GELIO_OK;
}

// Members that train at once: as many as keep the group's activations near
// 2 GiB (16 members of 16,384 rows; past 2^18 rows one, as much as a member
// always took), within the ensemble.
int group_size(const gelio_surrogate *s) {
  const size_t R = (size_t)s->rows;
  const size_t per = R * kInPad * 2 + 12 * R * kWidth * 2;
  return (int)std::max<size_t>(1, std::min(s->mem.size(), ((size_t)2 << 30) / per));
}

// Training buffers for G members; a refused or failed allocation leaves those
// there were.
int ensure_train(gelio_surrogate *s, int G) {
  if (G <= s->tb.G) return GELIO_OK;
  const size_t R = (size_t)s->rows, g = (size_t)G;
  TrainBuffers t;
  cudaError_t e = cudaSuccess;
  auto alloc = [&](auto **p, size_t n) {
    if (e == cudaSuccess) e = gelio::dev_malloc(p, n * sizeof(**p));
  };
  alloc(&t.X0, g * R * kInPad);
  for (int i = 0; i < 4; ++i) {
    alloc(&t.Z[i], g * R * kWidth);
    alloc(&t.X[i], g * R * kWidth);
    alloc(&t.dH[i], g * R * kWidth);
  }
  alloc(&t.yhat, g * R);
  alloc(&t.y, g * R);
  alloc(&t.dy, g * R);
  alloc(&t.cls, g * 5 * kClasses * kWidth);
  alloc(&t.loss_part, g * (R / kHeadRows));
  if (e == cudaSuccess) e = cudaMemsetAsync(t.X0, 0, g * R * kInPad * 2, s->stream);   // the padding columns
  bool ok = e == cudaSuccess;
  ok = ok && make_map3(&t.aX0, t.X0, kInPad, R, g, kTileM) && make_map3(&t.dw.x[0], t.X0, kInPad, R, g, kChunk);
  for (int i = 0; i < 4; ++i) {
    if (i < 3)
      ok = ok && make_map3(&t.aX[i], t.X[i], kWidth, R, g, kTileM) && make_map3(&t.dw.x[i + 1], t.X[i], kWidth, R, g, kChunk);
    ok = ok && make_map3(&t.adH[i], t.dH[i], kWidth, R, g, kTileM) && make_map3(&t.dw.dh[i], t.dH[i], kWidth, R, g, kChunk);
  }
  if (!ok) {
    free_train(t);
    return e != cudaSuccess ? cuda_status(e) : GELIO_ERR_CUDA;
  }
  t.G = G;
  if (s->tb.G) SUR_TRY(cudaStreamSynchronize(s->stream));
  free_train(s->tb);
  s->tb = t;
  return GELIO_OK;
}

// All that a group of G members needs to train on nrow rows.  The staging of
// the orders is plain memory where no pinned memory is to be had.  The group's
// buffers come last: where a part is refused, the smaller group that is tried
// next has the memory of the larger one's buffers to itself.
int ensure_group(gelio_surrogate *s, int G, int steps, size_t nrow) {
  const size_t n_loss = (size_t)G * steps, n_order = G * nrow;
  if (n_loss > s->step_loss_cap) {
    if (s->step_loss) cudaFree(s->step_loss);
    s->step_loss = nullptr;
    s->step_loss_cap = 0;
    SUR_TRY(gelio::dev_malloc(&s->step_loss, sizeof(float) * n_loss));
    s->step_loss_cap = n_loss;
  }
  if (n_order > s->order_cap) {
    if (s->order) cudaFree(s->order);
    s->order = nullptr;
    s->order_cap = 0;
    SUR_TRY(gelio::dev_malloc(&s->order, n_order * sizeof(int)));
    s->order_cap = n_order;
  }
  if (2 * n_order > s->h_order_cap) {
    free_orders(s);
    s->h_order_pinned = gelio::pinned_malloc(&s->h_order, 2 * n_order * sizeof(int)) == cudaSuccess;
    if (!s->h_order_pinned) {
      (void)cudaGetLastError();
      s->h_order = static_cast<int *>(std::malloc(2 * n_order * sizeof(int)));
      if (!s->h_order) return GELIO_ERR_OUT_OF_MEMORY;
    }
    s->h_order_cap = 2 * n_order;
  }
  return ensure_train(s, G);
}

template <int MODE>
int launch_train(gelio_surrogate *s, const CUtensorMap &A, const CUtensorMap &B, const TrainArgs &a) {
  // the same number of CTAs for each slot
  const int grid = a.G * std::max(1, std::min(s->sm_count / a.G, a.rows / kTileM));
  k_train_gemm<MODE><<<grid, kTrainThreads, kTrainSmem, s->stream>>>(A, B, a);
  return cuda_status(cudaGetLastError());
}

// One step of members [m0, m0 + G) on the gathered batches: forward, backward
// and the update that u describes (Adam's step, or the gradient of one member).
// The bias and head gradients run beside the weight gradients, on a stream of
// their own.
int train_step(gelio_surrogate *s, int m0, int G, int n_valid, UpdateArgs &u) {
  TrainBuffers &t = s->tb;
  const int R = s->rows;
  int rc;
  TrainArgs a{};
  a.rows = R; a.G = G; a.m0 = m0;
  a.error = s->error; a.timeout_ns = 2000000000ull;
  for (int g = 0; g < G; ++g) a.P[g] = s->mem[m0 + g].P;
  // forward
  a.K = kInPad; a.off_bias = kOffB1; a.z_out = t.Z[0]; a.x_out = t.X[0];
  if ((rc = launch_train<FWD>(s, t.aX0, s->tW1, a)) != GELIO_OK) return rc;
  a.K = kWidth; a.off_bias = kOffB2; a.z_out = t.Z[1]; a.x_out = t.X[1];
  if ((rc = launch_train<FWD>(s, t.aX[0], s->tW[0], a)) != GELIO_OK) return rc;
  a.off_bias = kOffB3; a.z_out = t.Z[2]; a.x_out = t.X[2];
  if ((rc = launch_train<FWD>(s, t.aX[1], s->tW[1], a)) != GELIO_OK) return rc;
  a.off_bias = kOffB4; a.z_out = t.Z[3]; a.x_out = t.X[3]; a.y_out = t.yhat;
  if ((rc = launch_train<FWD_LAST>(s, t.aX[2], s->tW[2], a)) != GELIO_OK) return rc;
  // head, then the hidden layers, top down
  k_head_backward<<<dim3(R / kHeadRows, G), 256, 0, s->stream>>>(t.yhat, t.y, n_valid, R, a, t.Z[3], t.dH[3], t.dy,
                                                                 t.loss_part);
  SUR_TRY(cudaGetLastError());
  // 64 inputs a tile while that is one item an SM or fewer (26 a member)
  const int n_tile = 26 * G <= s->sm_count ? 64 : 128;
  const int items = G * 2 * (3 * (kWidth / n_tile) + 1), dw_grid = std::min(items, s->sm_count);
  // The class sums start as their sources come where the weight gradients leave
  // them fewer than three tenths of the SMs, else all at once beside those.  Four
  // epochs of six batches, early / at once, ms: 5 members of 16,384 rows (130 of
  // 152 SMs) 8.95 / 9.74, 8 of 4,096 (112) 5.24 / 5.52; 4 of 16,384 and of 4,096
  // (104) 7.94 / 7.69 and 3.49 / 3.42, 1 of 4,096 (26; bound by its launches, three
  // more a step) 2.99 / 2.90.
  const bool early = 10 * dw_grid > 7 * s->sm_count;
  ClassSources c{};
  for (int li = 0; li < 4; ++li) c.src[li] = t.dH[li];
  c.src[4] = t.X[3];
  c.dy = t.dy;
  auto class_sums = [&](int k, int n) -> int {
    SUR_TRY(cudaEventRecord(s->ev_fork, s->stream));
    SUR_TRY(cudaStreamWaitEvent(s->side, s->ev_fork, 0));
    k_class_sums<<<dim3(kClasses / kClassBlock, kWidth / 64, n * G), 256, 0, s->side>>>(c, k, n, R, t.cls);
    return cuda_status(cudaGetLastError());
  };
  if (early && (rc = class_sums(3, 2)) != GELIO_OK) return rc;
  for (int li = 3; li > 0; --li) {
    a.K = kWidth; a.z_prev = t.Z[li - 1]; a.dh_out = t.dH[li - 1];
    if ((rc = launch_train<DX>(s, t.adH[li], s->tWT[li - 1], a)) != GELIO_OK) return rc;
    if (early && li > 1 && (rc = class_sums(li - 1, 1)) != GELIO_OK) return rc;
  }
  u.rows = R; u.G = G; u.m0 = m0;
  for (int li = 0; li < 4; ++li) {
    u.w[li] = (li == 0) ? s->W1 : s->W[li - 1];
    u.wt[li] = (li == 0) ? nullptr : s->WT[li - 1];
  }
  u.epi = s->epi;
  u.cls = t.cls;
  u.dy = t.dy;
  u.loss_part = t.loss_part;
  u.error = s->error;
  u.timeout_ns = a.timeout_ns;
  SUR_TRY(cudaEventRecord(s->ev_fork, s->stream));
  SUR_TRY(cudaStreamWaitEvent(s->side, s->ev_fork, 0));
  k_train_dw<<<dw_grid, kTrainThreads, kDwSmem, s->stream>>>(t.dw, u, n_tile);
  SUR_TRY(cudaGetLastError());
  const int left = early ? 1 : 5;
  k_class_sums<<<dim3(kClasses / kClassBlock, kWidth / 64, left * G), 256, 0, s->side>>>(c, 0, left, R, t.cls);
  k_update_biases<<<dim3(41, G), 256, 0, s->side>>>(u);
  SUR_TRY(cudaGetLastError());
  SUR_TRY(cudaEventRecord(s->ev_join, s->side));
  SUR_TRY(cudaStreamWaitEvent(s->stream, s->ev_join, 0));
  return GELIO_OK;
}

// A launch whose CTAs may start while the kernel before it on the stream still
// runs; the kernel itself waits for it (wait_for_previous_kernel).
template <class... P, class... A>
cudaError_t launch_early(gelio_surrogate *s, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s->stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Members [m0, m1) on the first c rows of the inference batch (s->Q0, zero
// past c up to a whole tile) in one launch of the fused network kernel; member
// m0 + e's outputs are added to y[e * stride + row].
int infer_fused(gelio_surrogate *s, int m0, int m1, int c, float *y, long long stride) {
  const int E = m1 - m0;
  if (E > kFusedMaxMembers) return GELIO_ERR_UNSUPPORTED;
  FusedMaps maps;
  maps.q0 = s->mQ0;
  FusedArgs a{};
  for (int e = 0; e < E; ++e) {
    maps.w[e][0] = s->mem[m0 + e].mW1;
    for (int l = 0; l < 3; ++l) maps.w[e][l + 1] = s->mem[m0 + e].mW[l];
    a.P[e] = s->mem[m0 + e].P;
  }
  a.M = c;
  a.n_pairs = (c + 2 * kTileM - 1) / (2 * kTileM);
  a.E = E;
  a.stride = stride;
  a.epi = s->epi + (size_t)m0 * kEpiFloats;
  a.y = y;
  a.error = s->error;
  a.timeout_ns = 2000000000ull;
  const int grid = std::max(1, std::min(E * a.n_pairs, s->sm_count));
  return cuda_status(launch_early(s, k_mlp_infer_fused, grid, kFusedThreads, kFusedSmem, maps, a));
}

// FLOP of the products over the rows actually multiplied (whole tiles of 128
// rows; first layer K padded to 64).
double gemm_flop(size_t padded, size_t members) {
  return 2.0 * (double)padded * (double)members * ((double)kInPad * kWidth + 3.0 * kWidth * kWidth + (double)kWidth);
}

bool valid_member(gelio_surrogate *s, int m) { return s && m >= 0 && m < (int)s->mem.size(); }

// Inference of one member on n rows x [n][7].
int infer_rows(gelio_surrogate *s, int m, const float *x, size_t n, float *y) {
  if (n == 0) return GELIO_OK;
  int rc = GELIO_OK;
  if (n > s->query_cap) {
    if (s->d_query) cudaFree(s->d_query);
    if (s->d_yq) cudaFree(s->d_yq);
    s->d_query = s->d_yq = nullptr;
    s->query_cap = 0;
    SUR_TRY(gelio::dev_malloc(&s->d_query, n * kFeatures * 4));
    SUR_TRY(gelio::dev_malloc(&s->d_yq, n * 4));
    s->query_cap = n;
  }
  SUR_TRY(cudaMemcpyAsync(s->d_query, x, n * kFeatures * 4, cudaMemcpyHostToDevice, s->stream));
  SUR_TRY(cudaEventRecord(s->ev0, s->stream));
  SUR_TRY(cudaMemsetAsync(s->d_yq, 0, n * 4, s->stream));
  size_t padded = 0;
  for (size_t off = 0; off < n; off += kQueryBatch) {
    const int c = (int)std::min<size_t>(kQueryBatch, n - off);
    const int M = (c + kTileM - 1) / kTileM * kTileM;     // only the tiles this chunk needs
    padded += (size_t)M;
    k_query_rows<<<(M + 127) / 128, 128, 0, s->stream>>>(s->d_query + off * kFeatures, c, M, s->Q0);
    SUR_TRY(cudaGetLastError());
    if ((rc = infer_fused(s, m, m + 1, c, s->d_yq + off, (long long)n)) != GELIO_OK) return rc;
  }
  SUR_TRY(cudaEventRecord(s->ev1, s->stream));
  SUR_TRY(cudaMemcpyAsync(y, s->d_yq, n * 4, cudaMemcpyDeviceToHost, s->stream));
  rc = check_error(s);
  float ms = 0.f;
  if (rc == GELIO_OK && cudaEventElapsedTime(&ms, s->ev0, s->ev1) == cudaSuccess) {
    s->last_ms = ms;
    s->last_flop = gemm_flop(padded, 1);
  }
  return rc;
}

// The epochs of members [m0, m0 + g).  Each member has its own shuffles; the
// host makes the next epoch's while the device runs this one's, a thread a
// member (a shuffle of 200,000 rows takes 1.5 ms, as long as the device's
// epoch).  Losses of the last epoch's steps: sl[member][step].
int train_group(gelio_surrogate *s, int m0, int g, int epochs, int steps, long long total, size_t nrow, float *sl) {
  const int R = s->rows;
  std::vector<std::vector<int>> order(g, std::vector<int>(nrow));
  std::vector<std::mt19937_64> rng;
  for (int k = 0; k < g; ++k) {
    rng.emplace_back(s->o.seed * 1000003ull + (unsigned)(m0 + k));
    for (size_t i = 0; i < nrow; ++i) order[k][i] = (int)i;
  }
  auto shuffle = [&](int k, int ep) {
    std::shuffle(order[k].begin(), order[k].end(), rng[k]);
    std::memcpy(s->h_order + ((size_t)(ep & 1) * g + k) * nrow, order[k].data(), nrow * sizeof(int));
  };
  std::vector<std::thread> workers;
  auto start_shuffles = [&](int ep) {
    for (int k = 0; k < g; ++k) {
      bool run = false;
      try {
        workers.emplace_back(shuffle, k, ep);
        run = true;
      } catch (...) {          // no thread to be had: shuffled here
      }
      if (!run) shuffle(k, ep);
    }
  };
  auto join = [&] {
    for (auto &w : workers) w.join();
    workers.clear();
  };
  int rc = GELIO_OK;
  UpdateArgs u{};
  u.b1 = 0.9f; u.b2 = 0.999f; u.eps = 1e-8f;
  for (int k = 0; k < g; ++k) {
    u.P[k] = s->mem[m0 + k].P;
    u.M1[k] = s->mem[m0 + k].M1;
    u.M2[k] = s->mem[m0 + k].M2;
  }
  u.loss_stride = steps;
  auto epoch = [&](int ep) -> int {
    SUR_TRY(cudaMemcpyAsync(s->order, s->h_order + (size_t)(ep & 1) * g * nrow, (size_t)g * nrow * sizeof(int),
                            cudaMemcpyHostToDevice, s->stream));
    SUR_TRY(cudaEventRecord(s->ev_copy[ep & 1], s->stream));
    if (ep + 1 < epochs) {
      // the other half of the staging was copied an epoch ago
      if (ep > 0) SUR_TRY(cudaEventSynchronize(s->ev_copy[(ep + 1) & 1]));
      start_shuffles(ep + 1);
    }
    for (int st = 0; st < steps; ++st) {
      const long long off = (long long)st * R;
      const int nv = (int)std::min<long long>(R, (long long)nrow - off);
      k_gather<<<dim3((R + 127) / 128, g), 128, 0, s->stream>>>(s->d_feats, s->d_targ, s->order, (long long)nrow, off,
                                                                R, s->tb.X0, s->tb.y, s->tb.yhat);
      SUR_TRY(cudaGetLastError());
      const long long t = (long long)ep * steps + st;
      const double frac = total > 1 ? (double)t / (double)(total - 1) : 1.0;
      const float lr = (float)(s->o.lr_final + 0.5 * (s->o.lr - s->o.lr_final) * (1.0 + std::cos(M_PI * frac)));
      for (int k = 0; k < g; ++k) {
        Member &m = s->mem[m0 + k];
        ++m.adam_t;
        u.lr[k] = lr;
        u.c1[k] = 1.0f - std::pow(0.9f, (float)m.adam_t);
        u.c2[k] = 1.0f - std::pow(0.999f, (float)m.adam_t);
      }
      u.loss = s->step_loss + st;
      const int r = train_step(s, m0, g, nv, u);
      if (r != GELIO_OK) return r;
    }
    return GELIO_OK;
  };
  if (epochs > 0) start_shuffles(0);
  for (int ep = 0; ep < epochs && rc == GELIO_OK; ++ep) {
    join();
    rc = epoch(ep);
  }
  join();
  if (rc != GELIO_OK) {
    cudaStreamSynchronize(s->side);
    cudaStreamSynchronize(s->stream);
    return rc;
  }
  SUR_TRY(cudaMemcpyAsync(sl, s->step_loss, sizeof(float) * (size_t)g * steps, cudaMemcpyDeviceToHost, s->stream));
  return check_error(s);
}

void default_opts(gelio_surrogate_opts &o) {
  std::memset(&o, 0, sizeof(o));
  o.members = 5;
  o.batch_rows = 16384;
  o.lis = 1;
  o.min_count = 64;
  o.lr = 2e-3f;
  o.lr_final = 2e-5f;
  o.fallback_std = 0.03f;
  o.t_min = 0.1f;
  o.t_max = 10.0f;
  o.seed = 1;
}

}  // namespace

extern "C" {

int32_t gelio_surrogate_features(const gelio_sim_params *sim, double T, float *out) {
  if (!sim || !out || !(T > 0.0)) return GELIO_ERR_INVALID_ARGUMENT;
  const double k0_cm2 = (double)sim->K0 / 4.4683705e-27;
  const double v_kms = (double)sim->V / 6.68458712e-9;
  const double rad = 180.0 / 3.14159265358979323846;
  out[0] = (float)((std::log10(k0_cm2) - 22.5) * 2.0);
  out[1] = (float)((v_kms - 550.0) / 200.0);
  out[2] = (float)(((double)sim->tilt * rad - 40.0) / 35.0);
  out[3] = (float)sim->polarity;
  out[4] = (float)(((double)sim->r_injection - 40.5) / 39.5);
  out[5] = (float)(((double)sim->theta_injection * rad - 90.0) / 80.0);
  out[6] = (float)(std::log10(T) / 2.0);
  return GELIO_OK;
}

int32_t gelio_surrogate_create(gelio_ctx *ctx, const gelio_surrogate_opts *opts, gelio_surrogate **out) {
  if (!ctx || !out) return GELIO_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  gelio_surrogate_opts o;
  default_opts(o);
  if (opts) {
    o = *opts;
    gelio_surrogate_opts d;
    default_opts(d);
    if (o.members <= 0) o.members = d.members;
    if (o.batch_rows <= 0) o.batch_rows = d.batch_rows;
    if (o.min_count <= 0) o.min_count = d.min_count;
    if (!(o.lr > 0.f)) o.lr = d.lr;
    if (!(o.lr_final > 0.f)) o.lr_final = d.lr_final;
    if (!(o.fallback_std > 0.f)) o.fallback_std = d.fallback_std;
    if (!(o.t_min > 0.f)) o.t_min = d.t_min;
    if (!(o.t_max > o.t_min)) o.t_max = d.t_max;
  }
  if (o.members > 16 || o.batch_rows % 256 != 0 || o.batch_rows > (1 << 20) || o.lis < 0 || o.lis > 2)
    return GELIO_ERR_INVALID_ARGUMENT;
  auto *s = new gelio_surrogate();
  s->ctx = ctx;
  s->o = o;
  s->device = gelio_internal_device(ctx);
  s->rows = o.batch_rows;
  int rc = GELIO_OK;
  auto fail = [&](int r) { free_all(s); delete s; return r; };
  if (cudaSetDevice(s->device) != cudaSuccess) return fail(GELIO_ERR_NO_DEVICE);
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  if (!encode_fn()) return fail(GELIO_ERR_UNSUPPORTED);
  if ((rc = set_smem_attrs()) != GELIO_OK) return fail(rc);
  cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, s->device);
  if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  if (cudaEventCreate(&s->ev0) != cudaSuccess || cudaEventCreate(&s->ev1) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  if (cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  for (cudaEvent_t *e : {&s->ev_copy[0], &s->ev_copy[1], &s->ev_fork, &s->ev_join})
    if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  const size_t R = (size_t)s->rows;
  auto alloc = [&](void **p, size_t bytes) {
    if (rc != GELIO_OK) return;
    cudaError_t e = gelio::dev_malloc(p, bytes);
    if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
    rc = cuda_status(e);
  };
  alloc((void **)&s->grad, (size_t)kParams * 4);
  alloc((void **)&s->ident, R * 4);
  alloc((void **)&s->Q0, kQueryBatch * kInPad * 2);
  alloc((void **)&s->error, 4);
  const size_t E = (size_t)o.members;
  alloc((void **)&s->epi, E * kEpiFloats * 4);
  alloc((void **)&s->W1, E * kWidth * kInPad * 2);
  for (int i = 0; i < 3; ++i) {
    alloc((void **)&s->W[i], E * kWidth * kWidth * 2);
    alloc((void **)&s->WT[i], E * kWidth * kWidth * 2);
  }
  s->mem.resize(E);
  for (size_t e = 0; e < E; ++e) {
    Member &m = s->mem[e];
    alloc((void **)&m.P, (size_t)kParams * 4);
    alloc((void **)&m.M1, (size_t)kParams * 4);
    alloc((void **)&m.M2, (size_t)kParams * 4);
    m.W1 = s->W1 + e * kWidth * kInPad;
    for (int i = 0; i < 3; ++i) {
      m.W[i] = s->W[i] + e * kWidth * kWidth;
      m.WT[i] = s->WT[i] + e * kWidth * kWidth;
    }
  }
  if (rc != GELIO_OK) return fail(rc);
  // one member's training memory is taken here, so that a surrogate there is can
  // be trained; a group's comes with its first training, where it is to be had
  if ((rc = ensure_train(s, 1)) != GELIO_OK) return fail(rc);
  bool ok = make_map(&s->mQ0, s->Q0, kInPad, kQueryBatch, kTileM);
  ok = ok && make_map3(&s->tW1, s->W1, kInPad, kWidth, E, kWidth);
  for (int i = 0; i < 3; ++i)
    ok = ok && make_map3(&s->tW[i], s->W[i], kWidth, kWidth, E, kWidth) &&
         make_map3(&s->tWT[i], s->WT[i], kWidth, kWidth, E, kWidth);
  for (auto &m : s->mem) {
    ok = ok && make_map(&m.mW1, m.W1, kInPad, kWidth, kWidth);
    for (int i = 0; i < 3; ++i) ok = ok && make_map(&m.mW[i], m.W[i], kWidth, kWidth, kWidth);
  }
  if (!ok) return fail(GELIO_ERR_CUDA);
  // initial weights: uniform(+-sqrt(3 / fan_in)), zero biases
  uint64_t st = o.seed * 0x2545F4914F6CDD1Dull + 12345;
  std::vector<float> p(kParams);
  for (size_t e = 0; e < s->mem.size(); ++e) {
    std::fill(p.begin(), p.end(), 0.0f);
    auto fill = [&](int off, int n, int fan_in) {
      const double a = std::sqrt(3.0 / fan_in);
      for (int i = 0; i < n; ++i) p[off + i] = (float)(a * (2.0 * ((splitmix(st) >> 11) * 0x1.0p-53) - 1.0));
    };
    fill(kOffW1, kWidth * kFeatures, kFeatures);
    fill(kOffW2, kWidth * kWidth, kWidth);
    fill(kOffW3, kWidth * kWidth, kWidth);
    fill(kOffW4, kWidth * kWidth, kWidth);
    fill(kOffW5, kWidth, kWidth);
    if (cudaMemcpy(s->mem[e].P, p.data(), (size_t)kParams * 4, cudaMemcpyHostToDevice) != cudaSuccess)
      return fail(GELIO_ERR_CUDA);
    if ((rc = pack(s, s->mem[e])) != GELIO_OK) return fail(rc);
  }
  {
    std::vector<int> id(R);
    for (size_t i = 0; i < R; ++i) id[i] = (int)i;
    if (cudaMemcpy(s->ident, id.data(), R * 4, cudaMemcpyHostToDevice) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  }
  if (cudaStreamSynchronize(s->stream) != cudaSuccess) return fail(GELIO_ERR_CUDA);
  *out = s;
  return GELIO_OK;
}

void gelio_surrogate_destroy(gelio_surrogate *s) {
  if (!s) return;
  cudaSetDevice(s->device);
  if (s->side) cudaStreamSynchronize(s->side);
  if (s->stream) cudaStreamSynchronize(s->stream);
  free_all(s);
  delete s;
}

int32_t gelio_surrogate_add_spectra(gelio_surrogate *s, const gelio_sim_params *sims, const gelio_spectra *spectra,
                                    int32_t n, int64_t *n_rows) {
  if (!s || n < 0 || (n > 0 && (!sims || !spectra))) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  for (int i = 0; i < n; ++i) {
    const gelio_sim_params &q = sims[i];
    if (q.model != GELIO_MODEL_2D_GELIOSPHERE || q.injection != GELIO_INJ_LOG_GRID || q.grid_bins != 0)
      return GELIO_ERR_INVALID_ARGUMENT;
  }
  for (int i = 0; i < n; ++i) {
    const gelio_sim_params &q = sims[i];
    for (int j = 0; j < q.inj_points; ++j) {
      const double cnt = spectra[i].grid_n[j];
      const double w = spectra[i].grid_w[s->o.lis][j];
      if (cnt < s->o.min_count || !(w > 0.0)) continue;
      const double T = grid_energy(q, j);
      float f[kFeatures];
      gelio_surrogate_features(&q, T, f);
      s->feats.insert(s->feats.end(), f, f + kFeatures);
      s->targ.push_back((float)std::log((w / cnt) / lis(s->o.lis, T)));
    }
  }
  s->dirty = true;
  if (n_rows) *n_rows = (int64_t)s->targ.size();
  return GELIO_OK;
}

int32_t gelio_surrogate_add_rows(gelio_surrogate *s, const float *x, const float *t, int64_t n, int64_t *n_rows) {
  if (!s || n < 0 || (n > 0 && (!x || !t))) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  s->feats.insert(s->feats.end(), x, x + (size_t)n * kFeatures);
  s->targ.insert(s->targ.end(), t, t + (size_t)n);
  s->dirty = true;
  if (n_rows) *n_rows = (int64_t)s->targ.size();
  return GELIO_OK;
}

int32_t gelio_surrogate_train(gelio_surrogate *s, int32_t epochs, float *last_loss) {
  if (!s || epochs < 0) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  const size_t nrow = s->targ.size();
  if (nrow == 0) return GELIO_ERR_NOT_TRAINED;
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  if (s->dirty) {
    if (nrow > s->d_rows_cap) {
      if (s->d_feats) cudaFree(s->d_feats);
      if (s->d_targ) cudaFree(s->d_targ);
      s->d_feats = s->d_targ = nullptr;
      SUR_TRY(gelio::dev_malloc(&s->d_feats, nrow * kFeatures * 4));
      SUR_TRY(gelio::dev_malloc(&s->d_targ, nrow * 4));
      s->d_rows_cap = nrow;
    }
    SUR_TRY(cudaMemcpy(s->d_feats, s->feats.data(), nrow * kFeatures * 4, cudaMemcpyHostToDevice));
    SUR_TRY(cudaMemcpy(s->d_targ, s->targ.data(), nrow * 4, cudaMemcpyHostToDevice));
    s->d_rows_used = nrow;
    s->dirty = false;
  }
  const int R = s->rows;
  const int steps = (int)std::max<size_t>(1, nrow / (size_t)R);
  // as large a group as the device has memory for
  const int E = (int)s->mem.size();
  int G = group_size(s), rc;
  while ((rc = ensure_group(s, G, steps, nrow)) == GELIO_ERR_OUT_OF_MEMORY && G > 1) {
    (void)cudaGetLastError();
    G = (G + 1) / 2;
  }
  if (rc != GELIO_OK) return rc;
  const long long total = (long long)epochs * steps;
  std::vector<float> sl((size_t)G * steps);
  for (int m0 = 0; m0 < E; m0 += G) {
    const int g = std::min(G, E - m0);
    if ((rc = train_group(s, m0, g, epochs, steps, total, nrow, sl.data())) != GELIO_OK) return rc;
    for (int k = 0; k < g; ++k) {
      double loss = 0.0;
      if (epochs > 0) {
        for (int st = 0; st < steps; ++st) loss += sl[(size_t)k * steps + st];
        loss /= (double)std::min<size_t>(nrow, (size_t)steps * R);
      }
      if (last_loss) last_loss[m0 + k] = (float)loss;
      s->mem[m0 + k].trained = true;
    }
  }
  return GELIO_OK;
}

static void touch_pages(void *p, size_t bytes) {
  volatile unsigned char *b = static_cast<volatile unsigned char *>(p);
  for (size_t i = 0; i < bytes; i += 4096) b[i] = b[i];
  if (bytes) b[bytes - 1] = b[bytes - 1];
}

// Ensemble inference of every LOG_GRID point of sims[0..n): the simulations
// and their row offsets go up (one copy from pinned staging), k_query builds the
// inputs of a batch, every member's layers run on it in one launch and
// k_ensemble forms mean and std.  Few rows come back through the staging, the
// error flag with them; many straight into the caller's arrays (through the
// staging the host's two copies of 3.2 MB took 200 us of an 870 us call), after
// the flag has been looked at: a call that fails leaves the arrays as they were.
// enqueue_infer_sims may return with work under way that reads or writes host
// memory; infer_sims does not.
int enqueue_infer_sims(gelio_surrogate *s, const gelio_sim_params *sims, int n, size_t rows, double *ln_ratio,
               double *ln_std) {
  const int E = (int)s->mem.size();
  const size_t stride = (rows + kTileM - 1) / kTileM * kTileM;
  // the simulations and their row offsets travel in one copy, so they share
  // one allocation (n * 96 bytes keeps the offsets 8-byte aligned)
  const size_t up = (size_t)n * sizeof(gelio_sim_params) + (size_t)(n + 1) * sizeof(long long);
  // staged / straight, us: 4,000 rows 65 / 77, 8,000 94 / 101, 16,000 118 / 122, 32,000 181 / 170
  constexpr size_t kStagedRows = 16384;
  const bool staged = rows <= kStagedRows;
  const size_t down = (staged ? 2 * rows * sizeof(double) : 0) + sizeof(double);   // ... and the error flag
  int rc = GELIO_OK;
  if (up > s->pup_cap) {
    unsigned char *fresh = nullptr;
    SUR_TRY(gelio::dev_malloc(&fresh, up));
    if (s->d_pup) cudaFree(s->d_pup);
    s->d_pup = fresh;
    s->pup_cap = up;
  }
  const gelio_sim_params *d_psims = reinterpret_cast<const gelio_sim_params *>(s->d_pup);
  const long long *d_pfirst = reinterpret_cast<const long long *>(s->d_pup + (size_t)n * sizeof(gelio_sim_params));
  if (stride > s->prows_cap) {
    if (s->d_py) cudaFree(s->d_py);
    if (s->d_pstat) cudaFree(s->d_pstat);
    s->d_py = nullptr;
    s->d_pstat = nullptr;
    s->prows_cap = 0;
    SUR_TRY(gelio::dev_malloc(&s->d_py, E * stride * sizeof(float)));
    SUR_TRY(gelio::dev_malloc(&s->d_pstat, (2 * stride + 1) * sizeof(double)));
    s->prows_cap = stride;
  }
  if (std::max(up, down) > s->pstage_cap) {
    if (s->h_pstage) cudaFreeHost(s->h_pstage);
    s->h_pstage = nullptr;
    s->pstage_cap = 0;
    SUR_TRY(gelio::pinned_malloc(&s->h_pstage, std::max(up, down)));
    s->pstage_cap = std::max(up, down);
  }
  std::memcpy(s->h_pstage, sims, (size_t)n * sizeof(gelio_sim_params));
  long long *first = reinterpret_cast<long long *>(s->h_pstage + (size_t)n * sizeof(gelio_sim_params));
  first[0] = 0;
  for (int i = 0; i < n; ++i) first[i + 1] = first[i] + sims[i].inj_points;
  SUR_TRY(cudaEventRecord(s->ev0, s->stream));
  SUR_TRY(cudaMemcpyAsync(s->d_pup, s->h_pstage, up, cudaMemcpyHostToDevice, s->stream));
  size_t padded = 0;
  for (size_t off = 0; off < rows; off += kQueryBatch) {
    const int c = (int)std::min<size_t>(kQueryBatch, rows - off);
    const int M = (c + kTileM - 1) / kTileM * kTileM;
    padded += (size_t)M;
    k_query<<<(M + kQueryBlock - 1) / kQueryBlock, kQueryBlock, 0, s->stream>>>(
        d_psims, d_pfirst, n, (long long)off, c, M, E, (long long)stride, s->Q0, s->d_py);
    SUR_TRY(cudaGetLastError());
    if ((rc = infer_fused(s, 0, E, c, s->d_py + off, (long long)stride)) != GELIO_OK) return rc;
  }
  SUR_TRY(launch_early(s, k_ensemble, (unsigned)((rows + 127) / 128), 128, 0, (const float *)s->d_py, E, (long long)rows,
                       (long long)stride, s->d_pstat, s->d_pstat + rows, (const unsigned *)s->error,
                       staged ? reinterpret_cast<unsigned *>(s->d_pstat + 2 * rows)
                              : reinterpret_cast<unsigned *>(s->h_pstage)));      // pinned: the kernel writes it
  SUR_TRY(cudaEventRecord(s->ev1, s->stream));
  const size_t bytes = rows * sizeof(double);
  if (staged) {
    SUR_TRY(cudaMemcpyAsync(s->h_pstage, s->d_pstat, down, cudaMemcpyDeviceToHost, s->stream));
  } else {
    // while the device works: the caller's pages are mapped, their values kept
    // (a copy into pages that no one has touched yet took 1.9 ms instead of 40 us)
    touch_pages(ln_ratio, bytes);
    if (ln_std) touch_pages(ln_std, bytes);
  }
  SUR_TRY(cudaStreamSynchronize(s->stream));
  unsigned error = 0;
  std::memcpy(&error, s->h_pstage + down - sizeof(double), sizeof(error));
  if (error) return check_error(s);
  if (staged) {
    std::memcpy(ln_ratio, s->h_pstage, bytes);
    if (ln_std) std::memcpy(ln_std, s->h_pstage + bytes, bytes);
  } else {
    SUR_TRY(cudaMemcpyAsync(ln_ratio, s->d_pstat, bytes, cudaMemcpyDeviceToHost, s->stream));
    if (ln_std) SUR_TRY(cudaMemcpyAsync(ln_std, s->d_pstat + rows, bytes, cudaMemcpyDeviceToHost, s->stream));
    SUR_TRY(cudaStreamSynchronize(s->stream));
  }
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, s->ev0, s->ev1) == cudaSuccess) {
    s->last_ms = ms;
    s->last_flop = gemm_flop(padded, (size_t)E);
  }
  return GELIO_OK;
}

int infer_sims(gelio_surrogate *s, const gelio_sim_params *sims, int n, size_t rows, double *ln_ratio,
               double *ln_std) {
  const int rc = enqueue_infer_sims(s, sims, n, rows, ln_ratio, ln_std);
  if (rc != GELIO_OK) cudaStreamSynchronize(s->stream);
  return rc;
}

// For tests of calls that fail: sets the device's error flag, as a kernel does
// one of whose waits ran out.
int32_t gelio_internal_surrogate_error(gelio_surrogate *s, uint32_t code) {
  if (!s) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  SUR_TRY(cudaSetDevice(s->device));
  SUR_TRY(cudaMemcpyAsync(s->error, &code, sizeof(code), cudaMemcpyHostToDevice, s->stream));
  SUR_TRY(cudaStreamSynchronize(s->stream));
  return GELIO_OK;
}

int32_t gelio_surrogate_forward(gelio_surrogate *s, int32_t member, const float *x, int32_t n, float *y) {
  if (!valid_member(s, member) || n < 0 || (n > 0 && (!x || !y))) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  return infer_rows(s, member, x, (size_t)n, y);
}

int32_t gelio_surrogate_gradient(gelio_surrogate *s, int32_t member, const float *x, const float *t, int32_t n,
                                 float *loss, float *grad) {
  if (!valid_member(s, member) || n <= 0 || !x || !t || !grad) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  if (n > s->rows) return GELIO_ERR_INVALID_ARGUMENT;
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  float *d_x = nullptr, *d_t = nullptr, *d_loss = nullptr;
  int rc = GELIO_OK;
  if (gelio::dev_malloc(&d_x, (size_t)n * kFeatures * 4) != cudaSuccess || gelio::dev_malloc(&d_t, (size_t)n * 4) != cudaSuccess ||
      gelio::dev_malloc(&d_loss, 4) != cudaSuccess)
    rc = GELIO_ERR_OUT_OF_MEMORY;
  if (rc == GELIO_OK && (cudaMemcpyAsync(d_x, x, (size_t)n * kFeatures * 4, cudaMemcpyHostToDevice, s->stream) !=
                             cudaSuccess ||
                         cudaMemcpyAsync(d_t, t, (size_t)n * 4, cudaMemcpyHostToDevice, s->stream) != cudaSuccess))
    rc = GELIO_ERR_CUDA;
  if (rc == GELIO_OK) rc = ensure_train(s, 1);
  if (rc == GELIO_OK) {
    k_gather<<<(s->rows + 127) / 128, 128, 0, s->stream>>>(d_x, d_t, s->ident, n, 0, s->rows, s->tb.X0, s->tb.y,
                                                           s->tb.yhat);
    UpdateArgs u{};
    u.P[0] = s->mem[member].P;
    u.grad = s->grad;
    u.loss = d_loss;
    rc = train_step(s, member, 1, n, u);
  }
  float l = 0.f;
  if (rc == GELIO_OK &&
      (cudaMemcpyAsync(grad, s->grad, (size_t)kParams * 4, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
       cudaMemcpyAsync(&l, d_loss, 4, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess))
    rc = GELIO_ERR_CUDA;
  if (rc == GELIO_OK) rc = check_error(s);
  cudaStreamSynchronize(s->side);
  cudaStreamSynchronize(s->stream);
  if (loss) *loss = l / (float)n;
  cudaFree(d_x);
  cudaFree(d_t);
  cudaFree(d_loss);
  return rc;
}

int32_t gelio_surrogate_last_inference(gelio_surrogate *s, double *device_ms, double *flop) {
  if (!s) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  if (device_ms) *device_ms = s->last_ms;
  if (flop) *flop = s->last_flop;
  return GELIO_OK;
}

int32_t gelio_surrogate_get_params(gelio_surrogate *s, int32_t member, float *params) {
  if (!valid_member(s, member) || !params) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  SUR_TRY(cudaMemcpyAsync(params, s->mem[member].P, (size_t)kParams * 4, cudaMemcpyDeviceToHost, s->stream));
  SUR_TRY(cudaStreamSynchronize(s->stream));
  return GELIO_OK;
}

int32_t gelio_surrogate_set_params(gelio_surrogate *s, int32_t member, const float *params) {
  if (!valid_member(s, member) || !params) return GELIO_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  Member &m = s->mem[member];
  SUR_TRY(cudaMemcpyAsync(m.P, params, (size_t)kParams * 4, cudaMemcpyHostToDevice, s->stream));
  SUR_TRY(cudaMemsetAsync(m.M1, 0, (size_t)kParams * 4, s->stream));
  SUR_TRY(cudaMemsetAsync(m.M2, 0, (size_t)kParams * 4, s->stream));
  m.adam_t = 0;
  int rc = pack(s, m);
  if (rc != GELIO_OK) return rc;
  SUR_TRY(cudaStreamSynchronize(s->stream));
  m.trained = true;
  return GELIO_OK;
}

int32_t gelio_surrogate_predict(gelio_surrogate *s, const gelio_sim_params *sims, int32_t n, double *ln_ratio,
                                double *ln_std) {
  if (!s || n < 0 || (n > 0 && (!sims || !ln_ratio))) return GELIO_ERR_INVALID_ARGUMENT;
  for (auto &m : s->mem)
    if (!m.trained) return GELIO_ERR_NOT_TRAINED;
  size_t rows = 0;
  for (int i = 0; i < n; ++i) {
    if (sims[i].injection != GELIO_INJ_LOG_GRID || sims[i].inj_points < 1 || sims[i].inj_points > GELIO_GRID_MAX ||
        !(sims[i].inj_min > 0.f) || !(sims[i].inj_max > 0.f))
      return GELIO_ERR_INVALID_ARGUMENT;
    rows += (size_t)sims[i].inj_points;
  }
  if (rows == 0) return GELIO_OK;
  std::lock_guard<std::mutex> lock(s->mu);
  SUR_TRY(cudaSetDevice(s->device));
  (void)cudaGetLastError();   // a launch check below must see only this call's errors
  return infer_sims(s, sims, n, rows, ln_ratio, ln_std);
}

int32_t gelio_surrogate_spectra(gelio_surrogate *s, const gelio_sim_params *sims, int32_t n,
                                const gelio_run_opts *mc_opts, double *ln_ratio, double *ln_std, int32_t *used_mc) {
  if (!s || n < 0 || (n > 0 && (!sims || !ln_ratio || !ln_std))) return GELIO_ERR_INVALID_ARGUMENT;
  int rc = gelio_surrogate_predict(s, sims, n, ln_ratio, ln_std);
  if (rc != GELIO_OK) return rc;
  std::vector<int> need;
  std::vector<size_t> first(n + 1, 0);
  for (int i = 0; i < n; ++i) first[i + 1] = first[i] + (size_t)sims[i].inj_points;
  for (int i = 0; i < n; ++i) {
    double worst = 0.0;
    for (int j = 0; j < sims[i].inj_points; ++j) {
      const double T = grid_energy(sims[i], j);
      if (T >= s->o.t_min && T <= s->o.t_max) worst = std::max(worst, ln_std[first[i] + j]);
    }
    const bool mc = worst > s->o.fallback_std;
    if (used_mc) used_mc[i] = mc ? 1 : 0;
    if (mc) need.push_back(i);
  }
  if (need.empty()) return GELIO_OK;
  std::vector<gelio_sim_params> sub;
  for (int i : need) sub.push_back(sims[i]);
  std::vector<gelio_spectra> out(sub.size());
  rc = gelio_run(s->ctx, sub.data(), (int32_t)sub.size(), mc_opts, out.data(), nullptr);
  if (rc != GELIO_OK && rc < GELIO_WARN_FIRST) return rc;
  for (size_t k = 0; k < need.size(); ++k) {
    const int i = need[k];
    for (int j = 0; j < sims[i].inj_points; ++j) {
      const double cnt = out[k].grid_n[j], w = out[k].grid_w[s->o.lis][j];
      const double T = grid_energy(sims[i], j);
      ln_ratio[first[i] + j] = (cnt > 0 && w > 0) ? std::log((w / cnt) / lis(s->o.lis, T)) : NAN;
      ln_std[first[i] + j] = 0.0;
    }
  }
  return GELIO_OK;
}

}  // extern "C"
