// matmul on strided row-major views and the three GEMMs of fl::linear's
// gradFunc (flashlight/fl/autograd/Functions.cpp:827-946, 1255-1309;
// TensorBackend::matmul, flashlight/fl/tensor/TensorBackend.h:213-217).
// STRICT mode runs the fp32-FMA kernel of simt_gemm.cuh; TF32 mode hands the
// shapes the tensor-core kernel covers to tc_gemm (tcgen05, fp32 accumulate in
// tensor memory) and everything else to the fp32 kernel.
#include "simt_gemm.cuh"
#include "tc_gemm.cuh"

namespace flb200 {
namespace {

// Which way an operand is read: 16-byte chunks along its unit stride where base, strides and
// extent allow it, single elements otherwise.
int loader_kind(const void* p, long long row, long long col, long long z, long long rows, long long K,
                long long batch) {
  const bool vec = aligned16(p) && (batch == 1 || z % 4 == 0);
  if (col == 1 && vec && row % 4 == 0 && K % 4 == 0) return kVecK;
  if (row == 1 && vec && col % 4 == 0 && rows % 4 == 0) return kVecRow;
  return row == 1 && col != 1 ? kElemRows : kElemK;
}

template <int AKIND, int BKIND>
int matmul_simt_as(const flb200_matmul_desc* d, const float* a, const float* b,
                   const StridedEpilogue& ep, void* ws, size_t ws_bytes, cudaStream_t st) {
  // Operand B is indexed (row = n, k): row stride is b_col, k stride is b_row.
  return launch_simt_gemm("matmul", StridedLoader<AKIND>{a, d->a_row, d->a_col, d->a_batch, (int)d->m},
                          StridedLoader<BKIND>{b, d->b_col, d->b_row, d->b_batch, (int)d->n}, ep, d->m,
                          d->n, d->k, d->batch, ws, ws_bytes, st);
}
template <int AKIND>
int matmul_simt_b(int bkind, const flb200_matmul_desc* d, const float* a, const float* b,
                  const StridedEpilogue& ep, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (bkind == kVecK) return matmul_simt_as<AKIND, kVecK>(d, a, b, ep, ws, ws_bytes, st);
  if (bkind == kVecRow) return matmul_simt_as<AKIND, kVecRow>(d, a, b, ep, ws, ws_bytes, st);
  if (bkind == kElemRows) return matmul_simt_as<AKIND, kElemRows>(d, a, b, ep, ws, ws_bytes, st);
  return matmul_simt_as<AKIND, kElemK>(d, a, b, ep, ws, ws_bytes, st);
}

int matmul_simt(const flb200_matmul_desc* d, const void* a, const void* b, void* c, void* ws,
                size_t ws_bytes, cudaStream_t st) {
  constexpr long long kMostK = 1LL << 30;  // the kernel counts k in 32 bits: longer sums in pieces
  if (d->k > kMostK) {
    flb200_matmul_desc part = *d;
    for (long long k0 = 0; k0 < d->k; k0 += kMostK) {
      part.k = d->k - k0 < kMostK ? d->k - k0 : kMostK;
      if (int rc = matmul_simt(&part, static_cast<const float*>(a) + k0 * d->a_col,
                               static_cast<const float*>(b) + k0 * d->b_row, c, ws, ws_bytes, st))
        return rc;
      part.beta = 1.f;
    }
    return FLB200_OK;
  }
  StridedEpilogue ep{static_cast<float*>(c), nullptr, d->alpha, d->beta, 0, 0, d->c_row, d->c_col,
                     d->c_batch};
  ep.along_m = d->c_row == 1 && d->c_col != 1;
  ep.vec = (ep.along_m ? d->m % 4 == 0 && d->c_col % 4 == 0 : d->c_col == 1 && d->n % 4 == 0 && d->c_row % 4 == 0) &&
           (d->batch == 1 || d->c_batch % 4 == 0) && aligned16(c);
  const int ak = loader_kind(a, d->a_row, d->a_col, d->a_batch, d->m, d->k, d->batch);
  const int bk = loader_kind(b, d->b_col, d->b_row, d->b_batch, d->n, d->k, d->batch);
  const float* ap = static_cast<const float*>(a);
  const float* bp = static_cast<const float*>(b);
  if (ak == kVecK) return matmul_simt_b<kVecK>(bk, d, ap, bp, ep, ws, ws_bytes, st);
  if (ak == kVecRow) return matmul_simt_b<kVecRow>(bk, d, ap, bp, ep, ws, ws_bytes, st);
  if (ak == kElemRows) return matmul_simt_b<kElemRows>(bk, d, ap, bp, ep, ws, ws_bytes, st);
  return matmul_simt_b<kElemK>(bk, d, ap, bp, ep, ws, ws_bytes, st);
}

int check_desc(const flb200_matmul_desc* d, const void* a, const void* b, const void* c) {
  FLB200_REQUIRE(d, "matmul: null descriptor");
  FLB200_REQUIRE(d->m >= 0 && d->n >= 0 && d->k >= 0 && d->batch >= 1, "matmul: negative extent");
  FLB200_REQUIRE(d->dtype == FLB200_F32 || d->dtype == FLB200_BF16,
                 "matmul: f32 and bf16 are built (dtype %d)", d->dtype);
  FLB200_REQUIRE(d->math_mode >= FLB200_MATH_STRICT_F32 && d->math_mode <= FLB200_MATH_F32X3,
                 "matmul: unknown math mode %d", d->math_mode);
  FLB200_REQUIRE((a && b && c) || d->m == 0 || d->n == 0, "matmul: null matrix");
  return FLB200_OK;
}

int run_matmul(const flb200_matmul_desc* d, const void* a, const void* b, void* c, void* ws,
               size_t ws_bytes, void* stream) {
  if (int st = check_desc(d, a, b, c)) return st;
  if (d->m == 0 || d->n == 0) return FLB200_OK;
  cudaStream_t st = as_stream(stream);
  if (d->dtype == FLB200_BF16) {
    // bf16 operands, fp32 accumulation, bf16 result: tensor cores only (no fp32-FMA kernel
    // reads bf16), whatever the math mode says
    if (!tc_gemm_supported(d, a, b, c))
      return fail(FLB200_UNSUPPORTED,
                  "matmul: bf16 needs the tensor-core path (sm_100, 16-byte aligned operands "
                  "with one unit stride each)");
    return tc_gemm_run(d, a, b, c, ws, ws_bytes, st);
  }
  tc::X3Scope x3(d->math_mode == FLB200_MATH_F32X3);
  if (d->math_mode != FLB200_MATH_STRICT_F32 && tc_gemm_supported(d, a, b, c))
    return tc_gemm_run(d, a, b, c, ws, ws_bytes, st);
  return matmul_simt(d, a, b, c, ws, ws_bytes, st);
}

}  // namespace
}  // namespace flb200

using namespace flb200;

extern "C" {

size_t flb200_matmul_workspace_bytes(const flb200_matmul_desc* d) {
  if (!d || d->m <= 0 || d->n <= 0 || d->batch <= 0) return 0;
  struct Key { long long m, n, k, batch; int mode, sm, cc, outer_x3; };
  static thread_local Memo<Key, size_t> memo;
  const DeviceInfo& di = device_info();
  const Key key = {d->m, d->n, d->k, d->batch, d->math_mode, di.sm_count, di.cc_major, tc::x3_enabled() ? 1 : 0};
  if (const size_t* known = memo.find(key)) return *known;
  size_t need = plan_simt(d->m, d->n, d->k, d->batch).workspace_bytes;
  const size_t tc = tc_gemm_workspace_bytes(d);
  return memo.put(key, need > tc ? need : tc);
}

size_t flb200_matmul_call_workspace_bytes(const flb200_matmul_desc* d, const void* a, const void* b,
                                          const void* c) {
  if (check_desc(d, a, b, c) || d->m == 0 || d->n == 0) return 0;
  tc::X3Scope x3(d->dtype == FLB200_F32 && d->math_mode == FLB200_MATH_F32X3);
  if ((d->dtype == FLB200_BF16 || d->math_mode != FLB200_MATH_STRICT_F32) && tc_gemm_supported(d, a, b, c))
    return tc_gemm_call_workspace_bytes(d, a, b, c);
  return flb200_matmul_workspace_bytes(d);
}

int flb200_matmul(const flb200_matmul_desc* d, const void* a, const void* b, void* c,
                  void* workspace, size_t workspace_bytes, void* stream) {
  return run_matmul(d, a, b, c, workspace, workspace_bytes, stream);
}

int flb200_matmul_wide(const flb200_matmul_desc* d, const void* a, const void* b, float* c,
                       void* workspace, size_t workspace_bytes, void* stream) {
  if (int st = check_desc(d, a, b, c)) return st;
  if (d->dtype == FLB200_F32) return run_matmul(d, a, b, c, workspace, workspace_bytes, stream);
  if (d->m == 0 || d->n == 0) return FLB200_OK;
  if (!tc_gemm_supported(d, a, b, c))
    return fail(FLB200_UNSUPPORTED, "matmul_wide: bf16 needs the tensor-core path");
  return tc_gemm_run(d, a, b, c, workspace, workspace_bytes, as_stream(stream), nullptr, 0, nullptr,
                     true);
}

// which: 0 forward, 1 backward-input, 2 backward-weight.  A NULL / short
// workspace is accepted by the three calls: the contraction then runs unsplit.
size_t flb200_linear_workspace_bytes(int64_t O, int64_t I, int64_t cols, int which) {
  flb200_matmul_desc d = {};
  d.batch = 1;
  if (which == 0) { d.m = cols; d.n = O; d.k = I; }
  else if (which == 1) { d.m = cols; d.n = I; d.k = O; }
  else { d.m = I; d.n = O; d.k = cols; }
  d.math_mode = FLB200_MATH_TF32;  // (the call may come in either tensor-core mode)
  const size_t tf32 = flb200_matmul_workspace_bytes(&d);
  d.math_mode = FLB200_MATH_F32X3;
  const size_t x3 = flb200_matmul_workspace_bytes(&d);
  return tf32 > x3 ? tf32 : x3;
}

// fl layout (column-major): weight (o,i) at o + i*O; x (i,col) at i + col*I;
// y (o,col) at o + col*O.  Row-major GEMM views used below:
//   forward          Y[col][o]  = sum_i X[col][i] * Wt[i][o]      (+ bias[o])
//   backward input   dX[col][i] = sum_o dY[col][o] * W(o,i)
//   backward weight  dWt[i][o]  = sum_col X[col][i] * dY[col][o]
int flb200_linear_forward(int64_t O, int64_t I, int64_t cols, const void* weight, const void* x,
                          const void* bias, void* y, int math_mode, void* workspace,
                          size_t workspace_bytes, void* stream) {
  flb200_matmul_desc d = {};
  d.m = cols; d.n = O; d.k = I; d.batch = 1;
  d.a_row = I; d.a_col = 1;
  d.b_row = O; d.b_col = 1;
  d.c_row = O; d.c_col = 1;
  d.alpha = 1.f; d.beta = 0.f;
  d.dtype = FLB200_F32; d.math_mode = math_mode;
  if (int st = run_matmul(&d, x, weight, y, workspace, workspace_bytes, stream)) return st;
  if (bias) return flb200_channel_bias_add(y, static_cast<const float*>(bias), y, cols, O, 1,
                                           FLB200_F32, stream);
  return FLB200_OK;
}

int flb200_linear_bias_act_forward(int64_t O, int64_t I, int64_t cols, const void* weight,
                                   const void* x, const float* bias, void* y, void* pre, int act,
                                   int dtype, int math_mode, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  FLB200_REQUIRE(act == FLB200_ACT_NONE || act == FLB200_ACT_GELU,
                 "linear_bias_act_forward: unknown activation %d", act);
  FLB200_REQUIRE(act != FLB200_ACT_NONE || pre == nullptr,
                 "linear_bias_act_forward: a pre-activation copy needs an activation");
  flb200_matmul_desc d = {};
  d.m = cols; d.n = O; d.k = I; d.batch = 1;
  d.a_row = I; d.a_col = 1;
  d.b_row = O; d.b_col = 1;
  d.c_row = O; d.c_col = 1;
  d.alpha = 1.f; d.beta = 0.f;
  d.dtype = dtype; d.math_mode = math_mode;
  if (int st = check_desc(&d, x, weight, y)) return st;
  if (cols == 0 || O == 0) return FLB200_OK;
  if ((dtype != FLB200_BF16 && math_mode == FLB200_MATH_STRICT_F32) ||
      !tc_gemm_supported(&d, x, weight, y) || (bias && !aligned16(bias)))
    return fail(FLB200_UNSUPPORTED,
                "linear_bias_act_forward: needs the tensor-core path (run linear, bias and "
                "activation one by one)");
  tc::X3Scope x3(dtype == FLB200_F32 && math_mode == FLB200_MATH_F32X3);
  return tc_gemm_run(&d, x, weight, y, workspace, workspace_bytes, as_stream(stream), bias, act,
                     pre);
}

int flb200_linear_backward_input(int64_t O, int64_t I, int64_t cols, const void* weight,
                                 const void* grad_y, void* grad_x, int math_mode, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  flb200_matmul_desc d = {};
  d.m = cols; d.n = I; d.k = O; d.batch = 1;
  d.a_row = O; d.a_col = 1;          // dY[col][o]
  d.b_row = 1; d.b_col = O;          // B(k=o, n=i) = W(o,i) at o + i*O
  d.c_row = I; d.c_col = 1;
  d.alpha = 1.f; d.beta = 0.f;
  d.dtype = FLB200_F32; d.math_mode = math_mode;
  return run_matmul(&d, grad_y, weight, grad_x, workspace, workspace_bytes, stream);
}

int flb200_linear_backward_weight(int64_t O, int64_t I, int64_t cols, const void* grad_y,
                                  const void* x, void* grad_w, int math_mode, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  flb200_matmul_desc d = {};
  d.m = I; d.n = O; d.k = cols; d.batch = 1;
  d.a_row = 1; d.a_col = I;          // A(m=i, k=col) = X[col][i]
  d.b_row = O; d.b_col = 1;          // B(k=col, n=o) = dY[col][o]
  d.c_row = O; d.c_col = 1;          // dWt[i][o]
  d.alpha = 1.f; d.beta = 0.f;
  d.dtype = FLB200_F32; d.math_mode = math_mode;
  return run_matmul(&d, x, grad_y, grad_w, workspace, workspace_bytes, stream);
}

}  // extern "C"
