// tsb200_linear: picks the kernel for LinearCompressed.forward
// (transformersurgeon/blocks/linear_compressed.py:81-105).
#include "tc_common.cuh"

namespace tsb {
int validate_linear(const tsb200_linear_desc* d, const void* x, void* y, int64_t M, bool& noop);
// Tensor-core path (linear_tc.cu); returns TSB200_ERR_UNSUPPORTED when the shape/dtype is
// outside what it implements, in which case the CUDA-core kernel takes the call.
int linear_tc(const tsb200_linear_desc* d, const void* x, void* y, int64_t M, void* workspace, size_t workspace_bytes,
              cudaStream_t s);
int linear_argmax_tc(const tsb200_linear_desc* d, const void* x, int64_t* tokens, int64_t M, void* amax, int* status, cudaStream_t s);
int argmax_rows(const void* y, int dtype, int64_t M, int64_t N, int64_t* tokens, cudaStream_t s);
}  // namespace tsb

using namespace tsb;

// Workspace of the greedy head: the linear layer's own workspace, then either the per-tile (maximum, column) pairs of
// the fused route or the logits of the general route (whichever is larger).
extern "C" size_t tsb200_linear_argmax_workspace_bytes(const tsb200_linear_desc* d, int64_t M) {
  if (!d || M <= 0) return tsb200_linear_workspace_bytes(d, M);
  const size_t lin = (tsb200_linear_workspace_bytes(d, M) + 255) / 256 * 256;
  const size_t tiles = (size_t)((d->out_features + 127) / 128);
  const size_t pairs = (size_t)M * tiles * 8;
  const size_t logits = (size_t)M * (size_t)d->out_features * (d->act_dtype == TSB200_F32 ? 4 : 2);
  return lin + (pairs > logits ? pairs : logits) + 256;
}

extern "C" int tsb200_linear_argmax(const tsb200_linear_desc* d, const void* x, int64_t* tokens, int64_t M, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!d || M < 0) return TSB200_ERR_ARG;
  if (M == 0) return TSB200_OK;
  if (!tokens || !x || !workspace || !aligned(workspace, 256)) return TSB200_ERR_ARG;
  if (workspace_bytes < tsb200_linear_argmax_workspace_bytes(d, M)) return TSB200_ERR_WORKSPACE;
  const size_t lin = (tsb200_linear_workspace_bytes(d, M) + 255) / 256 * 256;
  void* extra = (uint8_t*)workspace + lin;
  cudaStream_t s = as_stream(stream);
  int st = linear_argmax_tc(d, x, tokens, M, extra, (int*)workspace, s);
  if (st != TSB200_ERR_UNSUPPORTED) return st;
  st = tsb200_linear(d, x, extra, M, workspace, lin, stream);          // logits into the scratch, then their argmax
  if (st != TSB200_OK) return st;
  return argmax_rows(extra, d->act_dtype, M, d->out_features, tokens, s);
}

extern "C" int tsb200_argmax(const void* y, int dtype, int64_t M, int64_t N, int64_t* tokens, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (M < 0 || N <= 0) return TSB200_ERR_ARG;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (M == 0) return TSB200_OK;
  if (!y || !tokens) return TSB200_ERR_ARG;
  return argmax_rows(y, dtype, M, N, tokens, as_stream(stream));
}

namespace {
bool f32_factor(int bits) { return bits == 32 || (bits <= 8); }

// fp32 activations: both factors on the FMA kernel, the second launch chained to the first; n layers that read the same x go
// through together when their factors are alike.  h: the rank-r intermediates, one behind the other.
int linear_f32(const tsb200_linear_desc* const* d, int n, const void* x, void* const* y, int64_t M, float* h, cudaStream_t s,
               const tsb200_norm_desc* norm = nullptr) {
  GemmSpec v[4], u[4];
  const bool low = d[0]->rank > 0;
  for (int i = 0; i < n; ++i) {
    if (d[i]->act_dtype != TSB200_F32 || !f32_factor(d[i]->u_bits) || (low && !f32_factor(d[i]->v_bits))) return TSB200_ERR_UNSUPPORTED;
    const int64_t ku = low ? d[i]->rank : d[i]->in_features;
    v[i] = GemmSpec{d[i]->v, d[i]->v_scale, nullptr, x, h, d[i]->rank, d[i]->in_features};
    u[i] = GemmSpec{d[i]->u, d[i]->u_scale, d[i]->bias, low ? (const void*)h : x, y[i], d[i]->out_features, ku};
    h += M * d[i]->rank;
  }
  if (low) {
    const int st = gemm_f32(v, n, d[0]->v_bits, M, g_pdl != 0, s, norm);
    if (st != TSB200_OK) return st;
  }
  return gemm_f32(u, n, d[0]->u_bits, M, low || g_pdl, s, low ? nullptr : norm);
}

bool alike(const tsb200_linear_desc* a, const tsb200_linear_desc* b) {
  return a->act_dtype == b->act_dtype && a->in_features == b->in_features && a->rank == b->rank && a->u_bits == b->u_bits &&
         (a->rank == 0 || a->v_bits == b->v_bits);
}
size_t f32_intermediate_bytes(const tsb200_linear_desc* const* d, int n, int64_t M) {
  size_t b = 0;
  for (int i = 0; i < n; ++i) b += (size_t)M * (size_t)d[i]->rank * 4;
  return b;
}
}  // namespace

extern "C" size_t tsb200_linear_group_workspace_bytes(const tsb200_linear_desc* const* d, int n, int64_t M) {
  size_t b = tc::kWsHeader;
  if (!d || n <= 0 || M <= 0) return b;
  for (int i = 0; i < n; ++i) {
    const size_t one = d[i] ? tsb200_linear_workspace_bytes(d[i], M) : 0;
    if (one > b) b = one;
  }
  for (int i = 0; i < n; ++i)
    if (!d[i]) return b;
  const size_t f = tc::kWsHeader + f32_intermediate_bytes(d, n, M);
  return f > b ? f : b;
}

extern "C" int tsb200_linear_group(const tsb200_linear_desc* const* d, int n, const void* x, void* const* y, int64_t M, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!d || !y || n < 1) return TSB200_ERR_ARG;
  bool noop = false, group = n > 1 && n <= 4;
  for (int i = 0; i < n; ++i) {
    const int st = validate_linear(d[i], x, y[i], M, noop);
    if (st != TSB200_OK) return st;
    group = group && alike(d[0], d[i]);
  }
  if (noop) return TSB200_OK;
  if (!workspace || !aligned(workspace, 256)) return TSB200_ERR_ARG;
  if (workspace_bytes < tsb200_linear_group_workspace_bytes(d, n, M)) return TSB200_ERR_WORKSPACE;
  if (group && d[0]->act_dtype == TSB200_F32) {
    const int st = linear_f32(d, n, x, y, M, (float*)((uint8_t*)workspace + tc::kWsHeader), as_stream(stream));
    if (st != TSB200_ERR_UNSUPPORTED) return st;
  }
  for (int i = 0; i < n; ++i) {
    const int st = tsb200_linear(d[i], x, y[i], M, workspace, workspace_bytes, stream);
    if (st != TSB200_OK) return st;
  }
  return TSB200_OK;
}

extern "C" int tsb200_norm_linear_group(const tsb200_norm_desc* norm, const tsb200_linear_desc* const* d, int n, void* const* y, int64_t M, void* workspace,
                                        size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!norm || !norm->residual || !norm->weight || !norm->residual_out || !d || !y || n < 1) return TSB200_ERR_ARG;
  bool noop = false;
  for (int i = 0; i < n; ++i) {
    const int st = validate_linear(d[i], norm->residual, y[i], M, noop);
    if (st != TSB200_OK) return st;
    if (!alike(d[0], d[i])) return TSB200_ERR_UNSUPPORTED;
  }
  if (noop) return TSB200_OK;
  if (n > 4 || d[0]->act_dtype != TSB200_F32) return TSB200_ERR_UNSUPPORTED;
  if (!workspace || !aligned(workspace, 256)) return TSB200_ERR_ARG;
  if (workspace_bytes < tsb200_linear_group_workspace_bytes(d, n, M)) return TSB200_ERR_WORKSPACE;
  return linear_f32(d, n, nullptr, y, M, (float*)((uint8_t*)workspace + tc::kWsHeader), as_stream(stream), norm);
}

extern "C" int tsb200_linear(const tsb200_linear_desc* d, const void* x, void* y, int64_t M, void* workspace,
                             size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  bool noop;
  int st = validate_linear(d, x, y, M, noop);
  if (st != TSB200_OK || noop) return st;
  st = linear_tc(d, x, y, M, workspace, workspace_bytes, as_stream(stream));
  if (st != TSB200_ERR_UNSUPPORTED) return st;
  if (d->act_dtype == TSB200_F32) {
    if (d->rank > 0) {
      if (!workspace || !aligned(workspace, 16)) return TSB200_ERR_ARG;
      if (workspace_bytes < tsb200_linear_workspace_bytes(d, M)) return TSB200_ERR_WORKSPACE;
    }
    st = linear_f32(&d, 1, x, &y, M, d->rank > 0 ? (float*)((uint8_t*)workspace + tc::kWsHeader) : nullptr, as_stream(stream));
    if (st != TSB200_ERR_UNSUPPORTED) return st;
  }
  return tsb200_linear_simt(d, x, y, M, workspace, workspace_bytes, stream);
}
