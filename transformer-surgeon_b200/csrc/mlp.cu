// Gated MLP block: y = down(silu(gate(x)) * up(x)), the whole of
// transformersurgeon/blocks/mlp.py:171-185 (MLPGated.forward) behind one entry point.
//
// Up to 64 tokens through three layers packed alike (2, 4 or 8 bits, bf16) the block is [gate V | up V] -> [gate U, up U with
// SiLU(g) * u in the epilogue] -> [down V] -> [down U]: phases of ONE persistent tcgen05 launch (linear_tcq.cu) or, up to 16
// tokens and where that is faster, a chain of decode-sized launches (linear_gv.cu).  More than 128 tokens through gate and up packed
// alike take SiLU(g) * u into up's outputs; fp32 layers run as a chain on the FMA kernel (linear_f32.cu).  Otherwise the block is
// composed from tsb200_linear and tsb200_swiglu calls.
#include "tc_common.cuh"

namespace tsb {
int validate_linear(const tsb200_linear_desc* d, const void* x, void* y, int64_t M, bool& noop);
}  // namespace tsb

using namespace tsb;

namespace {
size_t align256(size_t v) { return (v + 255) / 256 * 256; }

bool fusable(const tsb200_linear_desc* g, const tsb200_linear_desc* u, const tsb200_linear_desc* d, int64_t M) {
  if (g->act_dtype != TSB200_BF16 || u->act_dtype != TSB200_BF16 || d->act_dtype != TSB200_BF16) return false;
  if (M < 1 || M > 64) return false;
  const int bits = g->u_bits;
  if (!(bits == 2 || bits == 4 || bits == 8)) return false;
  if (u->u_bits != bits || d->u_bits != bits) return false;
  if ((g->rank > 0) != (u->rank > 0) || g->rank != u->rank) return false;
  if (g->rank > 0 && (g->v_bits != bits || u->v_bits != bits)) return false;
  if (d->rank > 0 && d->v_bits != bits) return false;
  if (g->bias || u->bias) { /* biases are supported by the fused epilogue */ }
  const int64_t dims[] = {g->in_features, g->out_features, g->rank, d->rank, d->out_features};
  for (int64_t v : dims)
    if (v % 8) return false;
  // the gated phase keeps each tile's K range whole: it must fill the machine without a K split
  const int64_t tiles = (g->out_features + tc::BM - 1) / tc::BM;
  if (tiles < tc::kPlanSMs * 3 / 8) return false;
  return true;
}
// Gate and up packed alike and more tokens than a 128-token tile holds: their program takes SiLU(gate) * up along.
bool promptable(const tsb200_linear_desc* g, const tsb200_linear_desc* u, int64_t M) {
  const int bits = g->u_bits;
  if (g->act_dtype != TSB200_BF16 || M <= 128 || !(bits == 1 || bits == 2 || bits == 4 || bits == 8)) return false;
  if (u->u_bits != bits || g->rank != u->rank || g->out_features % 8) return false;
  if (g->rank > 0 && (g->v_bits != bits || u->v_bits != bits)) return false;
  const int64_t step = bits == 1 ? 128 : 8;                  // columns of a row pitch that the copy engine takes
  return g->in_features % step == 0 && g->rank % step == 0;
}
// Few enough tokens for the chain of decode-sized launches (linear_gv.cu); its results are those of the one-launch block, and
// gv_faster() chooses between the two.
bool chainable(const tsb200_linear_desc* g, const tsb200_linear_desc* u, const tsb200_linear_desc* d, int64_t M) {
  const int b = g->u_bits;
  return M <= kGvTokens && (g->rank == 0 || gv_supported(b, M, g->rank, g->in_features)) &&
         gv_supported(b, M, g->out_features, g->rank > 0 ? g->rank : g->in_features) &&
         (d->rank == 0 || gv_supported(b, M, d->rank, d->in_features)) &&
         gv_supported(b, M, d->out_features, d->rank > 0 ? d->rank : d->in_features);
}
// fp32 layers the FMA kernel takes as a chain: gate and up alike, dense or packed.
bool f32_chainable(const tsb200_linear_desc* g, const tsb200_linear_desc* u, const tsb200_linear_desc* d) {
  auto ok = [](const tsb200_linear_desc* l) {
    auto factor = [](int bits, const void* p, const float* scale, int64_t k) {
      return (bits == 32 && k % 8 == 0 && p) || ((bits == 1 || bits == 2 || bits == 4 || bits == 8) && p && scale);
    };
    if (l->act_dtype != TSB200_F32 || l->in_features <= 0 || l->out_features <= 0 || l->rank < 0) return false;
    if (l->rank > 0 && !(factor(l->v_bits, l->v, l->v_scale, l->in_features) && aligned(l->v, 16))) return false;
    return factor(l->u_bits, l->u, l->u_scale, l->rank > 0 ? l->rank : l->in_features) && aligned(l->u, 16);
  };
  return ok(g) && ok(u) && ok(d) && g->u_bits == u->u_bits && g->rank == u->rank && (g->rank == 0 || g->v_bits == u->v_bits);
}
// fp32: [gate V | up V] -> gated U -> down V -> down U on the FMA kernel, chained.  x: given, or normalised on the way in (norm).
struct F32Buffers {
  void *h0, *h1, *h2, *act;
};
int f32_chain(const tsb200_linear_desc* gate, const tsb200_linear_desc* up, const tsb200_linear_desc* down, const void* x, const tsb200_norm_desc* norm,
              void* y, int64_t M, const F32Buffers& b, cudaStream_t s) {
  const bool low = gate->rank > 0;
  const int64_t kgu = low ? gate->rank : gate->in_features;
  GemmSpec v[2] = {GemmSpec{gate->v, gate->v_scale, nullptr, x, b.h0, gate->rank, gate->in_features},
                   GemmSpec{up->v, up->v_scale, nullptr, x, b.h1, up->rank, up->in_features}};
  int st = low ? gemm_f32(v, 2, gate->v_bits, M, g_pdl != 0, s, norm) : TSB200_OK;
  if (st == TSB200_OK)
    st = gemm_f32_gated(GemmSpec{gate->u, gate->u_scale, gate->bias, low ? b.h0 : x, b.act, gate->out_features, kgu},
                        GemmSpec{up->u, up->u_scale, up->bias, low ? b.h1 : x, b.act, up->out_features, kgu}, gate->u_bits, M, low || g_pdl, s,
                        low ? nullptr : norm);
  const void* dx = b.act;
  if (st == TSB200_OK && down->rank > 0) {
    const GemmSpec dv{down->v, down->v_scale, nullptr, b.act, b.h2, down->rank, down->in_features};
    st = gemm_f32(&dv, 1, down->v_bits, M, true, s);
    dx = b.h2;
  }
  if (st == TSB200_OK) {
    const GemmSpec du{down->u, down->u_scale, down->bias, dx, y, down->out_features, down->rank > 0 ? down->rank : down->in_features};
    st = gemm_f32(&du, 1, down->u_bits, M, true, s);
  }
  return st;
}
}  // namespace

// Workspace layout: [region 0 | gate out | up out | act | h0 | h1 | h2].  Region 0 starts with the
// zero-between-calls header (status, grid barrier, split-K counters) and continues with scratch that
// needs no initialisation: split-K slices (fused path) or the body of the nested tsb200_linear
// workspace (composed path).  Keeping the header at offset 0 in both paths makes one workspace
// reusable across differently shaped blocks.
static size_t region0_bytes(const tsb200_linear_desc* gate, const tsb200_linear_desc* up, const tsb200_linear_desc* down,
                            int64_t M) {
  size_t scratch = 0;
  if (gate->rank > 0) {                        // V factors as one phase, or as two
    const size_t one = phase_scratch_bytes(M, gate->rank, gate->in_features, 2, false), two = 2 * phase_scratch_bytes(M, gate->rank, gate->in_features, 1, false);
    scratch += one > two ? one : two;
  }
  if (down->rank > 0) {
    scratch += phase_scratch_bytes(M, down->rank, down->in_features, 1, false);
    scratch += phase_scratch_bytes(M, down->out_features, down->rank, 1, false);
  } else {
    scratch += phase_scratch_bytes(M, down->out_features, down->in_features, 1, false);
  }
  size_t r0 = tc::kWsHeader + scratch;
  const size_t l1 = tsb200_linear_workspace_bytes(gate, M), l2 = tsb200_linear_workspace_bytes(up, M),
               l3 = tsb200_linear_workspace_bytes(down, M);
  if (l1 > r0) r0 = l1;
  if (l2 > r0) r0 = l2;
  if (l3 > r0) r0 = l3;
  return align256(r0);
}

namespace {
struct Buffers {
  uint8_t *g, *u, *a;                           // gate out (composed path) / act (fused path), up out, act (composed path)
  uint8_t *h0, *h1, *h2;
};
Buffers buffers(const tsb200_linear_desc* gate, const tsb200_linear_desc* up, const tsb200_linear_desc* down, int64_t M, uint8_t* ws) {
  const size_t elt = gate->act_dtype == TSB200_F32 ? 4 : 2;
  const size_t inter_b = align256((size_t)M * (size_t)gate->out_features * elt);
  const size_t r_b = align256((size_t)M * (size_t)(gate->rank > down->rank ? gate->rank : down->rank) * elt);
  Buffers b;
  b.g = ws + region0_bytes(gate, up, down, M);
  b.u = b.g + inter_b;
  b.a = b.u + inter_b;
  b.h0 = b.a + inter_b;
  b.h1 = b.h0 + r_b;
  b.h2 = b.h1 + r_b;
  return b;
}
bool block_ok(const tsb200_linear_desc* gate, const tsb200_linear_desc* up, const tsb200_linear_desc* down, int64_t M) {
  return gate && up && down && M >= 0 && gate->in_features == up->in_features && gate->out_features == up->out_features &&
         down->in_features == gate->out_features && gate->act_dtype == up->act_dtype && gate->act_dtype == down->act_dtype;
}
}  // namespace

extern "C" {

size_t tsb200_mlp_gated_workspace_bytes(const tsb200_linear_desc* gate, const tsb200_linear_desc* up,
                                        const tsb200_linear_desc* down, int64_t M) {
  if (!gate || !up || !down || M <= 0) return tc::kWsHeader;
  const size_t elt = gate->act_dtype == TSB200_F32 ? 4 : 2;
  size_t b = region0_bytes(gate, up, down, M);
  b += 3 * align256((size_t)M * (size_t)gate->out_features * elt);
  b += 3 * align256((size_t)M * (size_t)(gate->rank > down->rank ? gate->rank : down->rank) * elt);
  return b + 256;
}

int tsb200_mlp_gated(const tsb200_linear_desc* gate, const tsb200_linear_desc* up, const tsb200_linear_desc* down,
                     const void* x, void* y, int64_t M, void* workspace, size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!block_ok(gate, up, down, M)) return TSB200_ERR_ARG;
  if (M == 0) return TSB200_OK;
  if (!x || !y || !workspace || !aligned(workspace, 256)) return TSB200_ERR_ARG;
  if (workspace_bytes < tsb200_mlp_gated_workspace_bytes(gate, up, down, M)) return TSB200_ERR_WORKSPACE;
  cudaStream_t s = as_stream(stream);
  uint8_t* ws = (uint8_t*)workspace;
  const size_t r0 = region0_bytes(gate, up, down, M);
  const Buffers bufs = buffers(gate, up, down, M, ws);
  uint8_t *buf_g = bufs.g, *buf_u = bufs.u, *buf_a = bufs.a, *h0 = bufs.h0, *h1 = bufs.h1, *h2 = bufs.h2;

  if (fusable(gate, up, down, M)) {
    PhaseSpec ps[4];
    int n = 0;
    const void* gx = x;
    const void* ux = x;
    if (gate->rank > 0) {
      ps[n].nsub = 2; ps[n].gated = 0;
      ps[n].g[0] = GemmSpec{gate->v, gate->v_scale, nullptr, x, h0, gate->rank, gate->in_features};
      ps[n].g[1] = GemmSpec{up->v, up->v_scale, nullptr, x, h1, up->rank, up->in_features};
      ++n;
      gx = h0;
      ux = h1;
    }
    const int64_t kgu = gate->rank > 0 ? gate->rank : gate->in_features;
    ps[n].nsub = 2; ps[n].gated = 1;
    ps[n].g[0] = GemmSpec{gate->u, gate->u_scale, gate->bias, gx, buf_g, gate->out_features, kgu};
    ps[n].g[1] = GemmSpec{up->u, up->u_scale, up->bias, ux, buf_g, up->out_features, kgu};
    ++n;
    if (down->rank > 0) {
      ps[n].nsub = 1; ps[n].gated = 0;
      ps[n].g[0] = GemmSpec{down->v, down->v_scale, nullptr, buf_g, h2, down->rank, down->in_features};
      ++n;
      ps[n].nsub = 1; ps[n].gated = 0;
      ps[n].g[0] = GemmSpec{down->u, down->u_scale, down->bias, h2, y, down->out_features, down->rank};
      ++n;
    } else {
      ps[n].nsub = 1; ps[n].gated = 0;
      ps[n].g[0] = GemmSpec{down->u, down->u_scale, down->bias, buf_g, y, down->out_features, down->in_features};
      ++n;
    }
    const int bits[4] = {gate->u_bits, gate->u_bits, gate->u_bits, gate->u_bits};
    int st = TSB200_ERR_UNSUPPORTED;
    if (chainable(gate, up, down, M) && gv_faster(ps, bits, n, M)) {
      // [gate V | up V] -> [gate U, up U with SiLU(g) * u] -> [down V] -> [down U]: chained launches, the first two also request
      // codes of later ones into the L2
      auto span = [](const void* p, int bits, int64_t rows, int64_t cols) { return GvSpan{p, (size_t)rows * tsb200_packed_row_bytes(cols, bits)}; };
      const GvSpan down_u = span(down->u, down->u_bits, down->out_features, down->rank > 0 ? down->rank : down->in_features);
      const GvSpan first[3] = {span(gate->u, gate->u_bits, gate->out_features, kgu), span(up->u, up->u_bits, up->out_features, kgu),
                               down->rank > 0 ? span(down->v, down->v_bits, down->rank, down->in_features) : down_u};
      st = TSB200_OK;
      for (int p = 0; p < n && st == TSB200_OK; ++p) {
        const bool before_gated = !ps[p].gated && ps[p].nsub == 2;
        st = gv_gemm(ps[p], gate->u_bits, M, p > 0 || g_pdl != 0, before_gated ? first : &down_u, before_gated ? 3 : (ps[p].gated ? 1 : 0), s);
      }
      if (st != TSB200_ERR_UNSUPPORTED) return st;
    }
    st = run_program_tcq(ps, n, gate->u_bits, M, ws + tc::kWsHeader, (int*)(ws + tc::kWsCounters), (int*)(ws + tc::kWsGridBar), (int*)ws, s);
    if (st != TSB200_ERR_UNSUPPORTED) return st;
  }
  if (f32_chainable(gate, up, down)) {
    const int st = f32_chain(gate, up, down, x, nullptr, y, M, F32Buffers{h0, h1, h2, buf_g}, s);
    if (st != TSB200_ERR_UNSUPPORTED) return st;
  }
  bool noop_g = false, noop_u = false;
  if (promptable(gate, up, M) && aligned(x, 16) && validate_linear(gate, x, buf_g, M, noop_g) == TSB200_OK &&
      validate_linear(up, x, buf_a, M, noop_u) == TSB200_OK && !noop_g && !noop_u) {
    // Prompts: [gate V | up V] -> gate U -> up U with SiLU(gate) * up as its outputs leave -> down.  The separate SwiGLU pass over
    // [M, intermediate] (read twice, written once) and up's own round trip go away: 16384 tokens, 14336 features, 325 us of a
    // 1.97 ms block; the two V factors in one phase end in a fuller last wave (1024 tiles on 148 SMs, not twice 512).  Where a V
    // factor splits its K range the two stay apart: side by side they would split it differently and sum in another order than the
    // layers do by themselves.
    PhaseSpec ps[4];
    int n = 0;
    const bool low = gate->rank > 0;
    const int64_t kgu = low ? gate->rank : gate->in_features;
    if (low) {
      const bool together = tc::plan_gemm(M, gate->rank, gate->in_features, 1, false, gate->u_bits == 1 ? 2 : 1).splits == 1;
      const GemmSpec gv{gate->v, gate->v_scale, nullptr, x, h0, gate->rank, gate->in_features}, uv{up->v, up->v_scale, nullptr, x, h1, up->rank, up->in_features};
      ps[n].nsub = together ? 2 : 1; ps[n].gated = 0;
      ps[n].g[0] = gv;
      ps[n++].g[1] = uv;
      if (!together) {
        ps[n].nsub = 1; ps[n].gated = 0;
        ps[n++].g[0] = uv;
      }
    }
    ps[n].nsub = 1; ps[n].gated = 0;
    ps[n++].g[0] = GemmSpec{gate->u, gate->u_scale, gate->bias, low ? h0 : x, buf_g, gate->out_features, kgu};
    ps[n].nsub = 1; ps[n].gated = 0;
    ps[n++].g[0] = GemmSpec{up->u, up->u_scale, up->bias, low ? h1 : x, buf_a, up->out_features, kgu, buf_g};
    const int st = run_program_tcq(ps, n, gate->u_bits, M, ws + tc::kWsHeader, (int*)(ws + tc::kWsCounters), (int*)(ws + tc::kWsGridBar), (int*)ws, s);
    if (st == TSB200_OK) return tsb200_linear(down, buf_a, y, M, ws, r0, stream);
    if (st != TSB200_ERR_UNSUPPORTED) return st;
  }
  // composed path: three linear calls and the SwiGLU kernel; region 0 is their workspace
  int st = tsb200_linear(gate, x, buf_g, M, ws, r0, stream);
  if (st != TSB200_OK) return st;
  st = tsb200_linear(up, x, buf_u, M, ws, r0, stream);
  if (st != TSB200_OK) return st;
  const int64_t inter = gate->out_features;
  st = tsb200_swiglu(buf_g, buf_u, buf_a, gate->act_dtype, M, inter, inter, inter, inter, stream);
  if (st != TSB200_OK) return st;
  return tsb200_linear(down, buf_a, y, M, ws, r0, stream);
}

int tsb200_norm_mlp_gated(const tsb200_norm_desc* norm, const tsb200_linear_desc* gate, const tsb200_linear_desc* up,
                          const tsb200_linear_desc* down, void* y, int64_t M, void* workspace, size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!norm || !norm->residual || !norm->weight || !norm->residual_out) return TSB200_ERR_ARG;
  if (!block_ok(gate, up, down, M)) return TSB200_ERR_ARG;
  if (M == 0) return TSB200_OK;
  if (!y || !workspace || !aligned(workspace, 256)) return TSB200_ERR_ARG;
  if (workspace_bytes < tsb200_mlp_gated_workspace_bytes(gate, up, down, M)) return TSB200_ERR_WORKSPACE;
  if (!f32_chainable(gate, up, down)) return TSB200_ERR_UNSUPPORTED;
  const Buffers b = buffers(gate, up, down, M, (uint8_t*)workspace);
  return f32_chain(gate, up, down, nullptr, norm, y, M, F32Buffers{b.h0, b.h1, b.h2, b.g}, as_stream(stream));
}

}  // extern "C"
