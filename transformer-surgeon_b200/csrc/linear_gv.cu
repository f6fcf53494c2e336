// Host side of the decode-sized packed GEMM (linear_gv.cuh): choice of the work split, launch.
#include "linear_gv.cuh"
#include "tc_common.cuh"

namespace tsb {
namespace gv {
namespace {

int ceil_log2(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

int floor_log2(int v) {
  int l = 0;
  while ((2 << l) <= v) ++l;
  return l;
}

// Modelled time (about SM cycles) of a work split.  The constants are a fit to 2609 timings of 168 problems (N, K of 256 .. 18944,
// 4- and 8-bit codes, 1 .. 16 tokens, back to back under programmatic launch): the split it picks is on average 5 % slower than the
// fastest one.  A warp walks the blocks of its chain (widening per tile, MMAs per tile and token tile), an SM issues those of all
// its warps; staging costs the bytes of x, the epilogue the partial tiles, a cluster two barriers; CTAs run in rounds, and
// clusters leave SMs of a GPC unused.
float cost(int M, int nt, int mats, const Plan& q, int kb_split, int splits, int splits_rank) {
  const int regs = nt == 1 && q.R == 1 ? 64 : 96;
  int res = (int)((228 * 1024) / (q.smem + 1024));
  const int by_regs = 65536 / (regs * 32 * q.warps), by_warps = 64 / q.warps;
  if (by_regs < res) res = by_regs;
  if (by_warps < res) res = by_warps;
  if (res < 1) res = 1;
  const float usable = q.ranks <= 2 ? 1.f : (q.ranks <= 4 ? 0.887f : 0.8f);
  const int per = (q.grid + 147) / 148, conc = per < res ? per : res;
  float rounds = (float)((per + conc - 1) / conc);
  const float by_cap = (float)q.grid / (148.f * res * usable);
  if (by_cap > rounds) rounds = by_cap;
  const int kbc = (kb_split + 1) / 2;
  const float t_warp = kbc * (31.1f + 4 * q.R * (33.9f + nt * 25.1f));
  const float t_sm = kbc * 4.f * q.R * q.warps * conc * 4.06f;
  const float x_bytes = (float)M * splits_rank * kb_split * 128.f * mats;
  return rounds * ((t_warp > t_sm ? t_warp : t_sm) + 1024.f + x_bytes * conc / 46.8f + (q.ranks > 1 ? 5610.f : 0.f) +
                   (float)q.tg * M * mats * splits * 0.355f * conc / q.ranks + 1139.f);
}

bool make_plan(Plan& best, int bits, int M, int tiles_total, int kb_split, int splits, int mats, bool x_shared) {
  static const int kTiles[] = {1, 2, 3, 4, 6, 8, 12, 16};
  const int nt = token_tiles(M);
  float best_cost = 0.f;
  bool found = false;
  for (int ranks = 1; ranks <= 8 && ranks <= splits; ++ranks) {
    const int sr = (splits + ranks - 1) / ranks;
    if ((splits + sr - 1) / sr != ranks) continue;                   // every rank has work
    for (int R = 1; R <= 2; ++R)
      for (int rows : kTiles) {
        Plan q;
        q.R = R;
        q.tg = rows * R;
        q.ranks = ranks;
        q.warps = rows * 2 * mats * sr;
        if (q.warps > kMaxWarps) break;
        q.smem = smem_bytes(bits, R, nt, mats == 2, q.tg, M, kb_split, splits, ranks, sr, x_shared);
        if (q.smem > (size_t)kMaxSmem) continue;
        const int64_t grid = (int64_t)((tiles_total + q.tg - 1) / q.tg) * ranks;
        if (grid > 0x3fffffff) continue;
        q.grid = (int)grid;
        const float c = cost(M, nt, mats, q, kb_split, splits, sr);
        if (!found || c < best_cost) {
          found = true;
          best_cost = c;
          best = q;
        }
      }
  }
  return found;
}

// The plans of the shapes a thread met last (a model has a handful; the choice costs about 2 us of host time).
struct PlanKey {
  int bits, M, tiles, kb_total, kb_split, mats;
};
bool plan_for(Plan& out, int bits, int M, int tiles_total, int kb_total, int kb_split, int splits, int mats, bool x_shared) {
  struct Entry { PlanKey k; bool ok; Plan p; };
  static thread_local Entry table[64] = {};
  const PlanKey k{bits, M, tiles_total, kb_total, kb_split, mats * 2 + (x_shared ? 1 : 0)};
  const unsigned h = ((unsigned)tiles_total * 2654435761u ^ (unsigned)kb_total * 40503u ^ (unsigned)(M * 131 + bits * 17 + k.mats)) >> 3;
  Entry& e = table[h & 63];
  if (e.k.bits != k.bits || e.k.M != k.M || e.k.tiles != k.tiles || e.k.kb_total != k.kb_total || e.k.kb_split != k.kb_split || e.k.mats != k.mats) {
    e.ok = make_plan(e.p, bits, M, tiles_total, kb_split, splits, mats, x_shared);
    e.k = k;
  }
  out = e.p;
  return e.ok;
}

}  // namespace
}  // namespace gv

bool gv_supported(int bits, int64_t M, int64_t N, int64_t K) {
  return (bits == 1 || bits == 2 || bits == 4 || bits == 8) && M >= 1 && M <= gv::kMaxTokens && K % 8 == 0 && K >= 8 && N >= 1 &&
         N < (1 << 26) && K < (1 << 26);
}

int gv_gemm(const PhaseSpec& ps, int bits, int64_t M, bool pdl, const GvSpan* ahead, int n_ahead, cudaStream_t s) {
  const int64_t N = ps.g[0].N, K = ps.g[0].K;
  if (!gv_supported(bits, M, N, K)) return TSB200_ERR_UNSUPPORTED;
  for (int j = 0; j < ps.nsub; ++j)
    if (!aligned(ps.g[j].x, 16)) return TSB200_ERR_ARG;
  gv::Params p = {};
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.row_bytes = (int)tsb200_packed_row_bytes(K, bits);
  p.tiles = (int)((N + 15) / 16);
  p.tiles_total = p.tiles * (ps.nsub == 2 && !ps.gated ? 2 : 1);
  // the splits of the tcgen05 kernel: the sums are then its sums bit for bit
  const tc::GemmPlan g = tc::plan_gemm(M, N, K, ps.gated ? 1 : ps.nsub, ps.gated != 0, bits == 1 ? 2 : 1);
  p.kb_total = g.kb_total;
  p.kb_split = g.kb_per_split;
  p.splits = g.splits;
  p.x_shared = ps.gated && ps.g[0].x == ps.g[1].x;
  for (int j = 0; j < 2; ++j) {
    const GemmSpec& sp = ps.g[j < ps.nsub ? j : 0];
    p.sub[j] = gv::Sub{(const uint8_t*)sp.W, sp.scale, (const __nv_bfloat16*)sp.bias, (const __nv_bfloat16*)sp.x, (__nv_bfloat16*)sp.y};
  }
  gv::Plan plan;
  if (!gv::plan_for(plan, bits, p.M, p.tiles_total, p.kb_total, p.kb_split, p.splits, ps.gated ? 2 : 1, p.x_shared)) return TSB200_ERR_UNSUPPORTED;
  p.ranks = plan.ranks;
  p.splits_rank = (p.splits + plan.ranks - 1) / plan.ranks;
  p.tg = plan.tg;
  const int xk8 = p.splits_rank * p.kb_split * 8, fit = gv::floor_log2(plan.warps * 32);
  p.xk_log2 = gv::ceil_log2(xk8);
  if (p.xk_log2 > fit) p.xk_log2 = fit;
  p.mp_log2 = gv::ceil_log2(p.M);
  for (int i = 0; i < n_ahead && i < gv::kMaxSpans; ++i)
    if (ahead[i].bytes < (size_t)1 << 31 && aligned(ahead[i].p, 16)) p.ahead[i] = gv::Span{(const uint8_t*)ahead[i].p, (unsigned)ahead[i].bytes};
  cudaError_t e;
  switch (bits) {
    case 1: e = gv::launch<1>(p, plan, ps.gated != 0, pdl, s); break;
    case 2: e = gv::launch<2>(p, plan, ps.gated != 0, pdl, s); break;
    case 4: e = gv::launch<4>(p, plan, ps.gated != 0, pdl, s); break;
    default: e = gv::launch<8>(p, plan, ps.gated != 0, pdl, s); break;
  }
  TSB_CUDA(e);
  return TSB200_OK;
}

}  // namespace tsb
