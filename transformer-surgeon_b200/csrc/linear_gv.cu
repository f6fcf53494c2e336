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

// CTAs of a plan that one SM holds at a time.
int resident(int nt, const Plan& q) {
  const int regs = nt == 1 && q.R == 1 ? 64 : 96;
  int res = (int)((228 * 1024) / (q.smem + 1024));
  const int by_regs = 65536 / (regs * 32 * q.warps), by_warps = 64 / q.warps;
  if (by_regs < res) res = by_regs;
  if (by_warps < res) res = by_warps;
  return res < 1 ? 1 : res;
}

// Modelled time (about SM cycles) of a work split.  The constants are a fit to 2609 timings of 168 problems (N, K of 256 .. 18944,
// 4- and 8-bit codes, 1 .. 16 tokens, back to back under programmatic launch): the split it picks is on average 5 % slower than the
// fastest one of theirs, 8 % on 216 other problems.  A warp walks the blocks of its chain (widening per tile, MMAs per tile and token tile), an SM issues those of all
// its warps; staging costs the bytes of x, the epilogue the partial tiles, a cluster two barriers; CTAs run in rounds, and
// clusters leave SMs of a GPC unused.
float cost(int M, int nt, int mats, const Plan& q, int kb_split, int splits, int splits_rank) {
  const int res = resident(nt, q);
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

// Time of a work split in microseconds, to hold against tcq_time(): both are fits to 1906 timings of both kernels (11 K x 9 N of 896 .. 28672
// and 1024 .. 28672, all containers, 1 .. 16 tokens, dependent launches, codes from HBM; nine tenths of them within 14 and 12 %).
// Choosing by them takes 0.4 % longer in all than the faster kernel each time (at worst 1.36 times); always taking this kernel took up
// to 7.8 times the other's (4 bits, 11008 -> 18944, 10 tokens: beside the activations an SM has room for two warps).  `at_once`: CTAs per
// round when clusters of 1 .. 8 are placed one CTA to an SM.
float gv_time(int bits, int M, int nt, const Plan& q, int kb_split, int splits, bool two_x) {
  static const int at_once[] = {148, 128, 129, 128, 125, 96, 56, 64};
  const int res = resident(nt, q), per = (q.grid + at_once[q.ranks - 1] - 1) / at_once[q.ranks - 1], conc = per < res ? per : res;
  const int rounds = (per + conc - 1) / conc, kbc = (kb_split + 1) / 2, sr = (splits + q.ranks - 1) / q.ranks;
  const float x_kb = (float)M * sr * kb_split * (two_x ? 0.256f : 0.128f);
  return 0.58f + rounds * (1.94f + kbc * (0.0209f + 0.043f * q.R * nt + q.R * q.warps * conc * (bits == 8 ? 0.0229f : 0.0178f)) + 0.0251f * x_kb * conc) +
         (q.ranks > 1 ? 0.98f : 0.f);
}
// The tcgen05 kernel (linear_tcq.cu, 32-token tile) on the same phase: waves of items, a k-block of codes after the other.
float tcq_time(int bits, const tc::GemmPlan& g, int passes) {
  const float c = bits == 8 ? 0.394f : (bits == 4 ? 0.211f : (bits == 2 ? 0.203f : 0.175f));
  return 1.5f + (float)((g.items + tc::kPlanSMs - 1) / tc::kPlanSMs) * ((bits == 8 ? 1.58f : 2.1f) + c * g.kb_per_split * passes) + (g.splits > 1 ? 2.9f : 0.f);
}

// The plans of the shapes a thread met last (a model has a handful; the choice costs about 2 us of host time).
struct PlanKey {
  int bits, M, tiles, kb_total, kb_split, mats;
};
struct PlanEntry {
  PlanKey k;
  bool ok;
  Plan p;
  float us;
};
const PlanEntry& plan_for(int bits, int M, int tiles_total, int kb_total, int kb_split, int splits, int mats, bool x_shared) {
  static thread_local PlanEntry table[64] = {};
  const PlanKey k{bits, M, tiles_total, kb_total, kb_split, mats * 2 + (x_shared ? 1 : 0)};
  const unsigned h = ((unsigned)tiles_total * 2654435761u ^ (unsigned)kb_total * 40503u ^ (unsigned)(M * 131 + bits * 17 + k.mats)) >> 3;
  PlanEntry& e = table[h & 63];
  if (e.k.bits != k.bits || e.k.M != k.M || e.k.tiles != k.tiles || e.k.kb_total != k.kb_total || e.k.kb_split != k.kb_split || e.k.mats != k.mats) {
    e.ok = make_plan(e.p, bits, M, tiles_total, kb_split, splits, mats, x_shared);
    e.us = e.ok ? gv_time(bits, M, token_tiles(M), e.p, kb_split, splits, mats == 2 && !x_shared) : 0.f;
    e.k = k;
  }
  return e;
}

}  // namespace
}  // namespace gv

bool gv_supported(int bits, int64_t M, int64_t N, int64_t K) {
  return (bits == 1 || bits == 2 || bits == 4 || bits == 8) && M >= 1 && M <= gv::kMaxTokens && K % 8 == 0 && K >= 8 && N >= 1 &&
         N < (1 << 26) && K < (1 << 26);
}

namespace {
// A phase as this kernel sees it: the K splits of the tcgen05 kernel (the sums are then its sums bit for bit) and the plan.
struct GvPhase {
  tc::GemmPlan g;
  int tiles, tiles_total;
  bool x_shared;
  const gv::PlanEntry* plan;
};
bool gv_phase(GvPhase& f, const PhaseSpec& ps, int bits, int64_t M) {
  const int64_t N = ps.g[0].N, K = ps.g[0].K;
  if (!gv_supported(bits, M, N, K)) return false;
  f.tiles = (int)((N + 15) / 16);
  f.tiles_total = f.tiles * (ps.nsub == 2 && !ps.gated ? 2 : 1);
  f.g = tc::plan_gemm(M, N, K, ps.gated ? 1 : ps.nsub, ps.gated != 0, bits == 1 ? 2 : 1);
  f.x_shared = ps.gated && ps.g[0].x == ps.g[1].x;
  f.plan = &gv::plan_for(bits, (int)M, f.tiles_total, f.g.kb_total, f.g.kb_per_split, f.g.splits, ps.gated ? 2 : 1, f.x_shared);
  return f.plan->ok;
}
}  // namespace

bool gv_faster(const PhaseSpec* ps, const int* bits, int n, int64_t M) {
  float here = 0.f, there = 0.f;
  for (int i = 0; i < n; ++i) {
    GvPhase f;
    if (!gv_phase(f, ps[i], bits[i], M)) return false;
    here += f.plan->us;
    there += gv::tcq_time(bits[i], f.g, ps[i].gated ? 2 : 1);
  }
  return here < there;
}

int gv_gemm(const PhaseSpec& ps, int bits, int64_t M, bool pdl, const GvSpan* ahead, int n_ahead, cudaStream_t s) {
  const int64_t N = ps.g[0].N, K = ps.g[0].K;
  GvPhase f;
  if (!gv_phase(f, ps, bits, M)) return TSB200_ERR_UNSUPPORTED;
  for (int j = 0; j < ps.nsub; ++j)
    if (!aligned(ps.g[j].x, 16)) return TSB200_ERR_ARG;
  gv::Params p = {};
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.row_bytes = (int)tsb200_packed_row_bytes(K, bits);
  p.tiles = f.tiles;
  p.tiles_total = f.tiles_total;
  p.kb_total = f.g.kb_total;
  p.kb_split = f.g.kb_per_split;
  p.splits = f.g.splits;
  p.x_shared = f.x_shared;
  for (int j = 0; j < 2; ++j) {
    const GemmSpec& sp = ps.g[j < ps.nsub ? j : 0];
    p.sub[j] = gv::Sub{(const uint8_t*)sp.W, sp.scale, (const __nv_bfloat16*)sp.bias, (const __nv_bfloat16*)sp.x, (__nv_bfloat16*)sp.y};
  }
  const gv::Plan& plan = f.plan->p;
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
