// LinearCompressed.forward with fp32 activations (transformersurgeon/blocks/linear_compressed.py:96-100): dense fp32 or packed
// factors, fp32 accumulation on the FMA pipe (fp32 models keep fp32 products: no tensor-core path).
//
// What bounds it: one token is a stream of weights through launches of a few hundred KB, i.e. latency; a prompt is FMAs.  One
// kernel serves both.  A warp owns R weight rows and MT tokens; its lanes walk K in 16-byte pieces (dense) or words (codes), and
// the R x MT sums of the 32 lanes are reduced by a butterfly that halves the values with the lanes (31 shuffles for 32 sums
// instead of 160).  Activations are staged in shared memory once per CTA and K tile and shared by its 8 warps.  With one token,
// where the rows alone do not fill the machine, up to 8 warps split K.  Before the dependency wait of a programmatic launch every
// warp requests its rows into the L2.
//
// Up to four matrices that share the reduction length run as one launch (q | k | v, gate | up), and the second factors of a gate /
// up pair end in SiLU(g) * u (blocks/mlp.py:181-183).
#include <type_traits>
#include "tc_common.cuh"

namespace tsb {
namespace {

constexpr int kWarps = 8;
constexpr int kXFloats = 8192;               // staged activations: a K tile of this many floats over all tokens and matrices
constexpr int kMaxSegs = 4;

struct Seg {
  const uint8_t* w;
  const uint8_t* w2;                         // gated: the up matrix (w: gate)
  const float *scale, *scale2, *bias, *bias2;
  const float *x, *x2;
  float* y;
  int n, cta0;                               // rows; first CTA
};
struct Norm {                                // x = RMSNorm(residual + delta) * w; w: null where x is given
  const float *residual, *delta, *w;
  float* out;                                // residual + delta
  float eps;
};
struct F32Params {
  Seg seg[kMaxSegs];
  Norm norm;
  int nseg, M, K, ks_log2;
  int k_rank;                                // tiles: columns of a cluster rank
  int64_t row_bytes;
};

// Consecutive weights of a lane: a 16-byte piece of a dense row (4) or one 32-bit word of codes (4 / 8 / 16 / 32).  Bits are shared out
// eight to a lane where the products of four tokens or more outweigh the loads (a row of 896 bits is 28 words: 8 tokens, 896 rows:
// 12.9 us by words, 10.3 by halves, 7.5 by bytes).
template <int BITS, int MT> struct Piece {
  static constexpr int kCnt = BITS == 32 ? 4 : (BITS == 1 && MT >= 4 ? 8 : 32 / BITS);
  static constexpr int kBytes = BITS == 32 ? 16 : kCnt * BITS / 8;
  static constexpr int kWord = kBytes < 4 ? 4 : 1;              // pieces of less than a word: the word's address
};
// p: the 16 bytes or the word that piece i of a row lies in.
template <int BITS, int CNT> __device__ __forceinline__ void load_piece(const uint8_t* p, int i, float (&v)[CNT]) {
  if constexpr (BITS == 32) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else {
    const unsigned w = __ldg(reinterpret_cast<const unsigned*>(p));
    if constexpr (BITS == 8) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = (float)(int8_t)(w >> (8 * j));
    } else if constexpr (BITS == 1) {
      const unsigned x = w >> (i % (32 / CNT) * (CNT / 2));
#pragma unroll
      for (int j = 0; j < CNT / 2; ++j) {
        v[2 * j] = (float)(int)(((x >> j) & 1u) * 2u) - 1.0f;
        v[2 * j + 1] = (float)(int)(((x >> (j + 16)) & 1u) * 2u) - 1.0f;
      }
    } else {
      constexpr int half = 16 / BITS;          // pair-interleaved: field j = column 2 j, field j + half = column 2 j + 1
#pragma unroll
      for (int j = 0; j < half; ++j) {
        v[2 * j] = (float)sext((int)(w >> (BITS * j)), BITS);
        v[2 * j + 1] = (float)sext((int)(w >> (BITS * j + 16)), BITS);
      }
    }
  }
}

// Sums V values per lane over the 32 lanes; lane l returns the sum of value l % V (V a power of two up to 32).
template <int V> __device__ __forceinline__ float reduce_scatter(float (&v)[V]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = V / 2; n > 0; n /= 2) {
    const bool up = lane & n;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, n);
    }
  }
  float s = v[0];
#pragma unroll
  for (int o = V; o < 32; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Activations that are the RMSNorm of residual + delta, staged by every CTA for itself (rows of one K tile): a decode step's separate
// normalisation is a launch of its own in the chain, ~2.3 us, of which this adds back a reduction over the CTA.  The arithmetic and the
// order of its sums are tsb200_add_rmsnorm's (elementwise.cu): the same bits.  That order depends on the row: pieces of 16 bytes up to
// kNormPieceRow bytes (add_rmsnorm_hf_kernel), single elements beyond (add_rmsnorm_kernel; here only one token's row is that long).  The first
// CTA keeps the new residual.
template <int MATS, int MT, int KT>
__device__ __forceinline__ void stage_normalised(const F32Params& p, const float4& nw, float (&xs)[MATS][MT][KT], float (&red)[kWarps][32]) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float ss[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) ss[m] = 0.f;
  for (int i = tid * 4; i < ((p.K + 31) & ~31); i += kWarps * 128)
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m < p.M && i < p.K) {
        const int64_t at = (int64_t)m * p.K + i;
        v = *reinterpret_cast<const float4*>(p.norm.residual + at);
        if (p.norm.delta) {
          const float4 d = *reinterpret_cast<const float4*>(p.norm.delta + at);
          v.x = __fadd_rn(v.x, d.x); v.y = __fadd_rn(v.y, d.y); v.z = __fadd_rn(v.z, d.z); v.w = __fadd_rn(v.w, d.w);
        }
        if (blockIdx.x == 0) *reinterpret_cast<float4*>(p.norm.out + at) = v;
        ss[m] += v.x * v.x; ss[m] += v.y * v.y; ss[m] += v.z * v.z; ss[m] += v.w * v.w;
      }
      *reinterpret_cast<float4*>(&xs[0][m][i]) = v;
    }
  if constexpr (KT * 4 > kNormPieceRow) {
    if (p.K * 4 > kNormPieceRow) {
      __syncthreads();
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        ss[m] = 0.f;
        for (int i = tid; i < p.K; i += kWarps * 32) ss[m] += xs[0][m][i] * xs[0][m][i];
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    ss[m] = warp_sum(ss[m]);
    if (lane == 0) red[warp][m] = ss[m];
  }
  __syncthreads();
  float inv[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const float var = warp_sum(lane < kWarps ? red[lane][m] : 0.f) / (float)p.K;
    inv[m] = 1.0f / sqrtf(var + p.norm.eps);
  }
  for (int i = tid * 4; i < p.K; i += kWarps * 128) {                 // the pieces that this thread has staged
    const float4 w = i == tid * 4 ? nw : __ldg(reinterpret_cast<const float4*>(p.norm.w + i));
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      float4 v = *reinterpret_cast<const float4*>(&xs[0][m][i]);
      v.x = __fmul_rn(w.x, __fmul_rn(v.x, inv[m])); v.y = __fmul_rn(w.y, __fmul_rn(v.y, inv[m]));
      v.z = __fmul_rn(w.z, __fmul_rn(v.z, inv[m])); v.w = __fmul_rn(w.w, __fmul_rn(v.w, inv[m]));
#pragma unroll
      for (int mat = 0; mat < MATS; ++mat) *reinterpret_cast<float4*>(&xs[mat][m][i]) = v;
    }
  }
  if (MATS > 1)
    for (int i = p.K + tid; i < ((p.K + 31) & ~31); i += kWarps * 32)
#pragma unroll
      for (int m = 0; m < MT; ++m) xs[MATS - 1][m][i] = 0.f;
}

template <int BITS, int MT, int R, bool GATED, bool NORM>
__global__ void __launch_bounds__(kWarps * 32) linear_f32_kernel(const __grid_constant__ F32Params p) {
  constexpr int MATS = GATED ? 2 : 1;
  using P = Piece<BITS, MT>;
  constexpr int CNT = P::kCnt;
  constexpr int V = MATS * R * MT;
  constexpr int kKT = kXFloats / (MATS * MT);
  static_assert(V <= 32 && (V & (V - 1)) == 0, "one sum per lane");
  __shared__ __align__(16) float xs[MATS][MT][kKT];
  __shared__ float red[kWarps][32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ks_n = 1 << p.ks_log2, ks = warp & (ks_n - 1);
  int si = 0;
  while (si + 1 < p.nseg && (int)blockIdx.x >= p.seg[si + 1].cta0) ++si;
  const Seg& sg = p.seg[si];
  const int row0 = (((int)blockIdx.x - sg.cta0) * (kWarps >> p.ks_log2) + (warp >> p.ks_log2)) * R;
  const int m0 = blockIdx.y * MT;
  const uint8_t* rows[MATS][R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t o = (int64_t)min(row0 + r, sg.n - 1) * p.row_bytes;          // beyond the matrix: the last row, never stored
    rows[0][r] = sg.w + o;
    if (GATED) rows[MATS - 1][r] = sg.w2 + o;
  }
  pdl_launch_dependents();
  // One or two tokens: the first pieces of this warp's rows come ahead of the dependency wait (weights are constants), the rest of the
  // rows into the L2
  constexpr int kPre = MT <= 2 ? 16 / CNT / MATS : 0;           // 16 columns per row and matrix: 32 registers
  float pre[kPre ? kPre : 1][MATS][R][CNT];
  const int pre_end = (min(kKT, p.K) + CNT - 1) / CNT;
#pragma unroll
  for (int q = 0; q < kPre; ++q) {
    const int i = lane + 32 * (ks + q * ks_n);
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (i < pre_end) load_piece<BITS>(rows[mat][r] + (int64_t)(i / P::kWord * P::kWord) * P::kBytes, i, pre[q][mat][r]);
  }
  if (lane < MATS * R && ks == 0 && row0 < sg.n) {
    const uint8_t* q = rows[0][0];
#pragma unroll
    for (int i = 0; i < MATS * R; ++i)
      if (i == lane) q = rows[i / R][i % R];
    const uintptr_t a = (reinterpret_cast<uintptr_t>(q) + 15) & ~(uintptr_t)15, e = (reinterpret_cast<uintptr_t>(q) + p.row_bytes) & ~(uintptr_t)15;
    if (e > a) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
  }
  float4 nw = make_float4(0.f, 0.f, 0.f, 0.f);
  if (NORM && tid * 4 < p.K) nw = __ldg(reinterpret_cast<const float4*>(p.norm.w + tid * 4));
  pdl_wait();

  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  if constexpr (NORM) stage_normalised<MATS, MT, kKT>(p, nw, xs, red);
  for (int k0 = 0; k0 < p.K; k0 += kKT) {
    const int kt = min(kKT, p.K - k0);
    __syncthreads();
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat) {
      if (NORM) break;
      const float* x = mat ? sg.x2 : sg.x;
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const bool in = m0 + m < p.M;
        const float* xr = x + (int64_t)(m0 + m) * p.K + k0;
        const bool vec = (p.K & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
        const int stop = min(kKT, (kt + 31) & ~31);            // pieces of up to 32 columns are read beyond the end
        if (vec) {
          for (int i = tid * 4; i < stop; i += kWarps * 128) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in && i < kt) v = *reinterpret_cast<const float4*>(xr + i);
            *reinterpret_cast<float4*>(&xs[mat][m][i]) = v;
          }
        } else {
          for (int i = tid; i < stop; i += kWarps * 32) xs[mat][m][i] = in && i < kt ? xr[i] : 0.f;
        }
      }
    }
    __syncthreads();
    // pieces of this warp: lane + 32 ks, then every 32 * ks_n; beyond the row's end the activations are zero, and no piece is read
    const int pieces = (kt + CNT - 1) / CNT;
    const int64_t b0 = (int64_t)k0 * P::kBytes / CNT;
    auto use = [&](int i, const float (&w)[MATS][R][CNT]) {
#pragma unroll
      for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int c = 0; c < CNT; c += 4) {
            const float4 xv = *reinterpret_cast<const float4*>(&xs[mat][m][i * CNT + c]);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              float& a = acc[(mat * R + r) * MT + m];
              a += w[mat][r][c] * xv.x;
              a += w[mat][r][c + 1] * xv.y;
              a += w[mat][r][c + 2] * xv.z;
              a += w[mat][r][c + 3] * xv.w;
            }
          }
    };
    int i = lane + 32 * ks;
    if (kPre && k0 == 0) {
#pragma unroll
      for (int q = 0; q < kPre; ++q, i += 32 * ks_n)
        if (i < pieces) use(i, pre[q]);
    }
#pragma unroll(MT <= 2 ? 4 : 2)
    for (; i < pieces; i += 32 * ks_n) {
      float w[MATS][R][CNT];
#pragma unroll
      for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
        for (int r = 0; r < R; ++r) load_piece<BITS>(rows[mat][r] + b0 + (int64_t)(i / P::kWord * P::kWord) * P::kBytes, i, w[mat][r]);
      use(i, w);
    }
  }
  float s = reduce_scatter<V>(acc);
  if (ks_n > 1) {
    red[warp][lane] = s;
    __syncthreads();
    if (ks) return;
    for (int q = 1; q < ks_n; ++q) s += red[warp + q][lane];
  }
  // lane v: matrix v / (R MT), row v / MT % R, token v % MT
  const int r = lane / MT % R, m = m0 + lane % MT, n = row0 + r;
  const bool ok = lane < R * MT && n < sg.n && m < p.M;
  if constexpr (GATED) {
    const float u = __shfl_sync(0xffffffffu, s, (lane + R * MT) & 31);
    if (ok) {
      const float g = s * (sg.scale ? sg.scale[n] : 1.0f) + (sg.bias ? sg.bias[n] : 0.f);
      const float uv = u * (sg.scale2 ? sg.scale2[n] : 1.0f) + (sg.bias2 ? sg.bias2[n] : 0.f);
      sg.y[(int64_t)m * sg.n + n] = __fmul_rn(g / (1.0f + expf(-g)), uv);
    }
  } else if (ok) {
    sg.y[(int64_t)m * sg.n + n] = s * (sg.scale ? sg.scale[n] : 1.0f) + (sg.bias ? sg.bias[n] : 0.f);
  }
}

// Prompt-sized token counts on dense factors: TM tokens x TN rows per CTA, 4 x 4 sums per thread, K in steps of 64 through a ring of
// shared memory filled by cp.async (rows as they lie in memory; the pitch of 68 floats puts the eight rows of a read into different
// banks).  Bound by FMAs where the tiles fill the machine, by their number otherwise: with 32 x 32 tiles a CTA's four groups of 64
// threads take 16 of every step's 64 columns each, and where even those tiles are few a cluster of up to eight CTAs splits K and adds
// its partial tiles through distributed shared memory.
//
// Cold weights, both factors of a layer (before: 64 x 64 tiles transposed on their way into shared memory from 64 tokens on, the lane
// kernel below that and for few rows): 128 tokens, 896 -> 128 -> 4864 28.2 -> 14.9 us, 4864 -> 128 -> 896 43.2 -> 19.2; 64 tokens, 3584 -> 224 ->
// 3584 43.8 -> 17.9; full rank, 16 tokens, 4096 -> 6144 273 -> 77, 48 tokens, 14336 -> 4096 492 -> 262, 128 tokens, 18944 -> 3584 1249 -> 677 (26
// of the 70 TFLOP/s of the FMA pipe: eight 16-byte reads of shared memory to 64 FMAs).
constexpr int kTK = 64, kTPitch = kTK + 4;
template <bool GATED> struct TileCfg {
  static constexpr int kMats = GATED ? 2 : 1, kStages = GATED ? 2 : 3;
};
template <bool GATED, int TM, int TN> constexpr int tile_smem() { return TileCfg<GATED>::kStages * TileCfg<GATED>::kMats * (TM + TN) * kTPitch * 4; }

__device__ __forceinline__ void cp_async16(float* dst, const void* src, bool in) {   // !in: zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

template <bool GATED, int TM, int TN>
__global__ void __launch_bounds__(256, 2) linear_f32_tile_kernel(const __grid_constant__ F32Params p) {
  constexpr int MATS = TileCfg<GATED>::kMats, STAGES = TileCfg<GATED>::kStages;
  constexpr int TX = TN / 4, TY = TM / 4, KG = 256 / (TX * TY), KK = kTK / KG;
  constexpr int RP = TN + 8;                                         // pitch of a partial tile
  static_assert(KG * MATS * TM * RP * 4 <= tile_smem<GATED, TM, TN>(), "partial tiles replace the ring");
  extern __shared__ __align__(16) float tile_ring[];                 // [stage][matrix][x rows, then w rows][kTPitch]
  int si = 0;
  while (si + 1 < p.nseg && (int)blockIdx.x >= p.seg[si + 1].cta0) ++si;
  const Seg& sg = p.seg[si];
  const int n0 = ((int)blockIdx.x - sg.cta0) * TN, m0 = blockIdx.y * TM;
  const int tid = threadIdx.x, kg = tid / (TX * TY), tx = tid % TX, ty = tid / TX % TY;
  const int rank = blockIdx.z, ranks = gridDim.z;
  const int k_beg = rank * p.k_rank, k_end = min(p.K, k_beg + p.k_rank);   // (may be empty)
  const int steps = k_end > k_beg ? (k_end - k_beg + kTK - 1) / kTK : 0;
  pdl_launch_dependents();
  auto stage_at = [&](int slot, int mat, int row) { return tile_ring + ((slot * MATS + mat) * (TM + TN) + row) * kTPitch; };
  auto copy_w = [&](int st) {
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
      for (int i = tid; i < TN * (kTK / 4); i += 256) {
        const int row = i / (kTK / 4), k = k_beg + st * kTK + i % (kTK / 4) * 4;
        const float* w = reinterpret_cast<const float*>(mat ? sg.w2 : sg.w);
        const bool in = k < k_end && n0 + row < sg.n;
        cp_async16(stage_at(st % STAGES, mat, TM + row) + i % (kTK / 4) * 4, in ? w + (int64_t)(n0 + row) * p.K + k : w, in);
      }
  };
  auto copy_x = [&](int st) {
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
      for (int i = tid; i < TM * (kTK / 4); i += 256) {
        const int row = i / (kTK / 4), k = k_beg + st * kTK + i % (kTK / 4) * 4;
        const float* x = mat ? sg.x2 : sg.x;
        const bool in = k < k_end && m0 + row < p.M;
        cp_async16(stage_at(st % STAGES, mat, row) + i % (kTK / 4) * 4, in ? x + (int64_t)(m0 + row) * p.K + k : x, in);
      }
  };
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st)
    if (st < steps) copy_w(st);                                      // constants: ahead of the dependency wait
  pdl_wait();
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < steps) copy_x(st);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float acc[MATS][4][4] = {};
  for (int st = 0; st < steps; ++st) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                                 // the step has landed; every warp is done with the one before
    if (st + STAGES - 1 < steps) { copy_w(st + STAGES - 1); copy_x(st + STAGES - 1); }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat) {
      const float* xs = stage_at(st % STAGES, mat, ty) + kg * KK;
      const float* ws = stage_at(st % STAGES, mat, TM + tx) + kg * KK;
#pragma unroll 1
      for (int k0 = 0; k0 < KK; k0 += 16) {                          // sums of 8 products, added in pairs: chains of 8 and K / 16 additions, not of K
        float pair[4][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float part[4][4] = {};
#pragma unroll
          for (int k = k0 + 8 * half; k < k0 + 8 * half + 8; k += 4) {
            float4 xv[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              xv[i] = *reinterpret_cast<const float4*>(xs + i * TY * kTPitch + k);
              wv[i] = *reinterpret_cast<const float4*>(ws + i * TX * kTPitch + k);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                part[i][j] += xv[i].x * wv[j].x;
                part[i][j] += xv[i].y * wv[j].y;
                part[i][j] += xv[i].z * wv[j].z;
                part[i][j] += xv[i].w * wv[j].w;
              }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (half == 0) pair[i][j] = part[i][j];
              else acc[mat][i][j] += pair[i][j] + part[i][j];
            }
        }
      }
    }
  }
  // ---- partial tiles [group][matrix][token][row], then one value per (matrix, token, row)
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) tile_ring[((kg * MATS + mat) * TM + ty + TY * i) * RP + tx + TX * j] = acc[mat][i][j];
  __syncthreads();
  auto sum_groups = [&](int mat, int at) {
    static_assert(KG == 1 || KG == 4, "groups");
    auto part = [&](int g) { return tile_ring[((g * MATS + mat) * TM) * RP + at]; };
    return KG == 1 ? part(0) : (part(0) + part(1)) + (part(2) + part(3));
  };
  auto store = [&](int idx, float v, float u) {
    const int m = m0 + idx / TN, n = n0 + idx % TN;
    if (m >= p.M || n >= sg.n) return;
    v += sg.bias ? sg.bias[n] : 0.f;
    if (GATED) v = __fmul_rn(v / (1.0f + expf(-v)), u + (sg.bias2 ? sg.bias2[n] : 0.f));
    sg.y[(int64_t)m * sg.n + n] = v;
  };
  if (ranks == 1) {
#pragma unroll
    for (int idx = tid; idx < TM * TN; idx += 256) {
      const int at = idx / TN * RP + idx % TN;
      store(idx, sum_groups(0, at), GATED ? sum_groups(MATS - 1, at) : 0.f);
    }
    return;
  }
  if (KG > 1) {
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat)
#pragma unroll
      for (int idx = tid; idx < TM * TN; idx += 256) {
        const int at = idx / TN * RP + idx % TN;
        tile_ring[(mat * TM) * RP + at] = sum_groups(mat, at);       // read and written by this thread alone
      }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  for (int idx = rank * (TM * TN / ranks) + tid; idx < (rank + 1) * (TM * TN / ranks); idx += 256) {
    float v[MATS];
#pragma unroll
    for (int mat = 0; mat < MATS; ++mat) {
      const unsigned own = tc::smem_u32(&tile_ring[(mat * TM + idx / TN) * RP + idx % TN]);
      float f[8];                                                    // of the ranks, added in pairs
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        f[r] = 0.f;
        if (r < ranks) {
          unsigned a;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(own), "r"(r));
          asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(f[r]) : "r"(a) : "memory");
        }
      }
      v[mat] = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
    }
    store(idx, v[0], v[MATS - 1]);
  }
  // no CTA leaves while another one may still read its tile
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <int BITS, int MT, int R, bool GATED, bool NORM>
int launch_cfg(F32Params& p, bool pdl, cudaStream_t s) {
  // K split: enough CTAs for the machine with one token (148 SMs x 2), at least one piece per lane and warp
  int rows = 0;
  for (int i = 0; i < p.nseg; ++i) rows += p.seg[i].n;
  const int groups = (p.M + MT - 1) / MT;
  int ks = 0;
  while (ks < 3 && (int64_t)((rows + (kWarps >> ks) * R - 1) / ((kWarps >> ks) * R)) * groups < 296 &&
         p.K >= (64 << ks) * Piece<BITS, MT>::kCnt)
    ++ks;
  p.ks_log2 = ks;
  const int per = (kWarps >> ks) * R;
  int ctas = 0;
  for (int i = 0; i < p.nseg; ++i) {
    p.seg[i].cta0 = ctas;
    ctas += (p.seg[i].n + per - 1) / per;
  }
  if (groups > 65535) return TSB200_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, (unsigned)groups);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  TSB_CUDA(cudaLaunchKernelEx(&cfg, linear_f32_kernel<BITS, MT, R, GATED, NORM>, p));
  return TSB200_OK;
}

template <int BITS>
int launch_bits(F32Params& p, bool gated, bool pdl, cudaStream_t s) {
  if (p.norm.w && (p.M > 4 || p.K > kXFloats / ((gated ? 2 : 1) * (p.M == 1 ? 1 : (p.M == 2 ? 2 : 4))))) return TSB200_ERR_UNSUPPORTED;   // rows of one K tile
  // tokens per warp, and rows so that 32 sums fill the lanes where the tokens do not (few tokens: fewer rows, more warps)
  auto go = [&](auto norm) {
    constexpr bool N = decltype(norm)::value;
    if (gated) {
      if (p.M == 1) return launch_cfg<BITS, 1, 2, true, N>(p, pdl, s);
      if (p.M <= 2) return launch_cfg<BITS, 2, 2, true, N>(p, pdl, s);
      return launch_cfg<BITS, 4, 2, true, N>(p, pdl, s);
    }
    if (p.M == 1) return launch_cfg<BITS, 1, 2, false, N>(p, pdl, s);
    if (p.M <= 2) return launch_cfg<BITS, 2, 2, false, N>(p, pdl, s);
    return launch_cfg<BITS, 4, 4, false, N>(p, pdl, s);
  };
  if (p.norm.w) return go(std::true_type{});
  if (p.M <= 4) return go(std::false_type{});
  return gated ? launch_cfg<BITS, 8, 2, true, false>(p, pdl, s) : launch_cfg<BITS, 8, 4, false, false>(p, pdl, s);
}

// Whether the tiles take a call: dense factors and at least 16 tokens.  Where the lane kernel stages a row's activations once (K <= 1024) and a
// cluster cannot split K (many rows), only if the tokens, in the eights that it takes, fill more than three quarters of the tiles, which take
// as long for one token of their 32 as for all (896 -> 4864, tiles / lane kernel: 32 tokens 18.6 / 22.8 us, 24 tokens - / 17.0, 56 tokens 29.4 /
// 31.1, 40 tokens - / 24.2).  Elsewhere the lane kernel is the slower one by far (24 tokens, 4096 -> 14336 409 us, tiles 150; 3584 -> 3584 67, 41).
bool use_tiles(const F32Params& p, int bits) {
  if (bits != 32 || p.M < 16 || p.K % 4) return false;
  int64_t tiles = 0;
  for (int i = 0; i < p.nseg; ++i) {
    if (!aligned(p.seg[i].x, 16) || (p.seg[i].x2 && !aligned(p.seg[i].x2, 16))) return false;
    tiles += (p.seg[i].n + 31) / 32;
  }
  return p.K <= 256 || p.K > kXFloats / 8 || tiles <= 148 || (p.M + 7) / 8 * 4 > (p.M + 31) / 32 * 12;
}
template <bool GATED, int TM, int TN> int launch_tile(F32Params& p, int ranks, bool pdl, cudaStream_t s) {
  constexpr int smem = tile_smem<GATED, TM, TN>();
  static bool configured[64] = {false};
  int dev = 0;
  TSB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TSB200_ERR_DEVICE;
  if (!configured[dev]) {
    TSB_CUDA(cudaFuncSetAttribute(linear_f32_tile_kernel<GATED, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev] = true;
  }
  int ctas = 0;
  for (int i = 0; i < p.nseg; ++i) {
    p.seg[i].cta0 = ctas;
    ctas += (p.seg[i].n + TN - 1) / TN;
  }
  const int groups = (p.M + TM - 1) / TM;
  if (groups > 65535) return TSB200_ERR_UNSUPPORTED;
  p.k_rank = ((p.K + kTK - 1) / kTK + ranks - 1) / ranks * kTK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, (unsigned)groups, (unsigned)ranks);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (ranks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = (unsigned)ranks;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  TSB_CUDA(cudaLaunchKernelEx(&cfg, linear_f32_tile_kernel<GATED, TM, TN>, p));
  return TSB200_OK;
}
// 64 x 64 tiles (half the shared-memory reads a sum) from 296 of them on, two for every SM: at a time without a pair, whose 104 KB rings leave room for
// two CTAs, one after the other with one (139 KB).  Else 32 x 32, and K split over a cluster as long as the two CTAs an SM holds still go
// round once and K has a step for every rank; ranks take whole steps, the same number each, so that the last ones may have none (9
// steps: five ranks of eight work - as long as five would take).
int launch_tiles(F32Params& p, bool gated, bool pdl, cudaStream_t s) {
  int64_t t64 = 0, t32 = 0;
  for (int i = 0; i < p.nseg; ++i) {
    t64 += (p.seg[i].n + 63) / 64;
    t32 += (p.seg[i].n + 31) / 32;
  }
  t64 *= (p.M + 63) / 64;
  t32 *= (p.M + 31) / 32;
  if (t64 >= 296) return gated ? launch_tile<true, 64, 64>(p, 1, pdl, s) : launch_tile<false, 64, 64>(p, 1, pdl, s);
  int ranks = 1;
  while (ranks < 8 && t32 * ranks * 2 <= 296 && p.K >= 2 * ranks * kTK) ranks *= 2;
  return gated ? launch_tile<true, 32, 32>(p, ranks, pdl, s) : launch_tile<false, 32, 32>(p, ranks, pdl, s);
}

int launch_any(F32Params& p, int bits, bool gated, bool pdl, cudaStream_t s) {
  if (!p.norm.w && use_tiles(p, bits)) return launch_tiles(p, gated, pdl, s);
  switch (bits) {
    case 1: return launch_bits<1>(p, gated, pdl, s);
    case 2: return launch_bits<2>(p, gated, pdl, s);
    case 4: return launch_bits<4>(p, gated, pdl, s);
    case 8: return launch_bits<8>(p, gated, pdl, s);
    default: return launch_bits<32>(p, gated, pdl, s);
  }
}

// The first CTA stores the residual while others still read what it is the sum of: none of the two may share a byte with it.
bool overlap(const void* a, const void* b, int64_t bytes) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return (x < y ? y - x : x - y) < (uintptr_t)bytes;
}
int take_norm(F32Params& p, const tsb200_norm_desc* norm) {
  if (!norm) return TSB200_OK;
  const int64_t bytes = (int64_t)p.M * p.K * 4;
  if (overlap(norm->residual_out, norm->residual, bytes) || (norm->delta && overlap(norm->residual_out, norm->delta, bytes))) return TSB200_ERR_ARG;
  if (p.K % 4 || !aligned(norm->residual, 16) || !aligned(norm->residual_out, 16) || !aligned(norm->weight, 16) || !aligned(norm->delta, 16))
    return TSB200_ERR_UNSUPPORTED;
  p.norm = Norm{(const float*)norm->residual, (const float*)norm->delta, (const float*)norm->weight, (float*)norm->residual_out, norm->eps};
  return TSB200_OK;
}
int64_t row_bytes(int64_t K, int bits) { return bits == 32 ? K * 4 : (int64_t)tsb200_packed_row_bytes(K, bits); }

}  // namespace

// n matrices [N_i, K] of one container as one launch; x[i] [M, K], y[i] [M, N_i].
int gemm_f32(const GemmSpec* g, int n, int bits, int64_t M, bool pdl, cudaStream_t s, const tsb200_norm_desc* norm) {
  F32Params p = {};
  if (n < 1 || n > kMaxSegs || M < 1 || M > 65535 * 8 || g[0].K > (1 << 30)) return TSB200_ERR_UNSUPPORTED;
  for (int i = 0; i < n; ++i) {
    if (g[i].K != g[0].K || g[i].N > (1 << 28)) return TSB200_ERR_UNSUPPORTED;
    Seg& sg = p.seg[i];
    sg.w = (const uint8_t*)g[i].W;
    sg.scale = bits == 32 ? nullptr : g[i].scale;
    sg.bias = (const float*)g[i].bias;
    sg.x = (const float*)g[i].x;
    sg.y = (float*)g[i].y;
    sg.n = (int)g[i].N;
  }
  p.nseg = n;
  p.M = (int)M;
  p.K = (int)g[0].K;
  p.row_bytes = row_bytes(g[0].K, bits);
  const int st = take_norm(p, norm);
  if (st != TSB200_OK) return st;
  return launch_any(p, bits, false, pdl, s);
}

// y = silu(x_gate . gate^T) * (x_up . up^T), both [N, K] of one container.
int gemm_f32_gated(const GemmSpec& gate, const GemmSpec& up, int bits, int64_t M, bool pdl, cudaStream_t s, const tsb200_norm_desc* norm) {
  F32Params p = {};
  if (gate.K != up.K || gate.N != up.N || M < 1 || M > 65535 * 8 || gate.K > (1 << 30) || gate.N > (1 << 28)) return TSB200_ERR_UNSUPPORTED;
  Seg& sg = p.seg[0];
  sg.w = (const uint8_t*)gate.W; sg.w2 = (const uint8_t*)up.W;
  sg.scale = bits == 32 ? nullptr : gate.scale; sg.scale2 = bits == 32 ? nullptr : up.scale;
  sg.bias = (const float*)gate.bias; sg.bias2 = (const float*)up.bias;
  sg.x = (const float*)gate.x; sg.x2 = (const float*)up.x;
  sg.y = (float*)gate.y;
  sg.n = (int)gate.N;
  p.nseg = 1;
  p.M = (int)M;
  p.K = (int)gate.K;
  p.row_bytes = row_bytes(gate.K, bits);
  const int st = take_norm(p, norm);
  if (st != TSB200_OK) return st;
  return launch_any(p, bits, true, pdl, s);
}

}  // namespace tsb
