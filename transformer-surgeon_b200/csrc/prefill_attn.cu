// Causal attention of a PROMPT CHUNK on tcgen05: T query tokens per sequence over the L >= T tokens of the
// cache (query i sits at position L - T + i), reading the DEQUANTIZED cache - what every attention read of a
// quantized cache sees.  Replaces transformersurgeon/blocks/mha.py:9-103 (attention(): GQA, softmax(q k^T / sqrt d) v)
// for T > 1, i.e. what the reference hands to torch's scaled-dot-product attention during prefill.
//
// Inputs are produced by tsb200_kv_gather_heads (below): K as [B, hkv, L, d] and V TRANSPOSED as [B, hkv, d, Lp]
// (tokens contiguous, zero beyond L), both bf16, so that every MMA operand tile is K-major and one TMA box:
//     S[128 q, 128 keys]  = Q[128, d] . K_tile[128, d]^T          (tcgen05.mma kind::f16, fp32 in TMEM)
//     O[128 q, d]        += P[128, 128] . Vt_tile[d, 128]^T
// A persistent CTA works on TWO query tiles of one kv head at a time (their K / Vt tiles are shared), so that the tensor pipe multiplies
// for one while the other's softmax runs; the tiles of a kv head's query group are enumerated query-tile-major and paired in that
// order (two heads of one tile, now and then the last head of a tile with the first of the next), pairs go longest first.  11 warps:
//   warp 0      TMA: the pair's Q tiles, then K0, K1, V0, K2, V1, ... into a ring of three 128-key tiles, across pairs
//   warps 1, 2  one lane each: MMA issuer of a query tile (one lane needs ~114 cycles per MMA of 64 cycles of the pipe): S(j+1) as soon
//               as the softmax has moved S(j) to registers, then O += P(j) . V(j); warp 1 allocates the tensor memory (S, S', O, O')
//   warps 3..6, 7..10  softmax of a query tile: one thread = one query row (its TMEM lane): tcgen05.ld the 128 scores, mask the
//               diagonal tile, running maximum with LAZY rescaling (O and the row sum are rescaled only when the
//               maximum grew by more than 2^8; the final division uses the same reference maximum, so the result is
//               exact), exp2, row sum in fp32, P rounded to bf16 into shared memory in the swizzled K-major layout
//               the MMA descriptor expects; at the end O / l, rounded, while the next pair's scores are computed
// Bounds at 128 x 128 scores of a tile: 1024 cycles of the tensor pipe, 1024 of the exponential unit, ~1500 of shared memory.
// 8 x 2048 tokens, 32 / 8 heads of 128: 383 us (570 with one query tile per CTA, 4300 cycles a tile).  The softmax warps hold a row of 128
// scores: 168 registers a thread are all that 352 threads can have, and 128 bytes (head dimension 64: 108) spill.
// Every mbarrier wait is bounded; on expiry the CTA records a code in the status word, frees its TMEM and returns.
#include "tc_common.cuh"
#include "decode_attn_common.cuh"

namespace tsb {
using namespace tc;
namespace {

constexpr int kPfThreads = 352;
constexpr int BQ = 128, BKEY = 128, kRing = 3;

__device__ __forceinline__ void tmem_ld32(unsigned taddr, unsigned (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32f(unsigned taddr, const unsigned (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait_pf() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

struct PfParams {
  int64_t B, T, L;
  int H, hkv;
  int nq, pairs, items;      // query tiles per head, pairs per (sequence, kv head), pairs in all
  int per;                   // tiles of a pair: 2, or 1 where the tiles are fewer than the SMs
  float scale_log2;          // sm_scale * log2(e)
  __nv_bfloat16* out;        // [B, T, H, D]
  int* status;
};

template <int D> struct PfLayout {
  static constexpr int KB = D / 64;                    // 64-column blocks of the head dimension
  static constexpr int kQ = KB * BQ * 128;             // Q tile
  static constexpr int kTile = D * 256;                // K tile: KB blocks of [128 keys x 128 B]; Vt tile: 2 blocks (64 keys each) of [D rows x 128 B]
  static constexpr int kP = 2 * BQ * 128;              // P tile: 2 blocks (64 keys each) of [128 rows x 128 B]
  static constexpr int kBytes = 2 * kQ + kRing * kTile + 2 * kP + 1024 /*barriers*/ + 1024 /*alignment*/;
  static constexpr unsigned kSCol = 0;                 // S of tile i at columns 128 i
  static constexpr unsigned kOCol = 256;               // O of tile i at 256 + 128 i
  static_assert(kBytes <= 227 * 1024, "shared memory of one CTA");
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));   // below 2^-126: 0, which adds as little to a row's sum (at least 2^-8)
  return y;
}

// Two fp32 operations in one instruction, each rounded as the scalar one.
__device__ __forceinline__ void mul2(float& a, float& b, float y) {
  asm("{\n.reg .b64 p, q;\nmov.b64 p, {%0, %1};\nmov.b64 q, {%2, %2};\nmul.rn.f32x2 p, p, q;\nmov.b64 {%0, %1}, p;\n}\n" : "+f"(a), "+f"(b) : "f"(y));
}
__device__ __forceinline__ void add2(float& a, float& b, float y) {
  asm("{\n.reg .b64 p, q;\nmov.b64 p, {%0, %1};\nmov.b64 q, {%2, %2};\nadd.rn.f32x2 p, p, q;\nmov.b64 {%0, %1}, p;\n}\n" : "+f"(a), "+f"(b) : "f"(y));
}

template <int D>
__global__ void __launch_bounds__(kPfThreads, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_vt, PfParams p) {
  using Lt = PfLayout<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                                  // two tiles
  uint8_t* sKV = sQ + 2 * Lt::kQ;                      // ring
  uint8_t* sP = sKV + kRing * Lt::kTile;               // two tiles
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(sP + 2 * Lt::kP);
  unsigned long long* q_full = bars;                   // [1] the pair's Q tiles landed
  unsigned long long* q_empty = bars + 1;              // [1] both issuers: the pair's last score MMAs are complete
  unsigned long long* kv_full = bars + 2;              // [kRing] a K or Vt tile landed
  unsigned long long* kv_empty = kv_full + kRing;      // [kRing] both issuers: MMAs that read it are complete
  unsigned long long* s_full = kv_empty + kRing;       // [2] scores of query tile i are in TMEM
  unsigned long long* s_free = s_full + 2;             // [2] its four softmax warps have them in registers
  unsigned long long* p_full = s_free + 2;             // [2] ... have written P
  unsigned long long* o_done = p_full + 2;             // [2] P.V is complete: P and O may be touched
  unsigned long long* o_free = o_done + 2;             // [2] the four warps have read the finished O
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(o_free + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t off = p.L - p.T;                                   // position of query 0
  const int G = p.H / p.hkv;
  // Work item w: sequence, kv head and, for query tile i of the pair, its head, first query and number of key tiles (0: no tile).
  struct Work { int b, hk, pair; };
  struct Tile { int h, n; int64_t q0; };
  auto work = [&](int w) {
    const int per = p.hkv * (int)p.B, rest = w % per;
    return Work{rest / p.hkv, rest % p.hkv, p.pairs - 1 - w / per};   // longest first
  };
  auto tile = [&](const Work& k, int i) {
    const int u = p.per * k.pair + i, qt = u / G;
    const int64_t q0 = (int64_t)qt * BQ;
    return Tile{k.hk * G + u % G, i < p.per && qt < p.nq ? (int)((off + min(p.T - 1, q0 + BQ - 1)) / BKEY) + 1 : 0, q0};
  };

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);
    for (int i = 0; i < kRing; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 2); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 4); mbar_init(&p_full[i], 4); mbar_init(&o_done[i], 1); mbar_init(&o_free[i], 4); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int c = 0, it = 0;                                // tiles of the ring, work items so far
      bool ok = true;
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x, ++it) {
        const Work k = work(w);
        const Tile x = tile(k, 0), y = tile(k, 1);
        const int most = max(x.n, y.n);
        if (it > 0 && !mbar_wait(q_empty, (it - 1) & 1, abort_flag, 1)) break;
        mbar_expect_tx(q_full, (unsigned)((x.n > 0) + (y.n > 0)) * Lt::kQ);
        for (int kb = 0; kb < Lt::KB; ++kb) {
          if (x.n > 0) tma_load_3d(sQ + kb * BQ * 128, &map_q, kb * 64, x.h, (int)(k.b * p.T + x.q0), q_full);
          if (y.n > 0) tma_load_3d(sQ + Lt::kQ + kb * BQ * 128, &map_q, kb * 64, y.h, (int)(k.b * p.T + y.q0), q_full);
        }
        const int64_t krow0 = ((int64_t)k.b * p.hkv + k.hk) * p.L;
        const int64_t vrow0 = ((int64_t)k.b * p.hkv + k.hk) * D;
        auto slot = [&]() -> uint8_t* {
          const int s = c % kRing;
          if (c >= kRing && !mbar_wait(&kv_empty[s], (c / kRing - 1) & 1, abort_flag, 2)) { ok = false; return nullptr; }
          mbar_expect_tx(&kv_full[s], (unsigned)Lt::kTile);
          return sKV + s * Lt::kTile;
        };
        for (int j = 0; j <= most && ok; ++j) {         // K(j), V(j - 1)
          if (j < most) {
            uint8_t* st = slot();
            if (!ok) break;
            for (int kb = 0; kb < Lt::KB; ++kb)
              tma_load_2d(st + kb * BKEY * 128, &map_k, kb * 64, (int)(krow0 + (int64_t)j * BKEY), &kv_full[c % kRing]);
            ++c;
          }
          if (j > 0) {
            uint8_t* st = slot();
            if (!ok) break;
            for (int kb = 0; kb < 2; ++kb)
              tma_load_2d(st + kb * D * 128, &map_vt, (j - 1) * BKEY + kb * 64, (int)vrow0, &kv_full[c % kRing]);
            ++c;
          }
        }
      }
    }
  } else if (warp <= 2) {
    // ------------------------------------------------------------------ MMA issuer of query tile i
    if (lane == 0) {
      const int i = warp - 1;
      constexpr unsigned idesc_s = idesc_bf16(BKEY);
      constexpr unsigned idesc_o = idesc_bf16(D);
      const unsigned s_tmem = tmem_base + Lt::kSCol + 128 * i, o_tmem = tmem_base + Lt::kOCol + 128 * i;
      const unsigned q_addr = smem_u32(sQ + i * Lt::kQ), p_addr = smem_u32(sP + i * Lt::kP);
      int c = 0, it = 0;                                // tiles of the ring, work items so far
      int ts = 0, tp = 0, outs = 0;                     // scores issued, P.V issued, finished O tiles so far
      bool ok = true;
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x, ++it) {
        const Work k = work(w);
        const int n = tile(k, i).n, most = max(n, tile(k, 1 - i).n);
        ok = mbar_wait(q_full, it & 1, abort_flag, 3);
        for (int j = 0; j <= most && ok; ++j) {         // S(j), then P(j - 1) . V(j - 1)
          if (j < most) {
            const int s = c % kRing;
            ok = mbar_wait(&kv_full[s], (c / kRing) & 1, abort_flag, 4);
            if (ok && j < n && ts > 0) ok = mbar_wait(&s_free[i], (ts - 1) & 1, abort_flag, 5);
            if (!ok) break;
            if (j < n) {
              tc_fence_after();
              const unsigned k_addr = smem_u32(sKV + s * Lt::kTile);
#pragma unroll
              for (int kb = 0; kb < Lt::KB; ++kb) {
                const unsigned long long ad = smem_desc_sw128(q_addr + kb * BQ * 128);
                const unsigned long long bd = smem_desc_sw128(k_addr + kb * BKEY * 128);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) umma_bf16(s_tmem, ad + 2 * kk, bd + 2 * kk, idesc_s, (kb | kk) ? 1u : 0u);
              }
              umma_commit(&s_full[i]);
              umma_commit(&kv_empty[s]);
              ++ts;
            } else {
              mbar_arrive(&kv_empty[s]);
            }
            if (j == most - 1) umma_commit(q_empty);
            ++c;
          }
          if (j > 0) {
            const int s = c % kRing;
            ok = mbar_wait(&kv_full[s], (c / kRing) & 1, abort_flag, 6);
            if (ok && j - 1 < n) {
              ok = mbar_wait(&p_full[i], tp & 1, abort_flag, 7);
              if (ok && j == 1 && outs > 0) ok = mbar_wait(&o_free[i], (outs - 1) & 1, abort_flag, 8);
            }
            if (!ok) break;
            if (j - 1 < n) {
              tc_fence_after();
              const unsigned v_addr = smem_u32(sKV + s * Lt::kTile);
#pragma unroll
              for (int kb = 0; kb < 2; ++kb) {
                const unsigned long long ad = smem_desc_sw128(p_addr + kb * BQ * 128);
                const unsigned long long bd = smem_desc_sw128(v_addr + kb * D * 128);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) umma_bf16(o_tmem, ad + 2 * kk, bd + 2 * kk, idesc_o, (j > 1 || (kb | kk)) ? 1u : 0u);
              }
              umma_commit(&o_done[i]);
              umma_commit(&kv_empty[s]);
              ++tp;
            } else {
              mbar_arrive(&kv_empty[s]);
            }
            ++c;
          }
        }
        if (n > 0) ++outs;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue of query tile i
    const int i = (warp - 3) >> 2;
    const int quarter = warp & 3;                      // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;               // query row of the tile
    const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
    const unsigned s_tmem = lane_addr + Lt::kSCol + 128 * i, o_tmem = lane_addr + Lt::kOCol + 128 * i;
    uint8_t* my_p = sP + i * Lt::kP;
    const float scale = p.scale_log2;
    int t = 0;                                         // tiles so far
    bool ok = true;
    for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
      const Work k = work(w);
      const Tile mine = tile(k, i);
      const int n = mine.n;
      const int64_t q0 = mine.q0, qpos = off + q0 + row;           // position of this row's query
      float m_ref = -INFINITY, l_sum = 0.f;
      for (int j = 0; j < n && ok; ++j, ++t) {
        ok = mbar_wait(&s_full[i], t & 1, abort_flag, 9);
        if (!ok) break;
        tc_fence_after();
        float sc[128];
        {
          unsigned (&r)[4][32] = reinterpret_cast<unsigned (&)[4][32]>(sc);
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(s_tmem + c * 32, r[c]);
          tmem_ld_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[i]);
#pragma unroll
        for (int e = 0; e < 64; ++e) mul2(sc[2 * e], sc[2 * e + 1], scale);
        const int64_t key0 = (int64_t)j * BKEY;
        if (key0 + BKEY - 1 > off + q0) {                // a tile that reaches past the tile's first query: mask
          const int last = (int)min(qpos - key0, (int64_t)BKEY);   // last visible key of the tile
#pragma unroll
          for (int e = 0; e < 128; ++e)
            if (e > last) sc[e] = -INFINITY;
        }
        float mx[8];                                     // eight chains: one of 128 dependent steps takes longer than the exponentials
#pragma unroll
        for (int e = 0; e < 8; ++e) mx[e] = sc[e];
#pragma unroll
        for (int e = 8; e < 120; e += 16)
#pragma unroll
          for (int x = 0; x < 8; ++x) mx[x] = fmaxf(fmaxf(mx[x], sc[e + x]), sc[e + 8 + x]);
#pragma unroll
        for (int x = 0; x < 8; ++x) mx[x] = fmaxf(mx[x], sc[120 + x]);
        const float m_tile = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
        // lazy rescaling: keep the reference maximum until the true maximum has outgrown it by 2^8
        float alpha = 1.0f;
        const bool grow = m_tile > m_ref + 8.0f || m_ref == -INFINITY;
        if (grow && m_tile > -INFINITY) {
          alpha = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_tile);
          m_ref = m_tile;
          l_sum *= alpha;
        }
        const float mr = m_ref == -INFINITY ? 0.f : m_ref;
        float psum = 0.f;
        unsigned pk[64];
#pragma unroll
        for (int e = 0; e < 64; ++e) {
          add2(sc[2 * e], sc[2 * e + 1], -mr);
          const float p0 = ex2(sc[2 * e]), p1 = ex2(sc[2 * e + 1]);
          psum += p0 + p1;
          __nv_bfloat162 q2 = __floats2bfloat162_rn(p0, p1);
          pk[e] = *reinterpret_cast<unsigned*>(&q2);
        }
        l_sum += psum;
        // P(j - 1) . V must be complete before P is overwritten and before O is rescaled
        if (j > 0) {
          ok = mbar_wait(&o_done[i], (t - 1) & 1, abort_flag, 10);
          if (!ok) break;
          tc_fence_after();
          if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              unsigned r[32];
              tmem_ld32(o_tmem + c * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
              tmem_st32f(o_tmem + c * 32, r);
            }
            tmem_st_wait_pf();
          }
        }
#pragma unroll
        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            store_chunk(my_p + kb * BQ * 128, row, c, make_uint4(pk[kb * 32 + c * 4], pk[kb * 32 + c * 4 + 1], pk[kb * 32 + c * 4 + 2], pk[kb * 32 + c * 4 + 3]));
        fence_async_proxy();                             // generic-proxy writes -> visible to the MMA (async proxy)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[i]);
      }
      if (!ok || n == 0) continue;
      // ---- epilogue: O / l
      ok = mbar_wait(&o_done[i], (t - 1) & 1, abort_flag, 11);
      if (!ok) break;
      tc_fence_after();
      float o[D];
      {
        unsigned (&r)[D / 32][32] = reinterpret_cast<unsigned (&)[D / 32][32]>(o);
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld32(o_tmem + c * 32, r[c]);
        tmem_ld_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_free[i]);
      const float inv = l_sum > 0.f ? 1.0f / l_sum : 0.f;
      const int64_t tok = q0 + row;
      if (tok < p.T) {
        __nv_bfloat16* dst = p.out + (((int64_t)k.b * p.T + tok) * p.H + mine.h) * D;
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          unsigned v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            __nv_bfloat162 q2 = __floats2bfloat162_rn(o[c * 16 + 2 * e] * inv, o[c * 16 + 2 * e + 1] * inv);
            v[e] = *reinterpret_cast<unsigned*>(&q2);
          }
          *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<uint4*>(dst + c * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
        }
      }
    }
  }
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);   // error path only: let copies in flight land
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicMax(p.status, *abort_flag);
}

// ---- head-major gather: K [B, hkv, L, D], V transposed [B, hkv, D, Lp] (zeros beyond seq_lens[b] and in [L, Lp))
// One CTA per (64 tokens, kv head, sequence).  Bound by the pages in and the bf16 out: a unit is eight values that lie side by side in
// the output (K: elements of a token, V: tokens of an element), eight codes in, one 16-byte store out, all of a thread's units in
// flight together; eight lanes write 128 contiguous bytes of V^T.  8 x 2048 tokens, 8 heads, d 128, FP8 (33 MB in, 67 MB out):
// 25 us, 76 with one value per thread and store.
constexpr int kGatherTokens = 64;

// Codes of eight consecutive elements of a K vector / eight consecutive tokens of a V element -> their values (fp8: unscaled).
template <int D, int FMT>
__device__ __forceinline__ void k_eight(const uint8_t* __restrict__ rec, int t, int e, float (&v)[8]) {
  if constexpr (FMT == TSB200_KV_INT8 || FMT == TSB200_KV_FP8) {
    const uint2 c = *reinterpret_cast<const uint2*>(rec + t * D + e);
    const float s = FMT == TSB200_KV_INT8 ? reinterpret_cast<const float*>(rec + 16 * D)[t] : 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned b = ((i < 4 ? c.x : c.y) >> (8 * (i & 3))) & 0xffu;
      v[i] = FMT == TSB200_KV_INT8 ? (float)(int8_t)b * s : e4m3_byte_to_f32(b);
    }
  } else if constexpr (FMT == TSB200_KV_NVFP4) {
    const unsigned c = *reinterpret_cast<const unsigned*>(rec + t * (D / 2) + (e >> 1));
    const float s = e4m3_byte_to_f32(rec[16 * (D / 2) + t * (D / 16) + (e >> 4)]);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = e2m1_nibble_to_f32(c >> (4 * i)) * s;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = dense_elem<D>(rec, FMT, t, e + i);
  }
}
template <int D, int FMT>
__device__ __forceinline__ void v_eight(const uint8_t* __restrict__ rec, int t, int e, float (&v)[8]) {
  if constexpr (FMT == TSB200_KV_INT8 || FMT == TSB200_KV_FP8) {
    const uint2 c = *reinterpret_cast<const uint2*>(rec + e * 16 + t);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned b = ((i < 4 ? c.x : c.y) >> (8 * (i & 3))) & 0xffu;
      v[i] = FMT == TSB200_KV_INT8 ? (float)(int8_t)b * reinterpret_cast<const float*>(rec + 16 * D)[t + i] : e4m3_byte_to_f32(b);
    }
  } else if constexpr (FMT == TSB200_KV_NVFP4) {
    const uint2 c = *reinterpret_cast<const uint2*>(rec + (e >> 1) * 16 + t);
    const uint2 s = *reinterpret_cast<const uint2*>(rec + 16 * (D / 2) + (e >> 4) * 16 + t);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = e2m1_nibble_to_f32((i < 4 ? c.x : c.y) >> (8 * (i & 3) + (e & 1) * 4)) * e4m3_byte_to_f32(((i < 4 ? s.x : s.y) >> (8 * (i & 3))) & 0xffu);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = dense_elem<D>(rec, FMT, t + i, e);
  }
}
__device__ __forceinline__ uint4 pack_eight(const float (&v)[8], float s) {
  uint4 o;
  unsigned* u = reinterpret_cast<unsigned*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i] * s, v[2 * i + 1] * s);
    u[i] = *reinterpret_cast<const unsigned*>(&p);
  }
  return o;
}

template <int D, int FMT>
__global__ void __launch_bounds__(256)
kv_gather_heads_kernel(tsb200_kv_desc kv, __nv_bfloat16* __restrict__ k_out, __nv_bfloat16* __restrict__ vt_out, int64_t L, int64_t Lp) {
  constexpr int rec_bytes = FMT == TSB200_KV_INT8 ? 16 * D + 64 : FMT == TSB200_KV_FP8 ? 16 * D : FMT == TSB200_KV_NVFP4 ? 9 * D
                            : FMT == TSB200_KV_F32 ? 64 * D : 32 * D;
  constexpr int UNITS = kGatherTokens * D / 8, PER = UNITS / 256;
  pdl_launch_dependents();
  pdl_wait();
  const int64_t b = blockIdx.z, hk = blockIdx.y, t0 = (int64_t)blockIdx.x * kGatherTokens;
  const int64_t len = min((int64_t)kv.seq_lens[b], L);
  const float ks = FMT == TSB200_KV_FP8 ? kv.k_scale[b * kv.hkv + hk] : 1.0f;
  const float vs = FMT == TSB200_KV_FP8 ? kv.v_scale[b * kv.hkv + hk] : 1.0f;
  auto record = [&](const uint8_t* pool, int64_t t) {          // of token t's page (t < len)
    int64_t page = kv.block_table[b * kv.bt_stride + (t >> 4)];
    page = page < 0 ? 0 : (page >= kv.num_pages ? kv.num_pages - 1 : page);
    return pool + (page * kv.hkv + hk) * (int64_t)rec_bytes;
  };
  __nv_bfloat16* ko = k_out + (b * kv.hkv + hk) * L * D;
  __nv_bfloat16* vo = vt_out + (b * kv.hkv + hk) * (int64_t)D * Lp;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int u = threadIdx.x + i * 256;
    const int64_t t = t0 + u / (D / 8);
    const int e = u % (D / 8) * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t < len) k_eight<D, FMT>(record(kv.k_pool, t), (int)(t & 15), e, v);
    if (t < L) *reinterpret_cast<uint4*>(ko + t * D + e) = pack_eight(v, ks);
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int u = threadIdx.x + i * 256;
    const int64_t t = t0 + u % (kGatherTokens / 8) * 8;
    const int e = u / (kGatherTokens / 8);
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t < len) {
      v_eight<D, FMT>(record(kv.v_pool, t), (int)(t & 15), e, v);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (t + j >= len) v[j] = 0.f;
    }
    if (t < Lp) *reinterpret_cast<uint4*>(vo + e * Lp + t) = pack_eight(v, vs);   // Lp is a multiple of 8
  }
}

template <int D>
int launch_gather_heads(const tsb200_kv_desc& kv, void* k_out, void* vt_out, int64_t B, int64_t L, int64_t Lp, cudaStream_t s) {
  const dim3 grid((unsigned)((Lp + kGatherTokens - 1) / kGatherTokens), (unsigned)kv.hkv, (unsigned)B);
#define TSB_GO(F) TSB_CUDA(launch_kernel(kv_gather_heads_kernel<D, F>, grid, dim3(256), 0, s, kv, (__nv_bfloat16*)k_out, (__nv_bfloat16*)vt_out, L, Lp))
  switch (kv.format) {
    case TSB200_KV_INT8: TSB_GO(TSB200_KV_INT8); break;
    case TSB200_KV_FP8: TSB_GO(TSB200_KV_FP8); break;
    case TSB200_KV_NVFP4: TSB_GO(TSB200_KV_NVFP4); break;
    case TSB200_KV_F32: TSB_GO(TSB200_KV_F32); break;
    default: TSB_GO(TSB200_KV_BF16);
  }
#undef TSB_GO
  return TSB200_OK;
}

template <int D>
int launch_prefill(const void* q, int64_t q_token_stride, const void* k, const void* vt, void* out, int64_t B, int64_t T, int64_t L,
                   int64_t Lp, int H, int hkv, float sm_scale, int* status, cudaStream_t s) {
  using Lt = PfLayout<D>;
  static bool configured[64] = {false};
  int dev = 0;
  TSB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TSB200_ERR_DEVICE;
  if (!configured[dev]) {
    TSB_CUDA(cudaFuncSetAttribute(prefill_attn_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lt::kBytes));
    configured[dev] = true;
  }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return TSB200_ERR_CUDA;
  CUtensorMap mq, mk, mv;
  {   // q [B*T tokens][H heads][D]: box = 64 columns of one head for 128 tokens
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)(B * T)};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)q_token_stride * 2};
    cuuint32_t box[3] = {64, 1, BQ};
    cuuint32_t estr[3] = {1, 1, 1};
    if (fn(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return TSB200_ERR_CUDA;
  }
  if (!make_map(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, k, (uint64_t)D, (uint64_t)(B * hkv * L), (uint64_t)D * 2, 64, BKEY, CU_TENSOR_MAP_SWIZZLE_128B))
    return TSB200_ERR_CUDA;
  if (!make_map(&mv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, vt, (uint64_t)Lp, (uint64_t)(B * hkv * D), (uint64_t)Lp * 2, 64, D, CU_TENSOR_MAP_SWIZZLE_128B))
    return TSB200_ERR_CUDA;
  PfParams p;
  p.B = B; p.T = T; p.L = L; p.H = H; p.hkv = hkv;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.out = (__nv_bfloat16*)out;
  p.status = status;
  p.nq = (int)((T + BQ - 1) / BQ);
  // Two tiles to a CTA take up to 1.5 times the time of one: with a tile for at most every SM each gets its own (1 x 64 tokens at the end
  // of 4096, 32 / 8 heads: 92 us in pairs, 63 here).
  const int64_t tiles = (int64_t)p.nq * (H / hkv);
  p.per = tiles * hkv * B <= kPlanSMs ? 1 : 2;
  const int64_t pairs = (tiles + p.per - 1) / p.per, items = pairs * hkv * B;
  if (items > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  p.pairs = (int)pairs;
  p.items = (int)items;
  const dim3 grid((unsigned)(items < kPlanSMs ? items : kPlanSMs));        // one CTA per SM
  TSB_CUDA(launch_kernel(prefill_attn_kernel<D>, grid, dim3(kPfThreads), (size_t)Lt::kBytes, s, mq, mk, mv, p));
  return TSB200_OK;
}

}  // namespace
}  // namespace tsb

using namespace tsb;

extern "C" int tsb200_kv_gather_heads(const tsb200_kv_desc* kv, void* k_out, void* vt_out, int64_t B, int64_t L, int64_t Lp,
                                      void* stream) {
  TSB_REQUIRE_DEVICE();
  const int st = validate_kv(kv, true);
  if (st != TSB200_OK) return st;
  if (B < 0 || L < 0 || Lp < L || (Lp & 7)) return TSB200_ERR_ARG;
  if (B == 0 || L == 0) return TSB200_OK;
  if (!k_out || !vt_out || !aligned(k_out, 16) || !aligned(vt_out, 16)) return TSB200_ERR_ARG;
  if (B > 65535 || kv->hkv > 65535 || L > kv->bt_stride * 16) return TSB200_ERR_ARG;
  return kv->head_dim == 64 ? launch_gather_heads<64>(*kv, k_out, vt_out, B, L, Lp, as_stream(stream))
                            : launch_gather_heads<128>(*kv, k_out, vt_out, B, L, Lp, as_stream(stream));
}

extern "C" int tsb200_prefill_attn(const void* q, int64_t q_token_stride, const void* k, const void* vt, void* out, int64_t B,
                                   int64_t T, int64_t L, int64_t Lp, int H, int hkv, int head_dim, float sm_scale, int32_t* status,
                                   void* stream) {
  TSB_REQUIRE_DEVICE();
  if (B < 0 || T < 0 || L < T || Lp < L || (Lp & 7) || H <= 0 || hkv <= 0 || H % hkv) return TSB200_ERR_ARG;
  if (head_dim != 64 && head_dim != 128) return TSB200_ERR_UNSUPPORTED;
  if (B == 0 || T == 0) return TSB200_OK;
  if (!q || !k || !vt || !out || !aligned(q, 16) || !aligned(k, 16) || !aligned(vt, 16) || !aligned(out, 16)) return TSB200_ERR_ARG;
  const int64_t qs = q_token_stride ? q_token_stride : (int64_t)H * head_dim;
  if (qs < (int64_t)H * head_dim || (qs & 7)) return TSB200_ERR_ARG;
  if (B > 65535 || H > 65535 || B * T > 0x7fffffffLL || B * hkv * L > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  return head_dim == 64 ? launch_prefill<64>(q, qs, k, vt, out, B, T, L, Lp, H, hkv, sm_scale, status, s)
                        : launch_prefill<128>(q, qs, k, vt, out, B, T, L, Lp, H, hkv, sm_scale, status, s);
}
