// Split-K paged decode attention on tensor cores (int8, FP8-e4m3 and NVFP4 pages).
//
// Replaces transformersurgeon/blocks/mha.py:9-103 (attention(): GQA, softmax, @V) for the
// decode step.  One CTA = one (sequence, kv head, split); its warps (4, or 6 for int8 pages) take pages
// round-robin.  Each warp streams its pages through a private ring of shared-memory
// stages (two lanes, one cp.async.bulk per record, on an mbarrier; a page's number is looked up a
// page before its copy leaves), and computes, per 16-token page,
//     S^T[token, head] = K_page . Q^T          (8 x mma.m16n8k16, f16 in / f32 acc)
//     online softmax over tokens per head       (warp shuffles over the token lanes)
//     O^T[dim, head]  += V^T_page . P^T         (8 x mma.m16n8k16)
// so the whole GQA group (<= 8 query heads) shares one read of the page.  Codes are
// widened to f16 in registers (exact for e4m3 and int8); scales are applied in fp32.  NVFP4 pages:
// an e2m1 code times its e4m3 block scale is exact in f16 (2 x 4 significant bits), so K goes to
// the MMA as code * scale; for V the block scale of a token is folded into that token's softmax
// weight (one product per 16-dim block and token instead of one per element).
// Several splits leave partials (m, l, acc): in shared memory where a cluster merges them (launch_mma says when), else in the workspace for
// decode_attn_reduce_kernel.  That launch is resident before the last partial is there, and for few outputs 3-5 us faster than a merge by the
// last CTA of a pair (captured: int8, 2 sequences x 32 / 8 heads x 500 tokens 8.2 -> 5.5 us, NVFP4, 1 x 32 / 8 x 1000 9.6 -> 6.2); a
// call that is not captured pays 2 us for it on the host (1 x 12 x 1000, head_dim 64: 9.3 -> 11.2).
//
// Bound by the page loop's instructions.  Against copies by all 32 lanes (cp.async, 4 to 9 a lane and page), block scales widened by every
// lane and a rescale of the accumulators on every page, half to all of the stated tokens: int8, 64 x 8 kv heads x 4096 95.1 -> 89.6 us, 16 x 4 x
// 8192 35.7 -> 33.6; NVFP4, 64 x 8 x 4096 96.9 -> 86.9, 30 x 4 x 3000 31.3 -> 26.6, 8 x 4 x 32768 58.8 -> 54.3.
#include "tc_common.cuh"
#include "decode_attn_common.cuh"

namespace tsb {

template <typename T>
int launch_attn_fp8(const tsb200_kv_desc& kv, const void* q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S,
                    int64_t B, float* ws, void* out, int* status, cudaStream_t st);
int validate_attn_args(const tsb200_kv_desc* kv, const void* q, void* out, int dtype, int64_t B, int H,
                       int64_t max_seq_len, void* workspace, size_t workspace_bytes, bool& noop, size_t need_bytes);
int attn_dense(const tsb200_kv_desc* kv, const void* q, void* out, int dtype, int64_t qs, int64_t B, int H, float sm_scale,
               int64_t max_seq_len, float* ws, int* counters, cudaStream_t s);

namespace {

using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_try_wait;
using tc::smem_u32;

constexpr unsigned kWaitLimit = 1u << 22;
// Warps per CTA, ring stages (pages) per warp, CTAs per SM that registers are to allow.  What counts is how many CTAs an SM holds: the page
// loop is bound by the instructions that widen codes and by the chain of a page's softmax, and the warps of other CTAs fill its gaps.  int8,
// head_dim 64: 30 sequences x 2 kv heads x 1.5k-3k tokens 12.4 us at 5 CTAs, 13.5 at 4; head_dim 128 is limited by registers (3).
// VAR is another instance for some grids (the dispatch at the end counts CTAs; times of 1100 grids, captured):
//   * NVFP4, 128: 3 stages and 5 CTAs, or (VAR) 4 and 4, which has the registers for it.  VAR for up to 512 CTAs, which it holds at once too, from two an SM or
//     eight pages a split on (1 x 8 x 16k-32k tokens, 64 splits: 17.9 -> 15.1 us, 32 x 16 x 32-64, one split 0.91 of the time; below both
//     0.87 to 1.11, 64 x 4 x 32-64 5.0 -> 5.4), and for splits of 64 pages and more: on grids of two waves of
//     either 2-5 % faster, on 768 CTAs, one and a bit, 5 % faster to 4 % slower.  Shorter splits want the fifth CTA (16 x 8 x 250-500,
//     5 pages a split: 10.4 us, VAR 11.8; 21 pages 20.0 / 20.1).
//   * NVFP4 and FP8, 64: 88 registers and 5 CTAs, or (VAR) 64 and 8 (FP8: 24 bytes spilled).  VAR where there are more CTAs than the first holds and few
//     pages to each, so that what counts is how many start at a time (NVFP4, 128 x 12 x 32-64 tokens 9.5 -> 7.8 us, 128 x 4 x 65-130, 8
//     heads 11.6 -> 9.1); with long splits or few CTAs it is up to a third slower.
template <int FMT, int D, bool VAR> struct AttnCfg {
  static constexpr int kWarps = FMT == TSB200_KV_INT8 ? 6 : 4;
  static constexpr int kStages = FMT == TSB200_KV_INT8 && D == 128 ? 2 : (D == 128 && VAR ? 4 : 3);
  static constexpr int kCtas = FMT == TSB200_KV_INT8 ? (D == 128 ? 3 : 5) : D == 64 && VAR ? 8 : (FMT == TSB200_KV_NVFP4 && D == 128 && !VAR ? 5 : 4);
};

__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ float ex2(float x) {                       // (weights below 2^-126 are 0)
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned movmatrix_trans(unsigned a) {
  unsigned d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ unsigned pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&h);
}
// Two 8-bit codes (low 16 bits of w) -> f16x2, low byte in the low half.
template <int FMT> __device__ __forceinline__ unsigned widen2(unsigned w16) {
  if (FMT == TSB200_KV_FP8) {
    __half2_raw r = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w16 & 0xffffu), __NV_E4M3);
    return (unsigned)r.x | ((unsigned)r.y << 16);
  } else {
    // int8 -> f16: (code ^ 0x80) | 0x6400 is the f16 1024 + 128 + code; subtract 1152.
    const unsigned u = (w16 ^ 0x8080u);
    unsigned v = __byte_perm(u, 0x64646464u, 0x4140);   // {0x64, b1, 0x64, b0}
    const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6480));
    __half2 h = __hsub2(*reinterpret_cast<__half2*>(&v), bias);
    return *reinterpret_cast<unsigned*>(&h);
  }
}
// Two e4m3 codes (low 16 bits of w) -> f16x2 holding value * 2^-8, with integer instructions only:
// sign to bit 15, exponent+mantissa shifted to f16 bits 13..7 (e4m3 exponent bias 7 vs f16 bias 15,
// hence the 2^-8; e4m3 subnormals land on f16 subnormals, also exactly).  Used for the K operand so
// that only half of the widening work sits on the conversion pipe; the caller folds 2^8 into its scale.
__device__ __forceinline__ unsigned widen2_e4m3_alu(unsigned w16) {
  const unsigned t = __byte_perm(w16, 0u, 0x1404);          // {b1, 0, b0, 0}: each code in the high byte of a half
  return (t & 0x80008000u) | ((t >> 1) & 0x3f803f80u);
}
#ifndef TSB_ATTN_ALU_WIDEN
#define TSB_ATTN_ALU_WIDEN 1
#endif
template <int FMT> __device__ __forceinline__ unsigned widen2_k(unsigned w16) {
  return (FMT == TSB200_KV_FP8 && TSB_ATTN_ALU_WIDEN) ? widen2_e4m3_alu(w16) : widen2<FMT>(w16);
}

// e2m1 codes n_A and n_{A+4} of the 8 in a 32-bit word (16 bits apart, so one shift serves both) ->
// f16x2 holding value * 2^-14, with integer instructions only: the sign goes to bit 15 and the
// three magnitude bits (2 exponent, 1 mantissa; bias 1 against f16's 15) to f16 bits 11..9; code
// 0.5 lands on an f16 subnormal, also exactly.  The conversion instructions are far slower.
template <int A> __device__ __forceinline__ unsigned e2m1_pair_alu(unsigned w) {
  const unsigned m = A < 3 ? w << (9 - 4 * (A < 3 ? A : 0)) : w >> 3;
  return ((w << (12 - 4 * A)) & 0x80008000u) | (m & 0x0E000E00u);
}
// e4m3 codes in bytes 1 and 3 of t -> f16x2 of value * 2^-8 (see widen2_e4m3_alu)
__device__ __forceinline__ unsigned e4m3_hi_bytes_alu(unsigned t) { return (t & 0x80008000u) | ((t >> 1) & 0x3f803f80u); }
__device__ __forceinline__ unsigned hmul2_u(unsigned a, unsigned b) {
  __half2 h = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<unsigned*>(&h);
}
constexpr int kBarBytes = 256;                 // barriers of all warps, ahead of the rings; never anything else (an mbarrier's words may not be reused)
template <int FMT, int D> struct RecBytes {
  static constexpr int value = FMT == TSB200_KV_INT8 ? 16 * D + 64 : (FMT == TSB200_KV_NVFP4 ? 9 * D : 16 * D);
};

template <typename T, int D, int FMT, bool VAR>
__global__ void __launch_bounds__(AttnCfg<FMT, D, VAR>::kWarps * 32, AttnCfg<FMT, D, VAR>::kCtas)
decode_attn_mma_kernel(tsb200_kv_desc kv, const T* __restrict__ q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S,
                       float* __restrict__ ws, T* __restrict__ out, int* __restrict__ status) {
  constexpr bool FP4 = FMT == TSB200_KV_NVFP4;
  constexpr int REC = RecBytes<FMT, D>::value;
  constexpr int kWarps = AttnCfg<FMT, D, VAR>::kWarps, kStages = AttnCfg<FMT, D, VAR>::kStages;
  constexpr int STAGE = 2 * REC;                // K and V of a page
  constexpr int NC = D / 16;                    // k-steps of QK, m-tiles of PV
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_launch_dependents();

  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gid = lane >> 2, tid = lane & 3;
  const int b = blockIdx.x / kv.hkv, hk = blockIdx.x % kv.hkv, s = blockIdx.y;
  const int g = H / kv.hkv;
  const int g0 = blockIdx.z * 8, gn = min(8, g - g0);
  uint8_t* ring = smem + kBarBytes + (size_t)w * kStages * STAGE;
  uint2* vscales = reinterpret_cast<uint2*>(smem + kBarBytes + (size_t)kWarps * kStages * STAGE) + w * (D / 4);    // NVFP4
  const unsigned ring_a = smem_u32(ring), bar_a = smem_u32(smem) + w * kStages * 8;
  if (lane == 0) {
    for (int i = 0; i < kStages; ++i) mbar_init(reinterpret_cast<unsigned long long*>(smem) + w * kStages + i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  // lengths and block table do not come from the preceding launch (see tsb200_set_pdl): looked up ahead of the dependency wait
  int len = kv.seq_lens[b];
  len = len < 0 ? 0 : (len > max_seq_len ? (int)max_seq_len : len);
  int pb, pe;
  split_range(len, s, S, pb, pe);

  // ---- this warp's pages: pb + w, pb + w + kWarps, ...  Lane 0 copies K, lane 1 V; a page's number is looked up a page before its copy leaves.
  const int n_my = pe - pb > w ? (pe - pb - w + kWarps - 1) / kWarps : 0;
  const int64_t rec_stride = (int64_t)kv.hkv * REC;
  const uint8_t* pool = ((lane & 1) ? kv.v_pool : kv.k_pool) + (int64_t)hk * REC;
  const int* table = kv.block_table + (int64_t)b * kv.bt_stride + pb + w;
  auto look_up = [&](int it) { return lane < 2 && it < n_my ? table[it * kWarps] : 0; };
  auto issue = [&](int it, int page) {
    if (it < n_my) {
      if (lane == 0) mbar_expect_tx(reinterpret_cast<unsigned long long*>(smem) + w * kStages + it % kStages, 2u * REC);
      __syncwarp();
      if (lane < 2) {
        const int64_t at = page < 0 ? 0 : (page >= kv.num_pages ? kv.num_pages - 1 : page);
        bulk_g2s(ring_a + (it % kStages) * STAGE + lane * REC, pool + at * rec_stride, REC, bar_a + (it % kStages) * 8);
      }
    }
  };
  int ahead[kStages];
#pragma unroll
  for (int i = 0; i < kStages; ++i) ahead[i] = look_up(i);
  pdl_wait();     // q and the page just appended come from the preceding kernels
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) issue(i, ahead[i]);
  int next_page = ahead[kStages - 1];

  // Q^T fragments (B operand): this lane holds head g0+gid at the dims of its k-slots: 16 consecutive ones per four steps, fetched as
  // 16-byte pieces where q allows it (element by element: 32 loads, 2500 cycles before the first page of a short split).
  unsigned qf[NC][2];
  {
    const bool valid = gid < gn;
    const T* qp = q + (int64_t)b * qs + (int64_t)(hk * g + g0 + (valid ? gid : 0)) * D + 16 * tid;
    const bool vec = (reinterpret_cast<uintptr_t>(q) & 15) == 0 && qs * sizeof(T) % 16 == 0;
#pragma unroll
    for (int hh = 0; hh < NC / 4; ++hh) {
      __align__(16) T x[16];
      if (vec) {
#pragma unroll
        for (int i = 0; i < (int)sizeof(T); ++i) reinterpret_cast<uint4*>(x)[i] = reinterpret_cast<const uint4*>(qp + 64 * hh)[i];
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = qp[64 * hh + i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // int8 / fp8: the step's k-slots are 4 consecutive dims; NVFP4: dims (x, x + 4) and (x + 1, x + 5),
        // the pairs that e2m1_pair_alu extracts from a word of 8 codes
        const int base = FP4 ? 8 * (i >> 1) + 2 * (i & 1) : 4 * i;
        constexpr int o1 = FP4 ? 4 : 1, o2 = FP4 ? 1 : 2, o3 = FP4 ? 5 : 3;
        qf[4 * hh + i][0] = valid ? pack_h2(to_f32<T>(x[base]), to_f32<T>(x[base + o1])) : 0u;
        qf[4 * hh + i][1] = valid ? pack_h2(to_f32<T>(x[base + o2]), to_f32<T>(x[base + o3])) : 0u;
      }
    }
  }
  float kscale = 1.f, vscale = 1.f;
  if (FMT == TSB200_KV_FP8) { kscale = kv.k_scale[b * kv.hkv + hk]; vscale = kv.v_scale[b * kv.hkv + hk]; }
  // FP8 keys are widened to value * 2^-8 (widen2_e4m3_alu): 256 restores the scale
  // NVFP4 keys reach the MMA as code * block scale * 2^-7, values as code * 2^-14 (see below)
  if (FMT == TSB200_KV_NVFP4) vscale = 16384.0f;
  const float sc = sm_scale * 1.4426950408889634f * kscale *
                   ((FMT == TSB200_KV_FP8 && TSB_ATTN_ALU_WIDEN) ? 256.0f : (FMT == TSB200_KV_NVFP4 ? 128.0f : 1.0f));

  float oacc[NC][4];
#pragma unroll
  for (int i = 0; i < NC; ++i) { oacc[i][0] = oacc[i][1] = oacc[i][2] = oacc[i][3] = 0.f; }
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;   // heads 2*tid, 2*tid+1 (log2 domain)

  const int r1 = 4 * (gid >> 1) + (gid & 1), r2 = r1 + 2;   // token rows of this lane in S^T
  bool ok = true;
  for (int it = 0; it < n_my; ++it) {
    issue(it + kStages - 1, next_page);
    next_page = look_up(it + kStages);
    {
      unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem) + w * kStages + it % kStages;
      const unsigned parity = (it / kStages) & 1;
      unsigned spins = 0;
      while (!mbar_try_wait(bar, parity)) {
        if (++spins > kWaitLimit) { ok = false; break; }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
    }
    const int nt = min(16, len - (pb + w + it * kWarps) * 16);
    const uint8_t* sK = ring + (it % kStages) * STAGE;
    const uint8_t* sV = sK + REC;

    // ---- S^T = K . Q^T -----------------------------------------------------------
    float sacc[4] = {0.f, 0.f, 0.f, 0.f};
    if (FP4) {
      // the lane's 16 dims of a row = 8 bytes of codes = exactly one scale block
      // block scale * 2^-8 (integer widening) * 2^15 -> scale * 2^7 <= 57344; code * 2^-14 times that is
      // code * scale * 2^-7, exact in f16 (6 significant bits, >= 2^-17)
      const unsigned k215 = 0x78007800u, sel = tid * 0x1010u + 0x0404u;
      const unsigned* s1 = reinterpret_cast<const unsigned*>(sK + 16 * (D / 2) + r1 * (D / 16));
      const unsigned* s2 = reinterpret_cast<const unsigned*>(sK + 16 * (D / 2) + r2 * (D / 16));
#pragma unroll
      for (int hh = 0; hh < D / 64; ++hh) {
        const int j = tid + 4 * hh;
        const uint2 ka = *reinterpret_cast<const uint2*>(sK + r1 * (D / 2) + 8 * j);
        const uint2 kb = *reinterpret_cast<const uint2*>(sK + r2 * (D / 2) + 8 * j);
        const unsigned sa = hmul2_u(e4m3_hi_bytes_alu(__byte_perm(s1[hh], 0u, sel)), k215);
        const unsigned sb = hmul2_u(e4m3_hi_bytes_alu(__byte_perm(s2[hh], 0u, sel)), k215);
        mma16816(sacc, hmul2_u(e2m1_pair_alu<0>(ka.x), sa), hmul2_u(e2m1_pair_alu<0>(kb.x), sb), hmul2_u(e2m1_pair_alu<1>(ka.x), sa),
                 hmul2_u(e2m1_pair_alu<1>(kb.x), sb), qf[4 * hh][0], qf[4 * hh][1]);
        mma16816(sacc, hmul2_u(e2m1_pair_alu<2>(ka.x), sa), hmul2_u(e2m1_pair_alu<2>(kb.x), sb), hmul2_u(e2m1_pair_alu<3>(ka.x), sa),
                 hmul2_u(e2m1_pair_alu<3>(kb.x), sb), qf[4 * hh + 1][0], qf[4 * hh + 1][1]);
        mma16816(sacc, hmul2_u(e2m1_pair_alu<0>(ka.y), sa), hmul2_u(e2m1_pair_alu<0>(kb.y), sb), hmul2_u(e2m1_pair_alu<1>(ka.y), sa),
                 hmul2_u(e2m1_pair_alu<1>(kb.y), sb), qf[4 * hh + 2][0], qf[4 * hh + 2][1]);
        mma16816(sacc, hmul2_u(e2m1_pair_alu<2>(ka.y), sa), hmul2_u(e2m1_pair_alu<2>(kb.y), sb), hmul2_u(e2m1_pair_alu<3>(ka.y), sa),
                 hmul2_u(e2m1_pair_alu<3>(kb.y), sb), qf[4 * hh + 3][0], qf[4 * hh + 3][1]);
      }
    } else {
#pragma unroll
      for (int hh = 0; hh < D / 64; ++hh) {
        const int j = tid + 4 * hh;
        const uint4 ka = *reinterpret_cast<const uint4*>(sK + r1 * D + 16 * j);
        const uint4 kb = *reinterpret_cast<const uint4*>(sK + r2 * D + 16 * j);
        const unsigned wa[4] = {ka.x, ka.y, ka.z, ka.w};
        const unsigned wb[4] = {kb.x, kb.y, kb.z, kb.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = 4 * hh + i;
          mma16816(sacc, widen2_k<FMT>(wa[i]), widen2_k<FMT>(wb[i]), widen2_k<FMT>(wa[i] >> 16), widen2_k<FMT>(wb[i] >> 16),
                   qf[c][0], qf[c][1]);
        }
      }
    }
    // ---- online softmax over the page's tokens (rows) per head (column) -------------
    float ks1 = 1.f, ks2 = 1.f, vs1 = 1.f, vs2 = 1.f;
    if (FMT == TSB200_KV_INT8) {
      const float* ksc = reinterpret_cast<const float*>(sK + 16 * D);
      const float* vsc = reinterpret_cast<const float*>(sV + 16 * D);
      ks1 = ksc[r1]; ks2 = ksc[r2]; vs1 = vsc[r1]; vs2 = vsc[r2];
    }
    const bool ok1 = r1 < nt, ok2 = r2 < nt;
    const float s0 = ok1 ? sacc[0] * (sc * ks1) : -INFINITY;
    const float s1 = ok1 ? sacc[1] * (sc * ks1) : -INFINITY;
    const float s2 = ok2 ? sacc[2] * (sc * ks2) : -INFINITY;
    const float s3 = ok2 ? sacc[3] * (sc * ks2) : -INFINITY;
    float mx0 = fmaxf(s0, s2), mx1 = fmaxf(s1, s3);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
    }
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);   // finite: token 0 of a page is always valid
    const float c0 = ex2(m0 - mn0), c1 = ex2(m1 - mn1);
    const float p0 = ex2(s0 - mn0), p1 = ex2(s1 - mn1), p2 = ex2(s2 - mn0), p3 = ex2(s3 - mn1);
    l0 = __fmaf_rn(l0, c0, p0 + p2);
    l1 = __fmaf_rn(l1, c1, p1 + p3);
    m0 = mn0; m1 = mn1;
    if (__any_sync(0xffffffffu, c0 != 1.0f || c1 != 1.0f)) {  // (a product by 1 changes nothing)
#pragma unroll
      for (int mt = 0; mt < NC; ++mt) { oacc[mt][0] *= c0; oacc[mt][1] *= c1; oacc[mt][2] *= c0; oacc[mt][3] *= c1; }
    }
    // ---- O^T += V^T . P^T -----------------------------------------------------------
    {
      if (FP4) vs1 = vs2 = 256.0f;               // NVFP4: the block scales multiply P as scale * 2^-8
      const unsigned P1 = pack_h2(ok1 ? p0 * vs1 : 0.f, ok1 ? p1 * vs1 : 0.f);        // (a stale slot may hold any scale)
      const unsigned P2 = pack_h2(ok2 ? p2 * vs2 : 0.f, ok2 ? p3 * vs2 : 0.f);
      unsigned pb0 = movmatrix_trans(P1);         // tokens 4*tid, 4*tid+1 of head gid
      unsigned pb1 = movmatrix_trans(P2);         // tokens 4*tid+2, 4*tid+3
      if (FP4) {                                  // NVFP4 pairs tokens (4*tid, 4*tid+2) and (4*tid+1, 4*tid+3)
        const unsigned t0 = __byte_perm(pb0, pb1, 0x5410), t1 = __byte_perm(pb0, pb1, 0x7632);
        pb0 = t0; pb1 = t1;
      }
      if (FP4) {
        // the page's block scales, widened once for the warp (every lane for itself they were a seventh of the kernel's instructions: 8 sequences x
        // half to all of 32k tokens, 28 / 4 heads: 59 us against 52): f16 pairs of tokens (0, 2) and (1, 3) of four, value * 2^-8, stale slots +0
        if (lane < D / 4) {
          unsigned sw = *reinterpret_cast<const unsigned*>(sV + 16 * (D / 2) + lane * 4);
          if (nt < 16) {
            const int rest = nt - 4 * (lane & 3);
            sw &= rest >= 4 ? 0xffffffffu : (rest <= 0 ? 0u : (0xffffffffu >> (8 * (4 - rest))));
          }
          vscales[lane] = make_uint2(e4m3_hi_bytes_alu(__byte_perm(sw, 0u, 0x2404)), e4m3_hi_bytes_alu(__byte_perm(sw, 0u, 0x3414)));
        }
        __syncwarp();
#pragma unroll
        for (int mt = 0; mt < NC; ++mt) {
          // one word = tokens 4*tid..4*tid+3 of dims 16*mt + 2*gid (low nibbles) and + 1 (high nibbles):
          // MMA rows gid / gid + 8 are those two dims
          const unsigned wv = *reinterpret_cast<const unsigned*>(sV + (8 * mt + gid) * 16 + 4 * tid);
          const uint2 sc2 = vscales[mt * 4 + tid];
          // code pairs 16 bits apart = tokens (0, 2) and (1, 3) of the lane's four; values enter as code * 2^-14
          // (2^14 is restored with the split scale), weights as p * 2^8 * (block scale * 2^-8)
          mma16816(oacc[mt], e2m1_pair_alu<0>(wv), e2m1_pair_alu<1>(wv), e2m1_pair_alu<2>(wv), e2m1_pair_alu<3>(wv),
                   hmul2_u(pb0, sc2.x), hmul2_u(pb1, sc2.y));
        }
        __syncwarp();                            // the next page's take their place
      } else {
        // bytes of this lane's 4 tokens that are inside the sequence (stale slots -> +0)
        unsigned vmask = 0xffffffffu;
        if (nt < 16) {
          const int rest = nt - 4 * tid;
          vmask = rest >= 4 ? 0xffffffffu : (rest <= 0 ? 0u : (0xffffffffu >> (8 * (4 - rest))));
        }
#pragma unroll
        for (int mt = 0; mt < NC; ++mt) {
          unsigned w1 = *reinterpret_cast<const unsigned*>(sV + (16 * mt + gid) * 16 + 4 * tid);
          unsigned w2 = *reinterpret_cast<const unsigned*>(sV + (16 * mt + gid + 8) * 16 + 4 * tid);
          if (FMT == TSB200_KV_FP8) { w1 &= vmask; w2 &= vmask; }     // (an int8 code is finite whatever it is)
          mma16816(oacc[mt], widen2<FMT>(w1), widen2<FMT>(w2), widen2<FMT>(w1 >> 16), widen2<FMT>(w2 >> 16), pb0, pb1);
        }
      }
    }
    __syncwarp();                                // every lane has read the stage: the next round's copies may take it
  }
  if (!ok) {
    // error path only: a wait ran out.  Give the copies still in flight a bounded time to land before
    // shared memory is reused, and record the event.
    if (lane == 0 && status) atomicMax(status, 8);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  // row sums: add the partial sums of the 8 token lanes
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, o);
    l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  }
  const bool clustered = splits_are_cluster();
  __syncthreads();   // every warp is done with its ring; reuse shared memory for the merge
  constexpr int AR = D + 4;                                  // row pitch: the fragments' four head rows fall into different banks
  float* sm_m = reinterpret_cast<float*>(smem + kBarBytes);  // [warps][8]
  float* sm_l = sm_m + kWarps * 8;                           // [warps][8]
  float* sm_c = sm_l + kWarps * 8;                           // [warps][8]
  float* sm_acc = sm_c + kWarps * 8;                         // [warps][8][AR]
  float* sm_part = sm_acc + kWarps * 8 * AR;                 // [8][2 + D]: this split's partials where a cluster merges
  if (gid == 0) {
    sm_m[w * 8 + 2 * tid] = m0; sm_m[w * 8 + 2 * tid + 1] = m1;
    sm_l[w * 8 + 2 * tid] = l0; sm_l[w * 8 + 2 * tid + 1] = l1;
  }
#pragma unroll
  for (int mt = 0; mt < NC; ++mt) {
    float* a = sm_acc + (size_t)w * 8 * AR;
    const int da = FP4 ? 16 * mt + 2 * gid : 16 * mt + gid;         // dims of MMA rows gid and gid + 8
    const int db = FP4 ? da + 1 : da + 8;
    a[(2 * tid) * AR + da] = oacc[mt][0];
    a[(2 * tid + 1) * AR + da] = oacc[mt][1];
    a[(2 * tid) * AR + db] = oacc[mt][2];
    a[(2 * tid + 1) * AR + db] = oacc[mt][3];
  }
  __syncthreads();
  // merge the warps; with one split the result is final, otherwise it is this split's partial.  Coefficients once per (warp, head).
  if (threadIdx.x < kWarps * 8) {
    const int i = threadIdx.x & 7;
    float mm = -INFINITY;
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) mm = fmaxf(mm, sm_m[ww * 8 + i]);
    const float mw = sm_m[threadIdx.x];
    sm_c[threadIdx.x] = mw == -INFINITY ? 0.f : exp2f(mw - mm);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < gn * (D / 2); idx += blockDim.x) {
    const int i = idx / (D / 2), e = idx % (D / 2) * 2;
    float ll = 0.f, a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) {
      const float c = sm_c[ww * 8 + i];
      const float2 x = *reinterpret_cast<const float2*>(&sm_acc[((size_t)ww * 8 + i) * AR + e]);
      ll += sm_l[ww * 8 + i] * c;
      a0 += x.x * c;
      a1 += x.y * c;
    }
    const int64_t bh = (int64_t)b * H + hk * g + g0 + i;
    if (S == 1) {
      out[bh * D + e] = from_f32<T>(ll > 0.f ? a0 * vscale / ll : 0.f);
      out[bh * D + e + 1] = from_f32<T>(ll > 0.f ? a1 * vscale / ll : 0.f);
    } else {
      float* o = clustered ? sm_part + i * (2 + D) : ws + (bh * S + s) * (2 + D);
      if (e == 0) {                                          // natural-log domain (shared with the reducer kernel)
        float mm = -INFINITY;
#pragma unroll
        for (int ww = 0; ww < kWarps; ++ww) mm = fmaxf(mm, sm_m[ww * 8 + i]);
        *reinterpret_cast<float2*>(o) = make_float2(mm * 0.6931471805599453f, ll);
      }
      *reinterpret_cast<float2*>(o + 2 + e) = make_float2(a0 * vscale, a1 * vscale);
    }
  }
  if (clustered) merge_cluster<T, D>(sm_part, gn, S, out + ((int64_t)b * H + hk * g + g0) * D);
}

template <typename T, int D, int FMT, bool VAR>
int launch_mma(const tsb200_kv_desc& kv, const void* q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S, int64_t B, float* ws, void* out,
               int* status, cudaStream_t st) {
  constexpr int REC = RecBytes<FMT, D>::value;
  constexpr int kWarps = AttnCfg<FMT, D, VAR>::kWarps, kStages = AttnCfg<FMT, D, VAR>::kStages;
  static_assert(kWarps * kStages * 8 <= kBarBytes, "barriers");
  constexpr size_t pipe = (size_t)kWarps * (kStages * 2 * REC + (FMT == TSB200_KV_NVFP4 ? D * 2 : 0));
  constexpr size_t merge = (size_t)(kWarps * 24 + kWarps * 8 * (D + 4) + 8 * (2 + D)) * sizeof(float);
  constexpr size_t smem = kBarBytes + (pipe > merge ? pipe : merge);
  static bool configured[64] = {false};   // per device: the attribute lives in the device's context
  int dev = 0;
  TSB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TSB200_ERR_DEVICE;
  if (!configured[dev]) {
    TSB_CUDA(cudaFuncSetAttribute(decode_attn_mma_kernel<T, D, FMT, VAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev] = true;
  }
  const int g = H / kv.hkv;
  dim3 grid((unsigned)(B * kv.hkv), (unsigned)S, (unsigned)((g + 7) / 8));
  // A cluster merges without another launch, but its CTAs start together, in one group of SMs, and none leaves before the last: it is the faster
  // one as long as all of them fit the device at once (captured, NVFP4, head_dim 128: 16 sequences x 8 kv heads x 65-130 tokens, 2 splits, 6.3 us,
  // launch 7.7; 12 x 8 x 500-1000, 8 splits, one CTA in twenty-five too many, 14.9 / 11.9; int8, 64 x 8 x 1k-2k, 4 splits 67.8 / 58.7).  Beyond that it
  // depends on the outputs: the launch has a CTA per sequence and query head.  Two splits, more than one head to a CTA: 128 x 8 x 100-200, 8
  // heads 27.7 / 46.2; one head 21.7 / 20.8.  Up to four splits, more than four heads: 64 x 8 x 250-500, 8 heads 27.6 / 34.4, 4 heads 35.4 / 35.3.  Over
  // 2204 calls of several splits this choice is 0.7 % from the better of the two.
  static int held[64][kMaxCluster + 1] = {};
  const bool clusters = S > 1 && S <= kMaxCluster &&
                        ((S == 2 && g > 1) || (S <= 4 && g > 4) ||
                         (int64_t)grid.x * grid.z <= active_clusters(decode_attn_mma_kernel<T, D, FMT, VAR>, grid, kWarps * 32, smem, held[dev]));
  TSB_CUDA(launch_splits(attn_overlaps(kv), clusters, decode_attn_mma_kernel<T, D, FMT, VAR>, grid, dim3(kWarps * 32), smem, st, kv, (const T*)q, qs, H, sm_scale,
                         max_seq_len, S, ws, (T*)out, status));
  return S == 1 || clusters ? TSB200_OK : launch_reduce<T, D>(ws, B * H, S, out, st);
}

}  // namespace
}  // namespace tsb

using namespace tsb;

// Bytes that serve a problem: counters + partials of choose_splits() splits, which no format's own split count exceeds
// (tsb200_paged_decode_attn_workspace_bytes is the hkv-independent upper bound of this).
static size_t attn_exact_workspace_bytes(const tsb200_kv_desc* kv, int64_t B, int H, int64_t max_seq_len) {
  const int S = choose_splits(B, kv->hkv, max_seq_len);
  return kAttnCounterBytes + (size_t)(B * H * S * (2 + kv->head_dim)) * sizeof(float);
}

static int decode_attn_dispatch(const tsb200_kv_desc* kv, const void* q, void* out, int dtype, int64_t q_batch_stride, int64_t B,
                                int H, float sm_scale, int64_t max_seq_len, void* workspace, size_t workspace_bytes,
                                size_t need_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  bool noop;
  int st = validate_attn_args(kv, q, out, dtype, B, H, max_seq_len, workspace, workspace_bytes, noop, need_bytes);
  if (st != TSB200_OK || noop) return st;
  const int64_t qs = q_batch_stride ? q_batch_stride : (int64_t)H * kv->head_dim;
  if (qs < (int64_t)H * kv->head_dim) return TSB200_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  int* counters = (int*)workspace;                               // zero between calls
  float* ws = (float*)((char*)workspace + kAttnCounterBytes);
  const int D = kv->head_dim;
  const int64_t n_ctr = B * kv->hkv * ((H / kv->hkv + 7) / 8);
  // the last int of the counter block is the status word of the bounded waits, so one counter fewer is usable
  const bool room = n_ctr < (int64_t)(kAttnCounterBytes / sizeof(int));
  int* status = counters + kAttnStatusIndex;
  if (kv->format > TSB200_KV_NVFP4)    // unquantized pages: fp32 math (decode_attn_dense.cu)
    return attn_dense(kv, q, out, dtype, qs, B, H, sm_scale, max_seq_len, ws, room ? counters : nullptr, s);
  if (kv->format == TSB200_KV_FP8 && D == 128 && H / kv->hkv <= 4) {
    // e4m3 pages go to the tensor cores as FP8 (decode_attn_fp8.cu)
    const int S8 = choose_splits_fp8(B, kv->hkv, max_seq_len);   // never more than choose_splits(): the workspace fits
    return dtype == TSB200_F32 ? launch_attn_fp8<float>(*kv, q, qs, H, sm_scale, max_seq_len, S8, B, ws, out, status, s)
                               : launch_attn_fp8<__nv_bfloat16>(*kv, q, qs, H, sm_scale, max_seq_len, S8, B, ws, out, status, s);
  }
  const int S = choose_splits(B, kv->hkv, max_seq_len);
  // Instances: see AttnCfg
  const int64_t pages = (max_seq_len + 15) / 16, ctas = n_ctr * S;
  const bool var = kv->format != TSB200_KV_INT8 &&
                   (D == 64 ? (ctas > 5 * 148 && pages <= 2 * S) || (ctas > 6 * 148 && pages <= (kv->format == TSB200_KV_NVFP4 ? 16 : 8) * S)
                            : kv->format == TSB200_KV_NVFP4 && ((ctas <= 512 && (ctas > 2 * 148 || pages >= 8 * S)) || pages >= 64 * S));
#define TSB_GO(TT, DD, FF)                                                                                                       \
  if (var && FF != TSB200_KV_INT8 && (DD == 64 || FF == TSB200_KV_NVFP4))                                                        \
    return launch_mma<TT, DD, FF, (FF != TSB200_KV_INT8 && (DD == 64 || FF == TSB200_KV_NVFP4))>(*kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, out, status, s); \
  return launch_mma<TT, DD, FF, false>(*kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, out, status, s)
#define TSB_FMT(FF)                                                                                                       \
  if (dtype == TSB200_F32) { if (D == 64) { TSB_GO(float, 64, FF); } TSB_GO(float, 128, FF); }                               \
  if (D == 64) { TSB_GO(__nv_bfloat16, 64, FF); }                                                                            \
  TSB_GO(__nv_bfloat16, 128, FF)
  if (kv->format == TSB200_KV_NVFP4) { TSB_FMT(TSB200_KV_NVFP4); }
  if (kv->format == TSB200_KV_INT8) { TSB_FMT(TSB200_KV_INT8); }
  TSB_FMT(TSB200_KV_FP8);
#undef TSB_FMT
#undef TSB_GO
}

extern "C" int tsb200_paged_decode_attn(const tsb200_kv_desc* kv, const void* q, void* out, int dtype, int64_t q_batch_stride, int64_t B, int H,
                                        float sm_scale, int64_t max_seq_len, void* workspace, size_t workspace_bytes,
                                        void* stream) {
  return decode_attn_dispatch(kv, q, out, dtype, q_batch_stride, B, H, sm_scale, max_seq_len, workspace, workspace_bytes, 0, stream);
}


// ---------------------------------------------------------------------------------------------
// Allocation-free variant.
//
// Some callers may not allocate device memory at all: code running inside a CUDA-graph capture or
// under a framework that forbids cudaMalloc on its serving path, plugins handed a fixed memory
// budget, and host runtimes whose allocator cannot be re-entered from the calling thread.  For them
// the split partials live in the fixed array below instead of a caller-provided workspace.  Every
// GPU that loads this library carries the array (kStaticScratchBytes) until the process exits.
//
// In host code `g_attn_scratch` is only a stand-in for the symbol, not a device address; the
// address the kernels need is obtained once per device with cudaGetSymbolAddress while that device
// is current, and that pointer is what is passed to the launches.
namespace tsb {
namespace {
constexpr size_t kStaticScratchBytes = 8u << 20;     // 8 MiB: e.g. batch 32 x 32 heads x 15 splits x (2 + 128) floats
static __device__ __align__(256) unsigned char g_attn_scratch[kStaticScratchBytes];

int static_scratch_ptr(void** out) {
  static void* ptrs[64] = {nullptr};                 // one resolved address per device ordinal
  int dev = 0;
  TSB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TSB200_ERR_DEVICE;
  if (!ptrs[dev]) {
    void* p = nullptr;
    TSB_CUDA(cudaGetSymbolAddress(&p, g_attn_scratch));   // resolves the copy owned by the current device
    if (!p) return TSB200_ERR_CUDA;
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return TSB200_OK;
}
}  // namespace
}  // namespace tsb

extern "C" size_t tsb200_paged_decode_attn_static_capacity(void) { return tsb::kStaticScratchBytes; }

extern "C" int tsb200_paged_decode_attn_static(const tsb200_kv_desc* kv, const void* q, void* out, int dtype,
                                               int64_t q_batch_stride, int64_t B, int H, float sm_scale,
                                               int64_t max_seq_len, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (!kv || B < 0 || H <= 0) return TSB200_ERR_ARG;
  if (B == 0) return TSB200_OK;
  if (validate_kv(kv, true) != TSB200_OK || max_seq_len < 0) return TSB200_ERR_ARG;
  // sized by the split count this problem will really use, not by the hkv-independent bound that sizes a
  // caller's workspace: more problems fit the fixed array
  const size_t need = attn_exact_workspace_bytes(kv, B, H, max_seq_len);
  if (need > kStaticScratchBytes) return TSB200_ERR_WORKSPACE;   // problem too large for the built-in scratch
  void* scratch = nullptr;
  const int st = static_scratch_ptr(&scratch);
  if (st != TSB200_OK) return st;
  // The head of the array (split counters + status word) MUST be zero when the kernels start.  A finished call
  // leaves it zero, but a call that overlapped another one on the GPU, or was cut short, can leave a counter
  // stuck, after which the fused merge of that (sequence, head) would never fire again.  The caller cannot
  // reach the array, so every call clears the head itself, on its stream, ahead of its kernels.  The partials
  // behind the head need no clearing: each record the merge reads is written by the same call.
  TSB_CUDA(cudaMemsetAsync(scratch, 0, kAttnCounterBytes, as_stream(stream)));
  return decode_attn_dispatch(kv, q, out, dtype, q_batch_stride, B, H, sm_scale, max_seq_len, scratch, kStaticScratchBytes, need,
                              stream);
}
