// Packed-weight GEMM for decode-sized token counts: Y[M, N] = (X[M, K] . Wq[N, K]^T) * scale[N] + bias[N], bf16 activations,
// codes of 8 / 4 / 2 / 1 bits (transformersurgeon/blocks/linear_compressed.py:96-100 on packed codes).
//
// What bounds it: a call moves a few hundred KB to a few MB of codes, so it is a chain of latencies, and with one token the
// widening of the codes (half-rate logic operations) is longer than their transfer.  The kernel keeps the chain short instead of
// feeding tcgen05, whose operands pass through shared and tensor memory behind several barriers:
//   * one warp owns 16 R weight rows and one ACCUMULATION CHAIN (below) and runs warp-level m16n8k16 MMAs; it copies its codes
//     into a private ring of shared memory (cp.async, up to kRing steps in flight), all of the first ones before the dependency
//     wait of a programmatic launch: by the time the activations exist the codes have landed;
//   * the contraction index of an MMA may be permuted inside its 16 columns, so a lane takes columns 4 t .. 4 t + 3 of a block:
//     the codes of one 32-bit word (8 / 4 bits) or of a quarter of it, and 8 bytes of an activation row;
//   * activations are staged once per CTA in B-fragment order, one 16-byte read per two MMAs and token tile;
//   * where one CTA cannot hold the activations of all of K, a cluster of up to 8 CTAs deals the K splits out; the fragments go
//     straight to the shared memory of the CTA that owns the tile (one cluster barrier, no global scratch, no counters).
//
// Measured (chain of dependent calls, programmatic launches, codes from HBM, 4 bits): 4096 x 4096 at 1 / 8 / 16 tokens 6.1 / 6.6 / 7.9 us
// (tcgen05 kernel: 9.4 / 9.5 / 9.6), 1024 x 4096 twice 4.3 us, gated 14336 x 1024 9.5 us, 1024 x 14336 7.2 us, 4096 x 1024 2.9 us:
// the gated MLP of an 8B model 24 us at one token against 35.7 us.
//
// Results are those of the tcgen05 kernel (linear_tcq.cu) bit for bit: the same K splits, in each split one chain over its even
// and one over its odd 64-column blocks, 16 columns per MMA (mma.sync and tcgen05.mma round alike: compared on 1.8 million sums
// of 18944 products), chains added first, splits in order.
#pragma once
#include "common.cuh"

namespace tsb {
namespace gv {

constexpr int kMaxWarps = 16;
constexpr int kMaxTokens = 16;
constexpr int kMaxSmem = 227 * 1024;
constexpr int kRing = 8;                     // steps in flight per warp
constexpr int kRedStride = 20;               // floats per token column of a partial tile (16 rows + 4: conflict-free stores)
inline int token_tiles(int M) { return M <= 8 ? 1 : 2; }

struct Sub {
  const uint8_t* w;
  const float* scale;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* x;
  __nv_bfloat16* y;
};
struct Span {                                // constants of a later launch, brought into the L2 meanwhile, dealt out over the grid
  const uint8_t* p;
  unsigned bytes;
};
constexpr int kMaxSpans = 4;
struct Params {
  Sub sub[2];
  Span ahead[kMaxSpans];
  int M, N, K;                               // N: rows of one matrix
  int row_bytes;                             // bytes of one packed row
  int tiles, tiles_total;                    // 16-row tiles of one matrix; of the launch (stacked matrices add up)
  int kb_total, kb_split, splits;            // 64-column blocks; blocks per K split; K splits
  int ranks, splits_rank;                    // cluster size; K splits per rank
  int tg;                                    // tiles per CTA
  int x_shared;                              // gated: both matrices read the same activations
  int xk_log2;                               // log2 of the threads side by side on one token's columns while x is staged
  int mp_log2;                               // log2 of the tokens padded to a power of two
};

template <int BITS> struct Codes {
  static constexpr int kRow = 8 * BITS;                    // bytes of one row's 64-column block
  static constexpr int kBlocks = BITS >= 4 ? 1 : 4 / BITS; // 64-column blocks (of one chain) per step: a step copies 16 bytes per lane and tile or more
  static constexpr int kStep = kBlocks * 16 * kRow;        // bytes of a tile per step: 1024 / 512 / 512 / 512
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds_v4(unsigned a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ unsigned lds_u32(unsigned a) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_v2(unsigned a, unsigned x, unsigned y) {
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};\n" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int bytes) {   // bytes < 16: the rest is zero-filled
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* src, unsigned bytes) {
  if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned bsub2(unsigned a, unsigned b) {
  __nv_bfloat162 r = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<unsigned*>(&r);
}
__device__ __forceinline__ unsigned bfma2(unsigned a, unsigned b, unsigned c) {
  __nv_bfloat162 r = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b), *reinterpret_cast<__nv_bfloat162*>(&c));
  return *reinterpret_cast<unsigned*>(&r);
}

// Offset, in a 64-column block copied to shared memory, of the word that holds columns 16 b + 4 t .. + 3 of row g (row g + 8: 8 rows
// further, the same exchange).  The 16-byte pieces of a row are exchanged by row so that the eight rows of a read fall into
// different banks; what depends on the lane is computed once, the rest are immediates.
template <int BITS> struct WordAddr {
  unsigned lane[BITS == 8 ? 4 : 2];
  __device__ __forceinline__ WordAddr(int g, int t) {
    if (BITS == 8) {
#pragma unroll
      for (int b = 0; b < 4; ++b) lane[b & 3] = g * 64 + ((b ^ ((g >> 1) & 3)) << 4) + t * 4;
    } else if (BITS == 4) {
      lane[0] = g * 32 + (((g >> 2) & 1) << 4) + (t >> 1) * 4;
      lane[1] = g * 32 + ((1 ^ ((g >> 2) & 1)) << 4) + (t >> 1) * 4;
    } else {
      lane[0] = lane[1] = g * Codes<BITS>::kRow;
    }
  }
  __device__ __forceinline__ unsigned at(int b) const {
    if (BITS == 8) return lane[b & 3];
    if (BITS == 4) return lane[b >> 1] + (b & 1) * 8;
    return lane[0] + (BITS == 2 ? b * 4 : (b >> 1) * 4);
  }
};
// Where the copy of 16-byte piece `piece` of row `row` goes.
template <int BITS> __device__ __forceinline__ unsigned piece_off(int row, int piece) {
  if (BITS == 8) return row * 64 + ((piece ^ ((row >> 1) & 3)) << 4);
  if (BITS == 4) return row * 32 + ((piece ^ ((row >> 2) & 1)) << 4);
  return row * 16;
}

// The codes of columns 16 b + 4 t .. + 3 as two bf16 pairs, exact.  A code is placed in the low mantissa bits of bf16 128 and the
// offset taken off again; the pair-interleaved container puts the two codes of a pair 16 bits apart, so one logic operation
// extracts both.
template <int BITS>
__device__ __forceinline__ void widen4(unsigned w, int b, int t, unsigned& o0, unsigned& o1) {
  if (BITS == 4) {
    const unsigned v = w >> (8 * (t & 1));
    o0 = bsub2((v & 0x000f000fu) ^ 0x43084308u, 0x43084308u);              // 128 + (c + 8) - 136
    o1 = bsub2(((v >> 4) & 0x000f000fu) ^ 0x43084308u, 0x43084308u);
  } else if (BITS == 8) {
    // c = low seven bits - 128 * sign: bf16(128 + low7) - bf16(sign ? 256 : 128); the two constants differ in bit 7 alone
    const unsigned p0 = __byte_perm(w, 0x43434343u, 0x4140), p1 = __byte_perm(w, 0x43434343u, 0x4342);
    o0 = bsub2(p0 & 0xff7fff7fu, p0 & 0xff80ff80u);
    o1 = bsub2(p1 & 0xff7fff7fu, p1 & 0xff80ff80u);
  } else if (BITS == 2) {
    const unsigned v = w >> (4 * t);
    o0 = bsub2((v & 0x00030003u) ^ 0x43024302u, 0x43024302u);              // 128 + (c + 2) - 130
    o1 = bfma2((v & 0x000c000cu) ^ 0x43084308u, 0x3e803e80u, 0xc208c208u); // (128 + 4 (c + 2)) / 4 - 34
  } else {
    const int f = 8 * (b & 1) + 2 * t;
    o0 = ((w << (15 - f)) & 0x80008000u) ^ 0xbf80bf80u;                    // bit 1 -> +1, bit 0 -> -1
    o1 = ((w << (14 - f)) & 0x80008000u) ^ 0xbf80bf80u;
  }
}

template <int BITS, int NT, int R, bool GATED>
__global__ void __launch_bounds__(kMaxWarps * 32, NT == 1 && R == 1 ? 2 : 1) linear_gv_kernel(const __grid_constant__ Params p) {
  constexpr int MATS = GATED ? 2 : 1;
  using C = Codes<BITS>;
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, threads = blockDim.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x % p.ranks, group = blockIdx.x / p.ranks;
  const int tile0 = group * p.tg;
  const int crows = p.tg * 16;
  float* consts = reinterpret_cast<float*>(smem);                    // scale and bias words of the CTA's rows: [2][MATS][crows]
  uint8_t* ring = smem + 2 * MATS * crows * 4;                       // [warps][kRing][R][C::kStep]
  uint8_t* xs = ring + (threads >> 5) * (kRing * R * C::kStep);
  if (p.ranks > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");   // "has started": awaited before the first remote store

  // ---- this warp's item: tiles rw R .. + R - 1, matrix, split and chain
  const int rows_w = p.tg / R;                 // warps side by side on the tiles
  const int rw = warp % rows_w, rest = warp / rows_w;
  const int mat = GATED ? rest & 1 : 0, chain = (GATED ? rest >> 1 : rest) & 1, ls = (GATED ? rest >> 2 : rest >> 1);
  const int split = rank * p.splits_rank + ls;
  const int kb0 = split * p.kb_split;
  const int kb_n = split < p.splits ? (min(p.kb_split, p.kb_total - kb0) - chain + 1) / 2 : 0;     // the chain's blocks: kb0 + chain + 2 i
  const int steps = (kb_n + C::kBlocks - 1) / C::kBlocks;

  // ---- codes: this lane's pieces of a step
  const uint8_t* src[R];
  int src8[R];                                 // 8-bit codes: distance to the row 8 below
#pragma unroll
  for (int r = 0; r < R; ++r) {
    int tile = tile0 + rw * R + r, sub = mat;
    if (!GATED && tile >= p.tiles) { sub = 1; tile -= p.tiles; }
    if (tile >= p.tiles) { sub = 0; tile = p.tiles - 1; }            // beyond the launch's tiles: read, never stored
    const int lrow = BITS == 8 ? lane >> 2 : lane >> 1;
    const int row = min(tile * 16 + lrow, p.N - 1);
    src[r] = p.sub[sub].w + (int64_t)row * p.row_bytes;
    src8[r] = row + 8 < p.N ? 8 * p.row_bytes : 0;                   // beyond the matrix: the first row twice
  }
  const unsigned my_ring = smem_addr(ring) + warp * (kRing * R * C::kStep);
  int is_st = 0, is_slot = 0;
  auto issue = [&]() {
    if (is_st < steps) {
      const int kb = kb0 + chain + 2 * C::kBlocks * is_st;           // first block of the step
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned dst = my_ring + (is_slot * R + r) * C::kStep;
        if constexpr (BITS == 8) {
          const int byte = kb * 64 + (lane & 3) * 16;                // rows are padded to whole blocks
          cp_async16(dst + piece_off<8>(lane >> 2, lane & 3), src[r] + byte, 16);
          cp_async16(dst + piece_off<8>((lane >> 2) + 8, lane & 3), src[r] + src8[r] + byte, 16);
        } else if constexpr (BITS == 4) {
          cp_async16(dst + piece_off<4>(lane >> 1, lane & 1), src[r] + kb * 32 + (lane & 1) * 16, 16);
        } else if constexpr (BITS == 2) {
          const int sub = lane & 1;                                  // block of the step
          const bool in = C::kBlocks * is_st + sub < kb_n;
          cp_async16(dst + sub * 256 + (lane >> 1) * 16, src[r] + (in ? (kb + 2 * sub) * 16 : 0), in ? 16 : 0);
        } else {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int sub = (lane & 1) * 2 + q;
            const bool in = C::kBlocks * is_st + sub < kb_n;
            cp_async8(dst + sub * 128 + (lane >> 1) * 8, src[r] + (in ? (kb + 2 * sub) * 8 : 0), in ? 8 : 0);
          }
        }
      }
      ++is_st;
      is_slot = is_slot + 1 == kRing ? 0 : is_slot + 1;
    }
    cp_commit();
  };
  // Scales and biases of the CTA's rows (constants): asynchronous copies that join the first step's group.  A bias is copied as
  // the aligned word that holds it (copies are 4 bytes at least) where all of that word belongs to the bias; the epilogue picks the half.
  for (int i = tid; i < MATS * crows; i += threads) {
    const int lr = GATED && i >= crows ? i - crows : i;
    int tile = tile0 + lr / 16, sub = GATED && i >= crows ? 1 : 0;
    if (!GATED && tile >= p.tiles) { sub = 1; tile -= p.tiles; }
    const int n = min(tile * 16 + lr % 16, p.N - 1);
    cp_async4(smem_addr(consts + i), p.sub[sub].scale + n);
    if (const __nv_bfloat16* bias = p.sub[sub].bias) {
      const uintptr_t at = reinterpret_cast<uintptr_t>(bias + n), word = at & ~(uintptr_t)3;
      if (word >= reinterpret_cast<uintptr_t>(bias) && word + 4 <= reinterpret_cast<uintptr_t>(bias + p.N)) cp_async4(smem_addr(consts + crows * MATS + i), reinterpret_cast<const void*>(word));
      else reinterpret_cast<unsigned*>(consts)[crows * MATS + i] = (unsigned)__bfloat16_as_ushort(bias[n]) << ((at & 2) ? 16 : 0);
    }
  }
#pragma unroll
  for (int u = 0; u < kRing; ++u) issue();
  if (tid < kMaxSpans && p.ahead[tid].bytes) {                       // behind this launch's own codes
    const unsigned each = ((p.ahead[tid].bytes + gridDim.x - 1) / gridDim.x + 127) & ~127u;
    const unsigned at = each * blockIdx.x;
    if (at < p.ahead[tid].bytes) prefetch_l2(p.ahead[tid].p + at, min(each, p.ahead[tid].bytes - at) & ~15u);
  }

  // ---- activations of the CTA's splits in B-fragment order: slot (block pair u, token m, lane t) of 16 bytes = columns
  // 4 t .. + 3 of 16-column block 2 u, then of block 2 u + 1.  A thread keeps its 8 columns and walks the tokens.
  const int kbx0 = rank * p.splits_rank * p.kb_split;
  const int xk8 = min(p.splits_rank * p.kb_split, p.kb_total - kbx0) * 8;    // 8-column pieces of one token
  const int x_bytes = p.splits_rank * p.kb_split * p.M * 128;
  pdl_wait();
  // Only now: dependents that start earlier, and their dependents, would take the places of this grid's own CTAs on some SMs and
  // leave those SMs with two of them (a chain of 4096 x 4096 layers, one token: 6.1 us per call against 6.7)
  pdl_launch_dependents();
#pragma unroll
  for (int xm = 0; xm < MATS; ++xm) {
    if (GATED && xm == 1 && p.x_shared) break;
    const int tk = 1 << p.xk_log2;             // threads side by side on the columns of a token
    const int m_first = tid >> p.xk_log2, m_step = threads >> p.xk_log2;
    for (int k8 = tid & (tk - 1); k8 < xk8 && m_first < m_step; k8 += tk) {
      const int u = k8 >> 2, half = k8 & 1, blk = (k8 >> 1) & 1;
      const int k = kbx0 * 64 + k8 * 8;
      const __nv_bfloat16* xsrc = p.sub[xm].x + (int64_t)m_first * p.K + k;
      const unsigned base = smem_addr(xs) + xm * x_bytes + (u * p.M + m_first) * 64 + blk * 8;
      const unsigned d0 = base + ((2 * half) ^ (u & 3)) * 16, d1 = base + ((2 * half + 1) ^ (u & 3)) * 16;
      const bool in = k < p.K;                 // beyond K: zeros (the codes there are padding)
      constexpr int kBatch = NT == 1 ? 4 : 8;  // loads in flight per thread
      for (int m = m_first, q0 = 0; m < p.M; m += kBatch * m_step, q0 += kBatch) {
        uint4 v[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          v[q] = make_uint4(0, 0, 0, 0);
          if (in && m + q * m_step < p.M) v[q] = *reinterpret_cast<const uint4*>(xsrc + (int64_t)((q0 + q) * m_step) * p.K);
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
          if (m + q * m_step < p.M) {
            const unsigned o = (q0 + q) * m_step * 64;
            sts_v2(d0 + o, v[q].x, v[q].y);
            sts_v2(d1 + o, v[q].z, v[q].w);
          }
      }
    }
  }
  __syncthreads();

  float acc[R][NT][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[r][n][i] = 0.f;
  const unsigned xs_a = smem_addr(xs) + (GATED && !p.x_shared ? mat * x_bytes : 0);
  unsigned tok_off[NT];                        // tokens beyond M repeat the last one: their columns are never stored
#pragma unroll
  for (int n = 0; n < NT; ++n) tok_off[n] = (unsigned)min(n * 8 + g, p.M - 1) * 64;
  const WordAddr<BITS> words(g, t);
  int slot = 0;
#pragma unroll 1
  for (int st = 0; st < steps; ++st) {
    cp_wait<kRing - 1>();
    __syncwarp();                              // the step's codes were copied by all lanes
#pragma unroll
    for (int kk = 0; kk < C::kBlocks; ++kk) {
      const int i = C::kBlocks * st + kk;      // block of the chain
      if (C::kBlocks > 1 && i >= kb_n) break;
      const int u0 = (kb0 - kbx0 + chain + 2 * i) * 2;               // block pair of the CTA's activations
#pragma unroll
      for (int bp = 0; bp < 2; ++bp) {
        uint4 xf[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) xf[n] = lds_v4(xs_a + (unsigned)((u0 + bp) * p.M * 64) + tok_off[n] + ((t ^ ((u0 + bp) & 3)) << 4));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int b = bp * 2 + h;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const unsigned base = my_ring + (slot * R + r) * C::kStep + kk * 16 * C::kRow;
            unsigned a0, a1, a2, a3;
            widen4<BITS>(lds_u32(base + words.at(b)), b, t, a0, a2);
            widen4<BITS>(lds_u32(base + words.at(b) + 8 * C::kRow), b, t, a1, a3);
#pragma unroll
            for (int n = 0; n < NT; ++n) mma16816(acc[r][n], a0, a1, a2, a3, h ? xf[n].z : xf[n].x, h ? xf[n].w : xf[n].y);
          }
        }
      }
    }
    __syncwarp();                              // every lane has read the slot: the step kRing ahead takes it
    issue();
    slot = slot + 1 == kRing ? 0 : slot + 1;
  }

  // ---- partial tiles at the owning CTA (tile % ranks): [tile][mat][split][chain][token tile][8 tokens][kRedStride]
  constexpr int kTileF = NT * 8 * kRedStride;  // floats of one (tile, matrix, chain)
  const int entries = p.splits * 2;
  float* red = reinterpret_cast<float*>(xs + (GATED && !p.x_shared ? 2 : 1) * x_bytes);
  cp_wait<0>();                                // (a warp without blocks may have copied constants)
  if (p.ranks == 1) {
    __syncthreads();                           // ring and activations become the exchange area
    red = reinterpret_cast<float*>(ring);
  } else {
    asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
  }
  if (split < p.splits) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int lt = rw * R + r;
      const unsigned at = smem_addr(red) + ((((lt / p.ranks) * MATS + mat) * entries + split * 2 + chain) * kTileF) * 4;
      unsigned dst = at;
      if (p.ranks > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(dst) : "r"(at), "r"(lt % p.ranks));
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned d = dst + ((n * 8 + 2 * t + (i & 1)) * kRedStride + g + (i >> 1) * 8) * 4;
          if (p.ranks > 1) asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(d), "f"(acc[r][n][i]) : "memory");
          else asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(d), "f"(acc[r][n][i]) : "memory");
        }
    }
  }
  if (p.ranks == 1) __syncthreads();
  else asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");

  // ---- outputs by column (own tile, token): four threads to a column, four rows to a thread
  const int row = (tid & 3) * 4;
  const int own = (p.tg - rank + p.ranks - 1) / p.ranks;             // tiles rank, rank + ranks, ...
  const int cols = own << p.mp_log2;           // tokens padded to a power of two
  for (int col = tid >> 2; col < cols; col += threads >> 2) {
    const int ot = col >> p.mp_log2, m = col & ((1 << p.mp_log2) - 1);
    const int lt = ot * p.ranks + rank;
    int gt = tile0 + lt, sub = 0;
    if (!GATED && gt >= p.tiles) { sub = 1; gt -= p.tiles; }
    const int n = gt * 16 + row;
    if (m >= p.M || tile0 + lt >= p.tiles_total || n >= p.N) continue;
    float v[MATS][4];
#pragma unroll
    for (int mm = 0; mm < MATS; ++mm) {
      const float* e = red + (size_t)((ot * MATS + mm) * entries) * kTileF + m * kRedStride + row;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int q = 0; q < p.splits; ++q) {
        const float4 c0 = *reinterpret_cast<const float4*>(e + (2 * q) * kTileF), c1 = *reinterpret_cast<const float4*>(e + (2 * q + 1) * kTileF);
        a.x += c0.x + c1.x; a.y += c0.y + c1.y; a.z += c0.z + c1.z; a.w += c0.w + c1.w;
      }
      v[mm][0] = a.x; v[mm][1] = a.y; v[mm][2] = a.z; v[mm][3] = a.w;
      const __nv_bfloat16* bias = p.sub[GATED ? mm : sub].bias;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int ci = mm * crows + lt * 16 + row + i;
        float b = 0.f;
        if (bias) {
          const unsigned w = __float_as_uint(consts[crows * MATS + ci]);
          b = __uint_as_float((reinterpret_cast<uintptr_t>(bias + n + i) & 2) ? w & 0xffff0000u : w << 16);
        }
        v[mm][i] = v[mm][i] * consts[ci] + b;
      }
    }
    __align__(8) __nv_bfloat16 o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[i] = __float2bfloat16_rn(v[0][i]);
      if (GATED) {
        // the rounding points of separate gate / up / SiLU * up kernels (blocks/mlp.py:181-183)
        const float gq = __bfloat162float(o[i]);
        const float a = __bfloat162float(__float2bfloat16_rn(__fdividef(gq, 1.0f + __expf(-gq))));
        o[i] = __float2bfloat16_rn(__fmul_rn(a, __bfloat162float(__float2bfloat16_rn(v[MATS - 1][i]))));
      }
    }
    __nv_bfloat16* y = p.sub[sub].y + (int64_t)m * p.N + n;
    if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(y) & 7) == 0) {
      *reinterpret_cast<uint2*>(y) = *reinterpret_cast<const uint2*>(o);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < p.N) y[i] = o[i];
    }
  }
}

// Shared memory of one CTA: constants, code ring and activations; the partial tiles follow them (clusters) or replace them.
inline size_t smem_bytes(int bits, int R, int nt, bool gated, int tg, int M, int kb_split, int splits, int ranks, int splits_rank, bool x_shared) {
  const int mats = gated ? 2 : 1, warps = tg / R * 2 * mats * splits_rank;
  const size_t step = bits == 8 ? 1024 : 512;
  const size_t consts = (size_t)2 * mats * tg * 16 * 4;
  const size_t ring = (size_t)warps * kRing * R * step;
  const size_t xb = (size_t)splits_rank * kb_split * M * 128 * (gated && !x_shared ? 2 : 1);
  const size_t red = (size_t)((tg + ranks - 1) / ranks) * mats * splits * 2 * nt * 8 * kRedStride * 4;
  return consts + (ranks > 1 ? ring + xb + red : (ring + xb > red ? ring + xb : red));
}

struct Plan {
  int R, tg, ranks, grid, warps;
  size_t smem;
};
template <int BITS> cudaError_t launch(const Params& p, const Plan& plan, bool gated, bool pdl, cudaStream_t s);   // linear_gv_<bits>.cu

}  // namespace gv
}  // namespace tsb
