// Fused (RoPE on K +) quantize-and-append into the paged KV pools, and the FP8 scale
// reduction over a prompt.  One warp owns one (token, kv head) vector of d elements:
// lane l holds elements [l*d/32, (l+1)*d/32).  HBM-bound: reads 2*d*sizeof(act) bytes
// and writes 2*d*b_elem (+ scales) per vector.  Decode steps (one token per sequence) and small
// chunks use kv_append_kernel; larger prompt chunks use kv_append_pages_kernel, in which
// a CTA owns a whole page and writes the token-minor V record with 16-byte vectors.
//
// Quantization arithmetic (IEEE fp32, round-to-nearest-even) per format:
//   int8  : s = amax/127, code = clamp(rint(x/(s+1e-6)), +-127)   (the reference's weight
//           rule, compression/quantization_methods/vanilla.py:16-24, applied per vector)
//   fp8   : code = e4m3_satfinite(x / S[b, h])
//   nvfp4 : per 16 elements sb = e4m3_satfinite(amax/6), code = e2m1_satfinite(x/decode(sb))
#include <type_traits>
#include "common.cuh"

namespace tsb {

__device__ __forceinline__ float e4m3_to_f32(unsigned char c) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)c, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

template <int N> struct BytesN;
template <> struct BytesN<1> { using type = uint8_t; };
template <> struct BytesN<2> { using type = uint16_t; };
template <> struct BytesN<4> { using type = uint32_t; };

// This lane's EPL elements of a vector, as fp32 (one 8- or 16-byte load when the vector is aligned for it).
template <typename T, int D>
__device__ __forceinline__ void load_raw(const T* __restrict__ src, int lane, float (&x)[D / 32]) {
  constexpr int EPL = D / 32;
  const T* p = src + lane * EPL;
  if (sizeof(T) * EPL == 8 && (reinterpret_cast<uintptr_t>(p) & 7) == 0) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
    for (int i = 0; i < EPL; ++i) x[i] = to_f32<T>(e[i]);
  } else if (sizeof(T) * EPL == 16 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
    for (int i = 0; i < EPL; ++i) x[i] = to_f32<T>(e[i]);
  } else {
#pragma unroll
    for (int i = 0; i < EPL; ++i) x[i] = to_f32<T>(p[i]);
  }
}
// Rotate (optional) and round to T; returns this lane's EPL elements as fp32.
template <typename T, int D>
__device__ __forceinline__ void rope_vec(int lane, float (&x)[D / 32], bool rope, const float* __restrict__ cosr,
                                         const float* __restrict__ sinr) {
  constexpr int EPL = D / 32;
  if (rope) {
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, x[i], 16);
      const int e = (lane & 15) * EPL + i;             // index inside the half
      const float c = rnd<T>(cosr[e]), s = rnd<T>(sinr[e]);
      const float a = rnd<T>(__fmul_rn(x[i], c));       // own * cos
      const float b = rnd<T>(__fmul_rn(other, s));      // partner * sin
      x[i] = rnd<T>(lane < 16 ? __fsub_rn(a, b) : __fadd_rn(b, a));
    }
  }
}
template <typename T, int D>
__device__ __forceinline__ void load_vec(const T* __restrict__ src, int lane, float (&x)[D / 32], bool rope,
                                         const float* __restrict__ cosr, const float* __restrict__ sinr) {
  load_raw<T, D>(src, lane, x);
  rope_vec<T, D>(lane, x, rope, cosr, sinr);
}

// Unquantized pages (TSB200_KV_F32 / TSB200_KV_BF16): K and V records are both [16 tok][d] of T.
template <typename T, int D>
__device__ __forceinline__ void dense_store(const float (&x)[D / 32], int lane, uint8_t* __restrict__ rec, int slot) {
  constexpr int EPL = D / 32;
  T* dst = reinterpret_cast<T*>(rec) + slot * D + lane * EPL;
#pragma unroll
  for (int i = 0; i < EPL; ++i) dst[i] = from_f32<T>(x[i]);
}

template <int D, int FMT, bool IS_V>
__device__ __forceinline__ void quant_store(const float (&x)[D / 32], int lane, uint8_t* __restrict__ rec, int slot,
                                            float fp8_scale) {
  constexpr int EPL = D / 32;
  if (FMT == TSB200_KV_INT8 || FMT == TSB200_KV_FP8) {
    uint8_t code[EPL];
    if (FMT == TSB200_KV_INT8) {
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) m = fmaxf(m, fabsf(x[i]));
      m = warp_max(m);
      const float s = __fdiv_rn(m, 127.0f);
      const float den = __fadd_rn(s, 1e-6f);
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        float q = fminf(fmaxf(rintf(__fdiv_rn(x[i], den)), -127.f), 127.f);
        code[i] = (uint8_t)(int8_t)(int)q;
      }
      if (lane == 0) reinterpret_cast<float*>(rec + 16 * D)[slot] = s;
    } else {
#pragma unroll
      for (int i = 0; i < EPL; ++i)
        code[i] = (uint8_t)__nv_cvt_float_to_fp8(__fdiv_rn(x[i], fp8_scale), __NV_SATFINITE, __NV_E4M3);
    }
    if (!IS_V) {
      typename BytesN<EPL>::type packed = 0;
#pragma unroll
      for (int i = 0; i < EPL; ++i) packed |= (typename BytesN<EPL>::type)code[i] << (8 * i);
      *reinterpret_cast<typename BytesN<EPL>::type*>(rec + slot * D + lane * EPL) = packed;
    } else {
#pragma unroll
      for (int i = 0; i < EPL; ++i) rec[(lane * EPL + i) * 16 + slot] = code[i];
    }
  } else {  // NVFP4
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) m = fmaxf(m, fabsf(x[i]));
#pragma unroll
    for (int o = 1; o < 16 / EPL; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const uint8_t sb = (uint8_t)__nv_cvt_float_to_fp8(__fdiv_rn(m, 6.0f), __NV_SATFINITE, __NV_E4M3);
    const float sd = e4m3_to_f32(sb);
    uint8_t byte[EPL / 2];
#pragma unroll
    for (int i = 0; i < EPL / 2; ++i) {
      if (sd > 0.f) {
        float2 f = make_float2(__fdiv_rn(x[2 * i], sd), __fdiv_rn(x[2 * i + 1], sd));
        byte[i] = (uint8_t)__nv_cvt_float2_to_fp4x2(f, __NV_E2M1, cudaRoundNearest);
      } else {
        byte[i] = 0;
      }
    }
    const int blk = (lane * EPL) / 16;
    const bool blk_leader = ((lane * EPL) % 16) == 0;
    if (!IS_V) {
      typename BytesN<EPL / 2>::type packed = 0;
#pragma unroll
      for (int i = 0; i < EPL / 2; ++i) packed |= (typename BytesN<EPL / 2>::type)byte[i] << (8 * i);
      *reinterpret_cast<typename BytesN<EPL / 2>::type*>(rec + slot * (D / 2) + lane * (EPL / 2)) = packed;
      if (blk_leader) rec[16 * (D / 2) + slot * (D / 16) + blk] = sb;
    } else {
#pragma unroll
      for (int i = 0; i < EPL / 2; ++i) rec[(lane * (EPL / 2) + i) * 16 + slot] = byte[i];
      if (blk_leader) rec[16 * (D / 2) + blk * 16 + slot] = sb;
    }
  }
}

template <typename T, int D, int FMT>
__global__ void kv_append_kernel(tsb200_kv_desc kv, T* __restrict__ q, int64_t qs, int qheads,
                                 const T* __restrict__ k, const T* __restrict__ v, int64_t ks,
                                 int64_t vs_, int64_t B,
                                 int64_t Tn, const int32_t* __restrict__ new_lens, const float* __restrict__ rope_cos,
                                 const float* __restrict__ rope_sin, int64_t rope_rows, int64_t rec_bytes) {
  // Programmatic dependent launch: the write position, the page and the scales (inputs that the launch directly before
  // this one does not produce) are looked up while that launch drains; the wait stands in front of the first access to
  // q, k and v and of every store.
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t total = B * Tn * kv.hkv;
  if (warp >= total) {
    // extra warps: rotate the query heads in place (same rounding points as the key path)
    const int64_t qw = warp - total;
    if (q == nullptr || qw >= B * Tn * qheads || rope_cos == nullptr) return;
    const int qh = (int)(qw % qheads);
    const int64_t qbt = qw / qheads;
    const int64_t qb = qbt / Tn, qj = qbt - qb * Tn;
    if (new_lens && qj >= new_lens[qb]) return;
    int64_t qp = (int64_t)kv.seq_lens[qb] + qj;
    qp = qp < 0 ? 0 : (qp >= rope_rows ? rope_rows - 1 : qp);
    float xq[D / 32];
    T* dst = q + qbt * qs + (int64_t)qh * D;
    pdl_wait();
    load_vec<T, D>(dst, lane, xq, true, rope_cos + qp * (D / 2), rope_sin + qp * (D / 2));
#pragma unroll
    for (int i = 0; i < D / 32; ++i) dst[lane * (D / 32) + i] = from_f32<T>(xq[i]);
    return;
  }
  const int h = (int)(warp % kv.hkv);
  const int64_t bt = warp / kv.hkv;
  const int64_t b = bt / Tn, j = bt - b * Tn;
  if (new_lens && j >= new_lens[b]) return;
  const int64_t p = (int64_t)kv.seq_lens[b] + j;
  if (p < 0 || (p >> 4) >= kv.bt_stride) return;
  const int64_t page = kv.block_table[b * kv.bt_stride + (p >> 4)];
  if (page < 0 || page >= kv.num_pages) return;
  const int slot = (int)(p & 15);
  const int64_t rec = (page * kv.hkv + h) * rec_bytes;
  const bool rope = rope_cos != nullptr;
  const int64_t rp = p >= rope_rows ? rope_rows - 1 : p;
  float x[D / 32];
  float kscale = 1.f, vscale = 1.f;
  if (FMT == TSB200_KV_FP8) {
    kscale = kv.k_scale[b * kv.hkv + h];
    vscale = kv.v_scale[b * kv.hkv + h];
  }
  pdl_wait();
  load_vec<T, D>(k + bt * ks + (int64_t)h * D, lane, x, rope, rope ? rope_cos + rp * (D / 2) : nullptr, rope ? rope_sin + rp * (D / 2) : nullptr);
  if (FMT >= TSB200_KV_F32) dense_store<T, D>(x, lane, kv.k_pool + rec, slot);
  else quant_store<D, FMT, false>(x, lane, kv.k_pool + rec, slot, kscale);
  load_vec<T, D>(v + bt * vs_ + (int64_t)h * D, lane, x, false, nullptr, nullptr);
  if (FMT >= TSB200_KV_F32) dense_store<T, D>(x, lane, kv.v_pool + rec, slot);
  else quant_store<D, FMT, true>(x, lane, kv.v_pool + rec, slot, vscale);
}

// ---- prompt chunks -------------------------------------------------------------------------------------------------------
// Eight consecutive elements of a vector in the act dtype (bf16: as four packed pairs).
template <typename T> struct Raw8;
template <> struct Raw8<__nv_bfloat16> {
  unsigned u[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool vec) {
    if (vec) {
      const uint4 a = *reinterpret_cast<const uint4*>(p);
      u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = (unsigned)__bfloat16_as_ushort(p[2 * i]) | ((unsigned)__bfloat16_as_ushort(p[2 * i + 1]) << 16);
    }
  }
  __device__ __forceinline__ void load_shared(const __nv_bfloat16* p) { load(p, true); }
  __device__ __forceinline__ void store(__nv_bfloat16* p, bool vec) const {
    if (vec) {
      *reinterpret_cast<uint4*>(p) = make_uint4(u[0], u[1], u[2], u[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        p[2 * i] = __ushort_as_bfloat16((unsigned short)(u[i] & 0xffffu));
        p[2 * i + 1] = __ushort_as_bfloat16((unsigned short)(u[i] >> 16));
      }
    }
  }
  __device__ __forceinline__ void unpack(float (&v)[8]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
  }
  // into [-c, c], both halves of c2 holding c (NaN stays)
  __device__ __forceinline__ void clamp(unsigned c2) {
    const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&c2), lo = __hneg2(hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 r = __hmin2_nan(__hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&u[i]), lo), hi);
      u[i] = *reinterpret_cast<const unsigned*>(&r);
    }
  }
  // largest magnitude, as the bits of a positive bf16
  __device__ __forceinline__ float amax(float m) const {
    float v[8];
    unpack(v);
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
  }
};
template <> struct Raw8<float> {
  float f[8];
  __device__ __forceinline__ void load(const float* p, bool vec) {
    if (vec) {
      const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = p[i];
    }
  }
  __device__ __forceinline__ void load_shared(const float* p) { load(p, true); }
  __device__ __forceinline__ void store(float* p, bool vec) const {
    if (vec) {
      *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) p[i] = f[i];
    }
  }
  __device__ __forceinline__ void unpack(float (&v)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = f[i];
  }
  __device__ __forceinline__ float amax(float m) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(f[i]));
    return m;
  }
};
// fp32 elements rounded to the act dtype
__device__ __forceinline__ void round8(const Raw8<float>& f, Raw8<__nv_bfloat16>& r) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(f.f[2 * i], f.f[2 * i + 1]);
    r.u[i] = *reinterpret_cast<const unsigned*>(&b);
  }
}
__device__ __forceinline__ void round8(const Raw8<float>& f, Raw8<float>& r) { r = f; }
// Half-split rotation of elements (a[i], b[i]), i and i + d/2 of one vector: every product and sum rounded to the act dtype
// (blocks/rope.py:140-173).  bf16: packed arithmetic - one rounding per operation; the fp32 detour rounds the sum twice, which is
// the same, since two bf16 numbers whose sum has more than 24 bits are too far apart for it to lie near a midpoint.
__device__ __forceinline__ void rope8(Raw8<__nv_bfloat16>& a, Raw8<__nv_bfloat16>& b, const Raw8<__nv_bfloat16>& c, const Raw8<__nv_bfloat16>& s) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 x = *reinterpret_cast<__nv_bfloat162*>(&a.u[i]), y = *reinterpret_cast<__nv_bfloat162*>(&b.u[i]);
    const __nv_bfloat162 cc = *reinterpret_cast<const __nv_bfloat162*>(&c.u[i]), ss = *reinterpret_cast<const __nv_bfloat162*>(&s.u[i]);
    const __nv_bfloat162 r = __hsub2_rn(__hmul2_rn(x, cc), __hmul2_rn(y, ss)), q = __hadd2_rn(__hmul2_rn(x, ss), __hmul2_rn(y, cc));
    a.u[i] = *reinterpret_cast<const unsigned*>(&r);
    b.u[i] = *reinterpret_cast<const unsigned*>(&q);
  }
}
__device__ __forceinline__ void rope8(Raw8<float>& a, Raw8<float>& b, const Raw8<float>& c, const Raw8<float>& s) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = a.f[i], y = b.f[i];
    a.f[i] = __fsub_rn(__fmul_rn(x, c.f[i]), __fmul_rn(y, s.f[i]));
    b.f[i] = __fadd_rn(__fmul_rn(x, s.f[i]), __fmul_rn(y, c.f[i]));
  }
}

// Quotients by a divisor that many elements share, from its correctly rounded reciprocal, two at a time: q' = q + (x - d q) y is the
// rounded quotient when q is within an ulp of it (Markstein's theorem, Computation of elementary functions on the IBM RISC System/6000
// processor, 1990), which one correction of x y is.  Divisors near the ends of the exponent range divide.
//   * fp32 elements: corrected twice, correctly rounded.  An infinite product (of an infinite x, or a quotient beyond the type) stands as
//     it is where MAY_OVERFLOW: it saturates, and its corrections are NaN.
//   * bf16 elements: corrected once: what is rounded to fp32 is then within 2^-46 of the quotient, and only a quotient that close to
//     M + half an fp32 ulp, M the midpoint of two codes, could round to another code.  Codes have midpoints of up to eight significant
//     bits (M = 2 k + 1 for an int8 code k).  With M an odd number of B bits, the divisor as a 24-bit number D and x as X 2^t, X of eight
//     bits, such an x is M D + c + (less than 2^-18) for c = D 2^(B-25), a whole number below M; so D = c 2^(25-B) + e, |e| <= 8, and
//     X 2^t = M c 2^(25-B) + M e + c: the first term alone has up to 2 B - 1 bits above 2^(25-B) and X has eight in all, so M e = -c,
//     which no c between 0 and M is (D = 2^24 - 1, c = M = 1 is one: a divisor of all ones divides).  Quotients that overflow are kept
//     out by clamping x ahead (FP8: scales from elsewhere).
struct Divisor {
  float d, y;
  bool slow;
  template <bool TWICE, bool MAY_OVERFLOW> __device__ __forceinline__ void of(float x0, float x1, float& q0, float& q1) const {
    if (!TWICE) {
      asm("{\n.reg .b64 x, y, n, p, e;\n"
          "mov.b64 x, {%2, %3};\nmov.b64 y, {%4, %4};\nmov.b64 n, {%5, %5};\n"
          "mul.rn.f32x2 p, x, y;\n"
          "fma.rn.f32x2 e, p, n, x;\nfma.rn.f32x2 p, e, y, p;\n"
          "mov.b64 {%0, %1}, p;\n}\n"
          : "=f"(q0), "=f"(q1)
          : "f"(x0), "f"(x1), "f"(y), "f"(-d));
      return;
    }
    float p0, p1;
    asm("{\n.reg .b64 x, y, n, p, q, e;\n"
        "mov.b64 x, {%4, %5};\nmov.b64 y, {%6, %6};\nmov.b64 n, {%7, %7};\n"
        "mul.rn.f32x2 p, x, y;\n"
        "fma.rn.f32x2 e, p, n, x;\nfma.rn.f32x2 q, e, y, p;\n"
        "fma.rn.f32x2 e, q, n, x;\nfma.rn.f32x2 q, e, y, q;\n"
        "mov.b64 {%0, %1}, q;\nmov.b64 {%2, %3}, p;\n}\n"
        : "=f"(q0), "=f"(q1), "=f"(p0), "=f"(p1)
        : "f"(x0), "f"(x1), "f"(y), "f"(-d));
    if (MAY_OVERFLOW) {
      q0 = fabsf(p0) <= 3.4028235e38f ? q0 : p0;
      q1 = fabsf(p1) <= 3.4028235e38f ? q1 : p1;
    }
  }
};
__device__ __forceinline__ Divisor divisor(float v) {
  return Divisor{v, __frcp_rn(v), !(v >= 1e-18f && v <= 1e18f) || (__float_as_uint(v) & 0x7fffffu) == 0x7fffffu};
}

// Codes of one token's eight elements (half a lane's share): two words (8-bit formats) or one (NVFP4).
template <typename T, int FMT, bool SLOW> __device__ __forceinline__ void encode8_by(const float (&x)[8], const Divisor& d, unsigned& w0, unsigned& w1) {
  float q[8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    // FP8: a scale from elsewhere; the other formats' divisors come from the elements' own maximum
    if (SLOW) { q[i] = __fdiv_rn(x[i], d.d); q[i + 1] = __fdiv_rn(x[i + 1], d.d); }
    else d.of<sizeof(T) == 4, FMT == TSB200_KV_FP8>(x[i], x[i + 1], q[i], q[i + 1]);
  }
  if (FMT == TSB200_KV_FP8) {
    unsigned h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __nv_cvt_float2_to_fp8x2(make_float2(q[2 * i], q[2 * i + 1]), __NV_SATFINITE, __NV_E4M3);
    w0 = __byte_perm(h[0], h[1], 0x5410);
    w1 = __byte_perm(h[2], h[3], 0x5410);
  } else if (FMT == TSB200_KV_INT8) {
    unsigned c[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = __float_as_uint(fminf(fmaxf(q[i], -127.f), 127.f) + 12582912.0f);   // 1.5 * 2^23: half-to-even, in the low bits
    w0 = __byte_perm(__byte_perm(c[0], c[1], 0x0040), __byte_perm(c[2], c[3], 0x0040), 0x5410);
    w1 = __byte_perm(__byte_perm(c[4], c[5], 0x0040), __byte_perm(c[6], c[7], 0x0040), 0x5410);
  } else {
    w0 = w1 = 0;
    if (d.d > 0.f) {
#pragma unroll
      for (int i = 0; i < 4; ++i) w0 |= (unsigned)__nv_cvt_float2_to_fp4x2(make_float2(q[2 * i], q[2 * i + 1]), __NV_E2M1, cudaRoundNearest) << (8 * i);
    }
  }
}
template <typename T, int FMT> __device__ __forceinline__ void encode8(const float (&x)[8], const Divisor& d, unsigned& w0, unsigned& w1) {
  if (d.slow) encode8_by<T, FMT, true>(x, d, w0, w1);
  else encode8_by<T, FMT, false>(x, d, w0, w1);
}
// 4 x 4 byte transpose: out[j] = byte j of in[0..3]
__device__ __forceinline__ void transpose4(const unsigned (&in)[4], unsigned (&out)[4]) {
  const unsigned a = __byte_perm(in[0], in[1], 0x5140), b = __byte_perm(in[2], in[3], 0x5140);
  const unsigned c = __byte_perm(in[0], in[1], 0x7362), d = __byte_perm(in[2], in[3], 0x7362);
  out[0] = __byte_perm(a, b, 0x5410); out[1] = __byte_perm(a, b, 0x7632);
  out[2] = __byte_perm(c, d, 0x5410); out[3] = __byte_perm(c, d, 0x7632);
}

// Bulk append (quantized formats; launch_append says from which size on): a CTA owns the pages of 2048 / d consecutive slots of one sequence
// (d 128: one page, d 64: two), its 8 warps take the heads.  A lane holds four tokens x (8 + 8) elements, e and e + d/2, so that
//   * the rotation needs no other lane; cos and sin of the CTA's positions are rounded to the act dtype once, in shared memory, and
//     serve every key and query head;
//   * quantization shares one reciprocal per scale (the quotients the rules prescribe are IEEE divisions, ~10 instructions each
//     otherwise);
//   * V, stored token-minor, is transposed four bytes at a time in registers and leaves through a swizzled tile of shared memory as
//     16-byte rows, 512 contiguous bytes per warp.
// Pages that the range covers in part keep their other slots: those go out token by token.  A task is K or V of one head: both at once
// take 128 registers a thread and leave 24 % of the warps.  Instructions and their latencies bound it: a further instruction an element
// costs 2 to 4 us.  32 x 2048 tokens, 8 heads, d 128, FP8, 402 MB, with the scales' launch (48 us): 141.6 us; 147.6 with loads that a task
// waits for, two corrections a quotient and selects for what saturates; 290 with one warp per token vector and a byte-wise transpose.
template <typename T, int D, int FMT, bool AHEAD> struct AppendSmem {
  uint4 stage[8][AHEAD ? 8 : 1][32];                                      // per warp: a task's elements, 16-byte pieces by lane (bf16)
  T cos[2048 / D][D / 2], sin[2048 / D][D / 2];
  unsigned v[4][128 / D][(FMT == TSB200_KV_NVFP4 ? D / 2 : D) * 4];       // V records of the warps that have V (the odd ones)
};
template <typename T, int D, int FMT, bool AHEAD>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 3 : 1)
kv_append_pages_kernel(tsb200_kv_desc kv, T* __restrict__ q, int64_t qs, int qheads, const T* __restrict__ k,
                       const T* __restrict__ v, int64_t ks, int64_t vs_, int64_t Tn, const int32_t* __restrict__ new_lens,
                       const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int64_t rope_rows,
                       int64_t rec_bytes) {
  constexpr bool FP4 = FMT == TSB200_KV_NVFP4;
  constexpr int HALF = D / 2, PAGES = 128 / D, TOK = 16 * PAGES;          // tokens of the CTA
  constexpr int EG = HALF / 8;                                            // lanes side by side on a vector
  constexpr int ROWS = FP4 ? D / 2 : D;                                   // 16-byte rows of a V record
  extern __shared__ __align__(16) uint8_t append_smem[];
  auto& smem = *reinterpret_cast<AppendSmem<T, D, FMT, AHEAD>*>(append_smem);
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int eg = lane % EG, tq = lane / EG;                               // elements 8 eg .., tokens 4 tq .. of the CTA's
  const int64_t b = blockIdx.y;
  pdl_wait();
  const int64_t n_b = new_lens ? min((int64_t)new_lens[b], Tn) : Tn;
  const int64_t start = kv.seq_lens[b];
  const int64_t lp0 = (start >> 4) + (int64_t)blockIdx.x * PAGES;         // first logical page of the CTA
  const int64_t p0 = lp0 * 16;
  if (p0 >= start + n_b) return;
  const int page_of_lane = tq >> 2;                                       // of the CTA's PAGES
  const int slot0 = (tq & 3) * 4;                                         // first of the lane's four slots in that page
  const int64_t lp = lp0 + page_of_lane;
  const bool full = lp * 16 >= start && lp * 16 + 16 <= start + n_b;      // every slot of the page is appended
  const int64_t j0 = lp * 16 + slot0 - start;                             // index of the lane's first token in the chunk
  bool tok[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) tok[i] = j0 + i >= 0 && j0 + i < n_b;
  const bool kvec = (reinterpret_cast<uintptr_t>(k) & 15) == 0 && ks * sizeof(T) % 16 == 0;
  const bool vvec = (reinterpret_cast<uintptr_t>(v) & 15) == 0 && vs_ * sizeof(T) % 16 == 0;
  const int lt = page_of_lane * 16 + slot0;                               // the lane's first token in the tables

  // tasks: K or V of a head (half the registers of both at once; a warp's are all K or all V), then query heads; dealt out over the grid's
  // CTAs of these pages.  AHEAD: a task's elements are on their way while the task before it is encoded, the first one's while tables and page
  // numbers are fetched: every lane copies what it will read itself.  Not so with one task to a warp, which nothing hides the detour of
  // (NVFP4, 4 x 2048 tokens, 4 heads of 128: 12.5 us, 10.2 without), nor for fp32: a lane's 32 bytes would come from the L2 as two halves of a sector
  // (FP8, 32 x 2048 tokens, 4 heads of 128: 185 us, 118 without).
  const int tasks = 2 * kv.hkv + (q && rope_cos ? qheads : 0), task_step = 8 * (int)gridDim.z;
  int task = w + 8 * (int)blockIdx.z;
  auto staged = [&](int i, int half) { return &smem.stage[w][i * 2 + half][lane]; };
  float fp8_scale = 1.f;
  auto fetch = [&](int t) {
    if (t >= 2 * kv.hkv) return;
    const int h = t >> 1;
    const bool is_v = t & 1, vec = is_v ? vvec : kvec;
    if (FMT == TSB200_KV_FP8) fp8_scale = (is_v ? kv.v_scale : kv.k_scale)[b * kv.hkv + h];
    const int64_t stride = is_v ? vs_ : ks;
    const T* p = (is_v ? v : k) + (b * Tn + j0) * stride + (int64_t)h * D + eg * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i, p += stride)
      if (tok[i]) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (vec) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(staged(i, half))),
                         "l"(reinterpret_cast<const uint4*>(p + half * HALF)) : "memory");
          } else {
            Raw8<T> r;
            r.load(p + half * HALF, false);
            r.store(reinterpret_cast<T*>(staged(i, half)), true);
          }
        }
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  if constexpr (AHEAD) fetch(task);
  int64_t page = lp >= 0 && lp < kv.bt_stride ? (int64_t)kv.block_table[b * kv.bt_stride + lp] : -1;
  const bool page_ok = page >= 0 && page < kv.num_pages;
  if (rope_cos) {
    const bool rvec = ((reinterpret_cast<uintptr_t>(rope_cos) | reinterpret_cast<uintptr_t>(rope_sin)) & 15) == 0;
#pragma unroll 1
    for (int i = threadIdx.x * 8; i < 2 * TOK * HALF; i += 256 * 8) {      // eight elements of cos, then of sin
      const int at = i < TOK * HALF ? i : i - TOK * HALF;
      int64_t p = p0 + at / HALF;
      p = p < 0 ? 0 : (p >= rope_rows ? rope_rows - 1 : p);
      Raw8<float> f;
      f.load((i < TOK * HALF ? rope_cos : rope_sin) + p * HALF + at % HALF, rvec);
      Raw8<T> r;
      round8(f, r);
      r.store(&(i < TOK * HALF ? smem.cos : smem.sin)[at / HALF][at % HALF], true);
    }
    __syncthreads();
  }
  for (; task < 2 * kv.hkv; task += task_step) {
    const int h = task >> 1;
    const bool is_v = task & 1;
    uint8_t* rec = (is_v ? kv.v_pool : kv.k_pool) + ((page_ok ? page : 0) * kv.hkv + h) * rec_bytes;
    Raw8<T> x[4][2];
    if constexpr (AHEAD) {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (tok[i]) {
          x[i][0].load_shared(reinterpret_cast<const T*>(staged(i, 0))); x[i][1].load_shared(reinterpret_cast<const T*>(staged(i, 1)));
        } else {
          x[i][0] = x[i][1] = Raw8<T>{};
        }
      }
    } else {
      const int64_t stride = is_v ? vs_ : ks;
      const T* p = (is_v ? v : k) + (b * Tn + j0) * stride + (int64_t)h * D + eg * 8;
      const bool vec = is_v ? vvec : kvec;
#pragma unroll
      for (int i = 0; i < 4; ++i, p += stride) {
        if (tok[i] && page_ok) {
          x[i][0].load(p, vec); x[i][1].load(p + HALF, vec);
        } else {
          x[i][0] = x[i][1] = Raw8<T>{};
        }
      }
      if (FMT == TSB200_KV_FP8) fp8_scale = (is_v ? kv.v_scale : kv.k_scale)[b * kv.hkv + h];
    }
    const Divisor shared = divisor(fp8_scale);
    if constexpr (AHEAD) {
      __syncwarp();                            // read: the next task's elements may come
      fetch(task + task_step);
    }
    // FP8, bf16: what lies beyond 512 scales saturates as that does (e4m3 ends at 448), without an infinite quotient on the way
    unsigned bound = 0x7f807f80u;
    if (FMT == TSB200_KV_FP8 && sizeof(T) == 2 && !shared.slow) {
      const __nv_bfloat162 c2 = __bfloat162bfloat162(__float2bfloat16_ru(shared.d * 512.0f));
      bound = *reinterpret_cast<const unsigned*>(&c2);
    }
    // one vector's codes: per token two words per half (8-bit formats) or one, and its scale(s)
    auto encode = [&](Raw8<T> (&a)[2], unsigned (&c)[4], float& s8, unsigned (&sb)[2]) {
      float f[2][8];
      if constexpr (FMT == TSB200_KV_FP8 && sizeof(T) == 2) { a[0].clamp(bound); a[1].clamp(bound); }
      a[0].unpack(f[0]);
      a[1].unpack(f[1]);
      if (FMT == TSB200_KV_FP8) {
        encode8<T, FMT>(f[0], shared, c[0], c[1]);
        encode8<T, FMT>(f[1], shared, c[2], c[3]);
      } else if (FMT == TSB200_KV_INT8) {
        float m = a[1].amax(a[0].amax(0.f));
#pragma unroll
        for (int o = 1; o < EG; o *= 2) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        s8 = m > 0.f ? __fdiv_rn(m, 127.0f) : 0.f;         // 0 (slots outside the chunk) takes the division's slow path
        const Divisor d = divisor(__fadd_rn(s8, 1e-6f));
        encode8<T, FMT>(f[0], d, c[0], c[1]);
        encode8<T, FMT>(f[1], d, c[2], c[3]);
      } else {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float m = a[g].amax(0.f);
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));              // a block of 16 is two lanes' eights
          // 0 (slots outside the chunk) takes the division's slow path
          sb[g] = m > 0.f ? (unsigned)__nv_cvt_float_to_fp8(__fdiv_rn(m, 6.0f), __NV_SATFINITE, __NV_E4M3) : 0u;
          Divisor d = divisor(e4m3_to_f32((unsigned char)sb[g]));
          d.slow = m > 3.4028235e38f;                                    // the scale is one of e4m3's, or 0 and not divided by
          encode8<T, FMT>(f[g], d, c[2 * g], c[2 * g + 1]);
        }
      }
    };
    if (!is_v) {                             // K, token-major
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (rope_cos) {
          Raw8<T> cc, ss;
          cc.load_shared(&smem.cos[lt + i][eg * 8]);
          ss.load_shared(&smem.sin[lt + i][eg * 8]);
          rope8(x[i][0], x[i][1], cc, ss);
        }
        unsigned c[4], sb[2];
        float s8 = 0.f;
        encode(x[i], c, s8, sb);
        if (tok[i] && page_ok) {
          const int slot = slot0 + i;
          if (FP4) {
            *reinterpret_cast<unsigned*>(rec + slot * (D / 2) + eg * 4) = c[0];
            *reinterpret_cast<unsigned*>(rec + slot * (D / 2) + HALF / 2 + eg * 4) = c[2];
            if ((eg & 1) == 0) {
              rec[16 * (D / 2) + slot * (D / 16) + (eg >> 1)] = (uint8_t)sb[0];
              rec[16 * (D / 2) + slot * (D / 16) + HALF / 16 + (eg >> 1)] = (uint8_t)sb[1];
            }
          } else {
            *reinterpret_cast<uint2*>(rec + slot * D + eg * 8) = make_uint2(c[0], c[1]);
            *reinterpret_cast<uint2*>(rec + slot * D + HALF + eg * 8) = make_uint2(c[2], c[3]);
            if (FMT == TSB200_KV_INT8 && eg == 0) reinterpret_cast<float*>(rec + 16 * D)[slot] = s8;
          }
        }
      }
      continue;
    }
    // ---- V, token-minor
    unsigned vc[4][4], vsb[4][2];
    float vs8[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) encode(x[i], vc[i], vs8[i], vsb[i]);
    constexpr int GROUPS = FP4 ? 2 : 4;                                   // groups of four rows per lane
    unsigned t[GROUPS][4];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      const int src = FP4 ? 2 * g : g;
      const unsigned in[4] = {vc[0][src], vc[1][src], vc[2][src], vc[3][src]};
      transpose4(in, t[g]);
    }
    // row of word (g, j): 8-bit: element g / 2 * HALF + 8 eg + 4 (g & 1) + j; NVFP4: pair g * HALF / 2 + 4 eg + j
    auto row_of = [&](int g, int j) { return FP4 ? g * (HALF / 2) + eg * 4 + j : (g >> 1) * HALF + eg * 8 + (g & 1) * 4 + j; };
    // rows that a store meets fall into different banks: the low three bits of a row are exchanged by the next three
    auto swz = [](int r) { return (r & ~7) | ((r ^ (r >> 3)) & 7); };
    if (__any_sync(0xffffffffu, full && page_ok)) {
      unsigned* sv = smem.v[w >> 1][page_of_lane];
      __syncwarp();
#pragma unroll
      for (int g = 0; g < GROUPS; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) sv[swz(row_of(g, j)) * 4 + (slot0 >> 2)] = t[g][j];
      __syncwarp();
#pragma unroll
      for (int pg = 0; pg < PAGES; ++pg) {
        // the whole warp writes page pg: its address and state come from a lane of that page
        const int from = pg * 4 * EG;
        const bool go = __shfl_sync(0xffffffffu, (int)(full && page_ok), from);
        const unsigned long long dst = __shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)rec, from);
        if (go) {
#pragma unroll
          for (int r = lane; r < ROWS; r += 32)
            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>((uintptr_t)dst) + r * 16) = *reinterpret_cast<const uint4*>(&smem.v[w >> 1][pg][swz(r) * 4]);
        }
      }
    }
    if (page_ok && !full) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (tok[i]) {
#pragma unroll
          for (int g = 0; g < GROUPS; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) rec[row_of(g, j) * 16 + slot0 + i] = (uint8_t)(t[g][j] >> (8 * i));
        }
    }
    if (page_ok) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (tok[i]) {
          if (FMT == TSB200_KV_INT8 && eg == 0) reinterpret_cast<float*>(rec + 16 * D)[slot0 + i] = vs8[i];
          if (FP4 && (eg & 1) == 0) {
            rec[16 * (D / 2) + (eg >> 1) * 16 + slot0 + i] = (uint8_t)vsb[i][0];
            rec[16 * (D / 2) + (HALF / 16 + (eg >> 1)) * 16 + slot0 + i] = (uint8_t)vsb[i][1];
          }
        }
    }
  }
  // ---- query heads of the same positions, in place
  const bool qvec = (reinterpret_cast<uintptr_t>(q) & 15) == 0 && qs * sizeof(T) % 16 == 0;
  for (; task < tasks; task += task_step) {
    const int h = task - 2 * kv.hkv;
    Raw8<T> x[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (tok[i]) {
        const T* qp = q + (b * Tn + j0 + i) * qs + (int64_t)h * D + eg * 8;
        x[i][0].load(qp, qvec); x[i][1].load(qp + HALF, qvec);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (tok[i]) {
        T* qp = q + (b * Tn + j0 + i) * qs + (int64_t)h * D + eg * 8;
        Raw8<T> cc, ss;
        cc.load_shared(&smem.cos[lt + i][eg * 8]);
        ss.load_shared(&smem.sin[lt + i][eg * 8]);
        rope8(x[i][0], x[i][1], cc, ss);
        x[i][0].store(qp, qvec); x[i][1].store(qp + HALF, qvec);
      }
  }
}

// FP8 scales of a prompt: amax over the T tokens of a (sequence, kv head) -> amax / 448 (1 if 0).  A cluster of eight CTAs (for few
// tokens a single one) shares the tokens of G heads, D / 16 lanes a vector ((8 + 8) elements each, so the rotation needs no other lane;
// its cos and sin, as many bytes as K and V, are fetched and rounded once for the G heads), the maxima meet in distributed shared memory.
// Bound by the one trip of K and V from memory: 32 x 2048 tokens, 8 heads, d 128: 268 MB, 41 us at the copy rate; 50 us with four heads,
// 71 with one; one CTA per (sequence, head), a warp per vector and five shuffles per rotation took 343 us.
constexpr int kScaleRanks = 8;
template <typename T, int D, int G, int RANKS>
__global__ void __launch_bounds__(256)
kv_fp8_scales_kernel(const T* __restrict__ k, const T* __restrict__ v, int64_t ks, int64_t vs, int64_t Tn, int hkv,
                     const int32_t* __restrict__ pos0, const float* __restrict__ rope_cos,
                     const float* __restrict__ rope_sin, int64_t rope_rows, float* __restrict__ k_scale,
                     float* __restrict__ v_scale) {
  constexpr int HALF = D / 2, EG = HALF / 8, PER = 256 / EG;              // vectors of a CTA side by side
  __shared__ float sh[2 * G][8], srank[2 * G][RANKS];
  // "has started": a rank's shared memory may be written by another only once its CTA runs; awaited before the remote store below
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
  const int rank = blockIdx.x % RANKS, groups = (hkv + G - 1) / G;
  const int64_t item = blockIdx.x / RANKS, b = item / groups;
  const int h0 = (int)(item % groups) * G;
  const int eg = threadIdx.x % EG, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t start = pos0 ? (int64_t)pos0[b] : 0;
  const bool kvec = (reinterpret_cast<uintptr_t>(k) & 15) == 0 && ks * sizeof(T) % 16 == 0;
  const bool vvec = (reinterpret_cast<uintptr_t>(v) & 15) == 0 && vs * sizeof(T) % 16 == 0;
  const bool rvec = ((reinterpret_cast<uintptr_t>(rope_cos) | reinterpret_cast<uintptr_t>(rope_sin)) & 15) == 0;
  float mk[G], mv[G];
#pragma unroll
  for (int h = 0; h < G; ++h) mk[h] = mv[h] = 0.f;
  const int64_t t_first = (int64_t)rank * PER + threadIdx.x / EG, t_step = RANKS * PER;
  const T* kp = k + (b * Tn + t_first) * ks + h0 * D + eg * 8;
  const T* vp = v + (b * Tn + t_first) * vs + h0 * D + eg * 8;
#pragma unroll (G == 1 ? 4 : (G == 2 ? 2 : 1))
  for (int64_t t = t_first; t < Tn; t += t_step, kp += t_step * ks, vp += t_step * vs) {
    Raw8<T> x[G][2], y[G][2];
#pragma unroll
    for (int h = 0; h < G; ++h)
      if (G == 1 || h0 + h < hkv) {
        x[h][0].load(kp + h * D, kvec); x[h][1].load(kp + h * D + HALF, kvec);
        y[h][0].load(vp + h * D, vvec); y[h][1].load(vp + h * D + HALF, vvec);
      } else {
        x[h][0] = x[h][1] = y[h][0] = y[h][1] = Raw8<T>{};
      }
    if (rope_cos) {
      int64_t p = start + t;
      p = p >= rope_rows ? rope_rows - 1 : p;
      Raw8<T> cc, ss;
      Raw8<float> c, s;
      c.load(rope_cos + p * HALF + eg * 8, rvec);
      s.load(rope_sin + p * HALF + eg * 8, rvec);
      round8(c, cc);
      round8(s, ss);
#pragma unroll
      for (int h = 0; h < G; ++h) rope8(x[h][0], x[h][1], cc, ss);
    }
#pragma unroll
    for (int h = 0; h < G; ++h) {
      mk[h] = x[h][1].amax(x[h][0].amax(mk[h]));
      mv[h] = y[h][1].amax(y[h][0].amax(mv[h]));
    }
  }
#pragma unroll
  for (int h = 0; h < G; ++h) {
    const float a = warp_max(mk[h]), c = warp_max(mv[h]);
    if (lane == 0) { sh[2 * h][w] = a; sh[2 * h + 1][w] = c; }
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
  if (threadIdx.x < 2 * G) {
    float m = sh[threadIdx.x][0];
#pragma unroll
    for (int i = 1; i < 8; ++i) m = fmaxf(m, sh[threadIdx.x][i]);
    unsigned dst;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(dst) : "r"((unsigned)__cvta_generic_to_shared(&srank[threadIdx.x][rank])));
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(dst), "f"(m) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (rank == 0 && threadIdx.x < 2 * G && h0 + (int)threadIdx.x / 2 < hkv) {
    float m = srank[threadIdx.x][0];
#pragma unroll
    for (int i = 1; i < RANKS; ++i) m = fmaxf(m, srank[threadIdx.x][i]);
    ((threadIdx.x & 1) ? v_scale : k_scale)[b * hkv + h0 + threadIdx.x / 2] = m > 0.f ? __fdiv_rn(m, 448.0f) : 1.0f;
  }
}

template <typename T, int D>
int launch_append(const tsb200_kv_desc& kv, void* q, int64_t qs, int qheads, const void* k, const void* v, int64_t ks, int64_t vs, int64_t B, int64_t Tn, const int32_t* new_lens,
                  const float* rc, const float* rs, int64_t rr, cudaStream_t s) {
  const int64_t rec = (int64_t)tsb200_kv_record_bytes(kv.format, D);
  // By page from 2^17 K elements on (NVFP4, whose V is half as many scattered bytes: 2^18); below that the chain of a page's CTA (tables,
  // vectors, codes, staged V) is longer than that of a warp per vector, whose byte stores are still few.  8 heads, d 128, both kernels:
  // 64 tokens int8 5.5 us by page, 4.9 by vector; 192 tokens 5.6 / 6.3 (NVFP4 6.0 / 4.9); 512 tokens 6.1 / 10.2 (NVFP4 6.1 / 5.9).
  const int64_t elements = B * Tn * kv.hkv * D;
  if (Tn >= 16 && kv.format <= TSB200_KV_NVFP4 && B <= 65535 && elements >= (kv.format == TSB200_KV_NVFP4 ? 1 << 18 : 1 << 17)) {
    // one CTA per (sequence, page group touched); the range may straddle one more page than it fills
    constexpr int PAGES = 128 / D;
    const int64_t groups = ((Tn + 15) / 16 + 1 + PAGES - 1) / PAGES, tasks = 2 * (int64_t)kv.hkv + (q ? qheads : 0);
    // A short chunk leaves most SMs without a page: its heads are dealt out over as many CTAs per page as three an SM leave room for,
    // at most until a warp has one task.
    int64_t z = 444 / (groups * B);
    if (z > (tasks + 7) / 8) z = (tasks + 7) / 8;
    const dim3 grid((unsigned)groups, (unsigned)B, (unsigned)(z < 1 ? 1 : z));
    auto go = [&](auto fmt, auto ahead) {
      constexpr int FMT = decltype(fmt)::value;
      constexpr bool AHEAD = decltype(ahead)::value;
      constexpr size_t smem = sizeof(AppendSmem<T, D, FMT, AHEAD>);
      static bool configured[64] = {false};
      int dev = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e != cudaSuccess) return e;
      if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
      if (!configured[dev]) {
        e = cudaFuncSetAttribute(kv_append_pages_kernel<T, D, FMT, AHEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
      }
      return launch_kernel(kv_append_pages_kernel<T, D, FMT, AHEAD>, grid, dim3(256), smem, s, kv, (T*)q, qs, qheads, (const T*)k, (const T*)v, ks, vs, Tn, new_lens, rc, rs, rr, rec);
    };
    auto pick = [&](auto fmt) {
      if constexpr (sizeof(T) == 2)
        if (8 * (int)grid.z < 2 * kv.hkv) return go(fmt, std::true_type{});      // several tasks to a warp
      return go(fmt, std::false_type{});
    };
    if (kv.format == TSB200_KV_INT8) TSB_CUDA(pick(std::integral_constant<int, TSB200_KV_INT8>{}));
    else if (kv.format == TSB200_KV_FP8) TSB_CUDA(pick(std::integral_constant<int, TSB200_KV_FP8>{}));
    else TSB_CUDA(pick(std::integral_constant<int, TSB200_KV_NVFP4>{}));
    TSB_LAUNCH_CHECK();
    return TSB200_OK;
  }
  const int64_t warps = B * Tn * (kv.hkv + (q ? qheads : 0));
  const int64_t blocks = (warps + 7) / 8;
  if (blocks > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  switch (kv.format) {
    case TSB200_KV_INT8:
      TSB_CUDA(launch_kernel(kv_append_kernel<T, D, TSB200_KV_INT8>, dim3((unsigned)blocks), dim3(256), 0, s, kv, (T*)q, qs, qheads, (const T*)k, (const T*)v, ks, vs, B, Tn, new_lens, rc, rs, rr, rec));
      break;
    case TSB200_KV_FP8:
      TSB_CUDA(launch_kernel(kv_append_kernel<T, D, TSB200_KV_FP8>, dim3((unsigned)blocks), dim3(256), 0, s, kv, (T*)q, qs, qheads, (const T*)k, (const T*)v, ks, vs, B, Tn, new_lens, rc, rs, rr, rec));
      break;
    case TSB200_KV_NVFP4:
      TSB_CUDA(launch_kernel(kv_append_kernel<T, D, TSB200_KV_NVFP4>, dim3((unsigned)blocks), dim3(256), 0, s, kv, (T*)q, qs, qheads, (const T*)k, (const T*)v, ks, vs, B, Tn, new_lens, rc, rs, rr, rec));
      break;
    default:   // unquantized pages in the act dtype
      TSB_CUDA(launch_kernel(kv_append_kernel<T, D, TSB200_KV_F32>, dim3((unsigned)blocks), dim3(256), 0, s, kv, (T*)q, qs, qheads, (const T*)k, (const T*)v, ks, vs, B, Tn, new_lens, rc, rs, rr, rec));
  }
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

int validate_kv(const tsb200_kv_desc* kv, bool need_table) {
  if (!kv) return TSB200_ERR_ARG;
  if (kv->format < 0 || kv->format > TSB200_KV_BF16) return TSB200_ERR_UNSUPPORTED;
  if (kv->head_dim != 64 && kv->head_dim != 128) return TSB200_ERR_UNSUPPORTED;
  if (kv->hkv <= 0 || kv->num_pages < 0 || kv->bt_stride < 0) return TSB200_ERR_ARG;
  if (!kv->k_pool || !kv->v_pool || !aligned(kv->k_pool, 16) || !aligned(kv->v_pool, 16)) return TSB200_ERR_ARG;
  if (need_table && (!kv->block_table || !kv->seq_lens)) return TSB200_ERR_ARG;
  if (kv->format == TSB200_KV_FP8 && (!kv->k_scale || !kv->v_scale)) return TSB200_ERR_ARG;
  return TSB200_OK;
}

}  // namespace tsb

using namespace tsb;

extern "C" {

size_t tsb200_kv_record_bytes(int format, int head_dim) {
  if (head_dim <= 0 || head_dim % 32) return 0;
  switch (format) {
    case TSB200_KV_INT8: return (size_t)16 * head_dim + 64;
    case TSB200_KV_FP8: return (size_t)16 * head_dim;
    case TSB200_KV_NVFP4: return (size_t)16 * head_dim / 2 + (size_t)head_dim;
    case TSB200_KV_F32: return (size_t)16 * head_dim * 4;
    case TSB200_KV_BF16: return (size_t)16 * head_dim * 2;
    default: return 0;
  }
}

int tsb200_kv_fp8_scales(const void* k, const void* v, int dtype, int64_t B, int64_t T, int hkv, int head_dim,
                         const int32_t* pos0, const float* rope_cos, const float* rope_sin, int64_t rope_rows,
                         float* k_scale, float* v_scale, void* stream) {
  return tsb200_kv_fp8_scales_strided(k, v, dtype, 0, 0, B, T, hkv, head_dim, pos0, rope_cos, rope_sin, rope_rows, k_scale, v_scale, stream);
}

int tsb200_kv_fp8_scales_strided(const void* k, const void* v, int dtype, int64_t k_token_stride, int64_t v_token_stride, int64_t B,
                                 int64_t T, int hkv, int head_dim, const int32_t* pos0, const float* rope_cos, const float* rope_sin,
                                 int64_t rope_rows, float* k_scale, float* v_scale, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (B < 0 || T < 0 || hkv <= 0) return TSB200_ERR_ARG;
  if (head_dim != 64 && head_dim != 128) return TSB200_ERR_UNSUPPORTED;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (B == 0) return TSB200_OK;
  if (!k_scale || !v_scale || (T > 0 && (!k || !v))) return TSB200_ERR_ARG;
  if ((rope_cos != nullptr) != (rope_sin != nullptr) || (rope_cos && rope_rows <= 0)) return TSB200_ERR_ARG;
  const int64_t dense = (int64_t)hkv * head_dim;
  const int64_t ks = k_token_stride ? k_token_stride : dense, vs = v_token_stride ? v_token_stride : dense;
  if (ks < dense || vs < dense) return TSB200_ERR_ARG;
  if (B * hkv * kScaleRanks > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  // A single CTA where it takes all tokens at once (4096 / head_dim; 32 sequences x 17 tokens, 8 heads: 4.1 us, 6.6 with a cluster), and
  // heads per CTA: as many as leave every SM two CTAs.
  const int ranks = T <= 4096 / head_dim ? 1 : kScaleRanks;
  int g = 4;
  while (g > 1 && B * ((hkv + g - 1) / g) * ranks < 296) g /= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(B * ((hkv + g - 1) / g) * ranks));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
#define TSB_SR(TT, DD, GG, RR) TSB_CUDA(cudaLaunchKernelEx(&cfg, kv_fp8_scales_kernel<TT, DD, GG, RR>, (const TT*)k, (const TT*)v, ks, vs, T, hkv, pos0, rope_cos, rope_sin, rope_rows, k_scale, v_scale))
#define TSB_SG(TT, DD, GG) do { if (ranks == 1) TSB_SR(TT, DD, GG, 1); else TSB_SR(TT, DD, GG, kScaleRanks); } while (0)
#define TSB_SC(TT, DD) do { if (g == 4) TSB_SG(TT, DD, 4); else if (g == 2) TSB_SG(TT, DD, 2); else TSB_SG(TT, DD, 1); } while (0)
  if (dtype == TSB200_F32) { if (head_dim == 64) TSB_SC(float, 64); else TSB_SC(float, 128); }
  else { if (head_dim == 64) TSB_SC(__nv_bfloat16, 64); else TSB_SC(__nv_bfloat16, 128); }
#undef TSB_SR
#undef TSB_SG
#undef TSB_SC
  return TSB200_OK;
}

int tsb200_rope_append(const tsb200_kv_desc* kv, void* q, int q_heads, int64_t q_token_stride, const void* k,
                       const void* v, int dtype, int64_t k_token_stride, int64_t v_token_stride, int64_t B, int64_t T,
                       const int32_t* new_lens, const float* rope_cos, const float* rope_sin, int64_t rope_rows,
                       void* stream) {
  TSB_REQUIRE_DEVICE();
  int st = validate_kv(kv, true);
  if (st != TSB200_OK) return st;
  if (B < 0 || T < 0 || q_heads < 0) return TSB200_ERR_ARG;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (B == 0 || T == 0) return TSB200_OK;
  if (!k || !v) return TSB200_ERR_ARG;
  if ((kv->format == TSB200_KV_F32 && dtype != TSB200_F32) || (kv->format == TSB200_KV_BF16 && dtype != TSB200_BF16))
    return TSB200_ERR_UNSUPPORTED;   // unquantized pages hold the act dtype
  if ((rope_cos != nullptr) != (rope_sin != nullptr) || (rope_cos && rope_rows <= 0)) return TSB200_ERR_ARG;
  if (q && (!rope_cos || q_heads <= 0)) return TSB200_ERR_ARG;
  const int64_t dense = (int64_t)kv->hkv * kv->head_dim;
  const int64_t ks = k_token_stride ? k_token_stride : dense, vs = v_token_stride ? v_token_stride : dense;
  const int64_t qs = q_token_stride ? q_token_stride : (int64_t)q_heads * kv->head_dim;
  if (ks < dense || vs < dense || (q && qs < (int64_t)q_heads * kv->head_dim)) return TSB200_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (dtype == TSB200_F32)
    return kv->head_dim == 64 ? launch_append<float, 64>(*kv, q, qs, q_heads, k, v, ks, vs, B, T, new_lens, rope_cos, rope_sin, rope_rows, s)
                              : launch_append<float, 128>(*kv, q, qs, q_heads, k, v, ks, vs, B, T, new_lens, rope_cos, rope_sin, rope_rows, s);
  return kv->head_dim == 64 ? launch_append<__nv_bfloat16, 64>(*kv, q, qs, q_heads, k, v, ks, vs, B, T, new_lens, rope_cos, rope_sin, rope_rows, s)
                            : launch_append<__nv_bfloat16, 128>(*kv, q, qs, q_heads, k, v, ks, vs, B, T, new_lens, rope_cos, rope_sin, rope_rows, s);
}

int tsb200_kv_append(const tsb200_kv_desc* kv, const void* k, const void* v, int dtype, int64_t k_token_stride,
                     int64_t v_token_stride, int64_t B, int64_t T, const int32_t* new_lens, const float* rope_cos,
                     const float* rope_sin, int64_t rope_rows, void* stream) {
  return tsb200_rope_append(kv, nullptr, 0, 0, k, v, dtype, k_token_stride, v_token_stride, B, T, new_lens, rope_cos,
                            rope_sin, rope_rows, stream);
}

}  // extern "C"
