// Weight quantization, bit packing and reconstruction.
//
// Follows transformersurgeon/compression/quantization_methods/vanilla.py:5-37 step by
// step, in the parameter dtype: for bf16 parameters every intermediate (amax/qmax,
// scale+eps, w/(scale+eps)) is rounded to bf16 before the next op, exactly as the
// chain of torch ops does; rounding of the quotient to an integer is half-to-even.
#include "common.cuh"
#include <type_traits>

namespace tsb {

__device__ __forceinline__ float block_max(float v, float* sh) {
  v = warp_max(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (l < nw) ? sh[l] : 0.f;
  r = warp_max(r);
  __syncthreads();
  return r;
}
__device__ __forceinline__ double block_sum_d(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = (l < nw) ? sh[l] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  __syncthreads();
  return r;
}

struct TensorStats {       // lives in the caller's workspace (16 bytes)
  unsigned int amax_bits;  // max |w| as fp32 bits (non-negative floats order like uints)
  unsigned int pad;
  double abs_sum;
};

template <typename T>
__global__ void tensor_stats_kernel(const T* __restrict__ w, int64_t n, TensorStats* st) {
  __shared__ float shf[32];
  __shared__ double shd[32];
  float m = 0.f;
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float a = fabsf(to_f32<T>(w[i]));
    m = fmaxf(m, a);
    s += (double)a;
  }
  m = block_max(m, shf);
  s = block_sum_d(s, shd);
  if (threadIdx.x == 0) {
    atomicMax(&st->amax_bits, __float_as_uint(m));
    atomicAdd(&st->abs_sum, s);
  }
}

// One CTA per row.  precision 0 = binary.
template <typename T>
__global__ void quantize_rows_kernel(const T* __restrict__ w, int64_t rows, int64_t cols, int precision,
                                     int per_channel, float eps, int8_t* __restrict__ codes,
                                     float* __restrict__ scales, const TensorStats* st) {
  __shared__ float shf[32];
  __shared__ double shd[32];
  const int64_t r = blockIdx.x;
  const T* wr = w + r * cols;
  int8_t* cr = codes + r * cols;
  if (precision == 0) {
    float scale;
    if (per_channel) {
      double s = 0.0;
      for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) s += (double)fabsf(to_f32<T>(wr[c]));
      s = block_sum_d(s, shd);
      scale = rnd<T>((float)(s / (double)cols));
    } else {
      scale = rnd<T>((float)(st->abs_sum / (double)(rows * cols)));
    }
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
      float v = to_f32<T>(wr[c]);
      cr[c] = (int8_t)((v > 0.f) - (v < 0.f));
    }
    if (threadIdx.x == 0) scales[r] = scale;
    return;
  }
  const float qmax = (float)((1 << (precision - 1)) - 1);
  float amax;
  if (per_channel) {
    float m = 0.f;
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) m = fmaxf(m, fabsf(to_f32<T>(wr[c])));
    amax = block_max(m, shf);
  } else {
    amax = __uint_as_float(st->amax_bits);
  }
  const float scale = rnd<T>(__fdiv_rn(amax, qmax));
  const float denom = rnd<T>(__fadd_rn(scale, eps));
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    float q = rnd<T>(__fdiv_rn(to_f32<T>(wr[c]), denom));
    q = fminf(fmaxf(rintf(q), -qmax), qmax);
    cr[c] = (int8_t)(int)q;   // NaN (0/0 cannot occur: denom >= eps) -> not reached
  }
  if (threadIdx.x == 0) scales[r] = scale;
}

// One thread per packed 32-bit word (bits < 8) or per byte (bits == 8).
__global__ void pack_codes_kernel(const int8_t* __restrict__ codes, int64_t rows, int64_t cols, int bits,
                                  int64_t row_bytes, uint8_t* __restrict__ packed, int32_t* zero_flag) {
  if (bits == 8) {
    const int64_t total = rows * row_bytes;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
      const int64_t r = i / row_bytes, c = i - r * row_bytes;
      packed[i] = c < cols ? (uint8_t)codes[r * cols + c] : (uint8_t)0;
    }
    return;
  }
  const int per = 32 / bits;
  const int64_t row_words = row_bytes / 4;
  const int64_t total = rows * row_words;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / row_words, g = i - r * row_words;
    const int8_t* cr = codes + r * cols;
    unsigned int out = 0;
    for (int j = 0; j < per; ++j) {
      const int64_t c = g * per + j;
      const int q = (c < cols) ? (int)cr[c] : 0;
      const int f = field_of_column(j, per);
      if (bits == 1) {
        if (c < cols && q == 0 && zero_flag) *zero_flag = 1;
        out |= (unsigned)(q > 0) << f;
      } else {
        out |= ((unsigned)q & ((1u << bits) - 1u)) << (bits * f);
      }
    }
    reinterpret_cast<unsigned*>(packed)[i] = out;
  }
}

__global__ void unpack_codes_kernel(const uint8_t* __restrict__ packed, int64_t rows, int64_t cols, int bits,
                                    int64_t row_bytes, int8_t* __restrict__ codes) {
  const int64_t total = rows * cols;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / cols, c = i - r * cols;
    codes[i] = (int8_t)load_code(packed + r * row_bytes, c, bits);
  }
}

template <typename T>
__global__ void dequantize_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ scales, int64_t rows,
                                  int64_t cols, int bits, int64_t row_bytes, T* __restrict__ out) {
  const int64_t total = rows * cols;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / cols, c = i - r * cols;
    const int q = load_code(packed + r * row_bytes, c, bits);
    out[i] = from_f32<T>(__fmul_rn((float)q, scales[r]));
  }
}

// ---- quantize and pack in one pass --------------------------------------------------------------------------------------
// Bound by the weights' one trip from memory (a 14336 x 4096 bf16 matrix: 147 MB, 22 us) and, next to it, by the arithmetic: the
// quotient that vanilla.py prescribes is an IEEE division per element.  TPR threads own a row and keep it in registers between the
// statistic and the codes (IT units of 8 columns each), the codes never exist as bytes, and the quotient by a divisor that the
// whole row shares comes from its correctly rounded reciprocal y: for bf16 weights the product w y (unit_quotients), for fp32 ones
// q = w y, r = w - d q (exact), q + r y - correctly rounded by
// Markstein's theorem (Computation of elementary functions on the IBM RISC System/6000 processor, 1990) as long as nothing leaves
// the normal range, which the divisor's range guarantees for every quotient that does not round to zero; other divisors divide.
// Together with its packing launch the two-pass form took 177 us on that matrix; this one takes 33 us (36.9 with a correction of the
// quotients and codes placed one by one instead of in pairs).  The row stays in the weights'
// own type (as floats: 88 registers a thread, too few warps in flight, 108 us), and bf16 codes of up to four bits are rounded,
// clamped and placed in pairs.  CTAs that walk their rows and fetch the next one under the codes of this one were no faster (37.5 us: their warps
// keep step, and loads and arithmetic overlap less than those of independent CTAs do); 128 threads a row: 34.8, 256: 40.9.
//
// Eight columns in the weights' own type (bf16: as four packed pairs).
template <typename T> struct Unit;
template <> struct Unit<__nv_bfloat16> {
  unsigned u[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* row, int64_t c, int64_t cols, bool vec) {
    if (vec && c + 8 <= cols) {
      const uint4 a = __ldg(reinterpret_cast<const uint4*>(row + c));
      u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned lo = c + 2 * i < cols ? __bfloat16_as_ushort(row[c + 2 * i]) : 0, hi = c + 2 * i + 1 < cols ? __bfloat16_as_ushort(row[c + 2 * i + 1]) : 0;
        u[i] = lo | (hi << 16);
      }
    }
  }
  __device__ __forceinline__ float at(int j) const { return __uint_as_float((j & 1) ? u[j >> 1] & 0xffff0000u : u[j >> 1] << 16); }
  __device__ __forceinline__ float amax(float m) const {
    __nv_bfloat162 a = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&u[0]));
#pragma unroll
    for (int i = 1; i < 4; ++i) a = __hmax2(a, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&u[i])));
    return fmaxf(m, fmaxf(__low2float(a), __high2float(a)));
  }
};
template <> struct Unit<float> {
  float f[8];
  __device__ __forceinline__ void load(const float* row, int64_t c, int64_t cols, bool vec) {
    if (vec && c + 8 <= cols) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(row + c)), b = __ldg(reinterpret_cast<const float4*>(row + c + 4));
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = c + i < cols ? row[c + i] : 0.f;
    }
  }
  __device__ __forceinline__ float at(int j) const { return f[j]; }
  __device__ __forceinline__ float amax(float m) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(f[i]));
    return m;
  }
};

// The unit's quotients.  y: correctly rounded 1 / denom.  bf16: the quotient is rounded to bf16 next, whose midpoints no quotient of two
// 8-bit numbers hits (9 significant bits times the divisor's are more than 8) or comes closer to than 2^-17, so that the product,
// within 2^-23, rounds alike; fp32: corrected twice.
template <typename T, bool DIVIDE> __device__ __forceinline__ void unit_quotients(const Unit<T>& v, float denom, float y, float (&p)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float x = v.at(j);
    if (DIVIDE) {
      p[j] = __fdiv_rn(x, denom);
    } else {
      p[j] = x * y;
      if (sizeof(T) == 4) {
        p[j] = fmaf(fmaf(-p[j], denom, x), y, p[j]);
        p[j] = fmaf(fmaf(-p[j], denom, x), y, p[j]);
      }
    }
  }
}
// The unit's codes in the low BITS bits of q[0..7] (the other bits are anything).
template <typename T, bool DIVIDE> __device__ __forceinline__ void unit_codes(const Unit<T>& v, float denom, float y, float qmax, unsigned (&q)[8]) {
  float p[8];
  unit_quotients<T, DIVIDE>(v, denom, y, p);
#pragma unroll
  for (int j = 0; j < 8; ++j)       // the bounds are whole numbers: clamping before or after rounding is the same; 1.5 * 2^23: half-to-even
    q[j] = __float_as_uint(fminf(fmaxf(rnd<T>(p[j]), -qmax), qmax) + 12582912.0f);
}
// bf16 weights, codes of up to four bits: the codes of columns 2 i and 2 i + 1 in the low bits of the halves of h[i] (the other bits are
// anything).  Rounded to bf16, clamped and added to 192 in pairs: bf16 numbers of [128, 256) are whole, so the sum is rounded
// half-to-even to a whole number that stands in its low bits (|code| <= 7).
template <bool DIVIDE>
__device__ __forceinline__ void unit_code_pairs(const Unit<__nv_bfloat16>& v, float denom, float y, float qmax, unsigned (&h)[4]) {
  float p[8];
  unit_quotients<__nv_bfloat16, DIVIDE>(v, denom, y, p);
  const __nv_bfloat162 hi = __float2bfloat162_rn(qmax), lo = __float2bfloat162_rn(-qmax), magic = __float2bfloat162_rn(192.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 r = __floats2bfloat162_rn(p[2 * i], p[2 * i + 1]);
    r = __hadd2_rn(__hmin2(__hmax2(r, lo), hi), magic);
    h[i] = *reinterpret_cast<const unsigned*>(&r);
  }
}

// Reductions over the TPR threads of a row.
template <int TPR> __device__ __forceinline__ float row_max(float v, float* sh) {
  v = warp_max(v);
  if (TPR > 32) {
    const int w = threadIdx.x >> 5, w0 = w / (TPR / 32) * (TPR / 32);
    if ((threadIdx.x & 31) == 0) sh[w] = v;
    __syncthreads();
    v = sh[w0];
#pragma unroll
    for (int i = 1; i < TPR / 32; ++i) v = fmaxf(v, sh[w0 + i]);
  }
  return v;
}
template <int TPR> __device__ __forceinline__ double row_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (TPR > 32) {
    const int w = threadIdx.x >> 5, w0 = w / (TPR / 32) * (TPR / 32);
    if ((threadIdx.x & 31) == 0) sh[w] = v;
    __syncthreads();
    v = sh[w0];
#pragma unroll
    for (int i = 1; i < TPR / 32; ++i) v += sh[w0 + i];
  }
  return v;
}

// The unit's eight codes (as bits of `bits` each) in the pair-interleaved order of the container word that holds them.
template <int BITS> __device__ __forceinline__ unsigned place(const unsigned (&q)[8], int64_t c) {
  constexpr unsigned mask = BITS == 8 ? 0xffu : (1u << BITS) - 1u;
  constexpr int per = 32 / BITS;
  const int f0 = (int)(c % per) >> 1;          // first field of the unit's even columns
  unsigned w = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) w |= ((q[2 * i] & mask) << (BITS * i)) | ((q[2 * i + 1] & mask) << (BITS * (i + per / 2)));
  return BITS == 4 ? w : w << (BITS * f0);
}

// The same from pairs: the container word interleaves its columns in pairs too, field i and field i + per / 2, 16 bits apart.
template <int BITS> __device__ __forceinline__ unsigned place_pairs(const unsigned (&h)[4], int64_t c) {
  constexpr unsigned mask = ((1u << BITS) - 1u) * 0x10001u;
  unsigned w = h[0] & mask;
#pragma unroll
  for (int i = 1; i < 4; ++i) w |= (h[i] << (BITS * i)) & (mask << (BITS * i));
  return BITS == 4 ? w : w << (BITS * ((int)(c % (32 / BITS)) >> 1));
}

template <typename T, int TPR, int IT, int BITS>
__global__ void __launch_bounds__(256)
quantize_pack_kernel(const T* __restrict__ w, int64_t rows, int64_t cols, int precision, int per_channel, float eps, int64_t row_bytes,
                     uint8_t* __restrict__ packed, float* __restrict__ scales, const TensorStats* st, int32_t* zero_flag) {
  __shared__ float shf[8];
  __shared__ double shd[8];
  const int64_t r = (int64_t)blockIdx.x * (256 / TPR) + threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const bool live = r < rows;                  // every thread takes part in the reductions
  const T* row = w + (live ? r : rows - 1) * cols;
  const bool vec = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  const int64_t units = row_bytes / BITS;      // of 8 columns, the padding to 64 columns included
  Unit<T> v[IT];
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const int64_t u = t + (int64_t)i * TPR;
    if (u < units) v[i].load(row, u * 8, cols, vec);
    else v[i] = Unit<T>{};
  }
  float scale, denom = 1.f, y = 1.f;
  const float qmax = (float)((1 << ((precision ? precision : 2) - 1)) - 1);
  bool divide = false;
  if (precision == 0) {
    double s = 0.0;
    if (per_channel) {
#pragma unroll
      for (int i = 0; i < IT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) s += (double)fabsf(v[i].at(j));
      s = row_sum<TPR>(s, shd) / (double)cols;
    } else {
      s = st->abs_sum / (double)(rows * cols);
    }
    scale = rnd<T>((float)s);
  } else {
    float m = 0.f;
    if (per_channel) {
#pragma unroll
      for (int i = 0; i < IT; ++i)
        m = v[i].amax(m);
      m = row_max<TPR>(m, shf);
    } else {
      m = __uint_as_float(st->amax_bits);
    }
    scale = rnd<T>(__fdiv_rn(m, qmax));
    denom = rnd<T>(__fadd_rn(scale, eps));
    divide = !(denom >= 1e-18f && denom <= 1e18f);
    y = __frcp_rn(denom);
  }
  if (!live) return;
  if (t == 0) scales[r] = scale;
  uint8_t* out = packed + r * row_bytes;
  bool zero = false;
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const int64_t u = t + (int64_t)i * TPR;
    if constexpr (sizeof(T) == 2 && BITS > 1 && BITS < 8) {
      if (precision != 0) {
        unsigned h[4];
        if (divide) unit_code_pairs<true>(v[i], denom, y, qmax, h);
        else unit_code_pairs<false>(v[i], denom, y, qmax, h);
        unsigned word = u < units ? place_pairs<BITS>(h, u * 8) : 0u;
        if (BITS == 2) word |= __shfl_xor_sync(0xffffffffu, word, 1);      // a word is two units
        if (u < units && u % (4 / BITS) == 0) *reinterpret_cast<unsigned*>(out + u * BITS) = word;
        continue;
      }
    }
    unsigned q[8];
    if (precision == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = v[i].at(j);
        const int sgn = (x > 0.f) - (x < 0.f);
        if (BITS == 1) zero |= sgn == 0 && u < units && u * 8 + j < cols;
        q[j] = BITS == 1 ? (unsigned)(sgn > 0) : (unsigned)sgn;
      }
    } else if (divide) {
      unit_codes<T, true>(v[i], denom, y, qmax, q);
    } else {
      unit_codes<T, false>(v[i], denom, y, qmax, q);
    }
    if constexpr (BITS == 8) {
      if (u < units) {
        unsigned lo = 0, hi = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) { lo |= (q[j] & 0xffu) << (8 * j); hi |= (q[4 + j] & 0xffu) << (8 * j); }
        *reinterpret_cast<uint2*>(out + u * 8) = make_uint2(lo, hi);
      }
    } else {
      unsigned word = u < units ? place<BITS>(q, u * 8) : 0u;
      // a word of 2-bit codes is two units, one of 1-bit codes four: neighbouring lanes (units are a multiple of 8 per row)
      if (BITS <= 2) word |= __shfl_xor_sync(0xffffffffu, word, 1);
      if (BITS == 1) word |= __shfl_xor_sync(0xffffffffu, word, 2);
      constexpr int per = BITS == 4 ? 1 : (BITS == 2 ? 2 : 4);
      if (u < units && u % per == 0) *reinterpret_cast<unsigned*>(out + u * BITS) = word;
    }
  }
  if (BITS == 1 && zero && zero_flag) *zero_flag = 1;
}

// False: rows too long for the registers of 256 threads.
template <typename T, int BITS>
bool launch_quantize_pack(const T* w, int64_t rows, int64_t cols, int precision, int per_channel, float eps, uint8_t* packed, float* scales,
                          const TensorStats* st, int32_t* zero_flag, cudaStream_t s) {
  const int64_t rb = (int64_t)tsb200_packed_row_bytes(cols, BITS), units = rb / BITS;
  auto go = [&](auto tpr, auto it) {
    constexpr int TPR = decltype(tpr)::value, IT = decltype(it)::value;
    const int64_t blocks = (rows + 256 / TPR - 1) / (256 / TPR);
    quantize_pack_kernel<T, TPR, IT, BITS><<<(unsigned)blocks, 256, 0, s>>>(w, rows, cols, precision, per_channel, eps, rb, packed, scales, st, zero_flag);
    return true;
  };
  // as few threads per row as its units fit in registers, eight units to a thread where possible (64 registers)
  if (units <= 32 * 4) return go(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
  if (units <= 64 * 8) return go(std::integral_constant<int, 64>{}, std::integral_constant<int, 8>{});
  if (units <= 256 * 8) return go(std::integral_constant<int, 256>{}, std::integral_constant<int, 8>{});
  if (units <= 256 * 16) return go(std::integral_constant<int, 256>{}, std::integral_constant<int, 16>{});
  return false;
}

inline int grid_for(int64_t n, int block) {
  int64_t g = (n + block - 1) / block;
  const int64_t cap = 148 * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace tsb

using namespace tsb;

extern "C" {

size_t tsb200_packed_row_bytes(int64_t cols, int bits) {
  if (cols <= 0 || !(bits == 1 || bits == 2 || bits == 4 || bits == 8)) return 0;
  return (size_t)((cols + 63) / 64 * 64 * bits / 8);
}

int tsb200_quantize_weight(const void* w, int dtype, int64_t rows, int64_t cols, int precision,
                           int per_channel, float eps, int8_t* codes, float* scales,
                           void* workspace, size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (rows < 0 || cols < 0) return TSB200_ERR_ARG;
  if (rows == 0 || cols == 0) return TSB200_OK;
  if (!w || !codes || !scales) return TSB200_ERR_ARG;
  if (!(precision == 0 || (precision >= 2 && precision <= 8))) return TSB200_ERR_UNSUPPORTED;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (rows > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  TensorStats* st = nullptr;
  if (!per_channel) {
    if (!workspace || !aligned(workspace, 8)) return TSB200_ERR_ARG;
    if (workspace_bytes < sizeof(TensorStats)) return TSB200_ERR_WORKSPACE;
    st = (TensorStats*)workspace;
    TSB_CUDA(cudaMemsetAsync(st, 0, sizeof(TensorStats), s));
    const int64_t n = rows * cols;
    if (dtype == TSB200_F32) tensor_stats_kernel<float><<<grid_for(n, 256), 256, 0, s>>>((const float*)w, n, st);
    else tensor_stats_kernel<__nv_bfloat16><<<grid_for(n, 256), 256, 0, s>>>((const __nv_bfloat16*)w, n, st);
    TSB_LAUNCH_CHECK();
  }
  if (dtype == TSB200_F32)
    quantize_rows_kernel<float><<<(unsigned)rows, 256, 0, s>>>((const float*)w, rows, cols, precision, per_channel, eps, codes, scales, st);
  else
    quantize_rows_kernel<__nv_bfloat16><<<(unsigned)rows, 256, 0, s>>>((const __nv_bfloat16*)w, rows, cols, precision, per_channel, eps, codes, scales, st);
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

int tsb200_quantize_pack(const void* w, int dtype, int64_t rows, int64_t cols, int precision, int per_channel, float eps, int bits,
                         uint8_t* packed, float* scales, int32_t* zero_flag, void* workspace, size_t workspace_bytes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (rows < 0 || cols < 0) return TSB200_ERR_ARG;
  if (!(precision == 0 || (precision >= 2 && precision <= 8))) return TSB200_ERR_UNSUPPORTED;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (!(bits == 1 || bits == 2 || bits == 4 || bits == 8) || (precision != 0 && bits < precision) || (bits == 1 && precision != 0)) return TSB200_ERR_UNSUPPORTED;
  if (rows == 0 || cols == 0) return TSB200_OK;
  if (!w || !packed || !scales || !aligned(packed, 8)) return TSB200_ERR_ARG;
  if (rows > 0x7fffffffLL) return TSB200_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  TensorStats* st = nullptr;
  if (!per_channel) {
    if (!workspace || !aligned(workspace, 8)) return TSB200_ERR_ARG;
    if (workspace_bytes < sizeof(TensorStats)) return TSB200_ERR_WORKSPACE;
    st = (TensorStats*)workspace;
    TSB_CUDA(cudaMemsetAsync(st, 0, sizeof(TensorStats), s));
    const int64_t n = rows * cols;
    if (dtype == TSB200_F32) tensor_stats_kernel<float><<<grid_for(n, 256), 256, 0, s>>>((const float*)w, n, st);
    else tensor_stats_kernel<__nv_bfloat16><<<grid_for(n, 256), 256, 0, s>>>((const __nv_bfloat16*)w, n, st);
    TSB_LAUNCH_CHECK();
  }
  bool done;
#define TSB_GO(TT)                                                                                                                         \
  switch (bits) {                                                                                                                          \
    case 1: done = launch_quantize_pack<TT, 1>((const TT*)w, rows, cols, precision, per_channel, eps, packed, scales, st, zero_flag, s); break; \
    case 2: done = launch_quantize_pack<TT, 2>((const TT*)w, rows, cols, precision, per_channel, eps, packed, scales, st, zero_flag, s); break; \
    case 4: done = launch_quantize_pack<TT, 4>((const TT*)w, rows, cols, precision, per_channel, eps, packed, scales, st, zero_flag, s); break; \
    default: done = launch_quantize_pack<TT, 8>((const TT*)w, rows, cols, precision, per_channel, eps, packed, scales, st, zero_flag, s); break; \
  }
  if (dtype == TSB200_F32) { TSB_GO(float); } else { TSB_GO(__nv_bfloat16); }
#undef TSB_GO
  if (!done) return TSB200_ERR_UNSUPPORTED;
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

int tsb200_pack_codes(const int8_t* codes, int64_t rows, int64_t cols, int bits, uint8_t* packed,
                      int32_t* zero_flag, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (rows < 0 || cols < 0) return TSB200_ERR_ARG;
  const size_t rb = tsb200_packed_row_bytes(cols > 0 ? cols : 1, bits);
  if (rb == 0) return TSB200_ERR_UNSUPPORTED;
  if (rows == 0 || cols == 0) return TSB200_OK;
  if (!codes || !packed || !aligned(packed, 4)) return TSB200_ERR_ARG;
  pack_codes_kernel<<<grid_for(rows * (int64_t)(bits == 8 ? rb : rb / 4), 256), 256, 0, as_stream(stream)>>>(codes, rows, cols, bits, (int64_t)rb, packed, zero_flag);
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

int tsb200_unpack_codes(const uint8_t* packed, int64_t rows, int64_t cols, int bits, int8_t* codes, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (rows < 0 || cols < 0) return TSB200_ERR_ARG;
  const size_t rb = tsb200_packed_row_bytes(cols > 0 ? cols : 1, bits);
  if (rb == 0) return TSB200_ERR_UNSUPPORTED;
  if (rows == 0 || cols == 0) return TSB200_OK;
  if (!codes || !packed) return TSB200_ERR_ARG;
  unpack_codes_kernel<<<grid_for(rows * cols, 256), 256, 0, as_stream(stream)>>>(packed, rows, cols, bits, (int64_t)rb, codes);
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

int tsb200_dequantize_weight(const uint8_t* packed, const float* scales, int64_t rows, int64_t cols, int bits,
                             int dtype, void* w_out, void* stream) {
  TSB_REQUIRE_DEVICE();
  if (rows < 0 || cols < 0) return TSB200_ERR_ARG;
  const size_t rb = tsb200_packed_row_bytes(cols > 0 ? cols : 1, bits);
  if (rb == 0) return TSB200_ERR_UNSUPPORTED;
  if (dtype != TSB200_F32 && dtype != TSB200_BF16) return TSB200_ERR_UNSUPPORTED;
  if (rows == 0 || cols == 0) return TSB200_OK;
  if (!packed || !scales || !w_out) return TSB200_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (dtype == TSB200_F32)
    dequantize_kernel<float><<<grid_for(rows * cols, 256), 256, 0, s>>>(packed, scales, rows, cols, bits, (int64_t)rb, (float*)w_out);
  else
    dequantize_kernel<__nv_bfloat16><<<grid_for(rows * cols, 256), 256, 0, s>>>(packed, scales, rows, cols, bits, (int64_t)rb, (__nv_bfloat16*)w_out);
  TSB_LAUNCH_CHECK();
  return TSB200_OK;
}

}  // extern "C"
