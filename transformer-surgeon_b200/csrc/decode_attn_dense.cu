// Split-K paged decode attention over UNQUANTIZED pages (fp32 or bf16 values), fp32 math on the FMA pipe.
// Restates transformersurgeon/blocks/mha.py:9-103 for one query token per sequence; also serves the prompt of fp32 models, one
// "sequence" per query token.
//
// What bounds it: with the short contexts and few kv heads of the models that keep such pages (2 kv heads, a few hundred tokens) the
// latency of a page, not its bytes.  A warp takes whole pages (16 tokens).  Scores: two lanes per token, each with half of the head
// dimension, all query heads of the group against one read of the key (one shuffle per head and token, where a lane-per-element
// split needs five); weights go through shared memory to the lanes that own output elements, whose 16 value rows are requested
// before the scores are finished.  2 kv heads, 7 query heads, d 64, 150 tokens: 37 us (with
// its merge launch) -> 5.
#include "decode_attn_common.cuh"

namespace tsb {

template <typename T, int D> int launch_reduce(const float* ws, int64_t BH, int S, void* out, cudaStream_t st);

namespace {


template <typename PT> __device__ __forceinline__ float4 load4(const PT* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
template <typename PT> __device__ __forceinline__ float2 load2(const PT* p);
template <> __device__ __forceinline__ float2 load2<float>(const float* p) { return *reinterpret_cast<const float2*>(p); }
template <> __device__ __forceinline__ float2 load2<__nv_bfloat16>(const __nv_bfloat16* p) {
  const unsigned v = *reinterpret_cast<const unsigned*>(p);
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// grid (B * hkv, S, ceil(g / kHeads)).  S > 0: the last CTA of a (sequence, kv head, chunk) merges; S < 0: |S| splits, partials only.
// kWarps warps; kHeads query heads per CTA (a chunk of the group): 8 x 8, or 16 x 4 where the grid would leave most SMs idle (a
// page's instructions are then shared by two CTAs and all pages of a short context are in flight at once).
template <typename T, typename PT, int D, int kWarps, int kHeads>
__global__ void __launch_bounds__(kWarps * 32)
decode_attn_dense_kernel(tsb200_kv_desc kv, const T* __restrict__ q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S,
                         float* __restrict__ ws, int* __restrict__ counters, T* __restrict__ out) {
  constexpr int E2 = D / 64;                 // element pairs of a lane's outputs: elements 2 lane, 2 lane + 1 (+ 64)
  __shared__ __align__(16) float sq[kHeads][D];
  __shared__ __align__(16) float sp[kWarps][16][kHeads];
  __shared__ float sm_m[kWarps][kHeads], sm_l[kWarps][kHeads];
  __shared__ __align__(16) float sm_acc[kWarps][kHeads][D];
  pdl_launch_dependents();
  const int b = blockIdx.x / kv.hkv, hk = blockIdx.x % kv.hkv, s = blockIdx.y;
  const int g = H / kv.hkv, g0 = blockIdx.z * kHeads, gn = min(kHeads, g - g0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool fused = S > 0;
  S = S < 0 ? -S : S;
  int len = kv.seq_lens[b];
  len = len < 0 ? 0 : (len > max_seq_len ? (int)max_seq_len : len);
  int pb, pe;
  split_range(len, s, S, pb, pe);
  // lengths and block table do not come from the preceding launch (see tsb200_set_pdl): looked up ahead of the dependency wait
  auto page_of = [&](int pg) { return pg < pe ? kv.block_table[(int64_t)b * kv.bt_stride + pg] : 0; };
  int next_page = page_of(pb + w);
  pdl_wait();
  for (int i = threadIdx.x; i < kHeads * D; i += kWarps * 32) {
    const int h = i / D, e = i % D;
    sq[h][e] = h < gn ? to_f32<T>(q[(int64_t)b * qs + (int64_t)(hk * g + g0 + h) * D + e]) * sm_scale : 0.f;
  }
  __syncthreads();

  float m[kHeads], l[kHeads], acc[kHeads][E2 * 2];
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    m[h] = -INFINITY;
    l[h] = 0.f;
#pragma unroll
    for (int e = 0; e < E2 * 2; ++e) acc[h][e] = 0.f;
  }
  const int t = lane >> 1, half = lane & 1;
  const int64_t rec = (int64_t)16 * D;       // values of one page and head
  for (int pg = pb + w; pg < pe; pg += kWarps) {
    const int64_t page = next_page;
    next_page = page_of(pg + kWarps);
    if (page < 0 || page >= kv.num_pages) continue;
    const PT* kr = reinterpret_cast<const PT*>(kv.k_pool) + (page * kv.hkv + hk) * rec + t * D + half * 4;
    const PT* vr = reinterpret_cast<const PT*>(kv.v_pool) + (page * kv.hkv + hk) * rec + lane * 2;
    const int nt = min(16, len - pg * 16);
    float4 kx[D / 8];
    float2 vv[16][E2];
    float sc[kHeads];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) kx[i] = load4<PT>(kr + i * 8);
    auto load_v = [&]() {
#pragma unroll
      for (int u = 0; u < 16; ++u)
#pragma unroll
        for (int e = 0; e < E2; ++e) vv[u][e] = load2<PT>(vr + u * D + e * 64);
    };
    if (D == 64) load_v();                   // d 128: the key is used up first (registers)
#pragma unroll
    for (int h = 0; h < kHeads; ++h) sc[h] = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
#pragma unroll
      for (int h = 0; h < kHeads; ++h) {
        const float4 qx = *reinterpret_cast<const float4*>(&sq[h][i * 8 + half * 4]);
        sc[h] += kx[i].x * qx.x + kx[i].y * qx.y + kx[i].z * qx.z + kx[i].w * qx.w;
      }
    if (D != 64) load_v();
    float c[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) {
      sc[h] += __shfl_xor_sync(0xffffffffu, sc[h], 1);
      if (t >= nt) sc[h] = -INFINITY;
      float mx = sc[h];
#pragma unroll
      for (int o = 2; o < 32; o *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[h], mx);      // finite: token 0 of a page inside the range is valid
      c[h] = __expf(m[h] - mn);
      m[h] = mn;
      sc[h] = __expf(sc[h] - mn);
      l[h] = l[h] * c[h] + sc[h];            // per lane; both lanes of a token hold the same value
    }
    __syncwarp();                            // the previous page's weights have been read
    if (half == 0) {
#pragma unroll
      for (int h = 0; h < kHeads; h += 4) *reinterpret_cast<float4*>(&sp[w][t][h]) = make_float4(sc[h], sc[h + 1], sc[h + 2], sc[h + 3]);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kHeads; ++h)
#pragma unroll
      for (int e = 0; e < E2 * 2; ++e) acc[h][e] *= c[h];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      if (u < nt) {                          // stale slots hold anything finite: they must not count
        float ph[kHeads];
#pragma unroll
        for (int h = 0; h < kHeads; h += 4) {
          const float4 pv = *reinterpret_cast<const float4*>(&sp[w][u][h]);
          ph[h] = pv.x; ph[h + 1] = pv.y; ph[h + 2] = pv.z; ph[h + 3] = pv.w;
        }
#pragma unroll
        for (int h = 0; h < kHeads; ++h)
#pragma unroll
          for (int e = 0; e < E2; ++e) {
            acc[h][2 * e] += ph[h] * vv[u][e].x;
            acc[h][2 * e + 1] += ph[h] * vv[u][e].y;
          }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
#pragma unroll
    for (int o = 2; o < 32; o *= 2) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
    if (lane == 0) { sm_m[w][h] = m[h]; sm_l[w][h] = l[h]; }
#pragma unroll
    for (int e = 0; e < E2; ++e) *reinterpret_cast<float2*>(&sm_acc[w][h][e * 64 + lane * 2]) = make_float2(acc[h][2 * e], acc[h][2 * e + 1]);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < gn * D; idx += kWarps * 32) {
    const int i = idx / D, e = idx % D;
    float mm = -INFINITY;
#pragma unroll
    for (int u = 0; u < kWarps; ++u) mm = fmaxf(mm, sm_m[u][i]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int u = 0; u < kWarps; ++u) {
      const float cw = sm_m[u][i] == -INFINITY ? 0.f : __expf(sm_m[u][i] - mm);
      ll += sm_l[u][i] * cw;
      a += sm_acc[u][i][e] * cw;
    }
    const int64_t bh = (int64_t)b * H + hk * g + g0 + i;
    if (S == 1 && fused) {
      out[bh * D + e] = from_f32<T>(ll > 0.f ? a / ll : 0.f);
    } else {
      float* o = ws + (bh * S + s) * (2 + D);
      if (e == 0) { o[0] = mm; o[1] = ll; }
      o[2 + e] = a;
    }
  }
  if (S == 1 || !fused) return;
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  int* ctr = counters + ((int64_t)blockIdx.x * gridDim.z + blockIdx.z);
  if (threadIdx.x == 0) s_last = (atomicAdd(ctr, 1) == S - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int64_t bh0 = (int64_t)b * H + hk * g + g0;
  merge_splits<T, D>(ws + bh0 * S * (2 + D), gn, S, &sm_acc[0][0][0], out + bh0 * D);
  if (threadIdx.x == 0) *ctr = 0;
}

template <typename T, typename PT, int D, int W, int HC>
int launch_cfg(const tsb200_kv_desc& kv, const void* q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S, int64_t B, float* ws,
               int* counters, void* out, cudaStream_t st) {
  const dim3 grid((unsigned)(B * kv.hkv), (unsigned)S, (unsigned)((H / kv.hkv + HC - 1) / HC));
  TSB_CUDA(launch_kernel_if(attn_overlaps(kv), decode_attn_dense_kernel<T, PT, D, W, HC>, grid, dim3(W * 32), 0, st, kv, (const T*)q, qs, H, sm_scale, max_seq_len,
                         counters ? S : -S, ws, counters, (T*)out));
  return counters ? TSB200_OK : launch_reduce<T, D>(ws, B * H, S, out, st);
}
template <typename T, typename PT, int D>
int launch_dense(const tsb200_kv_desc& kv, const void* q, int64_t qs, int H, float sm_scale, int64_t max_seq_len, int S, int64_t B,
                 float* ws, int* counters, void* out, cudaStream_t st) {
  const int g = H / kv.hkv;
  if (B * kv.hkv * S * ((g + 3) / 4) <= 148)
    return launch_cfg<T, PT, D, 16, 4>(kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, counters, out, st);
  // (64 sequences of 17 tokens, 32 / 8 heads: 22 us with room for eight heads a CTA)
  if (g <= 4) return launch_cfg<T, PT, D, 8, 4>(kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, counters, out, st);
  return launch_cfg<T, PT, D, 8, 8>(kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, counters, out, st);
}

}  // namespace

// Unquantized pages.  Splits: one CTA's warps take a page each at a time, so a split keeps at least 16 pages (below that the
// merge costs more than the second round of pages); more splits than choose_splits() would take never happen (the workspace is
// sized for those).
int attn_dense(const tsb200_kv_desc* kv, const void* q, void* out, int dtype, int64_t qs, int64_t B, int H, float sm_scale,
               int64_t max_seq_len, float* ws, int* counters, cudaStream_t s) {
  int S = choose_splits(B, kv->hkv, max_seq_len);
  const int64_t cap = (max_seq_len + 255) / 256;
  if (S > cap) S = (int)(cap < 1 ? 1 : cap);
  if (!last_cta_merges(S, H, kv->hkv)) counters = nullptr;
#define TSB_GO(TT, PP)                                                                                                       \
  return kv->head_dim == 64 ? launch_dense<TT, PP, 64>(*kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, counters, out, s)    \
                            : launch_dense<TT, PP, 128>(*kv, q, qs, H, sm_scale, max_seq_len, S, B, ws, counters, out, s)
  if (kv->format == TSB200_KV_F32) {
    if (dtype == TSB200_F32) { TSB_GO(float, float); }
    TSB_GO(__nv_bfloat16, float);
  }
  if (dtype == TSB200_F32) { TSB_GO(float, __nv_bfloat16); }
  TSB_GO(__nv_bfloat16, __nv_bfloat16);
#undef TSB_GO
}

}  // namespace tsb
