// Shared pieces of the paged decode-attention kernels: split bookkeeping, the partial
// (m, l, acc) workspace layout and the cross-split reduction.
#pragma once
#include "common.cuh"

namespace tsb {

// Workspace: kAttnCounterBytes of int32 counters (zero between calls; one per (sequence, kv head,
// head chunk), used by the kernel of unquantized pages to let the last split merge the partials), then
// float [B][H][S][2 + d]  ->  m, l, acc[d] per (sequence, q head, split).
constexpr size_t kAttnCounterBytes = 16384;
// The last int32 of the counter block is a status word: a kernel that gave up on a bounded wait for its own
// copies records a non-zero code there (the result of that call is then not to be trusted).
constexpr int kAttnStatusIndex = (int)(kAttnCounterBytes / sizeof(int)) - 1;
// Whether an attention may start while the launch before it drains: it looks up lengths, block table and scales ahead of its wait.
inline bool attn_overlaps(const tsb200_kv_desc& kv) { return g_pdl != 0 && !(kv.flags & TSB200_KV_FRESH); }

inline int choose_splits(int64_t B, int hkv, int64_t max_seq_len) {
  const int64_t base = B * hkv;
  const int64_t pages = (max_seq_len + 15) / 16;
  int64_t s = (148 * 8 + base - 1) / (base > 0 ? base : 1);
  // few (sequence, kv head) pairs, long contexts: about 768 CTAs.  Fitted while the last CTA merged the splits and an SM held four CTAs (8 sequences x
  // 4 kv heads x 32k tokens, NVFP4 pages: 24 splits 99 us, 37 splits 115 us, 13 splits 128 us) and not since: 768 are 1.04 to 1.7 waves of
  // the 740 to 444 that fit now.  Another number would change the order of the sums.
  if (base > 0 && base < 148) {
    s = (768 + base - 1) / base;
  } else if (s >= 3) {
    // a power of two measured fastest (int8 / NVFP4 pages, 4k-32k tokens: 32 x 8 pairs 4 splits against 5: 5 % faster at
    // 4k; 64 x 8 pairs 4 against 3: 3-6 %; 128 x 8 pairs 2 stays): the nearest one
    int64_t p2 = 1;
    while (2 * p2 <= s) p2 *= 2;
    s = (2 * s >= 3 * p2) ? 2 * p2 : p2;
  }
  const int64_t cap = pages / 4 > 0 ? pages / 4 : 1;   // at least 4 pages per split
  if (s > cap) s = cap;
  if (s < 1) s = 1;
  if (s > 64) s = 64;
  return (int)s;
}

// Split count of the fp8-MMA kernel.  Two 6-warp CTAs fit an SM (296 slots): with that many (sequence, kv head)
// pairs or more, one split each is fastest (a second wave of CTAs costs more than it saves); below that the pairs
// are split so that the grid fills the slots without spilling into a second wave, each split keeping at least
// 24 pages (two page pairs per warp) to amortise the per-CTA query expansion and merge.
inline int choose_splits_fp8(int64_t B, int hkv, int64_t max_seq_len) {
  const int64_t base = B * hkv;
  const int64_t pages = (max_seq_len + 15) / 16;
  int64_t s = base > 0 ? 296 / base : 1;
  // two splits pay from about 1.5k tokens on (128 pairs: 1k tokens 18.8 us against 17.2 us for one split, 2k 25.9 / 28.5,
  // 4k 38.9 / 50.9, 8k 64.0 / 94.2 - one split leaves every SM with a single CTA)
  if (s == 2 && pages < 96) s = 1;
  const int64_t cap = pages / 24 > 0 ? pages / 24 : 1;
  if (s > cap) s = cap;
  if (s < 1) s = 1;
  if (s > 64) s = 64;
  return (int)s;
}

// Whether the last CTA of a (sequence, kv head, head chunk) of unquantized pages merges its splits (the quantized formats: a cluster or
// the reduction launch).  That takes ~80 cycles per (head, split) row - 35 k
// cycles, 20 us, at 7 heads and 63 splits -, a reduction launch that is resident before the partials are complete ~3 us whatever the
// shape: the launch from 64 rows on.
inline bool last_cta_merges(int splits, int H, int hkv) { return splits == 1 || splits * (H / hkv < 8 ? H / hkv : 8) < 64; }

// Pages [begin, end) of sequence with `len` tokens handled by split s of S.
__device__ __forceinline__ void split_range(int len, int s, int S, int& begin, int& end) {
  const int pages = (len + 15) >> 4;
  const int per = (pages + S - 1) / S;
  begin = s * per;
  end = min(pages, begin + per);
}

__device__ __forceinline__ float e4m3_byte_to_f32(unsigned int c) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)c, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}
__device__ __forceinline__ float e2m1_nibble_to_f32(unsigned int c) {
  __half_raw h = __nv_cvt_fp4_to_halfraw((__nv_fp4_storage_t)(c & 15), __NV_E2M1);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// Dequantized K / V element (token slot t, element e) of one page record; slow path used
// by the CUDA-core kernel.  fp8 scale is applied by the caller.
template <int D>
__device__ __forceinline__ float dense_elem(const uint8_t* __restrict__ rec, int fmt, int t, int e) {
  if (fmt == TSB200_KV_F32) return reinterpret_cast<const float*>(rec)[t * D + e];
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(rec)[t * D + e]);
}
template <int D>
__device__ __forceinline__ float k_elem(const uint8_t* __restrict__ rec, int fmt, int t, int e) {
  if (fmt >= TSB200_KV_F32) return dense_elem<D>(rec, fmt, t, e);
  if (fmt == TSB200_KV_INT8)
    return (float)(int8_t)rec[t * D + e] * reinterpret_cast<const float*>(rec + 16 * D)[t];
  if (fmt == TSB200_KV_FP8) return e4m3_byte_to_f32(rec[t * D + e]);
  const unsigned b = rec[t * (D / 2) + (e >> 1)];
  return e2m1_nibble_to_f32(b >> ((e & 1) * 4)) * e4m3_byte_to_f32(rec[16 * (D / 2) + t * (D / 16) + (e >> 4)]);
}
template <int D>
__device__ __forceinline__ float v_elem(const uint8_t* __restrict__ rec, int fmt, int t, int e) {
  if (fmt >= TSB200_KV_F32) return dense_elem<D>(rec, fmt, t, e);
  if (fmt == TSB200_KV_INT8)
    return (float)(int8_t)rec[e * 16 + t] * reinterpret_cast<const float*>(rec + 16 * D)[t];
  if (fmt == TSB200_KV_FP8) return e4m3_byte_to_f32(rec[e * 16 + t]);
  const unsigned b = rec[(e >> 1) * 16 + t];
  return e2m1_nibble_to_f32(b >> ((e & 1) * 4)) * e4m3_byte_to_f32(rec[16 * (D / 2) + (e >> 4) * 16 + t]);
}

// Splits of quantized pages whose CTAs are a cluster (1, S, 1) merge through distributed shared memory: `part` = this
// split's partials ([heads][2 + D], shared memory), `out` = the heads' outputs.  The arithmetic is decode_attn_reduce_kernel's, in its order: the
// same bits, without its launch.  No CTA leaves while another one may still read its partials.
constexpr int kMaxCluster = 8;
__device__ __forceinline__ bool splits_are_cluster() {
  unsigned n;
  asm("mov.u32 %0, %%cluster_nctaid.y;\n" : "=r"(n));
  return n > 1;
}
template <typename T, int D>
__device__ __forceinline__ void merge_cluster(const float* part, int heads, int S, T* __restrict__ out) {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  const unsigned own = (unsigned)__cvta_generic_to_shared(part);
  for (int idx = (int)(blockIdx.y * blockDim.x + threadIdx.x); idx < heads * (D / 2); idx += S * (int)blockDim.x) {
    const int h = idx / (D / 2), e = idx % (D / 2) * 2;
    float2 ml[kMaxCluster], v[kMaxCluster];
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s)
      if (s < S) {
        unsigned a;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(own + h * (2 + D) * 4), "r"(s));
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(ml[s].x), "=f"(ml[s].y) : "r"(a) : "memory");
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v[s].x), "=f"(v[s].y) : "r"(a + (2 + e) * 4) : "memory");
      }
    float mm = -INFINITY, ll = 0.f, a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s)
      if (s < S) mm = fmaxf(mm, ml[s].x);
#pragma unroll
    for (int s = 0; s < kMaxCluster; ++s)
      if (s < S) {
        const float c = ml[s].x == -INFINITY ? 0.f : __expf(ml[s].x - mm);
        ll += ml[s].y * c;
        a0 += v[s].x * c;
        a1 += v[s].y * c;
      }
    out[h * D + e] = from_f32<T>(ll > 0.f ? a0 / ll : 0.f);
    out[h * D + e + 1] = from_f32<T>(ll > 0.f ? a1 / ll : 0.f);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Clusters (1, S, 1) of `kernel` that the device holds at a time (0: none).  `cache`: of one instance and device, by S; 0 = not asked yet.
template <typename K>
inline int active_clusters(K* kernel, dim3 grid, int threads, size_t smem, int (&cache)[kMaxCluster + 1]) {
  if (cache[grid.y]) return cache[grid.y] - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = grid.y;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  cache[grid.y] = n + 1;
  return n;
}

// Launch of grid (pairs, S, chunks); `clusters`: one per (pair, chunk), its CTAs merge the splits themselves.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_splits(bool overlap, bool clusters, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (overlap) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (clusters) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1;
    attr[n].val.clusterDim.y = grid.y;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// The last CTA of a (sequence, kv head, head chunk) merges its S partials, in split order:
//   out[h][e] = sum_s acc_s[e] c_s / sum_s l_s c_s,  c_s = exp(m_s - max m).
// `part` = partials of the chunk's first head ([heads][S][2 + D], consecutive), `out` = its outputs, `sm` = shared scratch of
// 2 heads * S + heads floats.  Bound by the round trips to partials that other SMs have just written: every (m, l) is fetched
// once, all in flight together (it was two dependent loads per split and output element: 75 us of an 83 us launch at 63 splits,
// batch 1, 7 heads), the coefficients come from shared memory, and kFly partials of an element pair are in flight at once.
template <typename T, int D>
__device__ __forceinline__ void merge_splits(const float* __restrict__ part, int heads, int S, float* sm, T* __restrict__ out) {
  constexpr int kFly = 16;
  float* sc = sm;                                     // [heads][S] m, then c
  float* sl = sm + heads * S;                         // [heads][S] l
  float* ssum = sl + heads * S;                       // [heads]
  for (int i = threadIdx.x; i < heads * S; i += blockDim.x) {
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(part + (size_t)i * (2 + D)));
    sc[i] = ml.x;
    sl[i] = ml.y;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int h = warp; h < heads; h += blockDim.x >> 5) {
    float mm = -INFINITY;
    for (int s = lane; s < S; s += 32) mm = fmaxf(mm, sc[h * S + s]);
    mm = warp_max(mm);
    for (int s = lane; s < S; s += 32) {
      const float ms = sc[h * S + s];
      sc[h * S + s] = ms == -INFINITY ? 0.f : __expf(ms - mm);
    }
    __syncwarp();
    if (lane == 0) {
      float ll = 0.f;
      for (int s = 0; s < S; ++s) ll += sl[h * S + s] * sc[h * S + s];
      ssum[h] = ll;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < heads * (D / 2); i += blockDim.x) {
    const int h = i / (D / 2), e = i % (D / 2) * 2;
    const float* p = part + (size_t)h * S * (2 + D) + 2 + e;
    const float* c = sc + h * S;
    float a0 = 0.f, a1 = 0.f;
    for (int s0 = 0; s0 < S; s0 += kFly) {
      float2 v[kFly];
#pragma unroll
      for (int u = 0; u < kFly; ++u)
        if (s0 + u < S) v[u] = __ldcg(reinterpret_cast<const float2*>(p + (size_t)(s0 + u) * (2 + D)));
#pragma unroll
      for (int u = 0; u < kFly; ++u)
        if (s0 + u < S) {
          a0 += v[u].x * c[s0 + u];
          a1 += v[u].y * c[s0 + u];
        }
    }
    const float ll = ssum[h];
    out[h * D + e] = from_f32<T>(ll > 0.f ? a0 / ll : 0.f);
    out[h * D + e + 1] = from_f32<T>(ll > 0.f ? a1 / ll : 0.f);
  }
}

// Merges partials (decode_attn_simt.cu), chained to the attention launch.
template <typename T, int D> int launch_reduce(const float* ws, int64_t BH, int S, void* out, cudaStream_t st);
int validate_kv(const tsb200_kv_desc* kv, bool need_table);

}  // namespace tsb
