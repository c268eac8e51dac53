// Span means and scores of the cocktail-party head (model.py:258-296): for every row, the j-th [SPAN] token is
// paired with the j-th [ES] token, h_spans[b, j] = mean(x[b, st+1 : ed]) (zero when the pair is
// missing or st + 1 >= ed) and scores[b, j] = <x[b, first [MASK]], h_spans[b, j]>. The reference finds the markers with
// .nonzero() and walks the pairs in a Python loop over rows and spans; here
//   span_index_kernel      ranks the markers of a row with warp ballots and writes their positions,
//   cocktail_scores_kernel one CTA per (span, row): means and dot product from one read of the span's tokens,
//   cocktail_grad_kernel   one CTA per (32 tokens, row) and some for the [MASK]'s: the whole gradient, written once,
//   span_mean_fwd / _bwd   the means alone and their gradient (span_means).
// All are bound by HBM traffic; the gradient writes every token's row, of which most are zero.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "sm100_prims.cuh"

namespace kd {

constexpr int CK_THREADS = 256, CK_SCORE_THREADS = 512, CK_TOKENS = 32;

// positions of the r-th [SPAN] / [ES] of every row (-1 beyond the row's count), the row's [SPAN] and [ES] counts
// and the position of its first [MASK] (-1 if none); one CTA per row. counts_host, if given, receives the [SPAN] counts as
// well (pinned host memory, so that the caller needs no copy).
// Bound by the latency of a row's token loads: a warp takes 128 tokens of a chunk of 4096 with four loads in flight, and
// the tokens are read once (eight warps that walked the row 32 tokens at a time, twice, took 14 us at T = 4096).
constexpr int SI_THREADS = 1024, SI_WARPS = SI_THREADS / 32, SI_PER = 4, SI_CHUNK = SI_THREADS * SI_PER;
__global__ void __launch_bounds__(SI_THREADS)
span_index_kernel(const int64_t* __restrict__ tokens, int64_t stride_b, int T, int64_t tok_span, int64_t tok_es,
                  int64_t tok_mask, int32_t* __restrict__ starts, int32_t* __restrict__ ends, int32_t* __restrict__ n_starts,
                  int32_t* __restrict__ n_ends, int32_t* __restrict__ first_mask, int32_t* __restrict__ counts_host) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int s_span[SI_WARPS], s_es[SI_WARPS], s_mask[SI_WARPS];
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t* x = tokens + (size_t)b * stride_b;
  int32_t *row_st = starts + (size_t)b * T, *row_en = ends + (size_t)b * T;
  const uint32_t below = (1u << lane) - 1u;
  int c_span = 0, c_es = 0, first = T;   // of the chunks before
  for (int base = 0; base < T; base += SI_CHUNK) {
    const int t0 = base + warp * (32 * SI_PER) + lane;
    int64_t v[SI_PER];
#pragma unroll
    for (int r = 0; r < SI_PER; ++r) v[r] = t0 + 32 * r < T ? x[t0 + 32 * r] : 0;
    uint32_t bs[SI_PER], be[SI_PER];
    int n_span = 0, n_es = 0, fm = T;
#pragma unroll
    for (int r = 0; r < SI_PER; ++r) {
      const bool in = t0 + 32 * r < T;
      bs[r] = __ballot_sync(0xffffffffu, in && v[r] == tok_span);
      be[r] = __ballot_sync(0xffffffffu, in && v[r] == tok_es);
      const uint32_t bm = __ballot_sync(0xffffffffu, in && v[r] == tok_mask);
      if (bm != 0u && fm == T) fm = t0 - lane + 32 * r + __ffs(bm) - 1;
      n_span += __popc(bs[r]);
      n_es += __popc(be[r]);
    }
    if (lane == 0) { s_span[warp] = n_span; s_es[warp] = n_es; s_mask[warp] = fm; }
    __syncthreads();
    // every warp: totals of the chunk and of the warps before it
    const int w_span = s_span[lane], w_es = s_es[lane];
    const int tot_span = __reduce_add_sync(0xffffffffu, w_span), tot_es = __reduce_add_sync(0xffffffffu, w_es);
    int p_span = c_span + __reduce_add_sync(0xffffffffu, lane < warp ? w_span : 0);
    int p_es = c_es + __reduce_add_sync(0xffffffffu, lane < warp ? w_es : 0);
    first = min(first, __reduce_min_sync(0xffffffffu, s_mask[lane]));
    // the count is what the host waits for: it leaves as soon as it is known
    if (counts_host != nullptr && threadIdx.x == 0 && base + SI_CHUNK >= T) *const_cast<volatile int32_t*>(counts_host + b) = c_span + tot_span;
#pragma unroll
    for (int r = 0; r < SI_PER; ++r) {
      if ((bs[r] >> lane) & 1u) row_st[p_span + __popc(bs[r] & below)] = t0 + 32 * r;
      if ((be[r] >> lane) & 1u) row_en[p_es + __popc(be[r] & below)] = t0 + 32 * r;
      p_span += __popc(bs[r]);
      p_es += __popc(be[r]);
    }
    c_span += tot_span;
    c_es += tot_es;
    __syncthreads();   // the counts in shared memory are free for the next chunk
  }
  for (int r = c_span + threadIdx.x; r < T; r += SI_THREADS) row_st[r] = -1;
  for (int r = c_es + threadIdx.x; r < T; r += SI_THREADS) row_en[r] = -1;
  if (threadIdx.x == 0) {
    n_starts[b] = c_span;
    n_ends[b] = c_es;
    first_mask[b] = first < T ? first : -1;
  }
}

template <typename E> __device__ __forceinline__ float to_f(E v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename E> __device__ __forceinline__ E from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// the pair j of row b: true when it exists and holds at least one token between its markers
__device__ __forceinline__ bool span_pair(const int32_t* starts, const int32_t* ends, const int32_t* n_starts,
                                          const int32_t* n_ends, int b, int j, int T, int& st, int& ed) {
  if (j >= min(n_starts[b], n_ends[b])) return false;   // zip() of the reference stops at the shorter list
  st = starts[(size_t)b * T + j];
  ed = ends[(size_t)b * T + j];
  return st + 1 < ed;
}

// V consecutive elements as floats and back: one 16-byte access for V = 16 / sizeof(E)
template <typename E, int V> struct Vec;
template <typename E> struct Vec<E, 1> {
  static __device__ __forceinline__ void load(const E* p, float (&f)[1]) { f[0] = to_f<E>(*p); }
  static __device__ __forceinline__ void store(E* p, const float (&f)[1]) { *p = from_f<E>(f[0]); }
};
template <> struct Vec<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
};
template <typename E> struct Vec<E, 8> {
  static __device__ __forceinline__ void load(const E* p, float (&f)[8]) {
    uint4 v = *reinterpret_cast<const uint4*>(p);
    const E* e = reinterpret_cast<const E*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = to_f<E>(e[i]);
  }
  static __device__ __forceinline__ void store(E* p, const float (&f)[8]) {
    uint4 v;
    E* e = reinterpret_cast<E*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = from_f<E>(f[i]);
    *reinterpret_cast<uint4*>(p) = v;
  }
};

// scores[b, j] = <x[b, first_mask, :], mean over t in (st, ed) of x[b, t, :]>; grid (S, B).
// h, if given, keeps what the gradient needs in fp32: rows 0 .. S-1 of a batch row are the means, row S the embedding at
// the [MASK] (zero without one). `tpr` threads (a power of two) share a token's row, V columns each; the other
// blockDim / tpr groups take further tokens, so that a span of 100 tokens is a few dependent loads.
template <typename E, int V>
__global__ void __launch_bounds__(CK_SCORE_THREADS)
cocktail_scores_kernel(const E* __restrict__ x, int64_t x_sb, int64_t x_st, int T, int C, int S, int tpr,
                       const int32_t* __restrict__ starts, const int32_t* __restrict__ ends, const int32_t* __restrict__ n_starts,
                       const int32_t* __restrict__ n_ends, const int32_t* __restrict__ first_mask, E* __restrict__ scores,
                       float* __restrict__ h) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float part[CK_SCORE_THREADS * V];   // [group][column of the chunk]
  __shared__ float s_dot[CK_SCORE_THREADS / 32];
  const int j = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int groups = blockDim.x / tpr, g = tid / tpr, cols = tpr * V, mine = (tid - g * tpr) * V;
  int st = 0, ed = 0;
  const bool live = span_pair(starts, ends, n_starts, n_ends, b, j, T, st, ed);
  const float inv = live ? 1.f / static_cast<float>(ed - st - 1) : 0.f;
  const int fm = first_mask[b];
  const E* rows = x + (size_t)b * x_sb;
  float* hb = h == nullptr ? nullptr : h + (size_t)b * (S + 1) * C;
  float dot = 0.f;
  for (int c0 = 0; c0 < C; c0 += cols) {
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
    if (live && c0 + mine < C) {
      const E* col = rows + c0 + mine;
#pragma unroll 4
      for (int t = st + 1 + g; t < ed; t += groups) {
        float f[V];
        Vec<E, V>::load(col + (size_t)t * x_st, f);
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] += f[i];
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) part[g * cols + mine + i] = acc[i];
    __syncthreads();
    for (int c = tid; c < cols && c0 + c < C; c += blockDim.x) {
      float sum = 0.f;
      for (int k = 0; k < groups; ++k) sum += part[k * cols + c];
      const float mean = sum * inv, ctx = fm >= 0 ? to_f<E>(rows[(size_t)fm * x_st + c0 + c]) : 0.f;
      dot = fmaf(mean, ctx, dot);
      if (hb != nullptr) {
        hb[(size_t)j * C + c0 + c] = mean;
        if (j == 0) hb[(size_t)S * C + c0 + c] = ctx;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if ((tid & 31) == 0) s_dot[tid >> 5] = dot;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < static_cast<int>(blockDim.x) / 32; ++w) dot += s_dot[w];
    scores[(size_t)b * S + j] = from_f<E>(dot);
  }
}

// The coefficient of token t: the sum over the pairs covering it of ds_j / len_j. Starts and ends both ascend, so these pairs are the
// range [number of ends <= t, number of starts < t), found by two binary searches. False: no pair covers the token (a coefficient of
// zero does not say that: 0 times an infinity is not 0).
template <typename E>
__device__ __forceinline__ bool coefficient(const E* row_ds, const int32_t* row_st, const int32_t* row_en, int n, int t, float& c) {
  int lo = 0, hi = n, lo2 = 0, hi2 = n;   // both searches advance together: their loads overlap
  while (lo < hi || lo2 < hi2) {
    const int m = (lo + hi) >> 1, m2 = (lo2 + hi2) >> 1;
    const int en = lo < hi ? row_en[m] : 0, st = lo2 < hi2 ? row_st[m2] : 0;
    if (lo < hi) { if (en <= t) lo = m + 1; else hi = m; }
    if (lo2 < hi2) { if (st < t) lo2 = m2 + 1; else hi2 = m2; }
  }
  c = 0.f;
  for (int j = lo; j < lo2; ++j) c += to_f<E>(row_ds[j]) / static_cast<float>(row_en[j] - row_st[j] - 1);
  return lo < lo2;
}

// Gradient of the scores with respect to x; grid (ceil(C / CK_THREADS) + ceil(T / CK_TOKENS), B).
//   gx[b, t, :] = h_ctx * sum over the pairs covering t of ds_j / len_j   (+ sum_j ds_j h_j where t is the [MASK])
// Every pair multiplies the same h_ctx, so a token needs one coefficient: gx is written once, 16 bytes a store, and
// nothing but the [MASK]'s row reads the means. That row has the first CTAs to itself, a column per thread: walked by the CTA of its
// 32 tokens, between their stores, its chain of dependent loads made the kernel 30.6 us instead of 22.3 (16 x 4096 x 1024 bf16:
// 134 MB at 6.0 TB/s, as fast as a plain write; float32 48.8 -> 42.8, 4 x 1000 x 768 5.5 -> 4.2).
template <typename E, int V>
__global__ void __launch_bounds__(CK_THREADS)
cocktail_grad_kernel(const E* __restrict__ ds, const float* __restrict__ h, int S, int T, int C, int tpr,
                     const int32_t* __restrict__ starts, const int32_t* __restrict__ ends, const int32_t* __restrict__ n_starts,
                     const int32_t* __restrict__ n_ends, const int32_t* __restrict__ first_mask, E* __restrict__ gx) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float coef[CK_TOKENS];
  __shared__ bool covered[CK_TOKENS];
  const int mask_ctas = (C + CK_THREADS - 1) / CK_THREADS, block = static_cast<int>(blockIdx.x) - mask_ctas;
  const int b = blockIdx.y, tb = block * CK_TOKENS, tid = threadIdx.x;
  const int n = min(min(n_starts[b], n_ends[b]), S), fm = first_mask[b];
  const int32_t *row_st = starts + (size_t)b * T, *row_en = ends + (size_t)b * T;
  const E* row_ds = ds + (size_t)b * S;
  const float* hb = h + (size_t)b * (S + 1) * C;
  if (block < 0) {   // the [MASK]'s row
    const int c = static_cast<int>(blockIdx.x) * CK_THREADS + tid;
    if (fm < 0 || c >= C) return;
    float w, f = 0.f;
    if (coefficient<E>(row_ds, row_st, row_en, n, fm, w)) f = w * hb[(size_t)S * C + c];
#pragma unroll 8
    for (int j = 0; j < n; ++j) f = fmaf(to_f<E>(row_ds[j]), hb[(size_t)j * C + c], f);
    for (int j = n; j < S; ++j) f += 0.f * to_f<E>(row_ds[j]);   // the row's missing pairs, whose means are zero: what their gradients may add is a NaN
    gx[((size_t)b * T + fm) * C + c] = from_f<E>(f);
    return;
  }
  if (tid < CK_TOKENS) {
    float c;
    covered[tid] = coefficient<E>(row_ds, row_st, row_en, n, tb + tid, c);
    coef[tid] = c;
  }
  const int groups = CK_THREADS / tpr, g = tid / tpr, cols = tpr * V, mine = (tid - g * tpr) * V;
  __syncthreads();
  for (int c = mine; c < C; c += cols) {
    float ctx[V];
#pragma unroll
    for (int i = 0; i < V; ++i) ctx[i] = hb[(size_t)S * C + c + i];
    for (int k = g; k < CK_TOKENS && tb + k < T; k += groups) {
      if (tb + k == fm) continue;
      const float w = coef[k];
      float f[V];
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = covered[k] ? w * ctx[i] : 0.f;
      Vec<E, V>::store(gx + ((size_t)b * T + tb + k) * C + c, f);
    }
  }
}

// h[b, j, :] = mean over t in (st, ed) of x[b, t, :]; grid (S, B)
template <typename E>
__global__ void __launch_bounds__(CK_THREADS)
span_mean_fwd_kernel(const E* __restrict__ x, int64_t x_sb, int64_t x_st, int T, int C, const int32_t* __restrict__ starts,
                     const int32_t* __restrict__ ends, const int32_t* __restrict__ n_starts,
                     const int32_t* __restrict__ n_ends, E* __restrict__ h, int S) {
  pdl_wait();
  pdl_launch_dependents();
  const int j = blockIdx.x, b = blockIdx.y;
  int st = 0, ed = 0;
  const bool live = span_pair(starts, ends, n_starts, n_ends, b, j, T, st, ed);
  E* out = h + ((size_t)b * S + j) * C;
  const float inv = live ? 1.f / static_cast<float>(ed - st - 1) : 0.f;
  for (int c = threadIdx.x; c < C; c += CK_THREADS) {   // consecutive threads read consecutive columns
    float acc = 0.f;
    if (live) {
      const E* col = x + (size_t)b * x_sb + c;
      for (int t = st + 1; t < ed; ++t) acc += to_f<E>(col[(size_t)t * x_st]);
    }
    out[c] = from_f<E>(acc * inv);
  }
}

// grad_x[b, t, :] = sum_j [st_j < t < ed_j] grad_h[b, j, :] / (ed_j - st_j - 1); grid (ceil(T / 8), B)
template <typename E>
__global__ void __launch_bounds__(CK_THREADS)
span_mean_bwd_kernel(const E* __restrict__ gh, int S, int T, int C, const int32_t* __restrict__ starts,
                     const int32_t* __restrict__ ends, const int32_t* __restrict__ n_starts,
                     const int32_t* __restrict__ n_ends, E* __restrict__ gx, int64_t gx_sb, int64_t gx_st) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int TT = 8;
  const int b = blockIdx.y, tb = blockIdx.x * TT;
  const int n = min(min(n_starts[b], n_ends[b]), S);
  for (int tt = 0; tt < TT; ++tt) {
    const int t = tb + tt;
    if (t >= T) break;
    // pairs that cover t: none for most tokens, one for canonical data (the same for the whole CTA)
    int covers = 0, j0 = 0;
    for (int j = 0; j < n; ++j) {
      const int st = starts[(size_t)b * T + j], ed = ends[(size_t)b * T + j];
      if (st < t && t < ed) { if (covers == 0) j0 = j; ++covers; }
    }
    E* dst = gx + (size_t)b * gx_sb + (size_t)t * gx_st;
    if (covers == 0) {
      for (int c = threadIdx.x; c < C; c += CK_THREADS) dst[c] = from_f<E>(0.f);
    } else {
      for (int c = threadIdx.x; c < C; c += CK_THREADS) {
        float acc = 0.f;
        for (int j = j0; j < n; ++j) {
          const int st = starts[(size_t)b * T + j], ed = ends[(size_t)b * T + j];
          if (st < t && t < ed) acc += to_f<E>(gh[((size_t)b * S + j) * C + c]) / static_cast<float>(ed - st - 1);
          if (covers == 1) break;   // j0 was the only one
        }
        dst[c] = from_f<E>(acc);
      }
    }
  }
}

int launch_span_index(const int64_t* tokens, int64_t stride_b, int B, int T, int64_t tok_span, int64_t tok_es,
                      int64_t tok_mask, int32_t* starts, int32_t* ends, int32_t* n_starts, int32_t* n_ends,
                      int32_t* first_mask, int32_t* counts_host, cudaStream_t stream) {
  if (B == 0 || T == 0) return 0;
  const cudaError_t e = launch(span_index_kernel, B, SI_THREADS, 0, stream, tokens, stride_b, T, tok_span, tok_es, tok_mask, starts, ends, n_starts,
                                                  n_ends, first_mask, counts_host);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "span_index_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

// threads that share a row of C columns, V each: a power of two of at most `most`
static int threads_per_row(int C, int V, int most) {
  int tpr = 1;
  while (tpr * V < C && tpr < most) tpr *= 2;
  return tpr;
}

template <typename E, int V>
static cudaError_t scores_t(const kd_cocktail& p, cudaStream_t stream) {
  const int tpr = threads_per_row(p.C, V, CK_SCORE_THREADS);
  const int threads = std::min(CK_SCORE_THREADS, std::max(32, tpr * 32));   // at most 32 groups: they are added up one by one
  return launch(cocktail_scores_kernel<E, V>, dim3(p.S, p.B), threads, 0, stream,
      static_cast<const E*>(p.x), p.x_sb, p.x_st, p.T, p.C, p.S, tpr, p.starts, p.ends, p.n_starts, p.n_ends, p.first_mask,
      static_cast<E*>(p.scores), p.h);
}
template <typename E, int V>
static cudaError_t grad_t(const kd_cocktail& p, cudaStream_t stream) {
  return launch(cocktail_grad_kernel<E, V>, dim3((p.C + CK_THREADS - 1) / CK_THREADS + (p.T + CK_TOKENS - 1) / CK_TOKENS, p.B), CK_THREADS, 0, stream,
      static_cast<const E*>(p.scores), p.h, p.S, p.T, p.C, threads_per_row(p.C, V, CK_THREADS), p.starts, p.ends, p.n_starts, p.n_ends,
      p.first_mask, static_cast<E*>(p.gx));
}

// 16-byte accesses need rows that begin on 16 bytes; other widths and strides go element by element
int launch_cocktail(bool backward, const kd_cocktail& p, cudaStream_t stream) {
  const int es = p.dtype == KD_F32 ? 4 : 2, V = 16 / es;
  const bool wide = p.C % V == 0 && (backward ? reinterpret_cast<uintptr_t>(p.gx) % 16 == 0
                                              : reinterpret_cast<uintptr_t>(p.x) % 16 == 0 && p.x_sb % V == 0 && p.x_st % V == 0);
  auto run = [&](auto e, auto v) {
    using E = decltype(e);
    constexpr int W = decltype(v)::value;
    return backward ? grad_t<E, W>(p, stream) : scores_t<E, W>(p, stream);
  };
  using One = std::integral_constant<int, 1>;
  using Four = std::integral_constant<int, 4>;
  using Eight = std::integral_constant<int, 8>;
  const cudaError_t e = p.dtype == KD_F32   ? (wide ? run(float(), Four()) : run(float(), One()))
                        : p.dtype == KD_F16 ? (wide ? run(__half(), Eight()) : run(__half(), One()))
                                            : (wide ? run(__nv_bfloat16(), Eight()) : run(__nv_bfloat16(), One()));
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "cocktail kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

template <typename E>
static int span_mean_t(bool backward, const void* a, int64_t a_sb, int64_t a_st, void* out, int64_t o_sb, int64_t o_st, int B,
                       int T, int C, int S, const int32_t* starts, const int32_t* ends, const int32_t* n_starts,
                       const int32_t* n_ends, cudaStream_t stream) {
  const cudaError_t e =
      backward ? launch(span_mean_bwd_kernel<E>, dim3((T + 7) / 8, B), CK_THREADS, 0, stream, static_cast<const E*>(a), S, T, C, starts, ends, n_starts,
                        n_ends, static_cast<E*>(out), o_sb, o_st)
               : launch(span_mean_fwd_kernel<E>, dim3(S, B), CK_THREADS, 0, stream, static_cast<const E*>(a), a_sb, a_st, T, C, starts, ends, n_starts,
                        n_ends, static_cast<E*>(out), S);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "span_mean kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

int launch_span_mean(bool backward, const void* a, int64_t a_sb, int64_t a_st, void* out, int64_t o_sb, int64_t o_st, int B,
                     int T, int C, int S, int dtype, const int32_t* starts, const int32_t* ends, const int32_t* n_starts,
                     const int32_t* n_ends, cudaStream_t stream) {
  if (B == 0 || S == 0 || C == 0 || (backward && T == 0)) return 0;
  if (dtype == KD_F16) return span_mean_t<__half>(backward, a, a_sb, a_st, out, o_sb, o_st, B, T, C, S, starts, ends, n_starts, n_ends, stream);
  if (dtype == KD_BF16) return span_mean_t<__nv_bfloat16>(backward, a, a_sb, a_st, out, o_sb, o_st, B, T, C, S, starts, ends, n_starts, n_ends, stream);
  if (dtype == KD_F32) return span_mean_t<float>(backward, a, a_sb, a_st, out, o_sb, o_st, B, T, C, S, starts, ends, n_starts, n_ends, stream);
  return set_error(KD_ERR_ARG, "dtype %d not supported", dtype);
}

}  // namespace kd
