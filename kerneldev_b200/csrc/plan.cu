// Plan construction (two kernels: token descriptors; exact 128x128 tile classification with the work lists; one for short sequences)
// and the dense-mask materialiser. Integer-only kernels; HBM traffic is a few hundred KB.
#include "common.cuh"
#include "mask_rule.cuh"
#include "sm100_prims.cuh"

namespace kd {

// ---------------------------------------------------------------------------------------
// 1. pack: metadata -> descriptors + per-tile summaries
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ int tokens_of(const kd_meta& m, int b) { return m.lens != nullptr ? min(m.lens[b], m.T) : m.T; }
__device__ __forceinline__ bool out_of_range(int64_t sid) { return sid >= (1 << 23) || sid < -(1 << 23); }

// descriptor of token t of a sequence of n_b tokens
__device__ __forceinline__ uint32_t describe(const kd_meta& m, int b, int t, int n_b, bool& bad_id) {
  if (t >= n_b) return 0u;
  // no metadata: causal = every token is context; otherwise every token is prefix
  if (!m.rules) return pack_plain(m.causal != 0);
  const bool ins = m.in_span ? (m.in_span[b * m.in_span_stride_b + t] != 0) : false;
  const bool pre = m.is_prefix ? (m.is_prefix[b * m.is_prefix_stride_b + t] != 0) : false;
  const int64_t sid = m.span_id ? m.span_id[b * m.span_id_stride_b + t] : 0;
  bad_id = out_of_range(sid);
  return pack_token(ins, pre, sid, true);
}

// 128-bit class masks of a tile: bit t of mask k = descriptor bit k of token t (bits 0..2 = classes as a key, bits 5..7 = classes seen as
// a query, bit 4 = same-span armed); mask 7: span id out of range. Word w: from the warp that holds tokens 32 w ..
__device__ __forceinline__ void class_masks(uint32_t d, bool bad_id, int lane, int w, uint32_t* masks) {
  constexpr uint32_t src_bit[8] = {TD_PRE, TD_CTX, TD_INS, TD_PRE << TD_SEES_SHIFT, TD_CTX << TD_SEES_SHIFT,
                                   TD_INS << TD_SEES_SHIFT, TD_SIDPOS, 0u};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t bal = __ballot_sync(0xffffffffu, k < 7 ? (d & src_bit[k]) != 0u : bad_id);
    if (lane == 0) masks[k * 4 + w] = bal;
  }
}

// summary[b][tile] = { OR of flag bits, AND of flag bits, min span id, max span id } where
// the span id range is taken over the in_span tokens of the tile (sign-extended 24 bit).
__global__ void __launch_bounds__(KD_TILE) pack_kernel(kd_meta m, PlanView pv) {
  const int tile = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int t = tile * KD_TILE + tid;
  pdl_wait();
  pdl_launch_dependents();
  if (tile == 0 && b == 0 && tid == 0) {
    *pv.status = 0u;   // raised by the next kernel at the earliest
    *reinterpret_cast<uint32_t**>(pv.status + 2) = m.status_mirror;
  }
  bool bad_id = false;
  const uint32_t d = describe(m, b, t, tokens_of(m, b), bad_id);
  pv.desc[(size_t)b * pv.Tpad + t] = d;
  class_masks(d, bad_id, tid & 31, tid >> 5, pv.tilebits + ((size_t)b * pv.NT + tile) * 32);

  uint32_t f_or = d & TD_FLAGS, f_and = d & TD_FLAGS;
  int32_t smin = INT32_MAX, smax = INT32_MIN;
  if (d & TD_INS) {
    const int32_t s = static_cast<int32_t>(d) >> TD_SID_SHIFT;  // arithmetic shift sign-extends
    smin = s;
    smax = s;
  }
  for (int o = 16; o > 0; o >>= 1) {
    f_or |= __shfl_xor_sync(0xffffffffu, f_or, o);
    f_and &= __shfl_xor_sync(0xffffffffu, f_and, o);
    smin = min(smin, __shfl_xor_sync(0xffffffffu, smin, o));
    smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, o));
  }
  __shared__ uint32_t s_or[4], s_and[4];
  __shared__ int32_t s_min[4], s_max[4];
  if ((tid & 31) == 0) {
    s_or[tid >> 5] = f_or;
    s_and[tid >> 5] = f_and;
    s_min[tid >> 5] = smin;
    s_max[tid >> 5] = smax;
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t* out = pv.summary + ((size_t)b * pv.NT + tile) * 4;
    out[0] = s_or[0] | s_or[1] | s_or[2] | s_or[3];
    out[1] = s_and[0] & s_and[1] & s_and[2] & s_and[3];
    out[2] = static_cast<uint32_t>(min(min(s_min[0], s_min[1]), min(s_min[2], s_min[3])));
    out[3] = static_cast<uint32_t>(max(max(s_max[0], s_max[1]), max(s_max[2], s_max[3])));
    if (tile == 0) {
      pv.stats[b * 2 + 0] = 0;
      pv.stats[b * 2 + 1] = 0;
      pv.done[b] = 0;
      pv.len[b] = tokens_of(m, b);
    }
  }
}

// ---------------------------------------------------------------------------------------
// 2. classify and lists: one CTA per (b, pair of query tiles) and per (b, key tile)
// ---------------------------------------------------------------------------------------
// Tiles whose 128 query tokens share one flag combination and whose 128 key tokens share one
// are decided from the summaries; everything else is decided by evaluating the rule on all
// 128x128 pairs. Both routes give the exact reduction of the dense mask.
//
// A CTA classifies the tiles of its row pair (or of its column) and writes their list at once, so every tile is
// classified twice; in exchange the lists need no kernel of their own that walks the classes serially. The last CTA of a
// sequence sorts its items. All of it is latency: a step on 8 x 2048 tokens spent 21 us in a memset and three kernels, of
// which the serial lists took 8, and evaluating a tile pair by pair 5 (now a row's 128 bits are a few word operations).
// The pairs' CTAs also write the bits of their PARTIAL tiles, which the attention kernels mask with (0.1-1.5 us of a plan; each kernel
// and head formed them anew before, up to a tenth of a forward).
constexpr int CL_THREADS = 512, CL_WARPS = CL_THREADS / 32;

// exact class of tile (qt, kt) from all its pairs; one warp
// (desc, tilebits: of the sequence; words: null, or where a PARTIAL tile's bits go)
__device__ __forceinline__ int classify_exact(const uint32_t* desc, const uint32_t* tilebits, int qt, int kt, int lane, uint32_t* words) {
  const uint32_t *dq = desc + qt * KD_TILE, *dk = desc + kt * KD_TILE, *tb = tilebits + kt * 32;
  uint32_t pre[4], ctx[4], ins[4], kd[4], qd[4];
  uint32_t any_ins = 0u;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    pre[w] = tb[TB_PRE * 4 + w];
    ctx[w] = tb[TB_CTX * 4 + w];
    ins[w] = tb[TB_INS * 4 + w];
    any_ins |= ins[w];
    kd[w] = dk[w * 32 + lane];
    qd[w] = dq[w * 32 + lane];
  }
  uint32_t on = 0u, off = 0u, m[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    uint32_t (&mk)[4] = m[r];
    query_row_mask<4>(qd[r], qt * KD_TILE + r * 32 + lane, kt * KD_TILE, pre, ctx, ins, mk);
    add_same_span<4>(qd[r], any_ins != 0u, kd, mk);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      on |= mk[w];
      off |= ~mk[w];
    }
  }
  const bool w_on = __any_sync(0xffffffffu, on != 0u), w_off = __any_sync(0xffffffffu, off != 0u);
  if (words != nullptr && w_on && w_off) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int w = 0; w < 4; ++w) words[w * KD_TILE + r * 32 + lane] = m[r][w];
  }
  return w_on ? (w_off ? KD_TILE_PARTIAL : KD_TILE_FULL) : KD_TILE_EMPTY;
}

// class of tile (qt, kt) from the summaries of the two runs of tokens, or -1
__device__ __forceinline__ int classify_summary(uint4 q, uint4 k, int qt, int kt) {
  if (q.x == 0u || k.x == 0u) return KD_TILE_EMPTY;   // all queries or all keys are beyond the sequence length
  if (q.x != q.y || k.x != k.y) return -1;
  // flags only; the span id is handled below
  if (k.x & sees_of_flags(q.x)) return KD_TILE_FULL;
  if ((k.x & q.x & TD_CTX) != 0u) return qt > kt ? KD_TILE_FULL : (qt < kt ? KD_TILE_EMPTY : KD_TILE_PARTIAL);
  if ((q.x & TD_SIDPOS) && (k.x & TD_INS)) {
    const int32_t qmin = (int32_t)q.z, qmax = (int32_t)q.w, kmin = (int32_t)k.z, kmax = (int32_t)k.w;
    if (qmin == qmax && kmin == kmax) return (qmin == kmin) ? KD_TILE_FULL : KD_TILE_EMPTY;
    return (qmax < kmin || kmax < qmin) ? KD_TILE_EMPTY : -1;   // disjoint id ranges
  }
  return KD_TILE_EMPTY;
}

// places item t of n by decreasing count in row `kind` of the sequence's orders
__device__ __forceinline__ void order_item(const int* cnt, int kind, int t, int n, uint8_t* order, int NT) {
  if (t >= n) return;
  const int mine = cnt[t];
  int rank = 0;
  for (int u = 0; u < n; ++u) rank += (cnt[u] > mine) || (cnt[u] == mine && u < t);
  order[kind * NT + rank] = static_cast<uint8_t>(t);
}

// forward list: per (b, pair p of query tiles 2p, 2p+1) the key tiles that are non-empty for either
// backward list: per (b, key tile) the query tiles that are non-empty
// order: per b, the pairs / query tiles / key tiles sorted by decreasing list length, so that the
//        kernels can schedule the longest work items first
__global__ void __launch_bounds__(CL_THREADS) classify_kernel(PlanView pv) {
  __shared__ uint4 s_sum[128];        // summaries of all tiles of the sequence
  __shared__ uint8_t s_cls[2][128];   // [query tile of the pair][key tile], or [0][query tile]
  __shared__ int s_cnt[3][128];
  __shared__ int s_last;
  const int item = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NT = pv.NT, NP = pv.NP;
  const bool is_pair = item < NP;
  pdl_wait();
  pdl_launch_dependents();
  for (int t = tid; t < NT; t += CL_THREADS) s_sum[t] = *reinterpret_cast<const uint4*>(pv.summary + ((size_t)b * NT + t) * 4);
  __syncthreads();
  const int rows = is_pair ? min(2, NT - 2 * item) : 1, total = rows * NT;
  for (int e = warp; e < total; e += CL_WARPS) {
    const int r = e / NT, c = e - r * NT;
    const int qt = is_pair ? 2 * item + r : c, kt = is_pair ? c : item - NP;
    int cls = classify_summary(s_sum[qt], s_sum[kt], qt, kt);
    const bool writes = is_pair && pv.words != nullptr;   // a pair's CTA writes the bits of its PARTIAL tiles, where the plan has room for them
    if (cls < 0 || (writes && cls == KD_TILE_PARTIAL))
      cls = classify_exact(pv.desc + (size_t)b * pv.Tpad, pv.tilebits + (size_t)b * NT * 32, qt, kt, lane,
                           writes ? pv.words + (((size_t)b * NT + qt) * NT + kt) * KD_WORDS : nullptr);
    if (lane == 0) {
      s_cls[r][c] = static_cast<uint8_t>(cls);
      if (is_pair) pv.cls[((size_t)b * NT + qt) * NT + kt] = static_cast<uint8_t>(cls);
    }
  }
  __syncthreads();
  if (warp == 0) {
    int n = 0, full = 0, partial = 0;
    uint16_t* list = is_pair ? pv.fwd_list + ((size_t)b * NP + item) * NT : pv.bwd_list + ((size_t)b * NT + item - NP) * NT;
    for (int base = 0; base < NT; base += 32) {
      const int t = base + lane;
      const uint32_t c0 = t < NT ? s_cls[0][t] : KD_TILE_EMPTY, c1 = t < NT && rows == 2 ? s_cls[1][t] : KD_TILE_EMPTY;
      const uint32_t any = __ballot_sync(0xffffffffu, (c0 | c1) != 0u);
      if ((c0 | c1) != 0u) list[n + __popc(any & ((1u << lane) - 1u))] = static_cast<uint16_t>(t | (c0 << 8) | (c1 << 10));
      n += __popc(any);
      full += __popc(__ballot_sync(0xffffffffu, c0 == KD_TILE_FULL)) + __popc(__ballot_sync(0xffffffffu, c1 == KD_TILE_FULL));
      partial += __popc(__ballot_sync(0xffffffffu, c0 == KD_TILE_PARTIAL)) + __popc(__ballot_sync(0xffffffffu, c1 == KD_TILE_PARTIAL));
    }
    if (lane == 0) {
      if (is_pair) {
        pv.fwd_cnt[b * NP + item] = n;
        atomicAdd(&pv.stats[b * 2 + 0], static_cast<uint32_t>(full));
        atomicAdd(&pv.stats[b * 2 + 1], static_cast<uint32_t>(partial));
      } else {
        pv.bwd_cnt[b * NT + item - NP] = n;
        // span ids that do not fit the descriptors, found while packing
        const uint32_t* tb = pv.tilebits + ((size_t)b * NT + item - NP) * 32 + 28;
        if ((tb[0] | tb[1] | tb[2] | tb[3]) != 0u) report_status(pv.status, KD_STATUS_SPAN_RANGE);
      }
    }
  }
  // the last CTA of the sequence sorts its items
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&pv.done[b], 1u) == static_cast<uint32_t>(NP + NT - 1);
  __syncthreads();
  if (s_last == 0) return;
  __threadfence();
  for (int t = tid; t < NP; t += CL_THREADS) s_cnt[0][t] = __ldcg(pv.fwd_cnt + b * NP + t);
  for (int t = tid; t < NT; t += CL_THREADS) s_cnt[2][t] = __ldcg(pv.bwd_cnt + b * NT + t);
  for (int qt = warp; qt < NT; qt += CL_WARPS) {
    int n = 0;
    for (int kt = lane; kt < NT; kt += 32) n += __ldcg(pv.cls + ((size_t)b * NT + qt) * NT + kt) != KD_TILE_EMPTY;
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) s_cnt[1][qt] = n;
  }
  __syncthreads();
  for (int w = tid; w < 3 * NT; w += CL_THREADS) order_item(s_cnt[w / NT], w / NT, w % NT, w / NT == 0 ? NP : NT, pv.order + (size_t)b * 3 * NT, NT);
}

// ---------------------------------------------------------------------------------------
// 3. short sequences: the whole plan of a sequence by one CTA, in one launch
// ---------------------------------------------------------------------------------------
// Nothing but latency: the descriptors, class masks and tile classes of up to 1024 tokens stay in shared memory between the steps, where
// the two kernels above hand them over through global memory and a launch. For which calls: see launch_classify.
constexpr int PS_TILES = 8, PS_THREADS = 512, PS_WARPS = PS_THREADS / 32;
__global__ void __launch_bounds__(PS_THREADS) plan_small_kernel(kd_meta m, PlanView pv) {
  __shared__ uint32_t s_desc[PS_TILES * KD_TILE], s_bits[PS_TILES * 32];
  __shared__ uint32_t s_or[PS_TILES * 4], s_and[PS_TILES * 4];
  __shared__ int32_t s_min[PS_TILES * 4], s_max[PS_TILES * 4];
  __shared__ uint4 s_sum[PS_TILES];
  __shared__ uint8_t s_cls[PS_TILES][PS_TILES];   // [query tile][key tile]
  __shared__ int s_cnt[3][PS_TILES];              // entries of the lists of pairs, query tiles and key tiles
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NT = pv.NT, NP = pv.NP;
  pdl_wait();
  pdl_launch_dependents();
  const int n_b = tokens_of(m, b);
  if (tid == 0) pv.len[b] = n_b;
  for (int w = warp; w < 4 * NT; w += PS_WARPS) {   // 32 tokens: word w & 3 of tile w >> 2
    bool bad_id = false;
    const uint32_t d = describe(m, b, 32 * w + lane, n_b, bad_id);
    s_desc[32 * w + lane] = d;
    pv.desc[(size_t)b * pv.Tpad + 32 * w + lane] = d;
    class_masks(d, bad_id, lane, w & 3, s_bits + (w >> 2) * 32);
    const int32_t sid = static_cast<int32_t>(d) >> TD_SID_SHIFT;
    const uint32_t f_or = __reduce_or_sync(0xffffffffu, d & TD_FLAGS), f_and = __reduce_and_sync(0xffffffffu, d & TD_FLAGS);
    const int32_t lo = __reduce_min_sync(0xffffffffu, (d & TD_INS) ? sid : INT32_MAX), hi = __reduce_max_sync(0xffffffffu, (d & TD_INS) ? sid : INT32_MIN);
    if (lane == 0) { s_or[w] = f_or; s_and[w] = f_and; s_min[w] = lo; s_max[w] = hi; }
  }
  // The first CTA alone writes the status word, so it looks at every sequence's span ids: nothing orders the CTAs.
  bool any_bad = false;
  if (b == 0 && m.rules && m.span_id != nullptr)
    for (int s = 0; s < m.B; ++s)
      for (int t = tid, n = tokens_of(m, s); t < n; t += PS_THREADS) any_bad |= out_of_range(m.span_id[s * m.span_id_stride_b + t]);
  const bool bad = __syncthreads_or(any_bad) != 0;
  if (b == 0 && tid == 0) {
    *pv.status = 0u;
    *reinterpret_cast<uint32_t**>(pv.status + 2) = m.status_mirror;
    if (bad) report_status(pv.status, KD_STATUS_SPAN_RANGE);
  }
  if (tid < NT) {
    const int w = 4 * tid;
    s_sum[tid] = make_uint4(s_or[w] | s_or[w + 1] | s_or[w + 2] | s_or[w + 3], s_and[w] & s_and[w + 1] & s_and[w + 2] & s_and[w + 3],
                            static_cast<uint32_t>(min(min(s_min[w], s_min[w + 1]), min(s_min[w + 2], s_min[w + 3]))),
                            static_cast<uint32_t>(max(max(s_max[w], s_max[w + 1]), max(s_max[w + 2], s_max[w + 3]))));
    reinterpret_cast<uint4*>(pv.summary)[(size_t)b * NT + tid] = s_sum[tid];
  }
  for (int i = tid; i < NT * 32; i += PS_THREADS) pv.tilebits[(size_t)b * NT * 32 + i] = s_bits[i];
  __syncthreads();
  for (int e = warp; e < NT * NT; e += PS_WARPS) {
    const int qt = e / NT, kt = e - qt * NT;
    int cls = classify_summary(s_sum[qt], s_sum[kt], qt, kt);
    if (cls < 0 || cls == KD_TILE_PARTIAL) cls = classify_exact(s_desc, s_bits, qt, kt, lane, pv.words + ((size_t)b * NT * NT + e) * KD_WORDS);
    if (lane == 0) {
      s_cls[qt][kt] = static_cast<uint8_t>(cls);
      pv.cls[(size_t)b * NT * NT + e] = static_cast<uint8_t>(cls);
    }
  }
  __syncthreads();
  // lists: of pair w, of key tile w - NP; then the query tiles' counts and the statistics
  for (int w = warp; w < NP + 2 * NT + 1; w += PS_WARPS) {
    if (w < NP + NT) {
      const bool is_pair = w < NP;
      const int k = is_pair ? w : w - NP;
      const bool live = lane < NT;
      const uint32_t c0 = !live ? 0u : is_pair ? s_cls[2 * k][lane] : s_cls[lane][k], c1 = live && is_pair && 2 * k + 1 < NT ? s_cls[2 * k + 1][lane] : 0u;
      const uint32_t any = __ballot_sync(0xffffffffu, (c0 | c1) != 0u);
      uint16_t* list = is_pair ? pv.fwd_list + ((size_t)b * NP + k) * NT : pv.bwd_list + ((size_t)b * NT + k) * NT;
      if ((c0 | c1) != 0u) list[__popc(any & ((1u << lane) - 1u))] = static_cast<uint16_t>(lane | (c0 << 8) | (c1 << 10));
      if (lane == 0) {
        (is_pair ? pv.fwd_cnt + b * NP : pv.bwd_cnt + b * NT)[k] = __popc(any);
        s_cnt[is_pair ? 0 : 2][k] = __popc(any);
      }
    } else if (w < NP + 2 * NT) {
      const int qt = w - NP - NT;
      const uint32_t any = __ballot_sync(0xffffffffu, lane < NT && s_cls[qt][lane] != KD_TILE_EMPTY);
      if (lane == 0) s_cnt[1][qt] = __popc(any);
    } else {
      int full = 0, partial = 0;
      for (int e = lane; e < NT * NT; e += 32) {
        const int cls = s_cls[e / NT][e % NT];
        full += cls == KD_TILE_FULL;
        partial += cls == KD_TILE_PARTIAL;
      }
      full = __reduce_add_sync(0xffffffffu, full);
      partial = __reduce_add_sync(0xffffffffu, partial);
      if (lane == 0) {
        pv.stats[b * 2 + 0] = full;
        pv.stats[b * 2 + 1] = partial;
      }
    }
  }
  __syncthreads();
  if (tid < 3 * NT) order_item(s_cnt[tid / NT], tid / NT, tid % NT, tid / NT == 0 ? NP : NT, pv.order + (size_t)b * 3 * NT, NT);
}

// ---------------------------------------------------------------------------------------
// 4. dense mask materialiser
// ---------------------------------------------------------------------------------------
__global__ void mask_dense_kernel(PlanView pv, int T, uint8_t* out) {
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.z, i = blockIdx.y;
  const uint32_t* d = pv.desc + (size_t)b * pv.Tpad;
  const uint32_t qd = d[i];
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < T; j += gridDim.x * blockDim.x)
    out[((size_t)b * T + i) * T + j] = rule_allowed(qd, i, d[j], j) ? 1 : 0;
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
int launch_classify(const kd_meta& m, void* plan, cudaStream_t stream) {
  kd_plan_layout L;
  if (kd_plan_layout_get(m.B, m.T, &L) != 0) return KD_ERR_ARG;
  PlanView pv = make_plan_view(plan, L);
  cudaError_t e;
  // One launch where it is the faster one whatever the metadata says. Time of a plan in a chain of them (us), two launches | one; sections
  // of the model's layout, then flags and ids drawn for each token (every tile PARTIAL):
  //   1 x 173 6.6 | 3.6, 7.7 | 4.2    8 x 173 6.8 | 5.8, 7.3 | 6.4     12 x 173 6.9 | 7.2, 7.6 | 7.4
  //   1 x 512 5.7 | 3.9, 7.8 | 5.5    8 x 512 7.0 | 6.2, 7.6 | 7.5     12 x 512 7.1 | 7.6, 7.6 | 8.9
  //   1 x 640 6.6 | 4.2, 7.9 | 7.8    4 x 640 7.3 | 5.2, 8.1 | 8.7     1 x 1024 7.1 | 5.7, 7.5 | 12.9    16 x 1024 8.4 | 11.1, 10.7 | 18.1
  // Four tiles are one for each of the CTA's warps; with metadata the first CTA also looks at the span ids of one sequence after the other.
  // Without metadata neither counts: 1 x 173 6.6 | 2.8, 16 x 173 6.6 | 2.6, 1 x 1024 6.1 | 4.2, 16 x 1024 6.7 | 4.2, with lengths 7.4 | 6.3.
  const bool small = m.rules ? L.NT <= 4 && m.B <= 8 : L.NT <= PS_TILES && m.B <= 16;
  if (small) {
    e = launch(plan_small_kernel, m.B, PS_THREADS, 0, stream, m, pv);
  } else {
    e = launch(pack_kernel, dim3(L.NT, m.B), KD_TILE, 0, stream, m, pv);
    if (e == cudaSuccess) e = launch(classify_kernel, dim3(L.NP + L.NT, m.B), CL_THREADS, 0, stream, pv);
  }
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "plan kernels: %s", cudaGetErrorString(e));
  return 0;
}

int launch_mask_dense(const void* plan, int B, int T, uint8_t* out, cudaStream_t stream) {
  kd_plan_layout L;
  if (kd_plan_layout_get(B, T, &L) != 0) return KD_ERR_ARG;
  PlanView pv = make_plan_view(const_cast<void*>(plan), L);
  dim3 grid((T + 255) / 256, T, B);
  if (grid.x > 16) grid.x = 16;
  cudaError_t e = launch(mask_dense_kernel, grid, 256, 0, stream, pv, T, out);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "mask_dense_kernel: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace kd
