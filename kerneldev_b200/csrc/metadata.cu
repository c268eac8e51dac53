// Metadata from token ids on the device: the three per-token tensors of the hierarchical mask
// (in_span, span_id, is_prefix) for a batch of token rows, as the reference derives them when a
// caller passes token ids only (model.py:203-238):
//   in_span[t]   = (#[SPAN] in x[0..t]) - (#[ES] in x[0..t]) > 0
//   span_id[t]   = #[SPAN] in x[0..t] where in_span, else 0;  -1 at every [MASKQ]
//   is_prefix[t] = t <= position of the first [CLS] (all false without a [CLS])
// The reference does this with two cumulative sums and a host loop that synchronises once per row
// (.nonzero() / .item()). Here one CTA handles a row, 4096 tokens at a time: a warp takes 128 consecutive tokens with four
// coalesced loads in flight, the running marker counts come from warp ballots and a scan of the warps' totals, and every
// token is read once. Integer work, bound by the latency of the loads (with eight warps that walked the row twice it took
// 9 us at T = 2048). is_prefix needs the row's first [CLS], which a row longer than a chunk may have in a later one: it is
// looked for first then.
#include "common.cuh"
#include "sm100_prims.cuh"

namespace kd {

constexpr int MD_THREADS = 1024, MD_WARPS = MD_THREADS / 32, MD_PER = 4, MD_CHUNK = MD_THREADS * MD_PER;

__global__ void __launch_bounds__(MD_THREADS)
metadata_kernel(const int64_t* __restrict__ tokens, int64_t stride_b, int T, int64_t tok_span, int64_t tok_es,
                int64_t tok_cls, int64_t tok_maskq, uint8_t* __restrict__ in_span, int64_t* __restrict__ span_id,
                uint8_t* __restrict__ is_prefix) {
  __shared__ int s_span[MD_WARPS], s_es[MD_WARPS], s_cls[MD_WARPS];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t* x = tokens + (size_t)b * stride_b;
  uint8_t *o_ins = in_span + (size_t)b * T, *o_pre = is_prefix + (size_t)b * T;
  int64_t* o_sid = span_id + (size_t)b * T;
  const uint32_t upto = 0xFFFFFFFFu >> (31 - lane);   // lanes 0 .. lane
  pdl_wait();
  pdl_launch_dependents();
  int first_cls = T;   // T: none
  for (int base = 0; T > MD_CHUNK && base < T && first_cls == T; base += MD_CHUNK) {
    int mine = T;
    for (int r = MD_PER - 1; r >= 0; --r) {
      const int t = base + r * MD_THREADS + tid;
      if (t < T && x[t] == tok_cls) mine = t;
    }
    mine = __reduce_min_sync(0xffffffffu, mine);
    if (lane == 0) s_cls[warp] = mine;
    __syncthreads();
    first_cls = __reduce_min_sync(0xffffffffu, s_cls[lane]);
    __syncthreads();
  }
  int c_span = 0, c_es = 0;   // marker counts of the chunks before
  for (int base = 0; base < T; base += MD_CHUNK) {
    const int t0 = base + warp * (32 * MD_PER) + lane;
    int64_t v[MD_PER];
#pragma unroll
    for (int r = 0; r < MD_PER; ++r) v[r] = t0 + 32 * r < T ? x[t0 + 32 * r] : 0;
    uint32_t bs[MD_PER], be[MD_PER];
    int n_span = 0, n_es = 0, cls = T;
#pragma unroll
    for (int r = 0; r < MD_PER; ++r) {
      const bool live = t0 + 32 * r < T;
      bs[r] = __ballot_sync(0xffffffffu, live && v[r] == tok_span);
      be[r] = __ballot_sync(0xffffffffu, live && v[r] == tok_es);
      const uint32_t bc = __ballot_sync(0xffffffffu, live && v[r] == tok_cls);
      if (bc != 0u && cls == T) cls = t0 - lane + 32 * r + __ffs(bc) - 1;
      n_span += __popc(bs[r]);
      n_es += __popc(be[r]);
    }
    if (lane == 0) { s_span[warp] = n_span; s_es[warp] = n_es; s_cls[warp] = cls; }
    __syncthreads();
    const int w_span = s_span[lane], w_es = s_es[lane];
    int p_span = c_span + __reduce_add_sync(0xffffffffu, lane < warp ? w_span : 0);
    int p_es = c_es + __reduce_add_sync(0xffffffffu, lane < warp ? w_es : 0);
    c_span += __reduce_add_sync(0xffffffffu, w_span);
    c_es += __reduce_add_sync(0xffffffffu, w_es);
    if (T <= MD_CHUNK) first_cls = __reduce_min_sync(0xffffffffu, s_cls[lane]);
#pragma unroll
    for (int r = 0; r < MD_PER; ++r) {
      const int t = t0 + 32 * r;
      const int my_span = p_span + __popc(bs[r] & upto), my_es = p_es + __popc(be[r] & upto);   // inclusive counts at t
      p_span += __popc(bs[r]);
      p_es += __popc(be[r]);
      if (t < T) {
        const bool ins = (my_span - my_es) > 0;
        o_ins[t] = ins ? 1 : 0;
        o_sid[t] = (v[r] == tok_maskq) ? int64_t(-1) : (ins ? int64_t(my_span) : int64_t(0));
        o_pre[t] = (t <= first_cls && first_cls < T) ? 1 : 0;
      }
    }
    __syncthreads();   // the counts in shared memory are free for the next chunk
  }
}

int launch_metadata(const int64_t* tokens, int64_t stride_b, int B, int T, int64_t tok_span, int64_t tok_es,
                    int64_t tok_cls, int64_t tok_maskq, uint8_t* in_span, int64_t* span_id, uint8_t* is_prefix,
                    cudaStream_t stream) {
  if (B == 0 || T == 0) return 0;
  const cudaError_t e = launch(metadata_kernel, B, MD_THREADS, 0, stream, tokens, stride_b, T, tok_span, tok_es, tok_cls, tok_maskq, in_span,
                               span_id, is_prefix);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "metadata_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace kd
