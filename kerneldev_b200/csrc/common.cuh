// Shared host/device declarations of the library: plan view, error reporting, launch entry
// points of the individual translation units.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "../../include/kd_attention.h"

namespace kd {

// Visibility of a tile as bits: uint32 [4][128], bit k of word [w][q] = query q of the query tile sees key 32 w + k of the key tile. The last part of
// a plan has room for every tile of a sequence, [B][query tile][key tile], and holds the PARTIAL ones'.
constexpr size_t KD_WORDS = 4 * KD_TILE, KD_WORDS_BYTES = KD_WORDS * 4;
// ... if that is no more than KD_WORDS_LIMIT for the batch: a bit for each pair of tokens grows with the square of the length (64 x 16384 tokens 2 GB),
// whatever the heads and the head dim are, and would take the place of tensors. Beyond it the plan has no such part, and the kernels form the
// bits of a PARTIAL tile for every head (form_words), in instantiations of their own (kWords false). At the limit: 8 x 16384 tokens, 128 x 4096. Passes beyond it, us, with the bits in a
// plan of any size and so: hierarchical forward 9 x 4 x 16384 x 64 660 | 705, x 128 905 | 918, with the backward 2,050 | 2,220 and 3,215 | 3,230; deterministic 2,450 | 2,660;
// causal 2100 x 2 x 1000 x 64 with the backward 3,460 | 3,800.
constexpr size_t KD_WORDS_LIMIT = size_t(256) << 20;
inline size_t words_bytes(size_t B, size_t NT) {
  const size_t n = B * NT * NT * KD_WORDS_BYTES;
  return n <= KD_WORDS_LIMIT ? n : 0;
}

// Typed pointers into a plan buffer (see kd_plan_layout for the contents).
struct PlanView {
  int NT, NP, Tpad;
  uint32_t* desc;
  uint32_t* summary;
  uint8_t* cls;
  int32_t* fwd_cnt;
  uint16_t* fwd_list;
  int32_t* bwd_cnt;
  uint16_t* bwd_list;
  uint32_t* tilebits;
  uint8_t* order;
  uint32_t* stats;
  uint32_t* done;   // [B] CTAs of the classifier that have finished
  int32_t* len;     // [B] tokens of each sequence that are not padding
  uint32_t* status;
  uint32_t* words;   // null: see KD_WORDS_LIMIT
};

inline PlanView make_plan_view(void* plan, const kd_plan_layout& L) {
  char* base = static_cast<char*>(plan);
  PlanView v;
  v.NT = L.NT;
  v.NP = L.NP;
  v.Tpad = L.NT * KD_TILE;
  v.desc = reinterpret_cast<uint32_t*>(base + L.off_desc);
  v.summary = reinterpret_cast<uint32_t*>(base + L.off_summary);
  v.cls = reinterpret_cast<uint8_t*>(base + L.off_cls);
  v.fwd_cnt = reinterpret_cast<int32_t*>(base + L.off_fwd_cnt);
  v.fwd_list = reinterpret_cast<uint16_t*>(base + L.off_fwd_list);
  v.bwd_cnt = reinterpret_cast<int32_t*>(base + L.off_bwd_cnt);
  v.bwd_list = reinterpret_cast<uint16_t*>(base + L.off_bwd_list);
  v.tilebits = reinterpret_cast<uint32_t*>(base + L.off_tilebits);
  v.order = reinterpret_cast<uint8_t*>(base + L.off_order);
  v.stats = reinterpret_cast<uint32_t*>(base + L.off_stats);
  v.done = v.stats + 2 * (size_t)L.B;
  v.len = reinterpret_cast<int32_t*>(v.stats + 3 * (size_t)L.B);
  v.status = reinterpret_cast<uint32_t*>(base + L.off_status);
  const size_t words = words_bytes(L.B, L.NT);
  v.words = words > 0 ? reinterpret_cast<uint32_t*>(base + L.total - words) : nullptr;
  return v;
}

// Launches a kernel whose blocks may become resident while the kernel before it on the stream still runs (programmatic
// stream serialisation). Every kernel of this library is launched like this and executes pdl_wait(), which returns when
// the kernels before it are complete and their writes visible, before it reads or writes anything that they may write or read;
// most begin with it. Launch latency, barrier set-up, the TMEM allocation and in some the look-up of the work then overlap the
// predecessor, which is what a chain of short kernels consists of.
template <typename... P, typename... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// records a printf-style message for kd_last_error() and returns `code`
int set_error(int code, const char* fmt, ...);

// 4-D tensor map over a (B,H,T,D) tensor with box (64 elements along D, `box_rows` tokens),
// 128-byte swizzle, zero fill outside the tensor. box_bytes = 64: half the width and swizzle. name = NULL: a refusal leaves no message.
int encode_tensor_map(CUtensorMap* out, const kd_tensor& t, int B, int H, int T, int D, int dtype,
                      int box_rows, const char* name, int box_bytes = 128);

// 3-D tensor map over a contiguous fp32 (rows, T, D) array with box (32 elements along D, `box_rows` rows of
// one slice), 128-byte swizzle: the target of the fused backward's bulk reductions of dQ tiles.
int encode_tensor_map_f32_rows(CUtensorMap* out, float* base, int slices, int T, int D, int box_rows, const char* name);

// 4-D tensor map over a float32 (B,H,T,D) tensor with box (32 elements along D, `box_rows` tokens), 128-byte swizzle
int encode_tensor_map_f32(CUtensorMap* out, const kd_tensor& t, int B, int H, int T, int D, int box_rows, const char* name);

int launch_classify(const kd_meta& m, void* plan, cudaStream_t stream);
int launch_mask_dense(const void* plan, int B, int T, uint8_t* out, cudaStream_t stream);
// f32: NULL, or the call's float32 tensors (kd_attn_f32)
int launch_attn_fwd(const kd_attn_params& p, const kd_attn_f32* f32, cudaStream_t stream);
// signs: NULL, or of transformed Q and K (kd_attn_bwd_hadamard)
int launch_attn_bwd(const kd_attn_params& p, const kd_attn_f32* f32, const float* signs, cudaStream_t stream);
int static_delta_address(size_t rows_needed, float** out);
int launch_hadamard(const kd_tensor& x, const kd_tensor& y, int B, int H, int T, int D, int dtype,
                    const float* signs, int inverse, cudaStream_t stream);

int launch_grad_transform(const float* acc, int width, float scale, const int32_t* len, const float* signs, const kd_tensor& dq, const kd_tensor& dk,
                          int B, int H, int T, int D, int dtype, cudaStream_t stream);

int launch_cast(const kd_tensor* src, const kd_tensor* dst, int n, int B, int H, int T, int D, bool widen, cudaStream_t stream);

int launch_metadata(const int64_t* tokens, int64_t stride_b, int B, int T, int64_t tok_span, int64_t tok_es,
                    int64_t tok_cls, int64_t tok_maskq, uint8_t* in_span, int64_t* span_id, uint8_t* is_prefix,
                    cudaStream_t stream);

int launch_span_index(const int64_t* tokens, int64_t stride_b, int B, int T, int64_t tok_span, int64_t tok_es,
                      int64_t tok_mask, int32_t* starts, int32_t* ends, int32_t* n_starts, int32_t* n_ends,
                      int32_t* first_mask, int32_t* counts_host, cudaStream_t stream);
int launch_cocktail(bool backward, const kd_cocktail& p, cudaStream_t stream);
int launch_span_mean(bool backward, const void* a, int64_t a_sb, int64_t a_st, void* out, int64_t o_sb, int64_t o_st, int B,
                     int T, int C, int S, int dtype, const int32_t* starts, const int32_t* ends, const int32_t* n_starts,
                     const int32_t* n_ends, cudaStream_t stream);

}  // namespace kd
