// Declarations shared by the backward translation units.
#pragma once
#include "attn_common.cuh"

namespace kd {

struct BwdArgs {
  int B, H, T, NT, NP, Tpad;
  ItemOrder order_of;   // of the dQ kernel's items
  int after_dq;      // fused kernel without dQ: the dQ kernel of the same call is the kernel before this one on the stream
  int d_real;        // head dim of the tensors (a multiple of 16, <= HD); TMA zero-fills the tile columns beyond it
  float scale_log2;  // sm_scale * log2(e)
  float sm_scale;
  const uint32_t* words;   // [B][NT][NT][4][128] visibility bits of the PARTIAL tiles, or null
  const int32_t* fwd_cnt;
  const uint16_t* fwd_list;
  const int32_t* bwd_cnt;
  const uint16_t* bwd_list;
  const uint8_t* order;   // [B][3][NT]; row 1 = q tiles, row 2 = k tiles, by decreasing list length
  uint32_t* status;
  const void* o;
  int64_t o_sb, o_sh, o_st;
  void* d_o;         // with d_o32: written by the delta kernel
  int64_t do_sb, do_sh, do_st;
  const float* d_o32;   // null, or dO of a float32 call
  int64_t do32_sb, do32_sh, do32_st;
  int plan_ready;    // the plan may be read before the wait for the kernel ahead
  const float* lse;
  float* delta;
  float* dq_acc;     // fp32 (B,H,T,tile width) dQ accumulation scratch of the fused backward, else null
  bool grads_f32;    // dq, dk, dv are float32 (the fused backward then adds its dQ tiles into dq itself)
  bool zero_dq;      // ... and the delta kernel zeroes it
  void* dq;
  int64_t dq_sb, dq_sh, dq_st;
  void* dk;
  int64_t dk_sb, dk_sh, dk_st;
  void* dv;
  int64_t dv_sb, dv_sh, dv_st;
  const int32_t* len;   // [B] tokens that are not padding (at the end: the fused kernel of head dim 64 is 2 % slower with its other arguments elsewhere)
  const float* signs;   // null, or Q and K are Hadamard transforms with these signs, and dQ and dK are wanted of what they were made from
  int len_ready;     // the plan may be read by the delta kernel before the wait for the kernel ahead
  const uint32_t* desc;       // for kernels without words: the tokens' descriptors,
  const uint32_t* tilebits;   // [B][NT][8][4] class masks of every tile
#ifdef KD_TEST_DROP_LOAD
  int test_drop;     // wait time-out test build: what the producer of CTA 0 leaves out
#endif
};

// Wait time-out test build: whether the producer of this CTA leaves something out, so that waits run out and the CTA has to unwind. 2: the dQ kernel's
// first pair of K and V; the fused kernel's 3: first Q, 4: second header. Nothing is requested and no bytes are expected, so that nothing is in flight.
__device__ __forceinline__ bool test_drops(const BwdArgs& a, int what) {
#ifdef KD_TEST_DROP_LOAD
  return a.test_drop == what && blockIdx.x == 0;
#else
  return false;
#endif
}

// How the delta and the conversion kernel (256 threads) divide the rows: a block per ROWS rows of a head, HD / 8 threads to a row, three rows to a
// thread, all of whose loads are under way together. Both are bound by HBM traffic, and leave the rows of padding alone (delta kernel,
// hierarchical 16 x 16 x 4096 x 64 with a third of padding 84 -> 56 us; whole backward 1070 -> 1020, 8 x 16 x 2048 x 64 163 -> 151, 4 x 16 x 2048 x
// 128 140 -> 129). The block index gives head and sequence: with a flat row index, three 64-bit divisions a row and the length looked up for each
// the kernels lost 2 % of the backward without padding (causal 8 x 16 x 2048 x 64), with the length fetched a row ahead 10 %. One row to a thread
// 288 -> 303 us there, two 293, four 294.
template <int HD>
struct RowBlocks {
  static constexpr int TPR = HD / 8, RPB = 256 / TPR, STEPS = 3, ROWS = RPB * STEPS;
  static dim3 grid(int B, int H, int T) { return dim3((T + ROWS - 1) / ROWS, H, B); }
};

// 32 x 32 bits across a warp: lane l gives word l and gets bit l of every lane's word, lane 0's in bit 0
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
  constexpr uint32_t low[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int d = 16 >> i;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, d);
    x = (lane & d) ? ((x & ~low[i]) | ((y & ~low[i]) >> d)) : ((x & low[i]) | ((y & low[i]) << d));
  }
  return x;
}

// Fused backward (attn_bwd_fused.cu): one key-tile-major kernel that forms S and dP once per tile, accumulates dK and
// dV in TMEM and adds its dQ partials to a.dq_acc, then a conversion kernel.
int launch_bwd_fused(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                     const BwdArgs& a, int dtype, bool after_delta, cudaStream_t stream);

// The same kernel without dQ: dK and dV of the deterministic backward, behind a kernel for dQ (attn_bwd.cu).
int launch_bwd_dkdv(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                    const BwdArgs& a, int dtype, cudaStream_t stream);

}  // namespace kd
