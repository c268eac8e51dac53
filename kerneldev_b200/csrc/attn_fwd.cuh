// Declarations and the producer warp shared by the forward kernels (attn_fwd.cu for head dims up to 64, attn_fwd_wide.cu above).
#pragma once
#include "attn_common.cuh"
#include "fwd_rules.cuh"

namespace kd {

struct FwdArgs {
  int B, H, T, NT, NP, Tpad;
  ItemOrder order_of;
  int d_real;        // head dim of the tensors (a multiple of 16, <= HD); TMA zero-fills the tile columns beyond it
  float scale_log2;  // sm_scale * log2(e)
  const uint32_t* words;   // [B][NT][NT][4][128] visibility bits of the PARTIAL tiles, or null
  const int32_t* fwd_cnt;
  const uint16_t* fwd_list;
  const uint8_t* order;   // [B][3][NT]; row 0 = pairs sorted by decreasing list length
  uint32_t* status;
  int plan_ready;
  int split;         // 1: an item is one query tile of a pair (see launch_rules.cuh)
  void* o;           // null: O is wanted as float32 alone
  int64_t o_sb, o_sh, o_st;
  float* o32;        // null, or O of a float32 call
  int64_t o32_sb, o32_sh, o32_st;
  int o_tma;         // head dims up to 64: O leaves through shared memory and TMA stores
  float* lse;
  const uint32_t* desc;       // for kernels without words: the tokens' descriptors,
  const uint32_t* tilebits;   // [B][NT][8][4] class masks of every tile
#ifdef KD_TEST_DROP_LOAD
  int test_drop_load;   // wait time-out test build: the producer of CTA 0 leaves out its first K tile load
#endif
};

// wait-site codes reported in the status word
enum : uint32_t {
  W_F_QFULL = 0x101, W_F_KEMPTY = 0x102, W_F_VEMPTY = 0x103, W_F_KFULL = 0x104, W_F_VFULL = 0x105,
  W_F_PFULL = 0x106, W_F_SFULL = 0x107, W_F_PVDONE = 0x108, W_F_QEMPTY = 0x10A, W_F_OFREE = 0x10B,
  W_F_ITEMFULL = 0x10C, W_F_ITEMEMPTY = 0x10D, W_F_CLC = 0x10E, W_F_ALIGN = 0x10F,
};

// The producer warp: takes items (see the head of attn_fwd.cu), publishes their headers and lists and loads Q tiles and the rings of
// K and V tiles by TMA. C: the kernel's configuration. wait(barrier, parity, site): a warp's bounded wait. publish(slot, lst, n,
// units): writes the list of an item with n entries, 32 per register and lane (in a split pair with gaps: zeros), to its slot and counts
// the units of both query tiles.
template <typename C, typename Wait, typename Publish>
__device__ __forceinline__ void fwd_producer(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const FwdArgs& a, uint8_t* smem,
                                             AbortFlag* abortf, int lane, const Wait& wait, const Publish& publish) {
  constexpr int TILE = C::TILE_BYTES;
  const uint32_t s0 = smem_u32(smem), sQ = s0 + C::SMEM_Q, sK = s0 + C::SMEM_K, sV = s0 + C::SMEM_V;
  int4* items = reinterpret_cast<int4*>(smem + C::SMEM_ITEM);
  const uint16_t* sList = reinterpret_cast<const uint16_t*>(smem + C::SMEM_LIST);
  auto bar = [&](int i) -> uint32_t { return s0 + C::SMEM_BAR + i * 8; };
  if (lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  int q_cnt = 0, kv_cnt = 0, v_cnt = 0, k = 0, asked = 0;   // Q, K, V tiles requested, items published, cancellations asked for
  PhaseBits q_phases;   // of the Q tiles' "full" barriers
  uint32_t q_used = 0u;
  int k_dropped = -1;   // index of a K tile that was never requested (test builds only)
  bool ok = true, pending = false;
  uint32_t lst[4];      // the next item's list, 32 entries per register
  auto decode = [&](int idx) -> int4 {
    int4 it;
    int rank;
    a.order_of.decode(idx, a.NP << a.split, it.x, rank);
    it.y = it.x % a.H;
    it.x = it.x / a.H;
    const int pair = __ldcg(a.order + ((size_t)it.x * 3 + 0) * a.NT + (rank >> a.split)), only = a.split ? 1 + (rank & 1) : 0;
    it.z = pair | (only << 16);
    const uint16_t* list = a.fwd_list + ((size_t)it.x * a.NP + pair) * a.NT;
    it.w = __ldcg(a.fwd_cnt + it.x * a.NP + pair);
#pragma unroll
    for (int r = 0; r < 4; ++r) lst[r] = r * 32 + lane < a.NT ? __ldcg(list + r * 32 + lane) : 0u;   // does not wait for the count
#pragma unroll
    for (int r = 0; r < 4; ++r) lst[r] = r * 32 + lane < it.w ? lst[r] : 0u;
    if (only != 0) {   // the entries that are not EMPTY for the one tile
      it.w = 0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        lst[r] = entry_of_tile(lst[r], only - 1);
        it.w += __popc(__ballot_sync(0xffffffffu, lst[r] != 0u));
      }
    }
    return it;
  };
  // The next item is asked for three tiles before the end of this one (for a shorter one: when it is taken), which hides the
  // answer and the look-up of its list, and no earlier: an item held in reserve by a CTA with a long list is one that an idle CTA cannot take (claimed two
  // items ahead: 575 us for 519 with hierarchical masks at 16 x 16 x 4096 x 64).
  auto ask = [&]() {
    if (lane == 0) {
      fence_proxy_async_smem();   // the previous response has been read
      mbar_arrive_expect_tx(bar(C::B_CLC), 16);
      clc_try_cancel(s0 + C::SMEM_CLC, bar(C::B_CLC));
    }
    ++asked;
    pending = true;
  };
  auto take_next = [&](int4& nx) -> bool {
    if (!wait(C::B_CLC, (asked - 1) & 1, W_F_CLC)) return false;
    pending = false;
    const int idx = clc_first_ctaid_x(s0 + C::SMEM_CLC);
    __syncwarp();   // every lane has read the response that the next request overwrites
    nx.w = -1;
    if (idx >= 0) {
      nx = decode(idx);
      if (nx.w <= 2) ask();
    }
    return true;
  };
  auto load_tile = [&](const CUtensorMap* tm, uint32_t dst, int full, int tile, int h, int b) {
    if (lane != 0) return;
    mbar_arrive_expect_tx(bar(full), TILE);
    for (int kb = 0; kb < C::KBLK; ++kb) tma_load_4d(dst + kb * 16384, tm, bar(full), kb * 64, tile * KD_TILE, h, b);
  };
  int4 it = decode(blockIdx.x);
  if (it.w <= 2) ask();
  while (ok) {
    const int slot = k % C::NITEM;
    if (!(ok = wait(C::B_ITEMEMPTY + slot, ((k / C::NITEM) & 1) ^ 1, W_F_ITEMEMPTY))) break;
    const int b = it.x, h = it.y, pair = it.z & 0xFFFF, only = it.z >> 16, n = it.w;
    int units[2] = {0, 0};
    publish(slot, lst, n, units);
    if (lane == 0) items[slot] = make_int4(b, h, pair, n < 0 ? -1 : (n | (units[0] << 8) | (units[1] << 16) | (only << 24)));
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::B_ITEMFULL + slot));
    if (n < 0) break;
    if (k == 0) {   // Q, K and V are read from here on
      pdl_wait();
      pdl_launch_dependents();
    }
    ++k;
    const int ntile_q = (2 * pair + 1 < a.NT) ? 2 : 1;
    auto load_q = [&](int t) -> bool {
      const int s = C::QR::slot(q_cnt), full = C::QR::full(q_cnt, t);
      if (!wait(C::B_QEMPTY + s, C::QR::empty_parity(q_cnt), W_F_QEMPTY)) return false;
      load_tile(&tmQ, sQ + s * TILE, C::B_QFULL + full, 2 * pair + t, h, b);
      q_phases.take(full);
      q_used |= 1u << full;
      ++q_cnt;
      return true;
    };
    if (!(ok = load_q(0))) break;
    int4 nx = it;
#pragma unroll 1
    for (int e = 0; e < max(n, 1); ++e) {
      if (n > 2 && e == n - 3) ask();
      if (e >= n - 1 && !(ok = take_next(nx))) break;   // its list is looked up while this item's last tiles wait for slots
      if (n == 0) {
        if (ntile_q == 2) ok = load_q(1);
        break;
      }
      const int kt = sList[slot * 128 + e] & 0xFF;
#ifdef KD_TEST_DROP_LOAD
      // Test build only: this one K tile is never requested (no copy, no expected bytes), so the S issuer's
      // bounded wait for it runs out and the CTA has to unwind. Nothing is left in flight for the stage.
      if (a.test_drop_load && blockIdx.x == 0 && kv_cnt == 0) {
        k_dropped = kv_cnt++;
      } else
#endif
      {
        const int s = kv_cnt % C::KST;
        if (!(ok = wait(C::B_KEMPTY + s, ((kv_cnt / C::KST) & 1) ^ 1, W_F_KEMPTY))) break;
        load_tile(&tmK, sK + s * TILE, C::B_KFULL + s, kt, h, b);
        ++kv_cnt;
      }
      if (e == 0 && ntile_q == 2 && !(ok = load_q(1))) break;
      {
        const int s = v_cnt % C::VST;
        if (!(ok = wait(C::B_VEMPTY + s, ((v_cnt / C::VST) & 1) ^ 1, W_F_VEMPTY))) break;
        load_tile(&tmV, sV + s * TILE, C::B_VFULL + s, kt, h, b);
        ++v_cnt;
      }
    }
    it = nx;
  }
  if (abortf->v != 0 && lane == 0) {
    // unwinding: let every copy already in flight land (bounded) before the CTA exits
    for (int e = max(0, kv_cnt - C::KST); e < kv_cnt; ++e)
      if (e != k_dropped) drain_wait(bar(C::B_KFULL + e % C::KST), (e / C::KST) & 1);
    for (int e = max(0, v_cnt - C::VST); e < v_cnt; ++e) drain_wait(bar(C::B_VFULL + e % C::VST), (e / C::VST) & 1);
    for (int f = 0; f < C::QR::FULL; ++f)
      if ((q_used >> f) & 1u) drain_wait(bar(C::B_QFULL + f), q_phases.last(f));
    if (pending) drain_wait(bar(C::B_CLC), (asked - 1) & 1);
  }
}

// attn_fwd_wide.cu: head dims above 64
int launch_attn_fwd_wide(long long n_items, const FwdArgs& a, int dtype, const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                         cudaStream_t stream);

}  // namespace kd
