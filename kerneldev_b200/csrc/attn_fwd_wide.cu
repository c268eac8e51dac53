// Forward kernel for head dims above 64: O = softmax(mask(Q K^T * scale)) V and base-2 LSE, for sm_100a.
//
// Items, lists, units, the producer warp and the online softmax are those of the kernel for head dims up to 64 (attn_fwd.cu). What
// differs follows from TMEM: O takes 128 columns per query tile, so there are two score buffers, one for each query tile of the
// pair, and P lies over the scores it was made from. Tile i's unit u is then one chain: scores -> softmax -> P V(u), directly
// behind it the scores of unit u + 1 (the tensor pipe executes in issue order), and the two tiles take turns.
// Roles (384 threads):
//   warp 0      takes items, stages their lists, loads Q tiles and the K and V rings by TMA
//   warps 1, 2  issue both products of query tile 0, 1
//   warps 4-7   softmax of query tile 0, a thread per row
//   warps 8-11  softmax of query tile 1
//
// What bounds it: with long lists the power limit (bf16 causal 16 x 16384 x 128 runs at 1,600 MHz) and the chain above, of which 1,024
// cycles are the products and 1,024 the exponentials of a tile. A thread per row needs no exchange of row maxima and executes three
// quarters of the instructions that two threads per row do, and an issuing warp per tile does not make one tile's products wait
// for the other tile's P. Against sixteen softmax warps and one issuing warp (us, normally distributed inputs, at 1,600-1,680 MHz under the power
// limit; with outliers, whose sparse P draws less power, hierarchical 4 x 32 x 8192 x 128 955 -> 963):
//   bf16 causal 16 x 16384 x 128 977 -> 916          fp16 hierarchical 4 x 32 x 8192 x 128 1363 -> 1290
//   bf16 full 2 x 16 x 4096 x 128 280 -> 260         bf16 causal 8 x 16 x 2048 x 128 156 -> 157
// Masks formed after the scores had been loaded, from descriptors held in registers since the unit before: 916 -> 942 (registers).
// P handed over in quarters: 1026.
#include <algorithm>
#include <atomic>

#include "attn_fwd.cuh"

namespace kd {

struct FwdWideCfg {
  static constexpr int HD = 128;
  static constexpr int KBLK = HD / 64;                   // 64-element blocks along D
  static constexpr int TILE_BYTES = KD_TILE * HD * 2;    // one Q / K / V tile
  static constexpr int KST = 2, VST = 2;                 // K and V ring stages
  using QR = FwdWideQRing;                               // ring of Q tiles (two per item): three slots, a "full" barrier per slot and issuing warp
  static constexpr int NQ = QR::SLOTS;
  static constexpr int NPART = 2;                        // P is handed over in two halves of the keys
  static constexpr int NITEM = 2;                        // ring of item headers and lists
  static constexpr int SMEM_Q = 0;
  static constexpr int SMEM_K = SMEM_Q + NQ * TILE_BYTES;
  static constexpr int SMEM_V = SMEM_K + KST * TILE_BYTES;
  static constexpr int SMEM_LIST = SMEM_V + VST * TILE_BYTES;      // NITEM x <= 128 list entries
  static constexpr int SMEM_OWN = SMEM_LIST + NITEM * 128 * 2;     // NITEM x the units of query tile 0, then of tile 1: key tile | PARTIAL << 8
  static constexpr int SMEM_ITEM = SMEM_OWN + NITEM * 256 * 2;     // NITEM x {batch, head, pair, entries | units of tile 0 << 8 | of tile 1 << 16 | the item's only tile + 1 << 24}
  static constexpr int SMEM_CLC = SMEM_ITEM + NITEM * 16;
  static constexpr int SMEM_BAR = SMEM_CLC + 16;
  // barriers (8 bytes each)
  static constexpr int B_QFULL = 0, B_QEMPTY = B_QFULL + QR::FULL, B_KFULL = B_QEMPTY + NQ, B_KEMPTY = B_KFULL + KST, B_VFULL = B_KEMPTY + KST,
                       B_VEMPTY = B_VFULL + VST, B_SFULL = B_VEMPTY + VST, B_PFULL = B_SFULL + 2, B_PVDONE = B_PFULL + NPART * 2,
                       B_OFREE = B_PVDONE + 4, B_ITEMFULL = B_OFREE + 2, B_ITEMEMPTY = B_ITEMFULL + NITEM, B_CLC = B_ITEMEMPTY + NITEM,
                       NBAR = B_CLC + 1;
  static constexpr int SMEM_ALLOC = SMEM_BAR + NBAR * 8 + 16;
  static constexpr int THREADS = 384;                    // four light warps + four softmax warps per query tile
  // registers: 168 per thread at launch; light warps release down to 56, softmax warps take 224
  static constexpr int REGS_LAUNCH = 168, REGS_LIGHT = 56, REGS_COMPUTE = 224;
  static_assert(4 * 32 * REGS_LIGHT + 8 * 32 * REGS_COMPUTE <= THREADS * REGS_LAUNCH, "register pool");
  // TMEM columns: scores (and P) of the two query tiles, then O0 and O1
  static constexpr uint32_t TM_S = 0, TM_O = 2 * KD_TILE;
  static_assert(TM_O + 2 * HD <= 512, "TMEM budget");
  static_assert(SMEM_ALLOC <= 232448, "shared memory budget");
};

// kF32: of a float32 call; kWords: the plan has the PARTIAL tiles' bits (see attn_fwd.cu)
template <bool kBf16, bool kF32, bool kWords>
__global__ void __launch_bounds__(FwdWideCfg::THREADS, 1)
attn_fwd_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const FwdArgs a) {
  using C = FwdWideCfg;
  constexpr int HD = C::HD, TILE = C::TILE_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t s0 = smem_u32(smem);
  uint16_t* sList = reinterpret_cast<uint16_t*>(smem + C::SMEM_LIST);
  uint16_t* sOwn = reinterpret_cast<uint16_t*>(smem + C::SMEM_OWN);
  const int4* items = reinterpret_cast<const int4*>(smem + C::SMEM_ITEM);
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + C::SMEM_BAR + C::NBAR * 8);
  AbortFlag* abortf = reinterpret_cast<AbortFlag*>(tmem_base_s + 1);
  auto bar = [&](int i) -> uint32_t { return s0 + C::SMEM_BAR + i * 8; };

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  if ((s0 & 1023u) != 0u) {   // the swizzled tiles need it; the launch asks for it, so this never happens
    if (tid == 0) report_status(a.status, KD_DEV_TIMEOUT | W_F_ALIGN);
    return;
  }
  if (tid == 0) abortf->v = 0;
  if (tid < C::NBAR) {
    const int i = tid;
    uint32_t count = 1;
    if ((i >= C::B_KEMPTY && i < C::B_VFULL) || (i >= C::B_VEMPTY && i < C::B_SFULL)) count = 2;            // both issuers
    if ((i >= C::B_PFULL && i < C::B_PVDONE) || (i >= C::B_OFREE && i < C::B_ITEMFULL)) count = 4;          // the softmax warps of a tile
    if (i >= C::B_ITEMEMPTY && i < C::B_CLC) count = 10;                                                    // the issuers and eight softmax warps
    mbar_init(bar(i), count);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (!a.plan_ready) pdl_wait();   // (see attn_fwd.cu)
  // the whole of TMEM is allocated, so the allocation starts at column 0 and the addresses below are constants
  auto wait = [&](int i, uint32_t parity, uint32_t site) -> bool {
    return __all_sync(0xffffffffu, mbar_wait(bar(i), parity, abortf, site));
  };
  // header of this CTA's k-th item; false: there is none. The slot stays taken until item_done.
  auto next_item = [&](int k, int4& it) -> bool {
    const int slot = k % C::NITEM;
    // (Twice the limit: warps without work wait here for as long as the others wait for what is late, and those are to say what it is.)
    if (!__all_sync(0xffffffffu, mbar_wait(bar(C::B_ITEMFULL + slot), (k / C::NITEM) & 1, abortf, W_F_ITEMFULL, 2u * KD_WAIT_LIMIT_CYCLES))) return false;
    const int4 v = items[slot];
    it.x = __reduce_max_sync(0xffffffffu, v.x);   // warp-uniform for the compiler
    it.y = __reduce_max_sync(0xffffffffu, v.y);
    it.z = __reduce_max_sync(0xffffffffu, v.z);
    it.w = __reduce_max_sync(0xffffffffu, v.w);
    return it.w >= 0;
  };
  auto item_done = [&](int k) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::B_ITEMEMPTY + k % C::NITEM));
  };

  if (warp < 4) {
    reg_dealloc<C::REGS_LIGHT>();
    if (warp == 0) {
      // ------------------------------ producer warp ------------------------------
      const uint32_t below = (1u << lane) - 1u;
      // the list for the issuers, and each query tile's own for its softmax warps
      auto publish = [&](int slot, const uint32_t (&lst)[4], int, int (&units)[2]) {
        int e = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t any = __ballot_sync(0xffffffffu, lst[r] != 0u);
          if (lst[r] != 0u) sList[slot * 128 + e + __popc(any & below)] = static_cast<uint16_t>(lst[r]);
          e += __popc(any);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t cls = entry_class(lst[r], i), has = __ballot_sync(0xffffffffu, cls != 0u);
            if (cls != 0u)
              sOwn[slot * 256 + i * 128 + units[i] + __popc(has & below)] = static_cast<uint16_t>((lst[r] & 0xFFu) | (cls == KD_TILE_PARTIAL ? 0x100u : 0u));
            units[i] += __popc(has);
          }
        }
      };
      fwd_producer<C>(tmQ, tmK, tmV, a, smem, abortf, lane, wait, publish);
    } else if (warp <= 2) {
      // ------------------------------ issuers: a warp per query tile ------------------------------
      // All lanes follow the control flow and one elected lane issues (mma_ss_uniform).
      const int i = warp - 1;
      const uint32_t idesc_s = make_idesc_f16(kBf16, 0, 0, KD_TILE, KD_TILE), idesc_o = make_idesc_f16(kBf16, 0, 1, KD_TILE, HD);
      const uint32_t hi = desc_hi_sw128(), lo_q = desc_lo_kmajor(s0 + C::SMEM_Q), lo_k = desc_lo_kmajor(s0 + C::SMEM_K), lo_v = desc_lo_mnmajor(s0 + C::SMEM_V);
      const uint32_t tS = C::TM_S + i * KD_TILE, tO = C::TM_O + i * HD;
      constexpr uint32_t T16 = TILE >> 4;
      int kstage = 0, vstage = 0, q_cnt = 0;
      uint32_t kparity = 0u, vparity = 0u, pv_cnt = 0u, o_cnt = 0u;   // P V products issued; items with units
      PhaseBits q_phases;   // of this query tile's barriers
      bool first = false;   // no P V of the item has been issued
      auto next_k = [&]() { if (++kstage == C::KST) { kstage = 0; kparity ^= 1u; } };
      auto next_v = [&]() { if (++vstage == C::VST) { vstage = 0; vparity ^= 1u; } };
      auto issue_pv = [&]() -> bool {
        // the first product of an item overwrites O: the softmax warps must have read the previous item's result
        if (first && o_cnt++ > 0u && !wait(C::B_OFREE + i, o_cnt & 1u, W_F_OFREE)) return false;
        if (!wait(C::B_VFULL + vstage, vparity, W_F_VFULL)) return false;
        const uint32_t vlo = lo_v + vstage * T16, acc0 = first ? 0u : 1u;
        first = false;
#pragma unroll
        for (int part = 0; part < C::NPART; ++part) {
          if (!wait(C::B_PFULL + C::NPART * i + part, pv_cnt & 1u, W_F_PFULL)) return false;
          tc_fence_after_sync();
#pragma unroll
          for (int j = 0; j < 4; ++j) {   // P of 16 keys = 8 packed columns
            const int kk = 4 * part + j;
            mma_ts_uniform(tO, tS + kk * 8, vlo + koff_mnmajor(kk), hi, idesc_o, kk > 0 ? 1u : acc0);
          }
        }
        commit_uniform(bar(C::B_PVDONE + 2 * i + (pv_cnt & 1u)));
        commit_uniform(bar(C::B_VEMPTY + vstage));
        ++pv_cnt;
        next_v();
        return true;
      };
      bool ok = true;
      int4 it;
      for (int k = 0; ok && next_item(k, it); ++k) {
        // The waits for Q and K that follow are bounded, and the loads they wait for are issued behind the producer's wait for the
        // kernel ahead: the limit must not run while that kernel does (a caller's may let this one start early and take long).
        if (k == 0) pdl_wait();
        const int n = it.w & 0xFF, ntile_q = (2 * it.z + 1 < a.NT) ? 2 : 1;
        int left = (it.w >> (8 + 8 * i)) & 0xFF;   // units without scores
        const int q_slot = C::QR::slot(q_cnt + i);
        if (i < ntile_q) {
          const int full = C::QR::full(q_cnt + i, i);
          if (!(ok = wait(C::B_QFULL + full, q_phases.take(full), W_F_QFULL))) break;
          if (left == 0 && elect_one()) mbar_arrive(bar(C::B_QEMPTY + q_slot));
        }
        q_cnt += ntile_q;
        const uint16_t* list = sList + (k % C::NITEM) * 128;
        const uint32_t qlo = lo_q + q_slot * T16;
        uint32_t ahead = list[0];
        bool pending = false;   // a unit's P V has not been issued
        first = true;
        for (int e = 0; e < n; ++e) {
          const uint32_t ent = __reduce_or_sync(0xffffffffu, ahead);
          ahead = list[min(e + 1, 127)];
          // The unit in flight comes first: the next scores lie over its P, and an entry that is passed on may need the room its
          // K and V take.
          if (pending && !(ok = issue_pv())) break;
          pending = false;
          if (!(ok = wait(C::B_KFULL + kstage, kparity, W_F_KFULL))) break;
          if (entry_class(ent, i) == 0u) {   // not this tile's
            if (!(ok = wait(C::B_VFULL + vstage, vparity, W_F_VFULL))) break;
            if (elect_one()) {
              mbar_arrive(bar(C::B_KEMPTY + kstage));
              mbar_arrive(bar(C::B_VEMPTY + vstage));
            }
            next_k();
            next_v();
            continue;
          }
          // Tile 1's exponentials half a unit behind tile 0's. (With long lists that comes by itself, and the wait costs causal
          // 8 x 16 x 2048 x 128 0.7 %.)
          if (i == 1 && k == 0 && e == 0 && tiles_take_turns(ent, n)) {
            const uint32_t t0 = clock32();
            while (clock32() - t0 < 900u) {}
          }
          tc_fence_after_sync();
          const uint32_t klo = lo_k + kstage * T16;
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) mma_ss_uniform(tS, qlo + koff_kmajor(kk), klo + koff_kmajor(kk), hi, idesc_s, kk > 0 ? 1u : 0u);
          commit_uniform(bar(C::B_SFULL + i));
          commit_uniform(bar(C::B_KEMPTY + kstage));
          if (--left == 0) commit_uniform(bar(C::B_QEMPTY + q_slot));   // the tile's last product
          next_k();
          pending = true;
        }
        // (before the wait for the next header: the producer may need this unit to be finished to publish it)
        if (!ok || (pending && !(ok = issue_pv()))) break;
        item_done(k);
      }
    }
  } else {
    reg_alloc<C::REGS_COMPUTE>();
    // ------------------------------ softmax warps: a thread per row ------------------------------
    const int i = (warp - 4) >> 2;        // query tile of the pair
    const int wq = warp & 3;              // TMEM lane quadrant of this warp
    const int row = wq * 32 + lane;       // row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = lane_base + C::TM_S + i * KD_TILE, tO = lane_base + C::TM_O + i * HD;
    constexpr int NW = KD_TILE / 32;      // words of a row's mask; the scores are worked on 32 at a time
    const float c = a.scale_log2;
    const uint64_t c2 = pack_f32x2(c, c);
    bool ok = true;
    int n_seen = 0;   // units of this query tile so far, over all items
    // Waits for the P V of the unit `back` units before. The products signal on two barriers in turn; a parity wait is sound
    // while the barrier's phase before the awaited one is complete, that is the product two before it, and that one was
    // complete when the scores of the unit after it were ready.
    auto pv_done = [&](int back) -> bool {
      const int c = n_seen - back;
      return c < 0 || wait(C::B_PVDONE + 2 * i + (c & 1), (c >> 1) & 1, W_F_PVDONE);
    };
    // The next item's header and first unit's mask are fetched before the epilogue of the item in hand, and for the first
    // item before the wait for the kernel ahead, which hides their latency.
    int4 it = make_int4(0, 0, 0, 0);
    int n_next = 0, qi_next = 0;
    uint32_t ent_next = 0u;   // the first (then: the next) unit's entry
    const uint16_t* list = sOwn;
    // Visibility of the 128 keys of a PARTIAL tile for this thread's query, of the coming unit (from the plan, see attn_fwd.cu)
    uint32_t mk[NW] = {0u, 0u, 0u, 0u};
    const uint32_t* words = a.words;   // of this thread's query in the item's query tile
    uint32_t qd_next = 0u;             // without words: its descriptor
    auto fetch_words = [&](uint32_t ent) {
      if (!kWords || (ent & 0x100u) == 0u) return;
      const uint32_t* src = words + (ent & 0xFF) * static_cast<int>(KD_WORDS);
#pragma unroll
      for (int w = 0; w < NW; ++w) mk[w] = __ldcg(src + w * KD_TILE);
    };
    auto open_item = [&](int k) -> bool {
      if (!next_item(k, it)) return false;
      const int qtile = 2 * it.z + i;
      if (kWords) words = a.words + ((size_t)it.x * a.NT + qtile) * a.NT * KD_WORDS + row;
      else if (qtile < a.NT) qd_next = __ldcg(a.desc + (size_t)it.x * a.Tpad + qtile * KD_TILE + row);
      n_next = (it.w >> (8 + 8 * i)) & 0xFF;
      const int only = it.w >> 24;
      const bool mine = only == 0 || only == i + 1;
      qi_next = mine ? qtile * KD_TILE + row : INT_MAX;   // (written by the other item of the pair)
      list = sOwn + (k % C::NITEM) * 256 + i * 128;
      if (n_next > 0) {
        ent_next = list[0];
        fetch_words(ent_next);
      }
      return true;
    };

    bool have = open_item(0);
    pdl_wait();   // O and LSE are written from here on
    for (int k = 0; have; ++k) {
      const int b = it.x, h = it.y, n_own = n_next, qi = qi_next;   // qi: token index of this thread's query
      const uint32_t qd = qd_next;
      float m = -INFINITY, l = 0.f;
#pragma unroll 1
      for (int u = 0; u < n_own; ++u) {
        const uint32_t ent = ent_next;
        if (u + 1 < n_own) ent_next = list[u + 1];
        if (!kWords && (ent & 0x100u) != 0u) {   // (here, where no scores are held in registers: behind the exponentials every unit is 9 % longer)
          const KeyRun<NW> keys(a.desc + (size_t)b * a.Tpad, a.tilebits + (size_t)b * a.NT * 32, ent & 0xFF, 0, lane);
          keys.words(qd, qi, mk);
        }
        if (!(ok = wait(C::B_SFULL + i, n_seen & 1, W_F_SFULL))) break;
        tc_fence_after_sync();
        float sc[KD_TILE];
#pragma unroll
        for (int cb = 0; cb < NW; ++cb) {
          uint32_t r[32];
          tmem_ld32(tS + cb * 32, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) sc[cb * 32 + j] = __uint_as_float(r[j]);
        }
        tmem_wait_ld();
        if (ent & 0x100u) {
#pragma unroll
          for (int w = 0; w < NW; ++w) {
            if (__all_sync(0xffffffffu, mk[w] == 0xFFFFFFFFu)) continue;   // all 32 keys visible to all 32 queries
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if ((mk[w] & (1u << j)) == 0u) sc[w * 32 + j] = -INFINITY;
          }
        }
        // four independent chains for the row maximum: a single chain of dependent operations would be latency-bound
        float mx4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
        for (int j = 4; j + 8 <= KD_TILE; j += 8) {   // three-input maximum: two new scores per instruction
          mx4[0] = fmax3(mx4[0], sc[j + 0], sc[j + 4]);
          mx4[1] = fmax3(mx4[1], sc[j + 1], sc[j + 5]);
          mx4[2] = fmax3(mx4[2], sc[j + 2], sc[j + 6]);
          mx4[3] = fmax3(mx4[3], sc[j + 3], sc[j + 7]);
        }
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) mx4[k4] = fmaxf(mx4[k4], sc[KD_TILE - 4 + k4]);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // The running maximum is refreshed only when it would grow by more than 2^8 in the exponent (or is -inf: the difference is
        // then inf); until then the stale value is used consistently for P, l and O, which leaves the normalised result unchanged
        // and skips most O rescales.
        const bool grow = (mx - m) * c > 8.0f;
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = grow ? mx : m, alpha = (m == -INFINITY) ? 0.f : fast_exp2((m - m_new) * c);
          if (u > 0 && __any_sync(0xffffffffu, grow && m != -INFINITY)) {   // O may be touched only after the tile's previous product
            if (!(ok = pv_done(1))) break;
            tc_fence_after_sync();
            const float f = grow ? alpha : 1.f;
            // 64 columns at a time (the scores are still in registers). With outliers among Q and K a third of a warp's units come here,
            // and 16 columns loaded and awaited at a time made them 300 cycles longer: 4 x 32 x 8192 x 128 fp16, hierarchical, 0.1 %
            // outliers 1011 us -> 963 (32 columns 969), causal 2 x 16 x 4096 x 128 164 -> 154; normally distributed inputs are level.
            const uint64_t f2 = pack_f32x2(f, f);
#pragma unroll 1
            for (int cb = 0; cb < HD / 64; ++cb) {
              uint32_t r[4][16];
#pragma unroll
              for (int x = 0; x < 4; ++x) tmem_ld16(tO + cb * 64 + x * 16, r[x]);
              tmem_wait_ld();
#pragma unroll
              for (int x = 0; x < 4; ++x) {
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                  const uint64_t y = mul_f32x2(pack_u32x2(r[x][j], r[x][j + 1]), f2);
                  r[x][j] = __float_as_uint(lo_f32x2(y));
                  r[x][j + 1] = __float_as_uint(hi_f32x2(y));
                }
                tmem_st16(tO + cb * 64 + x * 16, r[x]);
              }
            }
          }
          if (grow) l *= alpha;
          m = m_new;
        }
        const float m_use = (m == -INFINITY) ? 0.f : m;
        const uint64_t neg_mc2 = pack_f32x2(-m_use * c, -m_use * c);
        uint64_t sum2[2] = {0u, 0u};
#pragma unroll
        for (int part = 0; part < C::NPART; ++part) {   // 64 keys at a time; P over the first columns of the scores, which are in registers
          uint32_t pk[32];
#pragma unroll
          for (int j = 0; j < 64; j += 2) {
            const uint64_t x = fma_f32x2(pack_f32x2(sc[part * 64 + j], sc[part * 64 + j + 1]), c2, neg_mc2);
            const float p0 = fast_exp2(lo_f32x2(x)), p1 = fast_exp2(hi_f32x2(x));
            sum2[(j / 2) & 1] = add_f32x2(sum2[(j / 2) & 1], pack_f32x2(p0, p1));
            pk[j / 2] = pack2<kBf16>(p0, p1);
          }
          tmem_st32(tS + part * 32, pk);
          // this part of P is complete: its product runs under the next exponentials
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_PFULL + C::NPART * i + part));
        }
        const uint64_t sum_pair = add_f32x2(sum2[0], sum2[1]);
        l += lo_f32x2(sum_pair) + hi_f32x2(sum_pair);
        ++n_seen;
        if (u + 1 < n_own) fetch_words(ent_next);   // while its scores are formed
      }
      if (!ok) break;
      item_done(k);
      have = open_item(k + 1);

      // epilogue of this item: normalise, convert, store this thread's row of O, and LSE
      if (n_own > 0 && !(ok = pv_done(2) && pv_done(1))) break;
      uint32_t r[HD / 32][32];   // (the scores' registers)
      if (n_own > 0) {
        tc_fence_after_sync();
#pragma unroll
        for (int cb = 0; cb < HD / 32; ++cb) tmem_ld32(tO + cb * 32, r[cb]);
        tmem_wait_ld();
        // this thread's row of O_i has been read out: the next item's first product may overwrite it
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_OFREE + i));
      } else {
#pragma unroll
        for (int cb = 0; cb < HD / 32; ++cb)
#pragma unroll
          for (int j = 0; j < 32; ++j) r[cb][j] = 0u;
      }
      if (qi < a.T) {
        const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
        uint16_t* orow = reinterpret_cast<uint16_t*>(a.o) + (size_t)b * a.o_sb + (size_t)h * a.o_sh + (size_t)qi * a.o_st;
#pragma unroll
        for (int cb = 0; cb < HD / 32; ++cb) {
          if (!kF32 || a.o != nullptr) store_row32_upto<kBf16>(orow + cb * 32, r[cb], inv_l, cb * 32, a.d_real);
          if (kF32)
            store_row32_f32_upto(a.o32 + (size_t)b * a.o32_sb + (size_t)h * a.o32_sh + (size_t)qi * a.o32_st + cb * 32, r[cb], inv_l, cb * 32, a.d_real);
        }
        if (a.lse != nullptr) a.lse[((size_t)b * a.H + h) * a.T + qi] = (l > 0.f) ? (m * c + log2f(l)) : -INFINITY;
      }
    }  // items
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(0, 512);
  if (tid == 0) report_abort(abortf, a.status);
}

template <bool kBf16, bool kF32, bool kWords>
static int launch_wide_t(long long n_items, const FwdArgs& a, const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, cudaStream_t stream) {
  using C = FwdWideCfg;
  auto kern = attn_fwd_wide_kernel<kBf16, kF32, kWords>;
  static SmemOptIn opt_in;
  cudaError_t e = opt_in(kern, C::SMEM_ALLOC);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fwd smem attribute: %s", cudaGetErrorString(e));
  // The warps re-divide the registers the CTA was launched with; a request beyond that pool would block for ever,
  // so a build whose per-thread count is below the one the division assumes is refused here.
  static std::atomic<int> launch_regs{0};
  int regs = launch_regs.load(std::memory_order_relaxed);
  if (regs == 0) {
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fwd attributes: %s", cudaGetErrorString(e));
    launch_regs.store(regs = fa.numRegs, std::memory_order_relaxed);
  }
  if (regs < C::REGS_LAUNCH) return set_error(KD_ERR_DEVICE, "fwd was built with %d registers per thread, needs %d", regs, C::REGS_LAUNCH);
  e = launch(kern, static_cast<unsigned>(n_items), C::THREADS, C::SMEM_ALLOC, stream, tmQ, tmK, tmV, a);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "attn_fwd_wide_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

int launch_attn_fwd_wide(long long n_items, const FwdArgs& a, int dtype, const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                         cudaStream_t stream) {
  auto run = [&](auto launch_fn) { return launch_fn(n_items, a, tmQ, tmK, tmV, stream); };
  if (a.words == nullptr) return a.o32 != nullptr ? run(launch_wide_t<false, true, false>) : dtype == KD_BF16 ? run(launch_wide_t<true, false, false>) : run(launch_wide_t<false, false, false>);
  return a.o32 != nullptr ? run(launch_wide_t<false, true, true>) : dtype == KD_BF16 ? run(launch_wide_t<true, false, true>) : run(launch_wide_t<false, false, true>);
}

}  // namespace kd
