// Forward kernel for head dims up to 64, and the dispatch: O = softmax(mask(Q K^T * scale)) V and base-2 LSE, for sm_100a.
//
// A work item is a pair of 128-row query tiles of one (batch, head); it walks the plan's list of key tiles that are
// non-empty for either of them. The grid has a CTA per item, but a running CTA takes further items by cancelling CTAs
// that have not been launched yet (clusterlaunchcontrol) and works on them without draining its pipeline. Items are
// numbered in chunks of heads that fit L2 together, inside a chunk by decreasing list length. (With one CTA per item or
// group of heads, a fifth of the time went into CTA starts and a last wave that was nearly empty.)
// Roles (warp-specialised, 640 threads):
//   warp 0      takes items, stages their lists, loads Q tiles and the K and V rings by TMA
//   warp 1      issues S = Q_i K^T (smem x smem -> TMEM) and O_i += P V (TMEM x smem -> TMEM)
//   warps 4-11  softmax of query tile 0: TMEM -> registers, rule on PARTIAL tiles, online softmax in base 2, P back to TMEM as
//   warps 12-19 softmax of query tile 1  16-bit operand. Two warps share 32 rows, 64 columns each, and exchange row maxima.
//
// What bounds it. An exponential per score: 1,024 cycles of the special-function units per 128 x 128 tile, twice what the
// tensor cores need at D = 64. With one warp per 32 rows (eight softmax warps) the units were busy 65 % of the time, because
// while a warp loads, masks and reduces its 128 columns only one other warp of its scheduler can compute exponentials. Two
// warps to a row spend half as long outside the exponentials, at the price of one exchange of row maxima per unit.
//
// A "unit" is one (key tile, query tile) product that is not EMPTY. Units are numbered in list order over all items; unit u
// computes its scores into TMEM buffer u % NBUF (128 fp32 columns), and P (32 columns of packed pairs for each half of the
// keys) is written over the same buffer. S(u + NBUF) is issued directly after P(u) V, so that a softmax warp that finishes
// unit u finds the scores of its tile's next unit in TMEM. The tensor pipe executes in issue order, which is what allows
// S(u + NBUF) to overwrite the buffer P(u) was read from.
// Measured, bf16: hierarchical masks 8 x 16 x 4096 x 64 215 us, causal 8 x 16 x 1000 x 64 38.9; 1,400 cycles a tile with full lists, of
// which the special-function units are busy 1,024. (The issuing warp's steps take as long one after the other, but a loop a fifth
// shorter, with what it needs of a unit in one byte, changed nothing.)
// Tried and slower: a quarter of the exponentials as polynomials on the FMA pipe (5-9 %); an issuing warp per query tile, or one for
// the scores and one for P V (the issuing warp's order is what keeps the exponentials of the two tiles apart: in phase, full lists
// 1,600, short ones +10 %); the first half of the exponentials before the exchange of maxima (1,550); the next scores loaded
// ahead (1,650); eight softmax warps with a thread per row, as above head dim 64 (1,465, short lists +10 %).
// EMPTY tiles never appear in the list: they are neither loaded nor multiplied.
//
// Replaces _flash_attn_fwd (original_kernel.py:278-626): same math (scores scaled by
// sm_scale*log2(e), exp2, LSE = m + log2(l)); rows without any visible key give O = 0 and
// LSE = -inf.
#include <algorithm>

#include "attn_fwd.cuh"
#ifdef KD_TEST_DROP_LOAD
#include <stdlib.h>
#endif

namespace kd {

#ifdef KD_TEST_DROP_LOAD
// Test build only: a caller's kernel that lets the next one start at once and goes on for `ns` nanoseconds.
__global__ void test_busy_kernel(uint64_t ns) {
  pdl_launch_dependents();
  auto now = [] {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
  };
  const uint64_t t0 = now();
  for (uint32_t i = 0; i < (1u << 20) && now() - t0 < ns; ++i) __nanosleep(1000);
}
#endif

struct FwdCfg {
  static constexpr int HD = 64;
  static constexpr int KBLK = HD / 64;                   // 64-element blocks along D
  static constexpr int TILE_BYTES = KD_TILE * HD * 2;    // one Q / K / V tile
  static constexpr int NBUF = 3;                         // score buffers in TMEM
  static constexpr int KST = NBUF;                       // K ring stages
  static constexpr int VST = 3;                          // V ring stages
  using QR = FwdQRing;                                   // ring of Q tiles (two per item): four slots, the next item's Q loads while this one computes
  static constexpr int NQ = QR::SLOTS;
  static constexpr int NPART = 2;                        // P is handed over in two parts: the first, then the second 32 columns of each half
  static constexpr int NITEM = 4;                        // ring of item headers and lists
  static constexpr int NXB = 2;                          // buffers of the row maxima that two warps exchange (see there)
  static constexpr int SMEM_Q = 0;
  static constexpr int SMEM_K = SMEM_Q + NQ * TILE_BYTES;
  static constexpr int SMEM_V = SMEM_K + KST * TILE_BYTES;
  static constexpr int SMEM_O = SMEM_V + VST * TILE_BYTES;         // O on its way out: per softmax warp a box [32 rows][32 columns], 64-byte swizzle
  static constexpr int SMEM_LIST = SMEM_O + 16 * 2048;             // NITEM x <= 128 list entries
  static constexpr int SMEM_ITEM = SMEM_LIST + NITEM * 128 * 2;    // NITEM x {batch, head, pair, entries | units of tile 0 << 8 | of tile 1 << 16 | the item's only tile + 1 << 24}
  static constexpr int SMEM_XCH = SMEM_ITEM + NITEM * 16;          // NXB x [query tile][half][row] fp32
  static constexpr int SMEM_CLC = SMEM_XCH + NXB * 4 * KD_TILE * 4;
  static constexpr int SMEM_BAR = SMEM_CLC + 16;
  // barriers (8 bytes each)
  static constexpr int B_QFULL = 0, B_QEMPTY = B_QFULL + QR::FULL, B_KFULL = B_QEMPTY + NQ, B_KEMPTY = B_KFULL + KST, B_VFULL = B_KEMPTY + KST,
                       B_VEMPTY = B_VFULL + VST, B_SFULL = B_VEMPTY + VST, B_PFULL = B_SFULL + 2 * NBUF,
                       B_PVDONE = B_PFULL + NPART * NBUF, B_OFREE = B_PVDONE + 4, B_ITEMFULL = B_OFREE + 2, B_ITEMEMPTY = B_ITEMFULL + NITEM,
                       B_CLC = B_ITEMEMPTY + NITEM, NBAR = B_CLC + 1;
  static constexpr int SMEM_ALLOC = SMEM_BAR + NBAR * 8 + 16;
  static constexpr int CW = KD_TILE / 2;                 // score columns per softmax thread: half a row
  static constexpr int THREADS = 640;                    // four light warps + eight softmax warps per query tile
  // registers: 96 per thread at launch; light warps release down to 56, softmax warps take 104
  static constexpr int REGS_LIGHT = 56, REGS_COMPUTE = 104;
  static_assert(4 * 32 * REGS_LIGHT + 16 * 32 * REGS_COMPUTE <= THREADS * 96, "register pool");
  // TMEM columns: NBUF score buffers of 128, then O0 and O1 (HD each)
  static constexpr uint32_t TM_O0 = NBUF * 128, TM_O1 = NBUF * 128 + HD;
  static_assert(TM_O1 + HD <= 512, "TMEM budget");
  static_assert(SMEM_O % 512 == 0, "a 64-byte swizzle repeats every 512 bytes");
  static_assert(SMEM_ALLOC <= 232448, "shared memory budget");
};

// kF32: of a float32 call: O goes to a float32 tensor, and to a 16-bit one where there will be a backward. (As a branch of the float16 kernels the
// second store cost short lists above head dim 64 4 %.)
// kWords: the plan has the PARTIAL tiles' bits (see KD_WORDS_LIMIT).
template <bool kBf16, bool kF32, bool kWords>
__global__ void __launch_bounds__(FwdCfg::THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdArgs a) {
  using C = FwdCfg;
  constexpr int HD = C::HD, TILE = C::TILE_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t s0 = smem_u32(smem);
  const uint32_t sQ = s0 + C::SMEM_Q, sK = s0 + C::SMEM_K, sV = s0 + C::SMEM_V;
  uint16_t* sList = reinterpret_cast<uint16_t*>(smem + C::SMEM_LIST);
  int4* items = reinterpret_cast<int4*>(smem + C::SMEM_ITEM);
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
  if (tid < C::NBAR) {   // a thread each: one after the other they took 900 cycles of a CTA's start
    const int i = tid;
    uint32_t count = 1;
    // One "scores ready" barrier per (buffer, query tile): each softmax warpgroup then sees every phase of the barriers it
    // waits on, which is what makes a parity wait sound. P and O barriers: one arrival per softmax warp.
    if ((i >= C::B_PFULL && i < C::B_PVDONE) || (i >= C::B_OFREE && i < C::B_ITEMFULL)) count = 8;
    if (i >= C::B_ITEMEMPTY && i < C::B_CLC) count = 17;   // the issuer and sixteen softmax warps
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
  // A plan that an earlier launch on this stream has used was complete when the kernel before this one let it start (a kernel
  // lets its successor start only when its own predecessors are complete): its lists and words may be read before the
  // wait, which hides three dependent look-ups under the predecessor (in a stack of layers, 2 us of each kernel's 9 at T = 173).
  // They are read past L1, which the start of a kernel that overlaps another need not have cleaned.
  if (!a.plan_ready) pdl_wait();
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
      uint32_t unit0 = 0u;  // score buffer of the next item's first unit
      // in shared memory an entry has the score buffer of its first unit << 12 as well
      auto publish = [&](int slot, const uint32_t (&lst)[4], int, int (&units)[2]) {
        int e = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t has0 = __ballot_sync(0xffffffffu, entry_class(lst[r], 0) != 0u), has1 = __ballot_sync(0xffffffffu, entry_class(lst[r], 1) != 0u);
          const uint32_t first = (unit0 + units[0] + units[1] + __popc(has0 & below) + __popc(has1 & below)) % C::NBUF;
          if (lst[r] != 0u) sList[slot * 128 + e + __popc((has0 | has1) & below)] = static_cast<uint16_t>(lst[r] | (first << 12));
          e += __popc(has0 | has1);
          units[0] += __popc(has0);
          units[1] += __popc(has1);
        }
        unit0 = (unit0 + units[0] + units[1]) % C::NBUF;
      };
      fwd_producer<C>(tmQ, tmK, tmV, a, smem, abortf, lane, wait, publish);
    } else if (warp == 1) {
      // ------------------------------ issuer ------------------------------
      // All lanes follow the control flow and one elected lane issues (mma_ss_uniform). One warp issues both products: the
      // scores of unit u + NBUF follow P(u) V directly, and what they need (the header, K, Q) has been waited for before
      // P(u) is. (In two warps, the hand-over cost a softmax warpgroup about 600 cycles per unit.)
      const uint32_t idesc_s = make_idesc_f16(kBf16, 0, 0, KD_TILE, KD_TILE), idesc_o = make_idesc_f16(kBf16, 0, 1, KD_TILE, HD);
      const uint32_t hi = desc_hi_sw128(), lo_q = desc_lo_kmajor(sQ), lo_k = desc_lo_kmajor(sK), lo_v = desc_lo_mnmajor(sV);
      constexpr uint32_t T16 = TILE >> 4;
      // A wait costs this warp 150-200 cycles even when the phase is complete, for it shares its scheduler with softmax warps; with
      // five of them one after the other and a walk over the list by entry and tile a unit took 1,550 cycles, more than the
      // exponentials. So the tests of an iteration are issued together, and the next list entry is fetched one entry ahead.
      // place in the stream of units: item k with n entries, `e` of them begun; unit = tile `i` of entry `ent`
      int k = 0, n = 0, e = 0, i = 1, kstage = -1, q_cnt = 0, ntile_q = 0;
      uint32_t ent = 0, ent_ahead = 0, kparity = 1u, left = 0, q_there = 0;   // units left of tile 0 | of tile 1 << 8; bit i: Q tile i has landed
      bool open = false;    // item k is being worked on
      bool new_k = false;   // the unit is the first of its entry
      int n_flight = 0;     // units whose scores have been issued and whose P V has not
      enum : int { UNIT, STALLED, ENDED, ABORTED };
      auto wait_q = [&](int t) -> bool {
        q_there |= 1u << t;
        const int g = q_cnt + t;
        return wait(C::B_QFULL + g % C::NQ, (g / C::NQ) & 1, W_F_QFULL);
      };
      // Closes the item in hand and opens the next one that has entries. With units in flight it does not wait for a header,
      // for the producer may need them to be finished to publish it (a run of empty items longer than the ring of headers).
      auto next_list = [&]() -> int {
        for (;;) {
          if (open) {
            for (int t = 0; t < ntile_q; ++t) {   // tiles without units
              if ((q_there >> t) & 1u) continue;
              if (!wait_q(t)) return ABORTED;
              if (elect_one()) mbar_arrive(bar(C::B_QEMPTY + (q_cnt + t) % C::NQ));
            }
            q_cnt += ntile_q;
            item_done(k);
            open = false;
            ++k;
          }
          if (n_flight > 0 && !__all_sync(0xffffffffu, mbar_test_wait(bar(C::B_ITEMFULL + k % C::NITEM), (k / C::NITEM) & 1))) return STALLED;
          int4 it;
          if (!next_item(k, it)) return abortf->v == 0u ? ENDED : ABORTED;
          // The waits for Q and K that follow are bounded, and the loads they wait for are issued behind the producer's wait for the
          // kernel ahead: the limit must not run while that kernel does (a caller's may let this one start early and take long).
          if (k == 0) pdl_wait();
          n = it.w & 0xFF;
          left = static_cast<uint32_t>(it.w) >> 8;
          ntile_q = (2 * it.z + 1 < a.NT) ? 2 : 1;
          e = 0;
          q_there = 0u;
          open = true;
          ent_ahead = sList[(k % C::NITEM) * 128];
          if (n > 0) return UNIT;
        }
      };
      // What P V needs to know of the units whose scores are in flight, oldest in the low byte
      constexpr uint32_t U_TILE = 1u, U_FIRST = 2u, U_NEW_V = 4u, U_LAST_V = 8u;
      uint32_t flight = 0u, pv_issued = 0u, used = 0u, used_par = 0u, vparity = 1u, pparity = 0u, began = 0u;
      int sbuf = 0, pbuf = 0, vstage = -1;
      for (;;) {
        int next = UNIT;
        if (i == 0 && entry_class(ent, 1) != 0u) {
          i = 1;
          new_k = false;
        } else {
          // (with every buffer taken a P V comes first: closing and opening an item takes this warp up to 1,800 cycles, which the
          // units in flight would wait for, to no purpose)
          if (e == n) next = n_flight == C::NBUF ? static_cast<int>(STALLED) : __reduce_max_sync(0xffffffffu, next_list());
          if (next == ABORTED) break;
          if (next == UNIT) {
            if (e == 0) began = 0u;
            ent = __reduce_or_sync(0xffffffffu, ent_ahead);
            ++e;
            ent_ahead = sList[(k % C::NITEM) * 128 + min(e, 127)];
            i = entry_class(ent, 0) != 0u ? 0 : 1;
            new_k = true;
            if (++kstage == C::KST) kstage = 0;
            if (kstage == 0) kparity ^= 1u;
          }
        }
        const bool s_now = next == UNIT, pv_now = n_flight == C::NBUF || (!s_now && n_flight > 0), new_v = pv_now && (flight & U_NEW_V) != 0u;
        if (new_v) {
          if (++vstage == C::VST) vstage = 0;
          if (vstage == 0) vparity ^= 1u;
        }
        bool there = true;
        if (s_now && new_k) there = mbar_test_wait(bar(C::B_KFULL + kstage), kparity);
        if (new_v) there &= mbar_test_wait(bar(C::B_VFULL + vstage), vparity);
        if (pv_now) there &= mbar_test_wait(bar(C::B_PFULL + C::NPART * pbuf), pparity);
        if (!__all_sync(0xffffffffu, there)) {
          if (s_now && new_k && !wait(C::B_KFULL + kstage, kparity, W_F_KFULL)) break;
          if (new_v && !wait(C::B_VFULL + vstage, vparity, W_F_VFULL)) break;
          if (pv_now && !wait(C::B_PFULL + C::NPART * pbuf, pparity, W_F_PFULL)) break;
        }
        if (s_now && ((q_there >> i) & 1u) == 0u && !wait_q(i)) break;
        if (pv_now) {
          const uint32_t t = flight & U_TILE;
          if (flight & U_FIRST) {
            // the first product of a query tile overwrites O: the softmax warps must have read the previous item's result
            if ((used >> t) & 1u) {
              if (!wait(C::B_OFREE + t, (used_par >> t) & 1u, W_F_OFREE)) break;
              used_par ^= 1u << t;
            }
            used |= 1u << t;
          }
          const uint32_t vlo = lo_v + vstage * T16, dO = C::TM_O0 + t * HD, acc0 = (flight & U_FIRST) ? 0u : 1u;
          tc_fence_after_sync();
#pragma unroll
          for (int part = 0; part < C::NPART; ++part) {
            if (part > 0) {
              if (!(there = wait(C::B_PFULL + C::NPART * pbuf + part, pparity, W_F_PFULL))) break;
              tc_fence_after_sync();
            }
            // P of 16 keys = 8 packed columns; a warp's 64 keys begin at the first of its score columns
#pragma unroll
            for (int kk = 0; kk < KD_TILE / 16; ++kk) {
              if (((kk >> 1) & 1) != part) continue;
              mma_ts_uniform(dO, pbuf * 128 + (kk >> 2) * C::CW + (kk & 3) * 8, vlo + koff_mnmajor(kk), hi, idesc_o, kk > 0 ? 1u : acc0);
            }
          }
          if (!there) break;
          commit_uniform(bar(C::B_PVDONE + 2 * t + ((pv_issued >> t) & 1u)));
          pv_issued ^= 1u << t;
          if (flight & U_LAST_V) commit_uniform(bar(C::B_VEMPTY + vstage));
          if (++pbuf == C::NBUF) { pbuf = 0; pparity ^= 1u; }
          flight >>= 8;
          --n_flight;
        }
        if (s_now) {
          const uint32_t qlo = lo_q + ((q_cnt + i) % C::NQ) * T16, klo = lo_k + kstage * T16;
          tc_fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) mma_ss_uniform(sbuf * 128, qlo + koff_kmajor(kk), klo + koff_kmajor(kk), hi, idesc_s, kk > 0 ? 1u : 0u);
          commit_uniform(bar(C::B_SFULL + 2 * sbuf + i));
          const bool last_of_entry = i == 1 || entry_class(ent, 1) == 0u;
          if (last_of_entry) commit_uniform(bar(C::B_KEMPTY + kstage));
          left -= 1u << (8 * i);
          if (((left >> (8 * i)) & 0xFFu) == 0u) commit_uniform(bar(C::B_QEMPTY + (q_cnt + i) % C::NQ));   // the tile's last product
          flight |= (static_cast<uint32_t>(i) | (((began >> i) & 1u) ? 0u : U_FIRST) | (new_k ? U_NEW_V : 0u) | (last_of_entry ? U_LAST_V : 0u)) << (8 * n_flight);
          began |= 1u << i;
          ++n_flight;
          if (++sbuf == C::NBUF) sbuf = 0;
        } else if (next == ENDED && n_flight == 0) {
          break;
        }
      }
    }
  } else {
    reg_alloc<C::REGS_COMPUTE>();
    // ------------------------------ softmax warpgroups ------------------------------
    // Two warpgroups per query tile; each thread owns half a row, 64 scores.
    constexpr int CW = C::CW, NW = CW / 32;
    const int i = (warp - 4) >> 3;        // query tile of the pair
    const int half = ((warp - 4) >> 2) & 1;   // columns 64 * half .. 64 * half + 63
    const int wq = warp & 3;              // TMEM lane quadrant of this warp
    const int row = wq * 32 + lane;       // row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tO = lane_base + (i == 0 ? C::TM_O0 : C::TM_O1) + half * (HD / 2);   // this thread's half of its row of O
    float* xch = reinterpret_cast<float*>(smem + C::SMEM_XCH) + i * (2 * KD_TILE) + row;
    // Both warps of 32 rows: hands over a value and takes the partner's. Whether some role has aborted is read behind the barrier and
    // looked at before the next exchange, off the chain. The barrier cannot hang: a warp that gives up arrives there once more
    // (below), and the partner sees the abort behind it.
    // A slot is written again two exchanges later, when the partner, which has been to the barrier in between, has read it.
    const uint32_t pair_bar = 1 + i * 4 + wq;
    int exchanges = 0;
    uint32_t aborted = 0u;   // looked at before the next exchange
    auto exchange = [&](float mine, float& other) {
      float* x = xch + (exchanges++ % C::NXB) * (4 * KD_TILE);
      x[half * KD_TILE] = mine;
      named_bar_sync(pair_bar, 64);
      other = x[(half ^ 1) * KD_TILE];
      aborted = abortf->v;
    };
    const float c = a.scale_log2;
    const uint64_t c2 = pack_f32x2(c, c);
    bool ok = true;
    // state that runs on across the items of this CTA
    uint32_t sfull_par = 0;     // bit j: parity of the next phase of this tile's score barrier on buffer j
    int pv_seen = 0;            // P V products of this query tile handed over so far
    // Waits for the last of them (back = 1), or the one before. Not for every unit: a product signals on one of two barriers in
    // turn. A parity wait is sound while the barrier's phase before the awaited one is complete, that is the tile's product two
    // before it. Once the scores of the tile's next unit are ready it is (products and scores execute in issue order, and at
    // most NBUF - 1 products precede those scores unfinished); at the end of an item it is after a wait with back = 2.
    auto pv_done = [&](int back) -> bool {
      const int c = pv_seen - back;
      return c < 0 || wait(C::B_PVDONE + 2 * i + (c & 1), (c >> 1) & 1, W_F_PVDONE);
    };
    // The next item's header and first unit are fetched before the epilogue of the item in hand, which
    // hides their latency (they took 2,000 cycles of an item, of 35,000 for one of nine tiles).
    int4 it = make_int4(0, 0, 0, 0);
    int n_next = 0, qi_next = 0, e = 0, buf_next = 0;
    uint32_t ent_next = 0u, fetched = 0u;   // fetched: entry e of the list, read one step ahead
    const uint16_t* list = sList;
    // this query tile's next unit, of which there is one: sets ent_next and, in buf_next, its buffer
    auto find_next = [&]() {
      do {
        ent_next = __reduce_or_sync(0xffffffffu, fetched);
        ++e;
        fetched = list[min(e, 127)];
      } while (entry_class(ent_next, i) == 0u);
      buf_next = static_cast<int>(ent_next >> 12) + ((i == 1 && entry_class(ent_next, 0) != 0u) ? 1 : 0);
      if (buf_next >= C::NBUF) buf_next -= C::NBUF;
    };
    // The visibility words of a PARTIAL tile (bit j: key j of 32) are fetched one unit ahead into registers, so that their latency overlaps
    // the previous tile's softmax. They come with the plan: formed here, for every head anew, from class masks and descriptors they were
    // half of what masking costs (us, before -> now: hierarchical 16 x 16 x 4096 x 64 397 -> 368, 8 x 16 x 2048 x 64 59.4 -> 54.4, causal
    // 8 x 16 x 1000 x 64 38.0 -> 33.7, no mask 8 x 16 x 2048 x 64 level). Asked for behind the exchange of maxima; ahead of it or behind
    // the exponentials +0.5-2.5 %.
    uint32_t mk[NW] = {0u, 0u};
    const uint32_t* words = a.words;   // of this thread's query in the item's query tile
    auto fetch_words = [&](uint32_t ent) {
      if (!kWords || entry_class(ent, i) != KD_TILE_PARTIAL) return;
      const uint32_t* src = words + (ent & 0xFF) * static_cast<int>(KD_WORDS);
#pragma unroll
      for (int w = 0; w < NW; ++w) mk[w] = __ldcg(src + w * KD_TILE);
    };
    auto open_item = [&](int k) -> bool {
      if (!next_item(k, it)) return false;
      const int qtile = 2 * it.z + i;
      if (kWords) words = a.words + ((size_t)it.x * a.NT + qtile) * a.NT * KD_WORDS + half * NW * KD_TILE + row;
      n_next = (it.w >> (8 + 8 * i)) & 0xFF;
      const int only = it.w >> 24;
      const bool mine = only == 0 || only == i + 1;
      qi_next = mine ? qtile * KD_TILE + row : INT_MAX;   // (written by the other item of the pair)
      list = sList + (k % C::NITEM) * 128;
      e = 0;
      if (n_next > 0) {
        fetched = list[0];
        find_next();
        fetch_words(ent_next);
      }
      return true;
    };

    bool have = open_item(0);
    pdl_wait();   // O and LSE are written from here on
    for (int k = 0; have; ++k) {
    const int b = it.x, h = it.y, n_own = n_next, qi = qi_next;   // qi: token index of this thread's query
    float m = -INFINITY, l = 0.f;
    int nact = 0;
#pragma unroll 1
    for (int u = 0; u < n_own; ++u) {
      const uint32_t ent = ent_next;
      const uint32_t cls = entry_class(ent, i);
      const int sbuf = buf_next;
      if (!kWords && cls == KD_TILE_PARTIAL)
        form_words<NW>(a.desc + (size_t)b * a.Tpad, a.tilebits + (size_t)b * a.NT * 32, qi, ent & 0xFF, half * NW, lane, mk);
      const uint32_t tS = lane_base + sbuf * 128 + half * CW;
      if (!(ok = wait(C::B_SFULL + 2 * sbuf + i, (sfull_par >> sbuf) & 1u, W_F_SFULL))) break;
      sfull_par ^= 1u << sbuf;
      tc_fence_after_sync();

      float sc[CW];
#pragma unroll
      for (int cb = 0; cb < NW; ++cb) {
        uint32_t r[32];
        tmem_ld32(tS + cb * 32, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) sc[cb * 32 + j] = __uint_as_float(r[j]);
      }
      if (u + 1 < n_own) find_next();   // while the scores are on their way
      tmem_wait_ld();
      if (cls == KD_TILE_PARTIAL) {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          if (__all_sync(0xffffffffu, mk[w] == 0xFFFFFFFFu)) continue;   // all 32 keys visible to all 32 queries
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if ((mk[w] & (1u << j)) == 0u) sc[w * 32 + j] = -INFINITY;
        }
      }
      // four independent chains for the row maximum and for the row sum: a single chain of
      // dependent operations would be latency-bound
      float mx4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
      for (int j = 4; j + 8 <= CW; j += 8) {   // three-input maximum: two new scores per instruction
        mx4[0] = fmax3(mx4[0], sc[j + 0], sc[j + 4]);
        mx4[1] = fmax3(mx4[1], sc[j + 1], sc[j + 5]);
        mx4[2] = fmax3(mx4[2], sc[j + 2], sc[j + 6]);
        mx4[3] = fmax3(mx4[3], sc[j + 3], sc[j + 7]);
      }
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) mx4[k4] = fmaxf(mx4[k4], sc[CW - 4 + k4]);
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      float mx_other;
      exchange(mx, mx_other);
      if (u + 1 < n_own) fetch_words(ent_next);
      mx = fmaxf(mx, mx_other);
      // The running maximum is refreshed only when it would grow by more than 2^8 in the exponent (or is -inf: the difference is then
      // inf); until then the stale value is used consistently for P, l and O, which leaves the normalised result unchanged, skips
      // most O rescales and keeps the refresh out of the chain.
      const bool grow = (mx - m) * c > 8.0f;
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? mx : m, alpha = (m == -INFINITY) ? 0.f : fast_exp2((m - m_new) * c);
        if (nact > 0 && __any_sync(0xffffffffu, grow && m != -INFINITY)) {   // O may be touched only after the tile's previous product
          if (!(ok = pv_done(1))) break;
          tc_fence_after_sync();
          const float f = grow ? alpha : 1.f;
#pragma unroll 1
          for (int cb = 0; cb < HD / 32; ++cb) {   // rare; 16 columns at a time, for the scores are still in registers
            uint32_t r[16];
            tmem_ld16(tO + cb * 16, r);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * f);
            tmem_st16(tO + cb * 16, r);
          }
        }
        if (grow) l *= alpha;
        m = m_new;
      }
      const float m_use = (m == -INFINITY) ? 0.f : m;
      const uint64_t neg_mc2 = pack_f32x2(-m_use * c, -m_use * c);
      uint64_t sum2[2] = {0u, 0u};
#pragma unroll
      for (int cb = 0; cb < NW; ++cb) {   // 32 columns at a time; P over the start of this thread's own score columns
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const uint64_t x = fma_f32x2(pack_f32x2(sc[cb * 32 + j], sc[cb * 32 + j + 1]), c2, neg_mc2);
          const float p0 = fast_exp2(lo_f32x2(x)), p1 = fast_exp2(hi_f32x2(x));
          sum2[(j / 2) & 1] = add_f32x2(sum2[(j / 2) & 1], pack_f32x2(p0, p1));
          pk[j / 2] = pack2<kBf16>(p0, p1);
        }
        tmem_st16(tS + cb * 16, pk);
        // this part of P is complete: its product runs under the next exponentials
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_PFULL + C::NPART * sbuf + cb));
      }
      const uint64_t sum_pair = add_f32x2(sum2[0], sum2[1]);
      l += lo_f32x2(sum_pair) + hi_f32x2(sum_pair);
      ++nact;
      ++pv_seen;
      if (!(ok = __all_sync(0xffffffffu, aborted == 0u))) break;
    }
    if (!ok) break;
    item_done(k);
    have = open_item(k + 1);

    // epilogue of this item: normalise, convert, store this thread's share of O, and LSE
    if (nact > 0 && !(ok = pv_done(2) && pv_done(1))) break;
    float l_other;
    exchange(l, l_other);
    if (!(ok = __all_sync(0xffffffffu, aborted == 0u))) break;
    l += l_other;
    if (half == 0 && qi < a.T && a.lse != nullptr) {
      a.lse[((size_t)b * a.H + h) * a.T + qi] = (l > 0.f) ? (m * c + log2f(l)) : -INFINITY;
    }
    {
      tc_fence_after_sync();
      const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
      uint16_t* orow = reinterpret_cast<uint16_t*>(a.o) + (size_t)b * a.o_sb + (size_t)h * a.o_sh + (size_t)qi * a.o_st;
#pragma unroll
      for (int cb = 0; cb < HD / 64; ++cb) {
        uint32_t r[32];
        if (nact > 0) {
          tmem_ld32(tO + cb * 32, r);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        if (cb == HD / 64 - 1 && nact > 0) {
          // this thread's share of O_i has been read out: the next item's first product may overwrite it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_OFREE + i));
        }
        const int col = half * (HD / 2) + cb * 32;
        if (a.o_tma != 0) {
          const int row0 = __reduce_min_sync(0xffffffffu, qi);   // INT_MAX: written by the other item of the pair
          if (row0 < a.T && col < a.d_real) {   // (both are the warp's)
            const uint32_t box = s0 + C::SMEM_O + (warp - 4) * 2048;
            if (lane == 0) bulk_wait_group_read0();   // the last item's rows have been read
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t at = box + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at),
                           "r"(pack2<kBf16>(__uint_as_float(r[8 * j + 0]) * inv_l, __uint_as_float(r[8 * j + 1]) * inv_l)),
                           "r"(pack2<kBf16>(__uint_as_float(r[8 * j + 2]) * inv_l, __uint_as_float(r[8 * j + 3]) * inv_l)),
                           "r"(pack2<kBf16>(__uint_as_float(r[8 * j + 4]) * inv_l, __uint_as_float(r[8 * j + 5]) * inv_l)),
                           "r"(pack2<kBf16>(__uint_as_float(r[8 * j + 6]) * inv_l, __uint_as_float(r[8 * j + 7]) * inv_l))
                           : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {   // rows at or beyond T and columns at or beyond d_real are not written
              tma_store_4d(&tmO, box, col, row0, h, b);
              bulk_commit_group();
            }
          }
        } else if (qi < a.T && (!kF32 || a.o != nullptr)) store_row32_upto<kBf16>(orow + col, r, inv_l, col, a.d_real);
        if (kF32 && qi < a.T)
          store_row32_f32_upto(a.o32 + (size_t)b * a.o32_sb + (size_t)h * a.o32_sh + (size_t)qi * a.o32_st + col, r, inv_l, col, a.d_real);
      }
    }
    }  // items
    if (abortf->v != 0u) named_bar_arrive(pair_bar, 64);
    if (lane == 0) bulk_wait_group0();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(0, 512);
  if (tid == 0) report_abort(abortf, a.status);
}

template <bool kBf16, bool kF32, bool kWords>
static int launch_fwd_t(long long n_items, const FwdArgs& a, const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmO,
                        cudaStream_t stream) {
  auto kern = attn_fwd_kernel<kBf16, kF32, kWords>;
  static SmemOptIn opt_in;
  cudaError_t e = opt_in(kern, FwdCfg::SMEM_ALLOC);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fwd smem attribute: %s", cudaGetErrorString(e));
  e = launch(kern, static_cast<unsigned>(n_items), FwdCfg::THREADS, FwdCfg::SMEM_ALLOC, stream, tmQ, tmK, tmV, tmO, a);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "attn_fwd_kernel launch: %s", cudaGetErrorString(e));
  return 0;
}

int launch_attn_fwd(const kd_attn_params& p, const kd_attn_f32* f32, cudaStream_t stream) {
  kd_plan_layout L;
  if (kd_plan_layout_get(p.B, p.T, &L) != 0) return KD_ERR_ARG;
  const PlanView pv = make_plan_view(const_cast<void*>(p.plan), L);
  CUtensorMap tmQ, tmK, tmV;
  int rc;
  if ((rc = encode_tensor_map(&tmQ, p.q, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "q")) != 0) return rc;
  if ((rc = encode_tensor_map(&tmK, p.k, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "k")) != 0) return rc;
  if ((rc = encode_tensor_map(&tmV, p.v, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "v")) != 0) return rc;
  FwdArgs a;
  a.B = p.B; a.H = p.H; a.T = p.T; a.NT = L.NT; a.NP = L.NP; a.Tpad = L.NT * KD_TILE;
  a.d_real = p.D;
  a.scale_log2 = scale_log2_of(p.sm_scale);
  a.split = split_pairs((long long)p.B * p.H * L.NP, L.NT, sm_count());
  const long long n_items = ((long long)p.B * p.H * L.NP) << a.split;
  if (n_items > 0x7FFFFFFF) return set_error(KD_ERR_LIMIT, "B * H * ceil(T / 256) exceeds 2^31 - 1");
  // Q, K, V and O. (64 and 110 MB: no difference outside the noise)
  a.order_of = ItemOrder::make(p.B * p.H, L.NP << a.split, (double)p.T * p.D * 2 * 4, 64e6);
  a.plan_ready = p.plan_ready;
  a.words = pv.words; a.fwd_cnt = pv.fwd_cnt; a.fwd_list = pv.fwd_list; a.status = pv.status;
  a.order = pv.order; a.desc = pv.desc; a.tilebits = pv.tilebits;
  a.o = p.o.ptr; a.o_sb = p.o.stride_b; a.o_sh = p.o.stride_h; a.o_st = p.o.stride_t;
  a.o32 = f32 ? static_cast<float*>(f32->o.ptr) : nullptr;
  if (f32) { a.o32_sb = f32->o.stride_b; a.o32_sh = f32->o.stride_h; a.o32_st = f32->o.stride_t; }
  a.lse = p.lse;
#ifdef KD_TEST_DROP_LOAD
  const char* drop = getenv("KD_TEST_DROP_LOAD");
  a.test_drop_load = (drop != nullptr && atoi(drop) == 1) ? 1 : 0;
#endif
  // head dims below the tile width run on the next wider kernel: TMA zero-fills the missing columns
  if (p.D > 64) return launch_attn_fwd_wide(n_items, a, p.dtype, tmQ, tmK, tmV, stream);
  // O through TMA stores: a thread's 16-byte stores to its own row are 32 lines an instruction, 1,240 cycles of an item's end with sixteen
  // warps at it (short bursts: hierarchical 16 x 16 x 4096 x 64 416 -> 406 us, 8 x 16 x 2048 x 64 66.3 -> 64.5; causal 113.9 -> 111.1; no mask
  // 187.6 -> 182.3; passes of 8 x 16 x 4096 x 64 one after the other 234 -> 229). Not where a CTA has one item: its rows leave as soon either way, and the map costs the host time. (Nor for strides
  // that a map cannot have: 0 or below.)
  CUtensorMap tmO = tmQ;
  a.o_tma = n_items > sm_count() && p.o.ptr != nullptr && encode_tensor_map(&tmO, p.o, p.B, p.H, p.T, p.D, p.dtype, 32, nullptr, 64) == 0 ? 1 : 0;
  auto run = [&](auto launch_fn) { return launch_fn(n_items, a, tmQ, tmK, tmV, tmO, stream); };
  if (a.words == nullptr) return f32 ? run(launch_fwd_t<false, true, false>) : p.dtype == KD_BF16 ? run(launch_fwd_t<true, false, false>) : run(launch_fwd_t<false, false, false>);
  return f32 ? run(launch_fwd_t<false, true, true>) : p.dtype == KD_BF16 ? run(launch_fwd_t<true, false, true>) : run(launch_fwd_t<false, false, true>);
}

}  // namespace kd

#ifdef KD_TEST_DROP_LOAD
extern "C" int kd_test_busy(uint64_t ns, void* stream) {
  kd::test_busy_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(ns);
  return static_cast<int>(cudaGetLastError());
}
#endif
