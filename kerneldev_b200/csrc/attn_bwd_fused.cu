// Fused backward on sm_100a: dK, dV and dQ from ONE pass over the non-empty tiles (head dims up to 128).
//
// The two-kernel backward (attn_bwd.cu) follows the reference's split into a dQ worker and a dK/dV
// worker (original_kernel.py:1173-1336, :1339-1525) and so forms S = Q K^T, dP = dO V^T and the
// exponentials twice per tile: 7 matrix products and two exponential passes. This kernel is key-tile
// major like the dK/dV worker and forms them once: per (query tile, key tile)
//     S^T = K Q^T, dP^T = V dO^T                           (smem x smem -> TMEM)
//     P^T = exp2(S^T c - LSE), dS^T = P^T (dP^T - delta)   (compute warps; 16-bit results)
//     dV += P^T dO                                         (P^T read from TMEM as the A operand)
//     dK += dS^T Q,  dQ_tile = dS K                        (dS^T written to shared memory once and read by
//                                                           the tensor core K-major for dK, MN-major for dQ)
// 5 products and one exponential pass. dK and dV stay in TMEM for the whole key tile; the dQ partial of
// every tile is added to an fp32 scratch (B,H,T,HD) by TMA bulk reductions (cp.reduce.async.bulk.tensor
// .add, fp32 adds performed in L2 on whole 128-byte lines; the additions of different key tiles arrive in
// no fixed order, so dQ is not bit-reproducible from run to run) and a bandwidth-bound kernel converts
// the scratch to the output dtype afterwards. The delta kernel, which runs first anyway, zeroes the
// scratch.
//
// What bounds it. Counters, cycles of an SM per tile: at HD = 64 (causal 8 x 16 x 2048, 2,790 a tile) 1,273 wavefronts of the threads in shared
// memory and 1,408 of the products' operands, tensor pipe 1,280, exponentials 1,030, instruction issue 1,280 of each scheduler; at HD = 128
// (hierarchical 1 x 32 x 8192, 4,290) 1,491 and 2,304, 2,560, 1,030, 1,330. So shared memory is the most loaded, and what is taken off it
// comes out of the time in part: timing-only builds that read the A operands of S^T and dP^T from TMEM (256 wavefronts of a tile less, 512 at HD
// = 128) took 3.5 % off the backward of causal 8 x 16 x 2048 x 64 and 6.5 % x 128, with dK's (384, 768) 5.5 % and 7.5 %: four to six tenths of
// those cycles. The rest is latency of the chain from scores to dS and hand-overs. Without the additions of dQ a tile at HD = 128 took 3,300 cycles for 3,900.
//  * Shared memory is kept free by the layout of the compute warps' registers: they read S^T and dP^T from TMEM in the
//    16x256b shape, in which a thread owns four key rows and a quarter of the columns, as in an mma fragment, so that a
//    warp needs LSE and delta of a column once and not 32 times; P^T goes back in the 16x128b shape and dS^T leaves
//    through stmatrix without bank conflicts. Arithmetic on column pairs uses the packed f32x2 instructions.
//  * The instruction cache: sixteen warps in six roles run different loops at the same time. With the waits' time-out
//    code inlined and more unrolling this kernel was 120 KB and took 5,600 cycles a tile (a loop back-edge cost 580);
//    at 75 KB the same schedule took 3,600. Loops of the issuing and dQ warps are therefore rolled where they can be, and
//    the waits are as short as they can be (mbar_wait_short): a first test ahead of the loop, a look at the flag that
//    another role has given up, and the raising of that flag at each wait made 64 KB at HD = 64 where it is 52 now; without
//    them the backward of 16 x 16 x 4096 x 64 hierarchical takes 954 us where it took 1093, of 8 x 16 x 2048 x 64 causal 278
//    where it took 301, of 8 x 16 x 2048 x 128 causal 485 where it took 492. Suspending the waiting threads for longer (20 us)
//    gives 2 % of it back, the test ahead of the loop 4 %.
//  * The products are issued by whole warps with warp-uniform operands (mma_ss_uniform).
//
// Schedule at HD = 64. The compute warps form dS^T of tile t - 1 and P^T of tile t in one instruction stream (see there).
//   warp 1   dP^T(t) as soon as dP^T(t - 1) has been loaded, S^T(t + 1) as soon as S^T(t) has
//   warp 3   dV += P^T(t) dO, a half of 64 queries at a time
//   warp 2   dK += dS^T(t - 1) Q by halves, dQ(t - 1)
// TMEM: S^T 128, dP^T 128, dV 64, dK 64, dQ 64, P^T 64 columns.
// Schedule at HD = 128. S^T, dP^T, dV and dK fill TMEM, so P^T lies over the S^T it was made from and dQ takes the columns
// of dP^T; the compute warps form P^T(t) while dQ(t - 1) is read out and dP^T(t) formed, then dS^T(t).
//   warp 1   dV += P^T(t) dO, then S^T(t + 1) over P^T(t) (the tensor pipe executes in issue order)
//   warp 2   dQ(t), dK += dS^T(t) Q; when dQ(t) has been read out, dP^T(t + 1); also requests the next item's K and V
//
// Work items. An item is one (batch, head, key tile). The grid has a CTA per item, but a CTA that is running takes
// further items by cancelling CTAs that have not been launched yet (clusterlaunchcontrol) and works on them without
// draining its pipeline: the rings of Q and dO tiles run on into the next item, K and V have two buffers at HD = 64
// (shared memory holds one at HD = 128; at HD = 64 the second V buffer takes the place of half of the dQ staging, which costs
// nothing), and dK and dV of the finished item leave through the dQ warps while the
// next item's first products run. Starting a CTA costs some 12,000 cycles (launch, TMEM, first loads, pipeline fill,
// drain), and a (batch, head, key tile) has around ten tiles.
// Items are numbered in chunks of heads whose scratch and operands fit L2 together (ItemOrder), inside a
// chunk by decreasing list length, so that the CTAs on the machine at one time add to dQ lines that stay in L2 and
// the last items are short.
//
// 512 threads: warp 0 takes items and streams Q and dO (lane 0 issues the TMA loads; all lanes copy LSE, delta
// and a PARTIAL tile's visibility words to shared memory); warps 1-3 as above; warps 4-11 are two compute
// warpgroups (64 query columns each); warps 12-15 move finished dQ tiles from TMEM to the scratch (each warp stages and
// reduces its own 32 rows) and write dK and dV of finished items.
//
// Measured against the two forms before it (us, delta and conversion kernels included): a fused kernel with a row per
// thread, sixteen compute warps and heads per CTA (HD = 64) and the two-kernel form (HD = 128):
//   bf16 B16 H16 T4096 D64 hierarchical 1291 -> 1175-1230    bf16 B8 H16 T2048 D64 causal 338 -> 284
//   bf16 B8 H16 T2048 D128 causal 644 -> 415                 fp16 B4 H32 T8192 D128 hierarchical 3944 -> 2420
// The first is 890-950 now, the second 230-280 (boxes differ, and the power limit's state).
#include <algorithm>
#include <type_traits>

#include "attn_bwd.cuh"

namespace kd {

struct FusedArgs {
  BwdArgs b;
  ItemOrder order_of;
  int after_delta;   // the delta kernel of the same call is the kernel before this one on the stream
  int direct;        // without dQ: dK or dV has strides that no tensor map describes, and is written row by row
};

template <int HD_>
struct FusedCfg {
  static constexpr int HD = HD_;
  static constexpr int KBLK = HD / 64;               // 64-element blocks along D
  static constexpr int TILE_BYTES = KD_TILE * HD * 2;
  static constexpr int NK = (HD == 64) ? 2 : 1;      // K buffers (K of the CTA's item m in buffer m % NK)
  static constexpr int QS = (HD == 64) ? 4 : 2;      // ring stages of Q tiles: held from S^T of a tile to its dK
  static constexpr int OS = (HD == 64) ? 2 : 1;      // ring stages of dO tiles: held from dP^T to dV
  static constexpr int SMEM_K = 0;
  static constexpr int NV = NK;                      // V buffers, as K's
  static constexpr int SMEM_V = SMEM_K + NK * TILE_BYTES;
  static constexpr int SMEM_Q = SMEM_V + NV * TILE_BYTES;
  static constexpr int SMEM_DO = SMEM_Q + QS * TILE_BYTES;
  static constexpr int SMEM_DS = SMEM_DO + OS * TILE_BYTES;   // dS^T: two blocks [128 keys][64 queries]
  static constexpr int SMEM_STG = SMEM_DS + 2 * 16384;        // dQ staging: per dQ warp NSTG boxes [32 rows][32 floats]
  static constexpr int NSTG = (HD == 64) ? 1 : 2;
  // per Q stage: LSE and delta of the 128 queries; HD = 64: the visibility words of a PARTIAL tile, [32 keys][query] (HD = 128 has no room: its
  // compute warps fetch them); the tile's list entry (4 words with padding)
  static constexpr int SIDE_BITS = 2 * KD_TILE, SIDE_ENT = SIDE_BITS + (HD == 64 ? static_cast<int>(KD_WORDS) : 0), SIDE_WORDS = SIDE_ENT + 4;
  static constexpr int SMEM_ZERO = SMEM_STG + 4 * NSTG * 4096;   // HD = 64: a box of zeros, what items without entries are written from
  static constexpr int ZERO_BYTES = (HD == 64) ? 4096 : 0;
  static constexpr int SMEM_SIDE = SMEM_ZERO + ZERO_BYTES;
  static constexpr int NITEM = 4;                    // ring of item headers
  static constexpr int SMEM_ITEM = SMEM_SIDE + QS * SIDE_WORDS * 4;   // NITEM x {batch, head, key tile | first entry << 16, entries}
  static constexpr int SMEM_CLC = SMEM_ITEM + NITEM * 16;             // response of a cancellation
  static constexpr int SMEM_BAR = SMEM_CLC + 16;
  // barriers (8 bytes each)
  static constexpr int NH = (HD == 64) ? 2 : 1;      // halves of 64 queries with barriers of their own
  static constexpr int B_KFULL = 0, B_KEMPTY = B_KFULL + NK, B_VFULL = B_KEMPTY + NK, B_VEMPTY = B_VFULL + NV, B_QFULL = B_VEMPTY + NV,
                       B_QEMPTY = B_QFULL + QS, B_DOFULL = B_QEMPTY + QS, B_DOEMPTY = B_DOFULL + OS, B_SFULL = B_DOEMPTY + OS,
                       B_SFREE = B_SFULL + NH, B_PFULL = B_SFREE + NH, B_PFREE = B_PFULL + NH, B_DPFULL = B_PFREE + NH, B_DPFREE = B_DPFULL + NH,
                       B_DSFULL = B_DPFREE + NH, B_DSFREE = B_DSFULL + NH, B_DQFULL = B_DSFREE + 1, B_DQEMPTY = B_DQFULL + 1,
                       B_ACCFULL = B_DQEMPTY + 1, B_ACCFREE = B_ACCFULL + 2, B_ITEMFULL = B_ACCFREE + 2, B_ITEMEMPTY = B_ITEMFULL + NITEM,
                       B_CLC = B_ITEMEMPTY + NITEM, NBAR = B_CLC + 1;
  static constexpr int ITEM_READERS = (HD == 64) ? 7 : 14;    // warps that read item headers
  static constexpr uint32_t ENT_END = 0xFFFFFFFFu;            // HD = 64: in place of a list entry, behind the last tile
  static constexpr int SMEM_ALLOC = SMEM_BAR + NBAR * 8 + 16;   // + TMEM base, abort flag
  static constexpr int THREADS = 512;
  // TMEM columns
  static constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = TM_DV + HD, TM_DQ = (HD == 64) ? TM_DK + HD : TM_DP,
                            TM_P = (HD == 64) ? TM_DQ + HD : TM_S;
  static constexpr uint32_t P_STRIDE = (HD == 64) ? 32 : 64;   // packed columns between the two warpgroups' P^T
  static_assert(TM_DK + HD <= 512 && TM_DQ + HD <= 512 && TM_P + P_STRIDE + 32 <= 512, "TMEM budget");
  static_assert(SMEM_ALLOC <= 232448, "shared memory budget");
  // registers: 128 per thread at launch; the light warps and the dQ warps release theirs down to REGS_LIGHT and REGS_DQ, the compute
  // warps take REGS_COMPUTE
  static constexpr int REGS_LAUNCH = 128, REGS_LIGHT = (HD == 64) ? 88 : 72, REGS_DQ = (HD == 64) ? 56 : 120, REGS_COMPUTE = (HD == 64) ? 184 : 160;
  static_assert(4 * 32 * REGS_LIGHT + 4 * 32 * REGS_DQ + 8 * 32 * REGS_COMPUTE <= THREADS * REGS_LAUNCH, "register pool");
};

enum : uint32_t {
  W_U_KFULL = 0x401, W_U_VFULL = 0x402, W_U_QFULL = 0x403, W_U_DOFULL = 0x404, W_U_QEMPTY = 0x405, W_U_DOEMPTY = 0x406, W_U_ITEMEMPTY = 0x407,
  W_U_SFULL = 0x408, W_U_SFREE = 0x409, W_U_PFULL = 0x40A, W_U_PFREE = 0x40B, W_U_DPFULL = 0x40C, W_U_DSFULL = 0x40D,
  W_U_DSFREE = 0x40E, W_U_DQFULL = 0x40F, W_U_DQEMPTY = 0x410, W_U_ACCFULL = 0x411, W_U_ACCFREE = 0x412, W_U_ALIGN = 0x413,
  W_U_ITEMFULL = 0x414, W_U_CLC = 0x415, W_U_KEMPTY = 0x416, W_U_VEMPTY = 0x417, W_U_DPFREE = 0x418,
};

__device__ __forceinline__ void st_shared_v4(uint32_t saddr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Two consecutive floats as two 4-byte loads. The lanes of a warp read four such pairs, eight lanes each: as 8-byte loads that
// took more than five shared-memory wavefronts, 690 of the 1,480 of a tile; a 4-byte load takes one.
__device__ __forceinline__ uint64_t ld_shared_pair(const float* p) {
  uint32_t lo, hi;
  const uint32_t a = smem_u32(p);
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(lo) : "r"(a));
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(hi) : "r"(a + 4u));
  return pack_u32x2(lo, hi);
}

// kF32: dQ, dK and dV are float32 tensors (of a float32 call). The dQ tiles are then scaled and added into dQ itself, which the delta kernel
// has zeroed: no scratch and no conversion (2 x 4 x 256 x 64: forward and backward 8 launches -> 4, 105 -> 86 us).
// kDq: false in the deterministic backward, which forms dQ in a kernel of its own (attn_bwd.cu). What is left here adds in a fixed order: the
// products of a key tile follow one another in the order of its list.
// kWords: the plan has the PARTIAL tiles' bits (see KD_WORDS_LIMIT); without them they are formed where they would be read.
template <int HD_, bool kBf16, bool kF32, bool kDq, bool kWords>
__global__ void __launch_bounds__(FusedCfg<HD_>::THREADS, 1)
attn_bwd_fused_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                      const __grid_constant__ CUtensorMap tmAcc, const __grid_constant__ CUtensorMap tmDK,
                      const __grid_constant__ CUtensorMap tmDV, const FusedArgs fa) {
  using C = FusedCfg<HD_>;
  const BwdArgs& a = fa.b;
  constexpr int HD = C::HD, TILE = C::TILE_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t s0 = smem_u32(smem);
  const uint32_t sK = s0 + C::SMEM_K, sV = s0 + C::SMEM_V, sQ = s0 + C::SMEM_Q, sDO = s0 + C::SMEM_DO, sDS = s0 + C::SMEM_DS;
  int4* items = reinterpret_cast<int4*>(smem + C::SMEM_ITEM);
  float* sSide = reinterpret_cast<float*>(smem + C::SMEM_SIDE);
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + C::SMEM_BAR + C::NBAR * 8);
  AbortFlag* abortf = reinterpret_cast<AbortFlag*>(tmem_base_s + 1);
  auto bar = [&](int i) -> uint32_t { return s0 + C::SMEM_BAR + i * 8; };

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if ((s0 & 1023u) != 0u) {   // the swizzled tiles need it; the launch asks for it, so this never happens
    if (tid == 0) report_status(a.status, KD_DEV_TIMEOUT | W_U_ALIGN);
    return;
  }
  if (tid == 0) abortf->v = 0;
  if (tid < C::NBAR) {   // a thread each: one after the other they took 900 cycles of a CTA's start
    const int i = tid;
    uint32_t count = 1;
    if (i >= C::B_QFULL && i < C::B_QEMPTY) count = 33;        // the TMA load and the producer lanes' own copies
    if (i >= C::B_DOEMPTY && i < C::B_SFULL) count = 2;        // dP^T and dV have read the tile
    if ((i >= C::B_DPFREE && i < C::B_DSFREE) || (i >= C::B_SFREE && i < C::B_PFREE)) count = 8 / C::NH;   // one arrival per compute warp
    if (i == C::B_DQEMPTY) count = 4;                          // one per dQ warp
    if (i == C::B_ACCFREE || i == C::B_ACCFREE + 1) count = 4; // dV, dK have been read out of TMEM
    if (i >= C::B_ITEMEMPTY && i < C::B_CLC) count = C::ITEM_READERS;
    mbar_init(bar(i), count);
    fence_barrier_init();
  }
  if (!kDq && tid == 0 && a.after_dq != 0) {   // see below
    __threadfence();
    fence_proxy_async_global();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // With the delta kernel directly before this one, everything that it does not write itself was complete before it let this one start:
  // the plan, Q, K, V and LSE may be read, and dK and dV written, before the wait (plain reads past L1, which the start of a kernel that
  // overlaps another need not have cleaned). Not so delta, the zeros of the dQ scratch or of a float32 dQ, and dO, which in a float32 call
  // the delta kernel rounds to 16 bits.
  // Without dQ, directly behind the dQ kernel of the same call, there is nothing to wait for at all: that kernel writes nothing that this one
  // reads, and lets it start when it has itself waited for the delta kernel. So the last CTAs of the one overlap the first of the other (both
  // together, with the wait here instead: 1 x 16 x 500 x 128 31.5 us, 23 so; 4 x 16 x 2048 x 64 110.2, 108.2; unmasked 1 x 4 x 2048 x 64 51.5, 34).
  // What orders delta, and the dO of a float32 call, before the reads here: CUDA promises visibility to the kernel that executes
  // griddepcontrol.wait behind the writer, which is the dQ kernel, and none through launch_dependents alone. Hence a device-wide
  // fence on both sides of that hand-over (there behind the wait, here ahead of the block's barrier, with one for the TMA loads); all reads
  // go past L1. That a dependent kernel starts after launch_dependents has been executed is what remains to be relied on.
  // The dQ kernel's end is awaited at this one's end, so that whatever comes next finds both complete (what a successor reads ahead of its
  // own wait is a plan, which no backward writes).
  if (kDq ? fa.after_delta == 0 : a.after_dq == 0) pdl_wait();
  // The site of this warp's wait that ran out, 0 while none has. There is no wait or product after it: every role ends at its first, with
  // its copies drained, and raises the flag where all roles meet. One exception: at HD = 64 the warp that issues S^T takes a header that stays out
  // for the end of the items and gives the signal that goes behind the last tile (another look at gave_up in its loop costs
  // the backward 3 %). The compute warps may then form a P^T that is no tile's; nobody reads it, for the other issuers wait for the same header. All waits of this kernel are such waits (there is no named
  // barrier), so a role whose partner has ended waits for its own limit and ends too.
  uint32_t gave_up = 0u;
  // the whole of TMEM is allocated, so the allocation starts at column 0 and the addresses below are constants
  auto wait = [&](int i, uint32_t parity, uint32_t site) -> bool {
    const bool there = __all_sync(0xffffffffu, mbar_wait_short(bar(i), parity));
    if (!there) gave_up = site;
    return there;
  };
  // two barriers of which both are complete as a rule: their tests overlap
  auto wait2 = [&](int i, uint32_t pi, uint32_t site_i, int j, uint32_t pj, uint32_t site_j) -> bool {
    const bool ri = mbar_try_wait(bar(i), pi), rj = mbar_try_wait(bar(j), pj);
    if (__all_sync(0xffffffffu, ri && rj)) return true;
    return wait(i, pi, site_i) && wait(j, pj, site_j);
  };

  // header of this CTA's k-th item with entries; entries < 0: there is none. The redux makes the fields warp-uniform for the compiler.
  auto next_item = [&](int k, int4& it) -> bool {
    const int slot = k % C::NITEM;
    if (!wait(C::B_ITEMFULL + slot, (k / C::NITEM) & 1, W_U_ITEMFULL)) return false;
    const int4 v = items[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::B_ITEMEMPTY + slot));
    it.x = __reduce_max_sync(0xffffffffu, v.x);
    it.y = __reduce_max_sync(0xffffffffu, v.y);
    it.z = __reduce_max_sync(0xffffffffu, v.z);
    it.w = __reduce_max_sync(0xffffffffu, v.w);
    return it.w >= 0;
  };

  // one thread: requests tile `tile` of (b, h); the barrier expects its bytes
  auto load_tile = [&](const CUtensorMap* tm, uint32_t dst, int full, int tile, int h, int b) {
    mbar_arrive_expect_tx(bar(full), TILE);
    for (int kb = 0; kb < C::KBLK; ++kb) tma_load_4d(dst + kb * 16384, tm, bar(full), kb * 64, tile * KD_TILE, h, b);
  };

  if (warp < 4) {
    reg_dealloc<C::REGS_LIGHT>();
    if (warp == 0) {
      // ------------------------------ producer warp ------------------------------
      if (lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmDO);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
      }
      for (int i = lane; i < C::ZERO_BYTES / 16; i += 32) st_shared_v4(s0 + C::SMEM_ZERO + 16 * i, 0u, 0u, 0u, 0u);
      if (C::ZERO_BYTES > 0) fence_proxy_async_smem();
      __syncwarp();
      int q_tiles = 0, do_tiles = 0, k_loads = 0, v_loads = 0, k = 0;   // Q / dO / K tiles requested and items published so far
      bool ok = true, pending = false;
      auto drops = [&](int what, bool here) -> bool { return test_drops(a, what) && here; };
      // decodes item number `idx` of the launch
      auto find_tile = [&](int idx, int4& it) {
        int bh, rank;
        fa.order_of.decode(idx, a.NT, bh, rank);
        it.x = bh / a.H;
        it.y = bh - it.x * a.H;
        it.z = __ldcg(a.order + ((size_t)it.x * 3 + 2) * a.NT + rank);   // longest lists first
        it.w = 0;
      };
      auto find_list = [&](int4& it, int& first) {
        first = __ldcg(a.bwd_list + ((size_t)it.x * a.NT + it.z) * a.NT);
        it.w = __ldcg(a.bwd_cnt + it.x * a.NT + it.z);
      };
      int asked = 0;   // cancellations asked for
      // The next item is asked for three tiles before the end of this one (for a shorter one: when it is taken), which hides the
      // answer and the look-up of its list, and no earlier: an item held in reserve by a CTA with a long list is one that an idle CTA cannot take.
      auto ask = [&]() {
        if (lane == 0) {
          fence_proxy_async_smem();   // the previous response has been read
          mbar_arrive_expect_tx(bar(C::B_CLC), 16);
          clc_try_cancel(s0 + C::SMEM_CLC, bar(C::B_CLC));
        }
        ++asked;
        pending = true;
      };
      // dK = dV = 0 for an item without entries
      auto write_zeros = [&](const int4& z) {
        using Out = std::conditional_t<kF32, float, uint16_t>;
        if (HD == 64 && (kDq || fa.direct == 0)) {
          // Items without entries come last and nothing hides them there: 14,500 of the 87,000 cycles of a CTA of hierarchical 4 x 16 x 2048
          // x 64 lie behind its last tile. So they leave through the copy engine, a lane per 32 rows, and cost this warp no more than
          // the look-up (stores by the lanes before: that backward 71.1 -> 67.8 us, 8 x 16 x 2048 x 64 141.7 -> 132.5, 16 x 16 x 4096 x 64
          // 978 -> 947, 8 x 8 x 1000 x 64 29.4 -> 28.5). At HD = 128 there is no room for the box; made in a Q stage that
          // is empty, it gives 1 to 4 % of longer hierarchical calls, and 3 x 6 x 1357 x 80 is 3.5 % slower for the longer code.
          if (lane < 4 && (z.z & 0xFFFF) * KD_TILE + lane * 32 < a.T) {   // rows at or beyond T and columns at or beyond d_real are not written
            for (int col = 0; col < a.d_real; col += 128 / static_cast<int>(sizeof(Out))) {
              tma_store_4d(&tmDK, s0 + C::SMEM_ZERO, col, (z.z & 0xFFFF) * KD_TILE + lane * 32, z.y, z.x);
              tma_store_4d(&tmDV, s0 + C::SMEM_ZERO, col, (z.z & 0xFFFF) * KD_TILE + lane * 32, z.y, z.x);
            }
            bulk_commit_group();
          }
          return;
        }
        constexpr int per = 16 / sizeof(Out);   // elements of a 16-byte chunk
        constexpr int CPR = HD / per;           // chunks of a tile's row
        const int row0 = (z.z & 0xFFFF) * KD_TILE, rows = min(KD_TILE, a.T - row0);
        Out* dk = reinterpret_cast<Out*>(a.dk) + (size_t)z.x * a.dk_sb + (size_t)z.y * a.dk_sh;
        Out* dv = reinterpret_cast<Out*>(a.dv) + (size_t)z.x * a.dv_sb + (size_t)z.y * a.dv_sh;
        for (int i = lane; i < rows * CPR; i += 32) {
          const int r = i / CPR, c = i % CPR * per;
          if (c >= a.d_real) continue;
          *reinterpret_cast<uint4*>(dk + (size_t)(row0 + r) * a.dk_st + c) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(dv + (size_t)(row0 + r) * a.dv_st + c) = make_uint4(0u, 0u, 0u, 0u);
        }
      };
      // the answer (nx.w < 0: there is no further item)
      // Takes the next item in three steps between the loads of this one's last tiles, which hide the look-ups (a round trip to L2 each):
      // the answer and the key tile (nx.w < 0: there is no further item), its list's length and first entry, and the header. At HD = 64
      // a tile lasts no longer than these: taken in one step ahead of the last tile's Q, that tile's S^T came 1,100 cycles late and the
      // next item's first, whose K was requested behind it, 600. With the steps, the next item's header, K and V ahead of the last
      // dO, and a second V buffer (one: the next item's second S^T waits for V, 600 cycles) backward us: causal 8 x 16 x 2048 x 64 280 -> 274,
      // 8 x 16 x 1000 x 64 90.2 -> 88.8, hierarchical 8 x 16 x 2048 x 64 132.2 -> 131.5, 16 x 16 x 4096 x 64 940 -> 937. Level at HD = 128.
      int first_entry = 0;
      auto next_tile = [&](int4& nx) -> bool {
        if (!wait(C::B_CLC, (asked - 1) & 1, W_U_CLC)) return false;
        pending = false;
        const int idx = clc_first_ctaid_x(s0 + C::SMEM_CLC);
        __syncwarp();   // every lane has read the response that the next request overwrites
        nx.w = -1;
        if (idx >= 0) find_tile(idx, nx);
        return true;
      };
      auto next_list = [&](int4& nx) {
        if (nx.w >= 0) find_list(nx, first_entry);
      };
      auto next_header = [&](int4& nx) {
        nx.z |= first_entry << 16;
        if (nx.w >= 0 && nx.w <= 2) ask();
      };
      int4 it;
      find_tile(blockIdx.x, it);
      next_list(it);
      next_header(it);
      int qs = 0, os = 0;
      uint32_t q_parity = 1u, do_parity = 1u;   // of the stages' "empty" phases
      // dO of a tile is requested after its Q; at HD = 64 that of an item's last tile behind the next item's header, K and V, none of which waits for it
      int do_tile = -1, do_h = 0, do_b = 0;
      auto load_do = [&]() -> bool {
        if (do_tile < 0) return true;
        if (!wait(C::B_DOEMPTY + os, do_parity, W_U_DOEMPTY)) return false;
        if (lane == 0) load_tile(&tmDO, sDO + os * TILE, C::B_DOFULL + os, do_tile, do_h, do_b);   // (behind pdl_wait())
        ++do_tiles;
        if (++os == C::OS) { os = 0; do_parity ^= 1u; }
        do_tile = -1;
        return true;
      };
      while (ok) {
        const int b = it.x, h = it.y, kt = it.z & 0xFFFF, n = it.w;
        if (HD == 64 && n <= 0 && !(ok = load_do())) break;
        if (n != 0) {   // (no other warp hears of an item without entries)
        const int slot = k % C::NITEM;
        if (!(ok = wait(C::B_ITEMEMPTY + slot, ((k / C::NITEM) & 1) ^ 1, W_U_ITEMEMPTY))) break;
        if (HD == 64 && n < 0) {   // the compute warps read no headers: the stage behind the last tile tells them
          if (!(ok = wait(C::B_QEMPTY + qs, q_parity, W_U_QEMPTY))) break;
          if (lane == 0) {
            st_shared_u32(s0 + C::SMEM_SIDE + qs * (C::SIDE_WORDS * 4) + C::SIDE_ENT * 4, C::ENT_END);
            if (k == 0) {   // no tile at all, and so no product that would wake them
              mbar_arrive(bar(C::B_SFULL));
              mbar_arrive(bar(C::B_SFULL + 1));
            }
          }
          __syncwarp();
        }
        if (lane == 0 && !drops(4, k == 1)) {
          items[slot] = it;
          mbar_arrive(bar(C::B_ITEMFULL + slot));
        }
        __syncwarp();
        if (n < 0) break;
        // K into the buffer of the item before the last (HD = 64; at HD = 128 the issuing warps request K as well as V)
        if (HD == 64 || k == 0) {
          if (!(ok = wait(C::B_KEMPTY + k % C::NK, ((k / C::NK) & 1) ^ 1, W_U_KEMPTY))) break;
          if (lane == 0) load_tile(&tmK, sK + (k % C::NK) * TILE, C::B_KFULL + k % C::NK, kt, h, b);
          ++k_loads;
        }
        if (HD == 64 || k == 0) {
          if (!(ok = wait(C::B_VEMPTY + k % C::NV, ((k / C::NV) & 1) ^ 1, W_U_VEMPTY))) break;
          if (lane == 0) load_tile(&tmV, sV + (k % C::NV) * TILE, C::B_VFULL + k % C::NV, kt, h, b);
          ++v_loads;
        }
        if (k == 0) {
          if (kDq) pdl_wait();   // delta and dO are read from here on
          pdl_launch_dependents();
        }
        ++k;
        if (HD == 64 && !(ok = load_do())) break;
        }
        const uint16_t* list = a.bwd_list + ((size_t)b * a.NT + kt) * a.NT;
        const size_t row = ((size_t)b * a.H + h) * a.T;
        // the rows of four scalars that the lanes copy begin on 16 bytes (the arrays need no alignment beyond a float's)
        const bool aligned = ((reinterpret_cast<uintptr_t>(a.lse + row) | reinterpret_cast<uintptr_t>(a.delta + row)) & 15u) == 0;
        uint32_t ent = static_cast<uint32_t>(it.z) >> 16;
        int4 nx = it;
#pragma unroll 1
        for (int e = 0; e < max(n, 1); ++e) {
          if (n > 2 && e == n - 3) ask();
          const bool last = e >= n - 1;
          if ((HD == 64 && n > 2 ? e == n - 2 : last) && !(ok = next_tile(nx))) break;
          if (last) next_list(nx);
          if (HD == 128 ? last : n == 0) next_header(nx);
          if (n == 0) {
            write_zeros(it);
            break;
          }
          const uint32_t this_ent = ent;
          if (e + 1 < n) ent = __ldcg(list + e + 1);
          const int qt = this_ent & 0xFF;
          if (!(ok = wait(C::B_QEMPTY + qs, q_parity, W_U_QEMPTY))) break;
          const uint32_t side = s0 + C::SMEM_SIDE + qs * (C::SIDE_WORDS * 4);
          if (lane == 0) {
            st_shared_u32(side + C::SIDE_ENT * 4, this_ent);   // published by the arrival that goes with the load
            if (!drops(3, q_tiles == 0)) load_tile(&tmQ, sQ + qs * TILE, C::B_QFULL + qs, qt, h, b);
          }
          // the scalars of four queries per lane, and a PARTIAL tile's words, copied asynchronously: the barrier counts the lanes' copies
          // (a query at or beyond the sequence length takes the last row's scalars: it sees nothing, so the tile is PARTIAL and the
          // mask removes it)
          const int q = qt * KD_TILE + 4 * lane;
          if (aligned && q + 3 < a.T) {
            cp_async16(side + 16 * lane, a.lse + row + q);
            cp_async16(side + KD_TILE * 4 + 16 * lane, a.delta + row + q);
          } else {
            if (kDq) {
#pragma unroll 1
              for (int j = 0; j < 4; ++j) {
                const size_t r = row + min(q + j, a.T - 1);
                cp_async4(side + 16 * lane + 4 * j, a.lse + r);
                cp_async4(side + KD_TILE * 4 + 16 * lane + 4 * j, a.delta + r);
              }
            } else {   // (copies of 4 bytes go through L1, which may hold delta of before the kernel ahead: see above)
              float l[4], d[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const size_t r = row + min(q + j, a.T - 1);
                l[j] = __ldcg(a.lse + r);
                d[j] = __ldcg(a.delta + r);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                st_shared_u32(side + 16 * lane + 4 * j, __float_as_uint(l[j]));
                st_shared_u32(side + KD_TILE * 4 + 16 * lane + 4 * j, __float_as_uint(d[j]));
              }
              __threadfence_block();   // the arrival below is ordered behind the asynchronous copies alone
            }
          }
          if (HD == 64 && (this_ent >> 8) == KD_TILE_PARTIAL) {
            if constexpr (kWords) {
              const uint32_t* src = a.words + (((size_t)b * a.NT + qt) * a.NT + kt) * KD_WORDS + 4 * lane;
#pragma unroll
              for (int w = 0; w < 4; ++w) cp_async16(side + (C::SIDE_BITS + w * KD_TILE) * 4 + 16 * lane, src + w * KD_TILE);
            } else {
              const uint32_t* desc = a.desc + (size_t)b * a.Tpad;
              const KeyRun<4> keys(desc, a.tilebits + (size_t)b * a.NT * 32, kt, 0, lane);
              uint32_t qd[4];
#pragma unroll
              for (int r = 0; r < 4; ++r) qd[r] = __ldcg(desc + qt * KD_TILE + r * 32 + lane);
#pragma unroll 1
              for (int r = 0; r < 4; ++r) {   // 32 queries at a time
                uint32_t mk[4];
                keys.words(r < 2 ? (r == 0 ? qd[0] : qd[1]) : (r == 2 ? qd[2] : qd[3]), qt * KD_TILE + r * 32 + lane, mk);
#pragma unroll
                for (int w = 0; w < 4; ++w) st_shared_u32(side + (C::SIDE_BITS + w * KD_TILE + r * 32 + lane) * 4, mk[w]);
              }
              __threadfence_block();   // (as above)
            }
          }
          cp_async_mbar_arrive(bar(C::B_QFULL + qs));
          ++q_tiles;
          if (++qs == C::QS) { qs = 0; q_parity ^= 1u; }
          do_tile = qt;
          do_h = h;
          do_b = b;
          if (HD == 64 && last) next_header(nx);
          if ((HD == 128 || !last) && !(ok = load_do())) break;
        }
        it = nx;
      }
      if (C::ZERO_BYTES > 0) bulk_wait_group_read0();   // the box of zeros has been read
      if (lane == 0 && (gave_up != 0u || abortf->v != 0u)) {   // let the copies in flight land before the CTA exits
        for (int f = max(0, k_loads - C::NK); f < k_loads; ++f) drain_wait(bar(C::B_KFULL + f % C::NK), (f / C::NK) & 1);
        for (int f = max(0, v_loads - C::NV); f < v_loads; ++f) drain_wait(bar(C::B_VFULL + f % C::NV), (f / C::NV) & 1);
        for (int f = max(0, q_tiles - C::QS); f < q_tiles; ++f) drain_wait(bar(C::B_QFULL + f % C::QS), (f / C::QS) & 1);
        for (int f = max(0, do_tiles - C::OS); f < do_tiles; ++f) drain_wait(bar(C::B_DOFULL + f % C::OS), (f / C::OS) & 1);
        if (pending) drain_wait(bar(C::B_CLC), (asked - 1) & 1);
      }
    } else {
      // ------------------------------ issuing warps ------------------------------
      // All lanes follow the control flow and one elected lane issues (mma_ss_uniform).
      const uint32_t hi = desc_hi_sw128();
      const uint32_t idesc_s = make_idesc_f16(kBf16, 0, 0, KD_TILE, KD_TILE);   // S^T, dP^T (of a half)
      const uint32_t idesc_dv = make_idesc_f16(kBf16, 0, 1, KD_TILE, a.d_real);      // dV, dK: B = dO / Q rows, MN-major
      const uint32_t idesc_dq = make_idesc_f16(kBf16, 1, 1, KD_TILE, a.d_real);      // A = dS^T read MN-major (M = queries)
      const uint32_t lo_k0 = desc_lo_kmajor(sK), lo_v = desc_lo_kmajor(sV), lo_q0 = desc_lo_kmajor(sQ), lo_do0 = desc_lo_kmajor(sDO);
      const uint32_t k_mn0 = desc_lo_mnmajor(sK), q_mn0 = desc_lo_mnmajor(sQ), do_mn0 = desc_lo_mnmajor(sDO);
      const uint32_t ds_k = desc_lo_kmajor(sDS), ds_mn = desc_lo_mnmajor(sDS);
      constexpr uint32_t T16 = TILE >> 4;
      bool ok = true;
      int4 it;
      int k = 0, m = 0, t = 0;   // headers read; current item; tiles so far
      bool have = false;
      auto advance = [&]() { have = next_item(k++, it); };
      auto product_kmajor = [&](uint32_t d, uint32_t a_lo, uint32_t b_lo) {   // d = A B^T over the head dim
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          mma_ss_uniform(d, a_lo + koff_kmajor(kk), b_lo + koff_kmajor(kk), hi, idesc_s, kk > 0 ? 1u : 0u);
      };
      auto product_dv = [&](int w, uint32_t do_mn, bool first) {   // dV += P^T dO over queries 64 w .. 64 w + 63
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          mma_ts_uniform(C::TM_DV, C::TM_P + w * C::P_STRIDE + kk * 8, do_mn + w * koff_mnmajor(4) + koff_mnmajor(kk), hi, idesc_dv, (kk > 0 || !first) ? 1u : 0u);
      };
      auto product_dk = [&](int w, uint32_t q_mn, bool first) {    // dK += dS^T Q over the same
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          mma_ss_uniform(C::TM_DK, ds_k + w * koff_kmajor(4) + koff_kmajor(kk), q_mn + w * koff_mnmajor(4) + koff_mnmajor(kk), hi, idesc_dv, (kk > 0 || !first) ? 1u : 0u);
      };
      auto product_dq = [&](uint32_t k_mn) {                                  // dQ = dS K
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) mma_ss_uniform(C::TM_DQ, ds_mn + koff_mnmajor(kk), k_mn + koff_mnmajor(kk), hi, idesc_dq, kk > 0 ? 1u : 0u);
      };
      if constexpr (HD == 64) {
        if (warp == 1) {
          // ---- dP^T(t) when dP^T(t - 1) has been loaded, S^T(t + 1) when S^T(t) has ----
          int q_stage = 0, do_stage = 0, e = 0;
          uint32_t q_parity = 0, do_parity = 0;
          auto issue_s = [&]() -> bool {   // of tile t + 1, the item's e-th; behind the last tile only the signal
            if (have) {
              if (e == 0 && !wait(C::B_KFULL + (m & 1), (m >> 1) & 1, W_U_KFULL)) return false;
              if (!wait(C::B_QFULL + q_stage, q_parity, W_U_QFULL)) return false;
            }
            if (t >= 0 && !wait2(C::B_SFREE, t & 1, W_U_SFREE, C::B_SFREE + 1, t & 1, W_U_SFREE)) return false;
            tc_fence_after_sync();
            if (have) product_kmajor(C::TM_S, lo_k0 + (m & 1) * T16, lo_q0 + q_stage * T16);
            commit_uniform(bar(C::B_SFULL));
            commit_uniform(bar(C::B_SFULL + 1));
            if (++q_stage == C::QS) { q_stage = 0; q_parity ^= 1u; }
            ++t;
            return true;
          };
          advance();
          t = -1;
          if (have) ok = issue_s();
          while (have && ok) {
            if (e == 0 && !(ok = wait(C::B_VFULL + (m & 1), (m >> 1) & 1, W_U_VFULL))) break;
            if (!(ok = wait(C::B_DOFULL + do_stage, do_parity, W_U_DOFULL))) break;
            if (t > 0 && !(ok = wait2(C::B_DPFREE, (t - 1) & 1, W_U_DPFREE, C::B_DPFREE + 1, (t - 1) & 1, W_U_DPFREE))) break;
            tc_fence_after_sync();
            product_kmajor(C::TM_DP, lo_v + (m & 1) * T16, lo_do0 + do_stage * T16);
            commit_uniform(bar(C::B_DPFULL));
            commit_uniform(bar(C::B_DPFULL + 1));
            commit_uniform(bar(C::B_DOEMPTY + do_stage));
            if (++do_stage == C::OS) { do_stage = 0; do_parity ^= 1u; }
            if (++e == it.w) {
              commit_uniform(bar(C::B_VEMPTY + (m & 1)));   // that was V's last reader in its item
              advance();
              ++m;
              e = 0;
            }
            ok = issue_s();
          }
        } else if (warp == 3) {
          // ---- dV, a half at a time ----
          int do_stage = 0;
          uint32_t do_parity = 0;
          advance();
          while (have && ok) {
            const int n = it.w;
            for (int e = 0; e < n && ok; ++e, ++t) {
              if (e == 0 && m > 0 && !(ok = wait(C::B_ACCFREE, (m - 1) & 1, W_U_ACCFREE))) break;
              if (!(ok = wait(C::B_DOFULL + do_stage, do_parity, W_U_DOFULL))) break;   // P^T does not imply it
#pragma unroll 1
              for (int w = 0; w < 2; ++w) {
                if (!(ok = wait(C::B_PFULL + w, t & 1, W_U_PFULL))) break;
                tc_fence_after_sync();
                product_dv(w, do_mn0 + do_stage * T16, e == 0 && w == 0);
                commit_uniform(bar(C::B_PFREE + w));
              }
              if (!ok) break;
              commit_uniform(bar(C::B_DOEMPTY + do_stage));
              if (e == n - 1) commit_uniform(bar(C::B_ACCFULL));
              if (++do_stage == C::OS) { do_stage = 0; do_parity ^= 1u; }
            }
            ++m;
            if (ok) advance();
          }
        } else {
          // ---- dK(t - 1), a half at a time, and dQ(t - 1) ----
          int q_stage = 0;
          bool first = false, last = false;   // of tile t - 1
          auto accumulate = [&](int item) -> bool {
            if (gave_up != 0u) return false;   // (a header stays out)
            if (first && item > 0 && !wait(C::B_ACCFREE + 1, (item - 1) & 1, W_U_ACCFREE)) return false;
#pragma unroll 1
            for (int w = 0; w < 2; ++w) {
              if (!wait(C::B_DSFULL + w, (t - 1) & 1, W_U_DSFULL)) return false;
              tc_fence_after_sync();
              product_dk(w, q_mn0 + q_stage * T16, first && w == 0);
            }
            if constexpr (kDq) {
              if (t > 1 && !wait(C::B_DQEMPTY, t & 1, W_U_DQEMPTY)) return false;
              tc_fence_after_sync();
              product_dq(k_mn0 + (item & 1) * T16);
              commit_uniform(bar(C::B_DQFULL));
            }
            commit_uniform(bar(C::B_DSFREE));
            commit_uniform(bar(C::B_QEMPTY + q_stage));
            if (last) {
              commit_uniform(bar(C::B_ACCFULL + 1));
              commit_uniform(bar(C::B_KEMPTY + (item & 1)));
            }
            if (++q_stage == C::QS) q_stage = 0;
            return true;
          };
          int e = 0;
          advance();
          while (have || t > 0) {
            if (t > 0 && !(ok = accumulate((have && e > 0) ? m : m - 1))) break;
            if (!have) break;   // that was the last tile
            first = e == 0;
            last = e == it.w - 1;
            ++t;
            ++e;
            if (last) {
              advance();
              ++m;
              e = 0;
            }
          }
        }
      } else if (warp == 1) {
        // ---- issuing warp A: S^T and dV ----
        int q_stage = 0, do_stage = 0;
        uint32_t q_parity = 0, do_parity = 0;
        auto issue_s = [&]() {
          tc_fence_after_sync();
          product_kmajor(C::TM_S, lo_k0, lo_q0 + q_stage * T16);
          commit_uniform(bar(C::B_SFULL));
          if (++q_stage == C::QS) { q_stage = 0; q_parity ^= 1u; }
        };
        advance();
        if (have && (ok = wait(C::B_KFULL, 0, W_U_KFULL) && wait(C::B_QFULL, 0, W_U_QFULL))) issue_s();
        while (have && ok) {
          const int n = it.w;
          for (int e = 0; e < n; ++e, ++t) {
            const bool last = (e == n - 1);
            if (e == 0 && m > 0 && !(ok = wait(C::B_ACCFREE, (m - 1) & 1, W_U_ACCFREE))) break;
            // (P^T does not imply that dO has landed)
            if (!(ok = wait2(C::B_PFULL, t & 1, W_U_PFULL, C::B_DOFULL + do_stage, do_parity, W_U_DOFULL))) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int w = 0; w < 2; ++w) product_dv(w, do_mn0 + do_stage * T16, e == 0 && w == 0);
            commit_uniform(bar(C::B_DOEMPTY + do_stage));
            if (last) commit_uniform(bar(C::B_ACCFULL));
            if (++do_stage == C::OS) { do_stage = 0; do_parity ^= 1u; }
            if (last) advance();
            if (have) {   // S^T of the next tile over P^T, whose reader precedes it in the pipe
              if (last && !(ok = wait(C::B_KFULL, (m + 1) & 1, W_U_KFULL))) break;
              if (!(ok = wait(C::B_QFULL + q_stage, q_parity, W_U_QFULL))) break;
              issue_s();
            }
          }
          ++m;
        }
      } else if (warp == 2) {
        // ---- issuing warp B: dP^T, dK and dQ ----
        int q_stage = 0, do_stage = 0, k_loads = 1, v_loads = 1;
        uint32_t do_parity = 0;
        auto issue_dp = [&]() {
          tc_fence_after_sync();
          product_kmajor(C::TM_DP, lo_v, lo_do0 + do_stage * T16);
          commit_uniform(bar(C::B_DPFULL));
          commit_uniform(bar(C::B_DOEMPTY + do_stage));
          if (++do_stage == C::OS) { do_stage = 0; do_parity ^= 1u; }
        };
        advance();
        if (have && (ok = wait(C::B_VFULL, 0, W_U_VFULL) && wait(C::B_DOFULL, 0, W_U_DOFULL))) issue_dp();
        while (have && ok) {
          const int n = it.w;
          for (int e = 0; e < n; ++e, ++t) {
            const bool last = (e == n - 1);
            if (e == 0 && m > 0 && !(ok = wait(C::B_ACCFREE + 1, (m - 1) & 1, W_U_ACCFREE))) break;
            if (!(ok = wait(C::B_DSFULL, t & 1, W_U_DSFULL))) break;
            // V's last reader in this item, dP^T(t), is done: the next item's V goes into the same buffer, before the products
            // below if that item is known
            bool v_asked = false;
            if (last && __all_sync(0xffffffffu, mbar_test_wait(bar(C::B_ITEMFULL + k % C::NITEM), (k / C::NITEM) & 1))) {
              advance();
              v_asked = true;
              if (have) {
                if (elect_one()) load_tile(&tmV, sV, C::B_VFULL, it.z & 0xFFFF, it.y, it.x);
                ++v_loads;
              }
            }
            tc_fence_after_sync();
            if (kDq) {
              product_dq(k_mn0);   // over dP^T(t), which dS^T(t) was made from
              commit_uniform(bar(C::B_DQFULL));
            }
#pragma unroll 1
            for (int w = 0; w < 2; ++w) product_dk(w, q_mn0 + q_stage * T16, e == 0 && w == 0);
            commit_uniform(bar(C::B_DSFREE));
            commit_uniform(bar(C::B_QEMPTY + q_stage));
            if (++q_stage == C::QS) q_stage = 0;
            if (last) {
              commit_uniform(bar(C::B_ACCFULL + 1));
              if (!v_asked) {
                advance();
                if (have) {
                  if (elect_one()) load_tile(&tmV, sV, C::B_VFULL, it.z & 0xFFFF, it.y, it.x);
                  ++v_loads;
                }
              }
              if (have) {   // one K buffer: the next item's K can only be requested when the products above are done
                if (!(ok = wait(C::B_DSFREE, t & 1, W_U_DSFREE))) break;
                if (elect_one()) load_tile(&tmK, sK, C::B_KFULL, it.z & 0xFFFF, it.y, it.x);
                ++k_loads;
              }
            }
            if (have) {
              if (kDq && !(ok = wait(C::B_DQEMPTY, t & 1, W_U_DQEMPTY))) break;
              if (last && !(ok = wait(C::B_VFULL, (m + 1) & 1, W_U_VFULL))) break;
              if (!(ok = wait(C::B_DOFULL + do_stage, do_parity, W_U_DOFULL))) break;
              issue_dp();
            }
          }
          ++m;
        }
        if (lane == 0 && (gave_up != 0u || abortf->v != 0u)) {   // let this warp's own copies in flight land before the CTA exits
          if (k_loads > 1) drain_wait(bar(C::B_KFULL), (k_loads - 1) & 1);
          if (v_loads > 1) drain_wait(bar(C::B_VFULL), (v_loads - 1) & 1);
        }
      }
    }
  } else if (warp < 12) {
    reg_alloc<C::REGS_COMPUTE>();
    // ------------------------------ compute warpgroups ------------------------------
    // Warpgroup w handles queries 64 w .. 64 w + 63 of every tile, a warp 32 keys of it in two halves of 16. In a half, this
    // thread holds keys lane / 4 and lane / 4 + 8 and, of every 8 queries, queries 2 (lane % 4) and + 1.
    const int w = (warp - 4) >> 2, wq = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = lane_base + C::TM_S + w * 64, tDP = lane_base + C::TM_DP + w * 64, tP = lane_base + C::TM_P + w * C::P_STRIDE;
    constexpr uint32_t ROW16 = 16u << 16;
    const uint64_t nc2 = pack_f32x2(-a.scale_log2, -a.scale_log2), minus1 = pack_f32x2(-1.f, -1.f);
    const int qcol = w * 64 + 2 * (lane & 3);       // this thread's first query
    // stmatrix: matrix m of four = (rows 8 (m & 1) .., 16-byte chunk n + (m >> 1)); lane l gives the address of row l % 8 of matrix l / 8
    const uint32_t ds_row = sDS + static_cast<uint32_t>(w) * 16384u + static_cast<uint32_t>(wq * 32 + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128u;
    const uint32_t ds_sw = static_cast<uint32_t>((lane >> 4) ^ (lane & 7)) << 4;
    bool ok = true;
    int t = 0, qs = 0;
    int4 it;
    // zeroes the hidden ones among this thread's 32 values of half hf
    auto apply_mask = [&](uint32_t (&p)[32], const uint32_t (&mk)[2], int hf) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int src = hf * 16 + r * 8 + (lane >> 2);   // the lane that holds this key's mask
        const uint32_t m0 = __shfl_sync(0xffffffffu, mk[0], src) >> (2 * (lane & 3));
        const uint32_t m1 = __shfl_sync(0xffffffffu, mk[1], src) >> (2 * (lane & 3));
        // A byte's top bit spread over a word by one permute, for the two queries of a byte: two instructions a value, where a test
        // and a select were three (hier T = 4096, D = 64: backward 1222 -> 1175 us; T = 2048 198 -> 192).
        const uint32_t e0 = m0 << 7, o0 = m0 << 6, e1 = m1 << 7, o1 = m1 << 6;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t sel = 0x8888u + 0x1111u * (j & 3);
          p[4 * j + 2 * r] &= prmt_sign(j < 4 ? e0 : e1, sel);
          p[4 * j + 2 * r + 1] &= prmt_sign(j < 4 ? o0 : o1, sel);
        }
      }
    };
    if constexpr (HD == 64) {
      // Iteration t forms dS^T of tile t - 1 and, LAG blocks behind it in the same instruction stream, P^T of tile t. Each product is issued as
      // soon as its predecessor has been loaded; dP^T(t) then has the P^T blocks behind the dS^T blocks' end, the masks and the stores
      // to be formed under, S^T(t + 1) the first LAG blocks of the next iteration. (Side by side from one barrier for both, every
      // iteration waits some 250 cycles for its products. Backward us on one box, lag 0 / 2 / 5 / 6 / 7 / 8: causal 8 x 16 x 1000 x 64 93.6 / 91.7 / 90.6 / 89.2 / 89.6 / 91.7,
      // 8 x 16 x 2048 280 / 290 / 281 / 273 / 276 / 281, hierarchical 8 x 16 x 2048 x 64 139.4 / 139.3 / 138.5 / 135.8 / 136.8 / 140.7, 16 x 16 x 4096 x 64 948 / 981 /
      // 966 / 930 / 943 / 983. The exponentials and the multiply-adds of one warp overlap less, so both want to be kept.) The two warpgroups
      // have barriers of their own and drift apart, so that one does arithmetic while the other waits, loads or stores:
      //   SFULL, DPFULL  the half of S^T, dP^T is there       SFREE, DPFREE  it has been loaded
      //   PFULL, DSFULL  its P^T, dS^T has been written       PFREE  dV has read P^T;  DSFREE  dK and dQ have read dS^T
      // P^T stays in registers as fp32 for a tile.
      uint32_t p[2][32];
#pragma unroll
      for (int j = 0; j < 32; ++j) p[0][j] = p[1][j] = 0u;
      constexpr int LAG = 6;
      bool dp_ready = true;
      const float* side_prev = sSide;
      // What the warps need to know of a tile's item lies beside its scalars: a header read at the start of every item is code that the
      // instruction cache has lost by then, and cost 900 cycles of it. (Read where PARTIAL tiles are masked; read ahead of the arithmetic the
      // entry makes every tile 4 % longer.) Behind the last tile, P^T is computed from whatever is there and read by nobody.
#pragma unroll 1
      for (;; ++t) {
        const float* side = sSide + qs * C::SIDE_WORDS;
        // 16 keys x 16 queries at a time, both halves of the keys for a group of queries. The next block is loaded while one is
        // worked on: with two warps to a scheduler a TMEM load of some 150 cycles that is waited for at once is not covered. (Four
        // blocks of 32 queries, each loaded and awaited: causal 8 x 16 x 1000 x 64 84.0 -> 80.7 us, 8 x 16 x 2048 241 -> 230.)
        // (In the first iteration dS^T is computed from whatever is there, and read by nobody.)
        uint32_t sb[2][8], db[2][8];
        uint64_t lse[2], delta[2];
        bool s_ready = false, out_ready = false;   // barriers are tested ahead: a test takes some 150 cycles under this load, and as a rule it finds the phase complete
        if (!__all_sync(0xffffffffu, dp_ready)) {
          if (t > 0 && !(ok = wait(C::B_DPFULL + w, (t - 1) & 1, W_U_DPFULL))) break;
          if (t > 1 && !(ok = wait(C::B_DSFREE, t & 1, W_U_DSFREE))) break;
        }
        tc_fence_after_sync();
        tmem_ld16x256_x2(tDP, db[0]);
#pragma unroll
        for (int c = 0; c < 8 + LAG; ++c) {
          const int hf = c & 1, g = c >> 1, cp = c - LAG, gp = cp >> 1, hp = cp & 1;
          if (c < 8 && hf == 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) delta[j] = ld_shared_pair(side_prev + KD_TILE + qcol + 16 * g + 8 * j);
          }
          if (cp >= 0 && hp == 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) lse[j] = ld_shared_pair(side + qcol + 16 * gp + 8 * j);
          }
          if (c == LAG - 2) s_ready = mbar_test_wait(bar(C::B_SFULL + w), t & 1);
          if (c == LAG - 1) {
            if (!__all_sync(0xffffffffu, s_ready) && !(ok = wait(C::B_SFULL + w, t & 1, W_U_SFULL))) break;
            tc_fence_after_sync();
          }
          tmem_wait_ld();
          if (c < 7) tmem_ld16x256_x2(tDP + ((c + 1) & 1) * ROW16 + ((c + 1) >> 1) * 16, db[(c + 1) & 1]);
          if (cp >= -1 && cp < 7) tmem_ld16x256_x2(tS + ((cp + 1) & 1) * ROW16 + ((cp + 1) >> 1) * 16, sb[(cp + 1) & 1]);
          if (c == 7) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0 && t > 0) mbar_arrive(bar(C::B_DPFREE + w));
          }
          if (cp == 7) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(C::B_SFREE + w));
            out_ready = mbar_test_wait(bar(C::B_PFREE + w), (t - 1) & 1);
          }
          if (c < 8) {
            uint32_t pk[4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint64_t d = fma_f32x2(delta[j], minus1, pack_u32x2(db[hf][4 * j + 2 * r], db[hf][4 * j + 2 * r + 1]));
                const uint64_t x = mul_f32x2(pack_u32x2(p[hf][8 * g + 4 * j + 2 * r], p[hf][8 * g + 4 * j + 2 * r + 1]), d);
                pk[2 * j + r] = pack2<kBf16>(lo_f32x2(x), hi_f32x2(x));
              }
            }
            stmatrix_x4(ds_row + hf * 2048u + ((static_cast<uint32_t>(2 * g) << 4) ^ ds_sw), pk[0], pk[1], pk[2], pk[3]);
          }
          if (cp >= 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint64_t y = fma_f32x2(pack_u32x2(sb[hp][4 * j + 2 * r], sb[hp][4 * j + 2 * r + 1]), nc2, lse[j]);   // LSE - c S
                p[hp][8 * gp + 4 * j + 2 * r] = __float_as_uint(fast_exp2(-lo_f32x2(y)));
                p[hp][8 * gp + 4 * j + 2 * r + 1] = __float_as_uint(fast_exp2(-hi_f32x2(y)));
              }
            }
          }
          if (c == 7) {
            fence_proxy_async_smem();   // the dK and dQ products read dS^T through the async proxy
            __syncwarp();
            if (lane == 0 && t > 0) mbar_arrive(bar(C::B_DSFULL + w));
          }
        }
        if (!ok) break;
        const uint32_t* side_u = reinterpret_cast<const uint32_t*>(side);
        const uint32_t ent = side_u[C::SIDE_ENT];
        if (ent == C::ENT_END) break;
        if ((ent >> 8) == KD_TILE_PARTIAL) {
          // The words of this thread's queries, one pair after the other: a shift brings this thread's keys to the top bits of the
          // bytes, and a byte's top bit spreads over a word by one permute. (Formed here from class masks and descriptors, key by
          // key, before the plan held them: hierarchical 16 x 16 x 4096 x 64 backward 1072 -> 1025 us, 8 x 16 x 2048 x 64 167 -> 162,
          // causal 8 x 16 x 1000 x 64 97.4 -> 94.5.)
          const uint32_t* words = side_u + C::SIDE_BITS + wq * KD_TILE + qcol;
          const int up = 7 - (lane >> 2);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint2 x = *reinterpret_cast<const uint2*>(words + 8 * j);
            const uint32_t even = x.x << up, odd = x.y << up;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint32_t sel = 0x8888u + 0x1111u * (2 * hf + r);
                p[hf][4 * j + 2 * r] &= prmt_sign(even, sel);
                p[hf][4 * j + 2 * r + 1] &= prmt_sign(odd, sel);
              }
          }
        }
        if (!__all_sync(0xffffffffu, out_ready) && t > 0 && !(ok = wait(C::B_PFREE + w, (t - 1) & 1, W_U_PFREE))) break;
        tc_fence_after_sync();
        dp_ready = mbar_test_wait(bar(C::B_DPFULL + w), t & 1) && mbar_test_wait(bar(C::B_DSFREE), (t + 1) & 1);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = pack2<kBf16>(__uint_as_float(p[hf][2 * j]), __uint_as_float(p[hf][2 * j + 1]));
          tmem_st16x128_x8(tP + hf * ROW16, pk);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_PFULL + w));
        side_prev = side;
        if (++qs == C::QS) qs = 0;
      }
    } else {
    for (int k = 0; ok && next_item(k, it); ++k) {
      const int b = it.x, kt = it.z & 0xFFFF, n = it.w;
      const uint16_t* list = a.bwd_list + ((size_t)b * a.NT + kt) * a.NT;
      uint32_t ent_next = static_cast<uint32_t>(it.z) >> 16;
      for (int e = 0; e < n; ++e, ++t) {
        const uint32_t ent = ent_next;
        if (e + 1 < n) ent_next = __ldcg(list + e + 1);
        const bool partial = (ent >> 8) == KD_TILE_PARTIAL;
        uint32_t mk[2] = {0u, 0u};   // of a PARTIAL tile: the words of queries 64 w + lane and + 32 for the warp's keys, requested ahead of the wait
        if (partial) {
          if constexpr (kWords) {
            const uint32_t* src = a.words + (((size_t)b * a.NT + (ent & 0xFF)) * a.NT + kt) * KD_WORDS + wq * KD_TILE + w * 64 + lane;
            mk[0] = __ldcg(src);
            mk[1] = __ldcg(src + 32);
          } else {
            const uint32_t* desc = a.desc + (size_t)b * a.Tpad;
            const int qi = static_cast<int>(ent & 0xFF) * KD_TILE + w * 64 + lane;
            const uint32_t qd[2] = {__ldcg(desc + qi), __ldcg(desc + qi + 32)};
            const KeyRun<1> keys(desc, a.tilebits + (size_t)b * a.NT * 32, kt, wq, lane);
#pragma unroll
            for (int r = 0; r < 2; ++r) keys.words(qd[r], qi + 32 * r, mk + r);
          }
        }
        // LSE and delta of the stage were copied by the producer warp, which the stage's barrier counts and for which the issuing warp waited before the product awaited here
        const float* side = sSide + qs * C::SIDE_WORDS;
        bool masked = false;
        if (partial) {   // before the wait for the scores: a word for each key (many a block of such a tile is visible as a whole)
          masked = __any_sync(0xffffffffu, (mk[0] & mk[1]) != 0xFFFFFFFFu);
          if (masked) {
            mk[0] = transpose_bits(mk[0], lane);
            mk[1] = transpose_bits(mk[1], lane);
          }
        }
        if (!(ok = wait(C::B_SFULL, t & 1, W_U_SFULL))) break;
        tc_fence_after_sync();
        if (++qs == C::QS) qs = 0;
        uint32_t s[2][32];
        tmem_ld16x256_x8(tS, s[0]);
        uint64_t col[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) col[j] = ld_shared_pair(side + qcol + 8 * j);   // LSE of this thread's columns
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {   // 16 keys at a time
          tmem_wait_ld();
          if (hf == 0) tmem_ld16x256_x8(tS + ROW16, s[1]);   // under the first half's arithmetic
#pragma unroll
          for (int j = 0; j < 8; ++j) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const uint64_t x = fma_f32x2(pack_u32x2(s[hf][4 * j + 2 * r], s[hf][4 * j + 2 * r + 1]), nc2, col[j]);   // LSE - c S
              s[hf][4 * j + 2 * r] = __float_as_uint(fast_exp2(-lo_f32x2(x)));
              s[hf][4 * j + 2 * r + 1] = __float_as_uint(fast_exp2(-hi_f32x2(x)));
            }
          }
          if (masked) apply_mask(s[hf], mk, hf);
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = pack2<kBf16>(__uint_as_float(s[hf][2 * j]), __uint_as_float(s[hf][2 * j + 1]));
          tmem_st16x128_x8(tP + hf * ROW16, pk);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_PFULL));

#pragma unroll
        for (int j = 0; j < 8; ++j) col[j] = ld_shared_pair(side + KD_TILE + qcol + 8 * j);   // delta
        // dP^T, and the products that read the previous tile's dS^T are done (long before, as a rule)
        if (!(ok = t == 0 ? wait(C::B_DPFULL, 0, W_U_DPFULL) : wait2(C::B_DPFULL, t & 1, W_U_DPFULL, C::B_DSFREE, (t - 1) & 1, W_U_DSFREE))) break;
        tc_fence_after_sync();
        // 16 keys x 32 queries at a time; the next block is loaded while one is worked on (causal 1 x 16 x 16384 x 128, whole backward: 2750 -> 2640 us)
        uint32_t dp[2][16];
        tmem_ld16x256_x4(tDP, dp[0]);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t pk[16];
#pragma unroll
          for (int ch = 0; ch < 2; ++ch) {
            tmem_wait_ld();
            if (hf + ch < 2) tmem_ld16x256_x4(tDP + (ch == 0 ? hf : 1) * ROW16 + (ch == 0 ? 32 : 0), dp[ch ^ 1]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint64_t d = fma_f32x2(col[4 * ch + j], minus1, pack_u32x2(dp[ch][4 * j + 2 * r], dp[ch][4 * j + 2 * r + 1]));
                const uint64_t x = mul_f32x2(pack_u32x2(s[hf][16 * ch + 4 * j + 2 * r], s[hf][16 * ch + 4 * j + 2 * r + 1]), d);
                pk[8 * ch + 2 * j + r] = pack2<kBf16>(lo_f32x2(x), hi_f32x2(x));
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 8; j += 2)
            stmatrix_x4(ds_row + hf * 2048u + ((static_cast<uint32_t>(j) << 4) ^ ds_sw), pk[2 * j], pk[2 * j + 1], pk[2 * j + 2], pk[2 * j + 3]);
        }
        fence_proxy_async_smem();   // the dK and dQ products read these shared-memory writes through the async proxy
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_DSFULL));
      }
    }
    }
  } else {
    reg_dealloc<C::REGS_DQ>();
    // ------------------------------ dQ warps: TMEM -> shared memory -> bulk reduction into the fp32 scratch ------------------------------
    if (kDq) pdl_wait();   // the scratch has been zeroed
    const int wq = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t stg = s0 + C::SMEM_STG + wq * (C::NSTG * 4096), st_row = static_cast<uint32_t>(lane) * 128u, st_sw = static_cast<uint32_t>(lane & 7);
    if (lane == 0) {
      tma_prefetch_desc(&tmAcc);
      tma_prefetch_desc(&tmDK);
      tma_prefetch_desc(&tmDV);
    }
    bool ok = true;
    int t = 0;
    const int np = (a.d_real + 31) / 32;   // 32-column pieces of a dQ tile
    auto stage_box = [&](int buf, const uint32_t (&r)[32]) {   // 32 columns as a box [32 rows][32 columns]
#pragma unroll
      for (int cch = 0; cch < 8; ++cch)
        st_shared_v4(stg + buf * 4096 + st_row + ((static_cast<uint32_t>(cch) ^ st_sw) << 4), r[4 * cch], r[4 * cch + 1], r[4 * cch + 2], r[4 * cch + 3]);
    };
    auto stage_scaled = [&](int buf, uint32_t (&r)[32], float f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * f);
      stage_box(buf, r);
    };
    // Writes dV or dK (is_k) of the item: 32 rows of a warp as boxes of 64 columns through the staging buffers and TMA stores. m: number of
    // the item; kt: its key tile. dV goes before the item's last dQ tile, which is formed an iteration after the last dV product: the next
    // item's first dV product waits for its columns, and with it P^T of the tile after. (dV behind that dQ tile, together with dK: the
    // second tile of an item took 2,300 cycles more than others.)
    auto write_out = [&](bool is_k, int b, int h, int kt, int m) -> bool {
      if (!wait(C::B_ACCFULL + (is_k ? 1 : 0), m & 1, W_U_ACCFULL)) return false;
      tc_fence_after_sync();
      const int key0 = kt * KD_TILE + wq * 32;
#pragma unroll 1
      for (int part = 0; part < HD / 64; ++part) {
        const int col = part * 64;
        const uint32_t buf = kF32 ? stg : stg + (part & 1) * 4096;   // 64 columns of float32 are two boxes
        const float f = is_k ? a.sm_scale : 1.0f;
        if (kF32 || (part & 1) == 0) {
          if (lane == 0) bulk_wait_group_read0();   // the staging buffers have been read
          __syncwarp();
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tmem_ld32(lane_base + (is_k ? C::TM_DK : C::TM_DV) + col + half * 32, r);
          tmem_wait_ld();
          if (col + 64 == HD && half == 1) {   // the accumulator is in registers: the next item's first product may overwrite it
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(C::B_ACCFREE + (is_k ? 1 : 0)));
          }
          if (!kDq && fa.direct != 0) {
            if (key0 + lane < a.T) {
              const size_t at = is_k ? (size_t)b * a.dk_sb + (size_t)h * a.dk_sh + (size_t)(key0 + lane) * a.dk_st : (size_t)b * a.dv_sb + (size_t)h * a.dv_sh + (size_t)(key0 + lane) * a.dv_st;
              void* out = is_k ? a.dk : a.dv;
              if constexpr (kF32) store_row32_f32_upto(static_cast<float*>(out) + at + col + half * 32, r, f, col + half * 32, a.d_real);
              else store_row32_upto<kBf16>(static_cast<uint16_t*>(out) + at + col + half * 32, r, f, col + half * 32, a.d_real);
            }
            continue;
          }
          if constexpr (kF32 && C::NSTG == 1) {   // a box at a time
            if (half == 1) {
              if (lane == 0) bulk_wait_group_read0();
              __syncwarp();
            }
            stage_scaled(0, r, f);
            if (half == 0) {
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0 && key0 < a.T) {
                tma_store_4d(is_k ? &tmDK : &tmDV, stg, col, key0, h, b);
                bulk_commit_group();
              }
            }
          } else if constexpr (kF32) {
            stage_scaled(half, r, f);
          } else {
            uint32_t pk[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) pk[j] = pack2<kBf16>(__uint_as_float(r[2 * j]) * f, __uint_as_float(r[2 * j + 1]) * f);
#pragma unroll
            for (int cch = 0; cch < 4; ++cch)
              st_shared_v4(buf + st_row + ((static_cast<uint32_t>(4 * half + cch) ^ st_sw) << 4), pk[4 * cch], pk[4 * cch + 1], pk[4 * cch + 2], pk[4 * cch + 3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && key0 < a.T && col < a.d_real && (kDq || fa.direct == 0)) {
          if (kF32 && C::NSTG == 1) {
            if (col + 32 < a.d_real) tma_store_4d(is_k ? &tmDK : &tmDV, buf, col + 32, key0, h, b);
          } else {
            tma_store_4d(is_k ? &tmDK : &tmDV, buf, col, key0, h, b);
          }
          if (kF32 && C::NSTG == 2 && col + 32 < a.d_real) tma_store_4d(is_k ? &tmDK : &tmDV, buf + 4096, col + 32, key0, h, b);
          bulk_commit_group();
        }
      }
      return true;
    };
    int4 it;
    int m = 0;
    for (int k = 0; ok && next_item(k, it); ++k) {
      const int b = it.x, h = it.y, kt = it.z & 0xFFFF, n = it.w;
      const int bh = b * a.H + h;
      const uint16_t* list = a.bwd_list + ((size_t)b * a.NT + kt) * a.NT;
      uint32_t ent_next = static_cast<uint32_t>(it.z) >> 16;
      auto dq_tile = [&](int e) -> bool {
        const int q0 = (ent_next & 0xFF) * KD_TILE + wq * 32;
        if (e + 1 < n) ent_next = list[e + 1];
        if (!wait(C::B_DQFULL, t & 1, W_U_DQFULL)) return false;
        tc_fence_after_sync();
        const uint32_t tDQ = lane_base + C::TM_DQ;
        auto drained = [&]() {   // the tile is in registers: the columns may be overwritten
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_DQEMPTY));
        };
        auto stage = [&](int buf, uint32_t (&r)[32]) {
          if constexpr (kF32) stage_scaled(buf, r, a.sm_scale);
          else stage_box(buf, r);
        };
        auto add = [&](uint32_t src, int col) {
          if constexpr (kF32) tma_reduce_add_4d(&tmAcc, src, col, q0, h, b);
          else tma_reduce_add_3d(&tmAcc, src, col, q0, bh);
        };
        auto reduce = [&](int g) {   // both boxes: columns 64 g .. 64 g + 63
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && q0 < a.T) {
            if (g * 2 < np) add(stg, g * 64);
            if (g * 2 + 1 < np) add(stg + 4096, g * 64 + 32);
            bulk_commit_group();
          }
        };
        if constexpr (HD == 64) {
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            uint32_t r[32];
            tmem_ld32(tDQ + p * 32, r);
            tmem_wait_ld();
            if (p == 1) drained();
            if (lane == 0) bulk_wait_group_read0();   // the staging buffer has been read
            __syncwarp();
            stage(0, r);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && q0 < a.T) {
              if (p < np) add(stg, p * 32);
              bulk_commit_group();
            }
          }
        } else {   // the next dP^T waits for these columns: the second half goes into registers before the first leaves
          uint32_t r[2][32];
          tmem_ld32(tDQ, r[0]);
          tmem_ld32(tDQ + 32, r[1]);
          tmem_wait_ld();
          if (lane == 0) bulk_wait_group_read0();   // the staging buffers have been read
          __syncwarp();
          stage(0, r[0]);
          stage(1, r[1]);
          tmem_ld32(tDQ + 64, r[0]);
          tmem_ld32(tDQ + 96, r[1]);
          tmem_wait_ld();
          drained();
          reduce(0);
          if (lane == 0) bulk_wait_group_read0();
          __syncwarp();
          stage(0, r[0]);
          stage(1, r[1]);
          reduce(1);
        }
        ++t;
        return true;
      };
      // the item's dQ tiles; dV before the last, dK behind it
      if constexpr (!kDq) {
#pragma unroll 1
        for (int step = 0; ok && step < 2; ++step) ok = write_out(step == 1, b, h, kt, m);
      } else if constexpr (HD == 64) {
        for (int e = 0; ok && e < n; ++e) {
          const bool last = e == n - 1;
          ok = (!last || write_out(false, b, h, kt, m)) && dq_tile(e) && (!last || write_out(true, b, h, kt, m));
        }
      } else {   // (two copies of write_out are 60 bytes of spills at this width, and 2 % of the kernel; one copy is 0.6 % slower at the other)
#pragma unroll 1
        for (int step = 0; ok && step < n + 2; ++step)
          ok = (step == n - 1 || step == n + 1) ? write_out(step == n + 1, b, h, kt, m) : dq_tile(min(step, n - 1));
      }
      ++m;
    }
    if (lane == 0) bulk_wait_group0();
  }

  if (gave_up != 0u) raise_abort(abortf, gave_up);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(0, 512);
  if (tid == 0) report_abort(abortf, a.status);
  if (!kDq && a.after_dq != 0) pdl_wait();
}

// dq[b, h, t, :] = dq_acc[b, h, t, :] * sm_scale in the output dtype; HD / 8 threads per row, 32 bytes in and 16 out each
template <int HD, bool kBf16>
__global__ void __launch_bounds__(256) attn_bwd_dq_convert_kernel(const BwdArgs a) {
  using R = RowBlocks<HD>;
  const int sub = threadIdx.x % R::TPR;
  const int b = blockIdx.z, h = blockIdx.y, t0 = blockIdx.x * R::ROWS;
  const int len = __ldcg(a.len + b);   // (the plan was complete before the fused kernel let this one start)
  pdl_wait();
  pdl_launch_dependents();
  if (sub * 8 >= a.d_real) return;
  const size_t row0 = ((size_t)b * a.H + h) * a.T;
  uint16_t* out = reinterpret_cast<uint16_t*>(a.dq) + (size_t)b * a.dq_sb + (size_t)h * a.dq_sh + sub * 8;
  float4 x[R::STEPS], y[R::STEPS];
#pragma unroll
  for (int i = 0; i < R::STEPS; ++i) {
    const int t = t0 + i * R::RPB + threadIdx.x / R::TPR;
    x[i] = y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < len) {   // (the scratch of padding has not been zeroed)
      const float4* src = reinterpret_cast<const float4*>(a.dq_acc + (row0 + t) * HD + sub * 8);
      x[i] = src[0];
      y[i] = src[1];
    }
  }
#pragma unroll
  for (int i = 0; i < R::STEPS; ++i) {
    const int t = t0 + i * R::RPB + threadIdx.x / R::TPR;
    uint4 v;
    v.x = pack2<kBf16>(x[i].x * a.sm_scale, x[i].y * a.sm_scale);
    v.y = pack2<kBf16>(x[i].z * a.sm_scale, x[i].w * a.sm_scale);
    v.z = pack2<kBf16>(y[i].x * a.sm_scale, y[i].y * a.sm_scale);
    v.w = pack2<kBf16>(y[i].z * a.sm_scale, y[i].w * a.sm_scale);
    if (t < a.T) *reinterpret_cast<uint4*>(out + (size_t)t * a.dq_st) = v;
  }
}

template <int HD, bool kBf16, bool kF32, bool kDq, bool kWords>
static int launch_fused_t(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                          const BwdArgs& a, int dtype, bool after_delta, cudaStream_t stream) {
  using C = FusedCfg<HD>;
  CUtensorMap tmAcc, tmDK, tmDV;
  const kd_tensor dq = {a.dq, a.dq_sb, a.dq_sh, a.dq_st}, dk = {a.dk, a.dk_sb, a.dk_sh, a.dk_st}, dv = {a.dv, a.dv_sb, a.dv_sh, a.dv_st};
  auto encode_out = [&](CUtensorMap* tm, const kd_tensor& t, const char* name) {
    return kF32 ? encode_tensor_map_f32(tm, t, a.B, a.H, a.T, a.d_real, 32, name) : encode_tensor_map(tm, t, a.B, a.H, a.T, a.d_real, dtype, 32, name);
  };
  FusedArgs fa;
  fa.direct = 0;
  int rc = 0;
  if (!kDq) {
    fa.direct = encode_out(&tmDK, dk, nullptr) != 0 || encode_out(&tmDV, dv, nullptr) != 0;
    if (fa.direct) tmDK = tmDV = tmQ;   // not used
    tmAcc = tmDK;                       // nor is this
  } else {
    rc = kF32 ? encode_out(&tmAcc, dq, "dq") : encode_tensor_map_f32_rows(&tmAcc, a.dq_acc, a.B * a.H, a.T, HD, 32, "dq_acc");
    if (rc == 0) rc = encode_out(&tmDK, dk, "dk");
    if (rc == 0) rc = encode_out(&tmDV, dv, "dv");
  }
  if (rc != 0) return rc;
  const long long n_items = (long long)a.B * a.H * a.NT;
  if (n_items > 0x7FFFFFFF) return set_error(KD_ERR_LIMIT, "B * H * ceil(T / 128) exceeds 2^31 - 1");
  fa.b = a;
  fa.after_delta = after_delta;
  // Q, K, V, dO and, if there is one, the dQ scratch. (64 MB: hier T = 8192, D = 128 2470 us instead of 2409; without chunks 3540)
  fa.order_of = ItemOrder::make(a.B * a.H, a.NT, (double)a.T * (4.0 * a.d_real * 2 + (kDq ? HD * 4.0 : 0.0)), 90e6);
  auto kern = attn_bwd_fused_kernel<HD, kBf16, kF32, kDq, kWords>;
  static SmemOptIn opt_in;
  cudaError_t e = opt_in(kern, C::SMEM_ALLOC);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fused bwd smem attribute: %s", cudaGetErrorString(e));
  // The warps re-divide the registers the CTA was launched with; a request beyond that pool would block for ever,
  // so a build whose per-thread count is below the one the division assumes is refused here.
  static int launch_regs = 0;
  if (launch_regs == 0) {
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fused bwd attributes: %s", cudaGetErrorString(e));
    launch_regs = fa.numRegs;
  }
  if (launch_regs < C::REGS_LAUNCH) return set_error(KD_ERR_DEVICE, "fused bwd was built with %d registers per thread, needs %d", launch_regs, C::REGS_LAUNCH);
  e = launch(kern, static_cast<unsigned>(n_items), C::THREADS, C::SMEM_ALLOC, stream, tmQ, tmK, tmV, tmDO, tmAcc, tmDK, tmDV, fa);
  if (e == cudaSuccess && kDq && !kF32 && a.signs != nullptr)
    return launch_grad_transform(a.dq_acc, HD, a.sm_scale, a.len, a.signs, dq, dk, a.B, a.H, a.T, a.d_real, dtype, stream);
  if (e == cudaSuccess && kDq && !kF32) e = launch(attn_bwd_dq_convert_kernel<HD, kBf16>, RowBlocks<HD>::grid(a.B, a.H, a.T), 256, 0, stream, a);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "fused bwd kernels launch: %s", cudaGetErrorString(e));
  return 0;
}

template <bool kDq, bool kWords>
static int launch_one_pass(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                           const BwdArgs& a, int dtype, bool after_delta, cudaStream_t stream) {
  auto run = [&](auto launch_fn) { return launch_fn(tmQ, tmK, tmV, tmDO, a, dtype, after_delta, stream); };
  const bool narrow = a.d_real <= 64;
  if (a.grads_f32) return narrow ? run(launch_fused_t<64, false, true, kDq, kWords>) : run(launch_fused_t<128, false, true, kDq, kWords>);
  if (dtype == KD_BF16) return narrow ? run(launch_fused_t<64, true, false, kDq, kWords>) : run(launch_fused_t<128, true, false, kDq, kWords>);
  return narrow ? run(launch_fused_t<64, false, false, kDq, kWords>) : run(launch_fused_t<128, false, false, kDq, kWords>);
}

int launch_bwd_fused(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                     const BwdArgs& a, int dtype, bool after_delta, cudaStream_t stream) {
  const auto run = a.words != nullptr ? launch_one_pass<true, true> : launch_one_pass<true, false>;
  return run(tmQ, tmK, tmV, tmDO, a, dtype, after_delta, stream);
}

int launch_bwd_dkdv(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                    const BwdArgs& a, int dtype, cudaStream_t stream) {
  const auto run = a.words != nullptr ? launch_one_pass<false, true> : launch_one_pass<false, false>;
  return run(tmQ, tmK, tmV, tmDO, a, dtype, false, stream);
}

}  // namespace kd
