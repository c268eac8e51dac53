// Backward for sm_100a: the delta kernel, the deterministic backward's dQ kernel (query-tile major), and the launches of both backwards.
//
// The dQ kernel recomputes P = exp2(S*scale*log2e - LSE) from Q, K and the saved base-2 LSE and
// forms dS = P * (dP - delta), as the reference's dQ worker does (_flash_attn_bwd_dq, original_kernel.py:1173-1336), but
// walks only the non-empty tiles of the plan and applies the rule only on PARTIAL tiles.
// delta = rowsum(O * dO) (the reference's _flash_attn_bwd_precompute, :629-710) is produced
// by a small bandwidth-bound kernel ahead of it. dK and dV (the reference's _flash_attn_bwd_dkdv, :1339-1525) come from the fused kernel
// without its dQ (attn_bwd_fused.cu), which forms them in a fixed order. (A kernel of the structure below in its place, all key-tile
// work in units of 64 queries: deterministic backward, us, before and with the fused kernel: hierarchical 4 x 16 x 2048 x 64 96.7 -> 82.8,
// 16 x 16 x 4096 x 64 1378 -> 1202, 4 x 16 x 2048 x 128 177 -> 154, 3 x 6 x 1357 x 80 37.4 -> 28.9, causal 8 x 16 x 1000 x 64 124 -> 113.)
//
// Structure of the dQ kernel (640 threads): warp 0 = TMA producer, warps 1-3 = MMA issuers, warps 4-19 =
// four compute warpgroups. The backward needs no row reductions, so a 128-column score tile is
// split by columns: a "unit" u = 2*entry + half is one 64-column half, and two warpgroups share a
// unit, 32 columns each, so that sixteen warps (four per scheduler) hide one another's
// tensor-memory, barrier and special-function latencies. A unit owns TMEM buffer u % NBUF
// (64 columns of scores + 64 of dP) and the issuers run NBUF units ahead, so that a warpgroup
// finishing unit u finds its next unit's scores already in TMEM:
//   M1(u): S_u, dP_u  (smem x smem -> TMEM, N = 64)      compute(u): dS_u -> TMEM (16 bit)
//   M2(u): dQ += dS_u K  (A from TMEM);   then M1(u + NBUF)
// Each warpgroup writes its 16 packed columns over the start of the 32 fp32 columns it has just
// read, so the 16-bit operand of a unit sits at columns [0,16) and [32,48) of the buffer.
// The tensor pipe executes in issue order, so M1(u + NBUF) may overwrite the buffer M2(u) read.
// M1 and M2 are issued by different single threads (warps 3 and 2 for M1, warp 1 for M2), so
// that none of them is on the critical path of the other.
#include <algorithm>
#include <mutex>
#ifdef KD_TEST_DROP_LOAD
#include <stdlib.h>
#endif

#include "attn_bwd.cuh"

namespace kd {


template <int HD>
struct BwdCfg {
  static constexpr int KBLK = HD / 64;
  static constexpr int TILE_BYTES = KD_TILE * HD * 2;
  static constexpr int NBUF = (HD == 64) ? 3 : 2;     // score / dP buffers in TMEM
  static constexpr int STAGES = NBUF;                 // ring of (tile, tile) pairs
  static constexpr int NFIX = (HD == 64) ? 2 : 1;     // buffers for the per-head resident tile pair
  static constexpr int SMEM_FIX = 0;                               // NFIX x two resident tiles
  static constexpr int SMEM_RING = SMEM_FIX + NFIX * 2 * TILE_BYTES;  // STAGES x two streamed tiles
  static constexpr int NSUB = 2;                      // warpgroups that share a 64-column unit
  static constexpr int CPT = 2 / NSUB;                // 32-column chunks per compute thread and unit
  static constexpr int THREADS = 128 + 256 * NSUB;    // four light warps + 2 * NSUB compute warpgroups
  static constexpr int REGS_COMPUTE = KD_REGS_COMPUTE_BWD;
  static constexpr int NITEM = 4;                     // ring of item headers and lists
  static constexpr int SMEM_ACT = SMEM_RING + STAGES * 2 * TILE_BYTES;  // NITEM x <= 128 list entries
  static constexpr int SMEM_TOTAL = SMEM_ACT + NITEM * 128 * 2;
  static constexpr int SMEM_ALLOC = SMEM_TOTAL + 1024;
  // TMEM columns
  // buffer j: scores at 128*j, dP at 128*j + 64; the accumulator behind the buffers
  static constexpr uint32_t TM_ACC0 = NBUF * 128;        // dQ
  static_assert(TM_ACC0 + HD <= 512, "TMEM budget");
  static_assert(SMEM_ALLOC <= 232448, "shared memory budget");
};

enum : uint32_t {
  W_Q_FIXFULL = 0x201, W_Q_RINGEMPTY = 0x202, W_Q_RINGFULL = 0x203, W_Q_PFULL = 0x204, W_Q_SFULL = 0x205,
  W_Q_ACCFULL = 0x206, W_Q_M2ISSUED = 0x207, W_Q_FIXEMPTY = 0x208, W_Q_ACCFREE = 0x209,
  W_Q_ITEMFULL = 0x20A, W_Q_ITEMEMPTY = 0x20B, W_Q_CLC = 0x20C,
};

// =========================================================================================
// delta kernel: delta[b, h, t] = sum_d O[b, h, t, d] * dO[b, h, t, d] in fp32 (the reference's
// _flash_attn_bwd_precompute, original_kernel.py:629-710). HD/8 threads share a row, 16 bytes of
// each tensor per thread, so a warp reads whole 128-byte lines; bound by HBM bandwidth. For the fused
// backward it also zeroes the row of the fp32 dQ accumulation scratch (8 floats per thread).
// =========================================================================================
// A float32 call (kF32) leaves two more passes to it: dO is rounded to the 16-bit operand on the way, and dQ, into which the fused
// backward then adds, is zeroed in place of a scratch.
// Rows of padding see nothing: neither their O and dO are read nor their scratch zeroed (the conversion writes zeros there without a look at it).
template <int HD, bool kBf16, bool kF32>
__global__ void __launch_bounds__(256) attn_bwd_delta_kernel(const BwdArgs a) {
  using R = RowBlocks<HD>;
  const int sub = threadIdx.x % R::TPR;
  const int b = blockIdx.z, h = blockIdx.y, t0 = blockIdx.x * R::ROWS;
  if (a.len_ready == 0) pdl_wait();
  const int len = __ldcg(a.len + b);
  pdl_wait();
  pdl_launch_dependents();
  const size_t row0 = ((size_t)b * a.H + h) * a.T;
  uint16_t* d_o = reinterpret_cast<uint16_t*>(a.d_o) + (size_t)b * a.do_sb + (size_t)h * a.do_sh + sub * 8;
  // the loops' bounds are the same for every thread of the block: the shuffles below need full warps
  uint4 ov[R::STEPS], dv[R::STEPS];
#pragma unroll
  for (int i = 0; i < R::STEPS; ++i) {   // all loads ahead of the stores
    const int t = t0 + i * R::RPB + threadIdx.x / R::TPR;
    ov[i] = dv[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t < len && sub * 8 < a.d_real) {
      ov[i] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.o) + (size_t)b * a.o_sb + (size_t)h * a.o_sh + (size_t)t * a.o_st + sub * 8);
      if (kF32 && a.d_o32 != nullptr) {
        const float4* src = reinterpret_cast<const float4*>(a.d_o32 + (size_t)b * a.do32_sb + (size_t)h * a.do32_sh + (size_t)t * a.do32_st + sub * 8);
        const float4 x = src[0], y = src[1];
        dv[i] = make_uint4(pack2<kBf16>(x.x, x.y), pack2<kBf16>(x.z, x.w), pack2<kBf16>(y.x, y.y), pack2<kBf16>(y.z, y.w));
      } else {
        dv[i] = *reinterpret_cast<const uint4*>(d_o + (size_t)t * a.do_st);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R::STEPS; ++i) {
    const int t = t0 + i * R::RPB + threadIdx.x / R::TPR;
    float acc = 0.f;
    const uint32_t ow[4] = {ov[i].x, ov[i].y, ov[i].z, ov[i].w}, dw[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = unpack2<kBf16>(ow[k]), y = unpack2<kBf16>(dw[k]);
      acc = fmaf(x.x, y.x, acc);
      acc = fmaf(x.y, y.y, acc);
    }
    if (!kF32 && a.dq_acc != nullptr && t < len && sub * 8 < a.d_real) {   // the columns beyond are never read (zeroed too: causal 8 x 16 x 2048 x 80 370 us, 365 without)
      float4* z = reinterpret_cast<float4*>(a.dq_acc + (row0 + t) * HD + sub * 8);
      z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (kF32 && t < a.T && sub * 8 < a.d_real) {
      if (a.d_o32 != nullptr) *reinterpret_cast<uint4*>(d_o + (size_t)t * a.do_st) = dv[i];   // of padding too (zeros): the fused kernel reads whole tiles
      if (a.zero_dq) {
        float4* z = reinterpret_cast<float4*>(static_cast<float*>(a.dq) + (size_t)b * a.dq_sb + (size_t)h * a.dq_sh + (size_t)t * a.dq_st + sub * 8);
        z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int d = R::TPR / 2; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (t < a.T && sub == 0) a.delta[row0 + t] = acc;
  }
}

// =========================================================================================
// The dQ kernel's barriers, items and producer warp.
//
// A work item is one tile of one (batch, head). The grid has a CTA per item, but a CTA that is running takes further items by cancelling CTAs that have not been launched yet
// (clusterlaunchcontrol), as in the forward and the fused backward: the rings, the issuers and the compute warps run on into the
// next item, and the start and drain of a CTA (launch, TMEM, first loads, pipeline fill, last products: 12,000 cycles) is paid once
// per SM instead of once per item, which has some ten tiles of 2,200-2,800 cycles. This kernel and one alike for dK and dV, before (a CTA per tile and one
// or more heads) and with this, bf16 (us): hierarchical 4 x 16 x 2048 x 64 114 -> 108, 16 x 16 x 4096 x 64 1570 -> 1500; causal 8 x 16 x
// 1000 x 64 146 -> 127, 8 x 16 x 2048 x 128 723 -> 685; no mask 4 x 16 x 2048 x 64 383 -> 331; causal 1 x 8 x 173 x 64 14.6 -> 11.7.
// =========================================================================================
template <typename C>
struct BwdShared {
  uint64_t fix_full[C::NFIX], fix_empty[C::NFIX], ring_full[C::STAGES], ring_empty[C::STAGES], s_full[C::NBUF], p_full[C::NBUF],
      m2_issued[C::NBUF], acc_full, acc_free, item_full[C::NITEM], item_empty[C::NITEM], clc;
  __align__(16) int4 items[C::NITEM];   // {batch, head, tile, entries}; entries < 0: there is no further item
  __align__(16) uint8_t answer[16];     // of a cancellation
  uint32_t tmem_base;
  AbortFlag abortf;
};

template <typename C>
__device__ __forceinline__ void bwd_init(BwdShared<C>& sh) {   // one thread
  sh.abortf.v = 0;
  for (int f = 0; f < C::NFIX; ++f) {
    mbar_init(smem_u32(&sh.fix_full[f]), 1);
    mbar_init(smem_u32(&sh.fix_empty[f]), 2);  // both M1 issuers are done with the item's resident tiles
  }
  for (int s = 0; s < C::STAGES; ++s) {
    mbar_init(smem_u32(&sh.ring_full[s]), 1);
    mbar_init(smem_u32(&sh.ring_empty[s]), 1);
  }
  for (int i = 0; i < C::NBUF; ++i) {
    mbar_init(smem_u32(&sh.s_full[i]), 2);     // one commit from each of the two M1 issuers
    mbar_init(smem_u32(&sh.p_full[i]), 4 * C::NSUB);   // one arrival per warp of the warpgroups that share the unit
    mbar_init(smem_u32(&sh.m2_issued[i]), 1);
  }
  mbar_init(smem_u32(&sh.acc_full), 1);
  mbar_init(smem_u32(&sh.acc_free), 8 * C::NSUB);      // every compute warp has read its part of the accumulators
  for (int i = 0; i < C::NITEM; ++i) {
    mbar_init(smem_u32(&sh.item_full[i]), 1);
    mbar_init(smem_u32(&sh.item_empty[i]), 3 + 8 * C::NSUB);   // the three issuers and every compute warp
  }
  mbar_init(smem_u32(&sh.clc), 1);
  fence_barrier_init();
}

// header of the CTA's k-th item for a single thread, which needs no list; false: an abort
template <typename C>
__device__ __forceinline__ bool bwd_header(BwdShared<C>& sh, int k, uint32_t site, int4& it) {
  const int slot = k % C::NITEM;
  if (!mbar_wait<true>(smem_u32(&sh.item_full[slot]), (k / C::NITEM) & 1, &sh.abortf, site)) return false;
  it = sh.items[slot];
  mbar_arrive(smem_u32(&sh.item_empty[slot]));
  return true;
}

// warp-uniform for the compiler
__device__ __forceinline__ int4 uniform(const int4& v) {
  return make_int4(__reduce_max_sync(0xffffffffu, v.x), __reduce_max_sync(0xffffffffu, v.y), __reduce_max_sync(0xffffffffu, v.z), __reduce_max_sync(0xffffffffu, v.w));
}

// The producer warp: items are query tiles; Q and dO resident, K and V streamed. wait_ahead: the plan may be read now, the tensors only behind pdl_wait().
template <int HD>
__device__ __forceinline__ void bwd_producer(const CUtensorMap& tmFix0, const CUtensorMap& tmFix1, const CUtensorMap& tmRing0, const CUtensorMap& tmRing1,
                                             const BwdArgs& a, uint32_t sFix, uint32_t sRing, uint16_t* lists, BwdShared<BwdCfg<HD>>& sh, int lane,
                                             bool wait_ahead) {
  using C = BwdCfg<HD>;
  if (lane == 0) {
    tma_prefetch_desc(&tmFix0);
    tma_prefetch_desc(&tmFix1);
    tma_prefetch_desc(&tmRing0);
    tma_prefetch_desc(&tmRing1);
  }
  auto wait = [&](const uint64_t& bar, uint32_t parity, uint32_t site) -> bool {
    return __all_sync(0xffffffffu, mbar_wait<true>(smem_u32(&bar), parity, &sh.abortf, site));
  };
  const uint32_t below = (1u << lane) - 1u;
  uint32_t lst[4];   // the decoded item's list, 32 entries per register: tile | class << 8, zeros where an entry is another tile's
  auto decode = [&](int idx) -> int4 {
    int bh, rank;
    a.order_of.decode(idx, a.NT, bh, rank);
    int4 it;
    it.x = bh / a.H;
    it.y = bh - it.x * a.H;
    it.z = __ldcg(a.order + ((size_t)it.x * 3 + 1) * a.NT + rank);   // longest lists first
    const int row = it.z >> 1;   // the list of the pair
    const uint16_t* list = a.fwd_list + ((size_t)it.x * a.NP + row) * a.NT;
    const int n = __ldcg(a.fwd_cnt + it.x * a.NP + row);
#pragma unroll
    for (int r = 0; r < 4; ++r) lst[r] = r * 32 + lane < a.NT ? __ldcg(list + r * 32 + lane) : 0u;   // does not wait for the count
    it.w = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r * 32 + lane >= n) lst[r] = 0u;
      const uint32_t cls = (lst[r] >> (8 + 2 * (it.z & 1))) & 3u;
      lst[r] = cls != 0u ? (lst[r] & 0xFFu) | (cls << 8) : 0u;
      it.w += __popc(__ballot_sync(0xffffffffu, lst[r] != 0u));
    }
    return it;
  };
  int k = 0, asked = 0, issued = 0, fixed = 0;   // items published, cancellations asked for, ring entries and resident pairs requested
  bool ok = true, pending = false;
  // The next item is asked for three tiles before the end of this one (for a shorter one: when it is taken), as in the other kernels.
  auto ask = [&]() {
    if (lane == 0) {
      fence_proxy_async_smem();   // the previous response has been read
      mbar_arrive_expect_tx(smem_u32(&sh.clc), 16);
      clc_try_cancel(smem_u32(sh.answer), smem_u32(&sh.clc));
    }
    ++asked;
    pending = true;
  };
  auto take_next = [&](int4& nx) -> bool {
    if (!wait(sh.clc, (asked - 1) & 1, W_Q_CLC)) return false;
    pending = false;
    const int idx = clc_first_ctaid_x(smem_u32(sh.answer));
    __syncwarp();   // every lane has read the response that the next request overwrites
    nx.w = -1;
    if (idx >= 0) {
      nx = decode(idx);
      if (nx.w <= 2) ask();
    }
    return true;
  };
  auto load_pair = [&](const CUtensorMap& t0, const CUtensorMap& t1, uint32_t dst, const uint64_t& full, int tile, int h, int b) {
    if (lane != 0) return;
    const uint32_t bar = smem_u32(&full);
    mbar_arrive_expect_tx(bar, 2 * C::TILE_BYTES);
    for (int kb = 0; kb < C::KBLK; ++kb) {
      tma_load_4d(dst + kb * 16384, &t0, bar, kb * 64, tile * KD_TILE, h, b);
      tma_load_4d(dst + C::TILE_BYTES + kb * 16384, &t1, bar, kb * 64, tile * KD_TILE, h, b);
    }
  };
  int4 it = decode(blockIdx.x);
  if (it.w <= 2) ask();
  while (ok) {
    const int slot = k % C::NITEM, b = it.x, h = it.y, n = it.w;
    if (!(ok = wait(sh.item_empty[slot], ((k / C::NITEM) & 1) ^ 1, W_Q_ITEMEMPTY))) break;
    uint16_t* list = lists + slot * 128;
    int at = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t has = __ballot_sync(0xffffffffu, lst[r] != 0u);
      if (n > 0 && lst[r] != 0u) list[at + __popc(has & below)] = static_cast<uint16_t>(lst[r]);
      at += __popc(has);
    }
    if (lane == 0) sh.items[slot] = it;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sh.item_full[slot]));
    if (n < 0) break;
    if (k == 0 && wait_ahead) pdl_wait();
    ++k;
    int4 nx = it;
#pragma unroll 1
    for (int e = 0; e < max(n, 1); ++e) {
      if (n > 2 && e == n - 3) ask();
      if (e >= n - 1 && !(ok = take_next(nx))) break;   // its list is looked up while this item's last tiles wait for slots
      if (n == 0) break;
      if (e == 0) {   // the item's resident tiles: into the buffer of the item before the last (NFIX = 2)
        const int f = fixed % C::NFIX;
        if (!(ok = wait(sh.fix_empty[f], ((fixed / C::NFIX) & 1) ^ 1, W_Q_FIXEMPTY))) break;
        load_pair(tmFix0, tmFix1, sFix + f * 2 * C::TILE_BYTES, sh.fix_full[f], it.z, h, b);
        ++fixed;
      }
      const int st = issued % C::STAGES;
      if (!(ok = wait(sh.ring_empty[st], ((issued / C::STAGES) & 1) ^ 1, W_Q_RINGEMPTY))) break;
      if (!(test_drops(a, 2) && issued == 0)) load_pair(tmRing0, tmRing1, sRing + st * 2 * C::TILE_BYTES, sh.ring_full[st], list[e] & 0xFF, h, b);
      ++issued;
    }
    it = nx;
  }
  if (lane == 0 && sh.abortf.v != 0) {   // let the copies in flight land before the CTA exits
    for (int e = max(0, issued - C::STAGES); e < issued; ++e) drain_wait(smem_u32(&sh.ring_full[e % C::STAGES]), (e / C::STAGES) & 1);
    for (int f = max(0, fixed - C::NFIX); f < fixed; ++f) drain_wait(smem_u32(&sh.fix_full[f % C::NFIX]), (f / C::NFIX) & 1);
    if (pending) drain_wait(smem_u32(&sh.clc), (asked - 1) & 1);
  }
}

// =========================================================================================
// dQ kernel: items are query tiles; streams = key halves of the current key
// tile.   M1(i): S_i = Q K_i^T, dP_i = dO V_i^T      M2(i): dQ += dS_i K_i
// The producer and the issuers run on into the next item while the compute warps finish the current one.
// kF32: of a float32 call, whose gradients are float32. (As a branch of the float16 kernels: causal 8 x 16 x 2048 x 128 610.8 us, 609.4 so; level at head dim 64.)
// kWords: the plan has the PARTIAL tiles' bits (see KD_WORDS_LIMIT).
// =========================================================================================
template <int HD, bool kBf16, bool kF32, bool kWords>
__global__ void __launch_bounds__(BwdCfg<HD>::THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const BwdArgs a) {
  using C = BwdCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sFix = smem_u32(smem + C::SMEM_FIX);    // buffer f: Q at +0, dO at +TILE_BYTES
  const uint32_t sRing = smem_u32(smem + C::SMEM_RING);  // stage s: K at +0, V at +TILE_BYTES
  uint16_t* lists = reinterpret_cast<uint16_t*>(smem + C::SMEM_ACT);
  __shared__ BwdShared<C> sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) bwd_init<C>(sh);
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh.tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // With the delta kernel ahead the plan may be read before the wait, past L1: the start of a kernel that overlaps another
  // need not have cleaned it, and a plan's memory may have held another one.
  const bool wait_ahead = a.plan_ready != 0;
  if (!wait_ahead) pdl_wait();
  const uint32_t tbase = sh.tmem_base;

  if (warp < 4) {
    reg_dealloc<KD_REGS_ISSUE>();
    if (warp == 0) {
      bwd_producer<HD>(tmQ, tmDO, tmK, tmV, a, sFix, sRing, lists, sh, lane, wait_ahead);
    } else if ((warp == 3 || warp == 2) && lane == 0) {
      // ------------------------------ M1 issuers: warp 3: S_u = Q K_u^T; warp 2: dP_u = dO V_u^T ------------------------------
      const bool dp_part = (warp == 2);
      const uint32_t idesc_m1 = make_idesc_f16(kBf16, 0, 0, KD_TILE, 64);   // N = 64 keys
      const uint32_t hi = desc_hi_sw128();
      const uint32_t loRingK = desc_lo_kmajor(sRing);
      bool ok = true;
      int buf = 0, round = 0, stage = 0, item = 0;   // run on across the items; item: of those with entries
      uint32_t ring_parity = 0;
      int4 it;
      for (int k = 0; ok && bwd_header<C>(sh, k, W_Q_ITEMFULL, it) && it.w >= 0; ++k) {
        if (it.w == 0) continue;
        const int U = 2 * it.w, fb = item % C::NFIX;
        ok = mbar_wait<true>(smem_u32(&sh.fix_full[fb]), (item / C::NFIX) & 1, &sh.abortf, W_Q_FIXFULL);
        ++item;
        if (!ok) break;
        const uint32_t loA = desc_lo_kmajor(sFix + fb * 2 * C::TILE_BYTES + (dp_part ? C::TILE_BYTES : 0));   // dO or Q
        uint64_t adesc[HD / 16];   // A descriptors of the item's k-steps
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) adesc[kk] = desc64(loA + koff_kmajor(kk), hi);
        for (int u = 0; u < U && ok; ++u) {
          const int i = u & 1;
          // operands of the unit, formed ahead of the waits
          // key rows 64i.. of K (scores) or V (dP)
          const uint32_t blo = loRingK + stage * (2 * C::TILE_BYTES >> 4) + i * (64 * 128 >> 4) + (dp_part ? (C::TILE_BYTES >> 4) : 0);
          uint64_t bdesc[HD / 16];
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) bdesc[kk] = desc64(blo + koff_kmajor(kk), hi);
          const uint32_t dst = tbase + buf * 128 + (dp_part ? 64 : 0);
          if (round > 0) {   // buffer free once M2 of its previous unit has been issued
            ok = mbar_wait<true>(smem_u32(&sh.m2_issued[buf]), (round - 1) & 1, &sh.abortf, W_Q_M2ISSUED);
            if (!ok) break;
          }
          if (i == 0) {      // first unit of a new entry: its K and V tiles must have landed
            ok = mbar_wait<true>(smem_u32(&sh.ring_full[stage]), ring_parity, &sh.abortf, W_Q_RINGFULL);
            if (!ok) break;
          }
          tc_fence_after_sync();
          mma_ss64<false>(dst, adesc[0], bdesc[0], idesc_m1);
#pragma unroll
          for (int kk = 1; kk < HD / 16; ++kk) mma_ss64<true>(dst, adesc[kk], bdesc[kk], idesc_m1);
          mma_commit(smem_u32(&sh.s_full[buf]));
          if (++buf == C::NBUF) { buf = 0; ++round; }
          if (i == 1 && ++stage == C::STAGES) { stage = 0; ring_parity ^= 1; }
        }
        if (ok) mma_commit(smem_u32(&sh.fix_empty[fb]));   // this issuer's products of the item no longer read Q / dO
      }
    } else if (warp == 1 && lane == 0) {
      // ------------------------------ M2 issuer: dQ += dS_u K_u ------------------------------
      const uint32_t idesc_m2 = make_idesc_f16(kBf16, 0, 1, KD_TILE, HD);   // B = K rows, MN-major
      const uint32_t tAcc = tbase + C::TM_ACC0;
      const uint32_t hi = desc_hi_sw128();
      const uint32_t loRingMN = desc_lo_mnmajor(sRing);
      bool ok = true;
      int buf = 0, stage = 0, item = 0;
      uint32_t round_parity = 0;
      int4 it;
      for (int k = 0; ok && bwd_header<C>(sh, k, W_Q_ITEMFULL, it) && it.w >= 0; ++k) {
        if (it.w == 0) continue;
        const int U = 2 * it.w;
        if (item++ > 0) {   // the previous item's dQ must have been read out of the accumulator
          ok = mbar_wait<true>(smem_u32(&sh.acc_free), item & 1, &sh.abortf, W_Q_ACCFREE);
          if (!ok) break;
        }
        for (int u = 0; u < U && ok; ++u) {
          const int i = u & 1;
          // operands of the unit, formed ahead of the wait
          const uint32_t kb = loRingMN + stage * (2 * C::TILE_BYTES >> 4) + i * (64 * 128 >> 4);
          const uint32_t aS = tbase + buf * 128;   // dS_u sits on top of S_u: keys 0-31 at columns [0,16), keys 32-63 at [32,48)
          uint64_t bdesc[4];
          uint32_t aop[4];
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {  // 64 keys of this unit, 16 per MMA
            bdesc[kk] = desc64(kb + koff_mnmajor(kk), hi);
            aop[kk] = aS + (kk >> 1) * 32 + (kk & 1) * 8;
          }
          ok = mbar_wait<true>(smem_u32(&sh.p_full[buf]), round_parity, &sh.abortf, W_Q_PFULL);
          if (!ok) break;
          tc_fence_after_sync();
          mma_ts64_p(tAcc, aop[0], bdesc[0], idesc_m2, u > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 1; kk < 4; ++kk) mma_ts64<true>(tAcc, aop[kk], bdesc[kk], idesc_m2);
          if (i == 1) mma_commit(smem_u32(&sh.ring_empty[stage]));
          tc_fence_before_sync();
          mbar_arrive(smem_u32(&sh.m2_issued[buf]));
          if (++buf == C::NBUF) { buf = 0; round_parity ^= 1; }
          if (i == 1 && ++stage == C::STAGES) stage = 0;
        }
        if (ok) mma_commit(smem_u32(&sh.acc_full));
      }
    }
  } else {
    reg_alloc<C::REGS_COMPUTE>();
    // ------------------------------ compute warpgroups ------------------------------
    constexpr int CPT = C::CPT;      // 32-column chunks of a unit this thread handles
    const int g = (warp - 4) >> 2;   // warpgroup
    const int i = g / C::NSUB;       // stream: key half (64 keys) of each key tile
    const int c0 = (g % C::NSUB) * CPT;   // first 32-key chunk of that half handled here
    const int wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const float c = a.scale_log2;
    const int first_word = 2 * i + c0;   // of this thread's chunks among the four of a key tile
    bool ok = true;

    int4 it = make_int4(0, 0, 0, 0);   // the item in hand; behind its last unit the next one
    // The visibility words of a PARTIAL tile (of the plan; bit j: key j of a chunk) are fetched one entry ahead into registers.
    uint32_t mk_next[CPT];
    const uint32_t* words = a.words;   // of this thread's query and chunks in the item's query tile
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc) mk_next[cc] = 0u;
    auto fetch_words = [&](uint32_t entry) {
      if ((entry >> 8) != KD_TILE_PARTIAL) return;
      if constexpr (kWords) {
        const uint32_t* src = words + (entry & 0xFFu) * static_cast<uint32_t>(KD_WORDS);
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) mk_next[cc] = __ldcg(src + cc * KD_TILE);
      } else {
        form_words<CPT>(a.desc + (size_t)it.x * a.Tpad, a.tilebits + (size_t)it.x * a.NT * 32, it.z * KD_TILE + row, entry & 0xFFu, first_word, lane, mk_next);
      }
    };
    // The next item's header, first entry and scalars are fetched before the epilogue.
    uint32_t ent_next = 0u;
    float delta = 0.f, lse = 0.f;
    const uint16_t* list = lists;
    auto open_item = [&](int k) -> bool {
      const int slot = k % C::NITEM;
      if (!__all_sync(0xffffffffu, mbar_wait<true>(smem_u32(&sh.item_full[slot]), (k / C::NITEM) & 1, &sh.abortf, W_Q_ITEMFULL))) return false;
      it = uniform(sh.items[slot]);
      if (it.w < 0) return false;
      list = lists + slot * 128;
      if (kWords) words = a.words + ((size_t)it.x * a.NT + it.z) * a.NT * KD_WORDS + first_word * KD_TILE + row;
      if (it.w > 0) {
        ent_next = list[0];
        fetch_words(ent_next);
        const int qi = it.z * KD_TILE + row;
        const size_t at = ((size_t)it.x * a.H + it.y) * a.T + min(qi, a.T - 1);   // (rows beyond the last see nothing)
        delta = __ldcg(a.delta + at);
        lse = __ldcg(a.lse + at);
      }
      return true;
    };
    if (wait_ahead) pdl_wait();
    if (warp == 4) {
      __threadfence();   // for the kernel behind it, which does not wait for the delta kernel itself
      pdl_launch_dependents();
    }
    int n_acc = 0;   // items with units so far
    // this stream's next unit, counted over all items, as (unit / NBUF, unit % NBUF)
    int buf = i % C::NBUF;
    uint32_t rnd = i / C::NBUF;
    const uint32_t sfull0 = smem_u32(&sh.s_full[0]), pfull0 = smem_u32(&sh.p_full[0]);
    const uint32_t tcol = tbase + lane_base + c0 * 32;   // this thread's first chunk inside a buffer

    bool have = open_item(0);
    for (int k = 0; have && ok; ++k) {
      const int b = it.x, h = it.y, na = it.w, qi = it.z * KD_TILE + row;
      for (int e = 0; e < na; ++e) {
        const uint32_t ent = ent_next;
        const uint32_t cls = ent >> 8;
        uint32_t mk[CPT];   // visibility of the chunks' keys for this query row, where the tile is PARTIAL
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) mk[cc] = mk_next[cc];
        if (e + 1 < na) {
          ent_next = list[e + 1];
          fetch_words(ent_next);
        }
        const uint32_t tS = tcol + buf * 128, tP = tS + 64;
        ok = mbar_wait<true>(sfull0 + buf * 8, rnd & 1u, &sh.abortf, W_Q_SFULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();

#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          uint32_t pk[16];
          uint32_t rs[32], rp[32];
          tmem_ld32(tS + cc * 32, rs);
          tmem_ld32(tP + cc * 32, rp);
          tmem_wait_ld();
          if (cls != KD_TILE_PARTIAL) {   // warp-uniform: the common case carries no mask code at all
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const float p0 = fast_exp2(fmaf(__uint_as_float(rs[j]), c, -lse));
              const float p1 = fast_exp2(fmaf(__uint_as_float(rs[j + 1]), c, -lse));
              pk[j / 2] = pack2<kBf16>(p0 * (__uint_as_float(rp[j]) - delta), p1 * (__uint_as_float(rp[j + 1]) - delta));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float p0 = fast_exp2(fmaf(__uint_as_float(rs[j]), c, -lse));
              float p1 = fast_exp2(fmaf(__uint_as_float(rs[j + 1]), c, -lse));
              if ((mk[cc] & (1u << j)) == 0u) p0 = 0.f;
              if ((mk[cc] & (2u << j)) == 0u) p1 = 0.f;
              pk[j / 2] = pack2<kBf16>(p0 * (__uint_as_float(rp[j]) - delta), p1 * (__uint_as_float(rp[j + 1]) - delta));
            }
          }
          // dS of the chunk as 16-bit A operand over the start of the scores it was made from (this thread's own row)
          tmem_st16(tS + cc * 32, pk);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(pfull0 + buf * 8);
        buf += 2;
        if (buf >= C::NBUF) { buf -= C::NBUF; ++rnd; }
      }
      if (!ok) break;

      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh.item_empty[k % C::NITEM]));
      have = open_item(k + 1);
      // epilogue of this item: warpgroup g stores EC columns of dQ from column g * EC
      if (na > 0) {
        ok = mbar_wait<true>(smem_u32(&sh.acc_full), n_acc++ & 1, &sh.abortf, W_Q_ACCFULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      tc_fence_after_sync();
      constexpr int EC = HD / (2 * C::NSUB);
      constexpr int ECH = EC < 32 ? EC : 32;   // columns per TMEM load
      uint16_t* drow = reinterpret_cast<uint16_t*>(a.dq) + (size_t)b * a.dq_sb + (size_t)h * a.dq_sh + (size_t)qi * a.dq_st + g * EC;
      uint32_t r[EC / ECH][ECH];
      if (na > 0) {
#pragma unroll
        for (int cb = 0; cb < EC / ECH; ++cb) {
          if constexpr (ECH == 16) tmem_ld16(tbase + lane_base + C::TM_ACC0 + g * EC + cb * ECH, r[cb]);
          else tmem_ld32(tbase + lane_base + C::TM_ACC0 + g * EC + cb * ECH, r[cb]);
        }
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sh.acc_free));   // the next item's first product may overwrite the accumulator
      } else {
#pragma unroll
        for (int cb = 0; cb < EC / ECH; ++cb)
#pragma unroll
          for (int j = 0; j < ECH; ++j) r[cb][j] = 0u;
      }
      if (qi < a.T) {
#pragma unroll
        for (int cb = 0; cb < EC / ECH; ++cb) {
          const int col = g * EC + cb * ECH;
          if constexpr (kF32) {
            float* wide = static_cast<float*>(a.dq) + (size_t)b * a.dq_sb + (size_t)h * a.dq_sh + (size_t)qi * a.dq_st + col;
            if constexpr (ECH == 16) store_row16_f32_upto(wide, r[cb], a.sm_scale, col, a.d_real);
            else store_row32_f32_upto(wide, r[cb], a.sm_scale, col, a.d_real);
          } else if constexpr (ECH == 16) {
            store_row16_upto<kBf16>(drow + cb * ECH, r[cb], a.sm_scale, col, a.d_real);
          } else {
            store_row32_upto<kBf16>(drow + cb * ECH, r[cb], a.sm_scale, col, a.d_real);
          }
        }
      }
    }  // items
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tbase, 512);
  if (tid == 0) report_abort(&sh.abortf, a.status);
}

template <int HD, bool kBf16, bool kF32>
static int launch_bwd_t(const kd_attn_params& p, const kd_attn_f32* f32, const float* signs, const kd_plan_layout& L, const PlanView& pv, cudaStream_t stream) {
  using C = BwdCfg<HD>;
  CUtensorMap tmQ, tmK, tmV, tmDO;
  int rc;
  if ((rc = encode_tensor_map(&tmQ, p.q, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "q")) != 0) return rc;
  if ((rc = encode_tensor_map(&tmK, p.k, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "k")) != 0) return rc;
  if ((rc = encode_tensor_map(&tmV, p.v, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "v")) != 0) return rc;
  if ((rc = encode_tensor_map(&tmDO, p.d_o, p.B, p.H, p.T, p.D, p.dtype, KD_TILE, "do")) != 0) return rc;
  BwdArgs a;
  a.B = p.B; a.H = p.H; a.T = p.T; a.NT = L.NT; a.NP = L.NP; a.Tpad = L.NT * KD_TILE;
  a.d_real = p.D;
  a.scale_log2 = scale_log2_of(p.sm_scale);
  a.sm_scale = p.sm_scale;
  a.words = pv.words; a.len = pv.len; a.fwd_cnt = pv.fwd_cnt; a.fwd_list = pv.fwd_list;
  a.bwd_cnt = pv.bwd_cnt; a.bwd_list = pv.bwd_list; a.status = pv.status; a.order = pv.order;
  a.desc = pv.desc; a.tilebits = pv.tilebits;
  a.o = p.o.ptr; a.o_sb = p.o.stride_b; a.o_sh = p.o.stride_h; a.o_st = p.o.stride_t;
  a.d_o = p.d_o.ptr; a.do_sb = p.d_o.stride_b; a.do_sh = p.d_o.stride_h; a.do_st = p.d_o.stride_t;
  a.lse = p.lse; a.delta = p.delta;
  // with the delta kernel ahead of them in this call, the plan was complete before the kernels may start
  a.plan_ready = ((p.bwd_phases & 3) == 0 || (p.bwd_phases & 1)) ? 1 : 0;
  a.len_ready = p.plan_ready;
  a.signs = signs;
#ifdef KD_TEST_DROP_LOAD
  const char* drop = getenv("KD_TEST_DROP_LOAD");
  a.test_drop = drop != nullptr ? atoi(drop) : 0;
#endif
  a.after_dq = 0;
  const bool fused = (p.bwd_mode == KD_BWD_FUSED);
  a.grads_f32 = f32 != nullptr;
  a.zero_dq = f32 != nullptr && fused;
  a.dq_acc = fused && !f32 ? p.dq_acc : nullptr;
  const kd_tensor &dq = f32 ? f32->dq : p.dq, &dk = f32 ? f32->dk : p.dk, &dv = f32 ? f32->dv : p.dv;
  a.dq = dq.ptr; a.dq_sb = dq.stride_b; a.dq_sh = dq.stride_h; a.dq_st = dq.stride_t;
  a.dk = dk.ptr; a.dk_sb = dk.stride_b; a.dk_sh = dk.stride_h; a.dk_st = dk.stride_t;
  a.dv = dv.ptr; a.dv_sb = dv.stride_b; a.dv_sh = dv.stride_h; a.dv_st = dv.stride_t;
  a.d_o32 = f32 ? static_cast<const float*>(f32->d_o.ptr) : nullptr;
  if (f32) { a.do32_sb = f32->d_o.stride_b; a.do32_sh = f32->d_o.stride_h; a.do32_st = f32->d_o.stride_t; }
 
  auto kq = pv.words != nullptr ? attn_bwd_dq_kernel<HD, kBf16, kF32, true> : attn_bwd_dq_kernel<HD, kBf16, kF32, false>;
  static SmemOptIn opt_in[2];
  cudaError_t e = opt_in[pv.words != nullptr](kq, C::SMEM_ALLOC);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "bwd smem attribute: %s", cudaGetErrorString(e));
  const long long n_items = fused ? 0 : (long long)p.B * p.H * L.NT;
  if (n_items > 0x7FFFFFFF) return set_error(KD_ERR_LIMIT, "B * H * ceil(T / 128) exceeds 2^31 - 1");
  const unsigned grid = static_cast<unsigned>(n_items);
  a.order_of = ItemOrder::make(p.B * p.H, L.NT, (double)p.T * p.D * 2 * 5, 64e6);   // Q, K, V, dO and a gradient (32 and 128 MB: within 1 %; no chunks: up to 6 % slower)
  const int phases = (p.bwd_phases & 3) ? (p.bwd_phases & 3) : 3;
  if (phases & 1) {
    e = launch(attn_bwd_delta_kernel<HD, kBf16, kF32>, RowBlocks<HD>::grid(p.B, p.H, p.T), 256, 0, stream, a);
    if (!fused && e == cudaSuccess) e = launch(kq, grid, C::THREADS, C::SMEM_ALLOC, stream, tmQ, tmK, tmV, tmDO, a);
  }
  if (fused && e == cudaSuccess) {
    // bwd_phases 1: the delta kernel alone (it also zeroes dq_acc); 2: the fused kernel and the conversion
    if (phases & 2) return launch_bwd_fused(tmQ, tmK, tmV, tmDO, a, p.dtype, (phases & 1) != 0, stream);
  } else if ((phases & 2) && e == cudaSuccess) {
    a.after_dq = phases & 1;
    return launch_bwd_dkdv(tmQ, tmK, tmV, tmDO, a, p.dtype, stream);
  }
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "attn_bwd kernels launch: %s", cudaGetErrorString(e));
  return 0;
}

// ---------------------------------------------------------------------------------------
// Library-owned scratch for kd_attn_bwd_static.
//
// Some hosts may not allocate device memory on the path that calls the backward: an inference or
// training engine that hands every byte of HBM to its own arena at start-up and forbids plugin
// code to call cudaMalloc afterwards, or a caller that is already inside a region where the
// allocator must not run. For them the `delta` scratch of the backward (one float per
// (batch, head, token) row) lives in this fixed array instead of in a caller-supplied buffer.
// Every GPU that loads the library holds the array (4 MiB) until the process exits.
//
// In host code the name of a __device__ array is only a handle; the device address a kernel can
// use is obtained with cudaGetSymbolAddress, once per device, with that device current.
// ---------------------------------------------------------------------------------------
constexpr size_t KD_STATIC_DELTA_ROWS = size_t(1) << 20;   // B*H*T may not exceed this
static __device__ __align__(256) float g_static_delta[KD_STATIC_DELTA_ROWS];

constexpr int KD_MAX_DEVICES = 64;
static float* g_static_delta_addr[KD_MAX_DEVICES] = {};
static std::mutex g_static_delta_mutex;

// Device address of the static scratch on the current device (looked up on first use per device).
int static_delta_address(size_t rows_needed, float** out) {
  if (rows_needed > KD_STATIC_DELTA_ROWS)
    return set_error(KD_ERR_LIMIT, "kd_attn_bwd_static: B*H*T = %zu rows exceed the built-in scratch of %zu rows; "
                     "use kd_attn_bwd with a caller-provided delta buffer", rows_needed, KD_STATIC_DELTA_ROWS);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error(KD_ERR_DEVICE, "cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= KD_MAX_DEVICES) return set_error(KD_ERR_LIMIT, "device ordinal %d beyond %d", dev, KD_MAX_DEVICES);
  std::lock_guard<std::mutex> lock(g_static_delta_mutex);
  if (g_static_delta_addr[dev] == nullptr) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_delta);
    if (e != cudaSuccess || ptr == nullptr)
      return set_error(KD_ERR_DEVICE, "cudaGetSymbolAddress(static delta scratch): %s", cudaGetErrorString(e));
    g_static_delta_addr[dev] = ptr;
  }
  *out = g_static_delta_addr[dev];
  return 0;
}

int launch_attn_bwd(const kd_attn_params& p, const kd_attn_f32* f32, const float* signs, cudaStream_t stream) {
  kd_plan_layout L;
  if (kd_plan_layout_get(p.B, p.T, &L) != 0) return KD_ERR_ARG;
  PlanView pv = make_plan_view(const_cast<void*>(p.plan), L);
  if (!p.d_o.ptr) return set_error(KD_ERR_ARG, "d_o is null");
  auto run = [&](auto launch_fn) { return launch_fn(p, f32, signs, L, pv, stream); };
  const bool narrow = p.D <= 64;
  if (f32) return narrow ? run(launch_bwd_t<64, false, true>) : run(launch_bwd_t<128, false, true>);
  if (p.dtype == KD_BF16) return narrow ? run(launch_bwd_t<64, true, false>) : run(launch_bwd_t<128, true, false>);
  return narrow ? run(launch_bwd_t<64, false, false>) : run(launch_bwd_t<128, false, false>);
}

}  // namespace kd
