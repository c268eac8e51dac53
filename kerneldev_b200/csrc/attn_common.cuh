// Device helpers shared by the forward and backward attention kernels: pre-split shared-memory
// descriptors (so the single MMA-issuing thread spends two integer adds per MMA, not a 64-bit
// descriptor build), work-list staging, 16-bit row stores.
#pragma once
#include <algorithm>
#include <atomic>
#include <cfloat>

#include "common.cuh"
#include "launch_rules.cuh"
#include "mask_rule.cuh"
#include "sm100_prims.cuh"

// Registers of the light warps (producer, MMA issuers) of the two-kernel backward.
#ifndef KD_REGS_ISSUE
#define KD_REGS_ISSUE 56
#endif
// The backward kernels run sixteen compute warps (640 threads, 96 registers each at launch):
// 4*32*(96 - ISSUE) released registers cover 16*32*(COMPUTE_BWD - 96).
#ifndef KD_REGS_COMPUTE_BWD
#define KD_REGS_COMPUTE_BWD 104
#endif

namespace kd {

// The factor of the scores in base 2. The kernels flush numbers below FLT_MIN to zero, and a factor of zero makes NaN of a hidden
// score and of a row maximum without keys (-inf both); raised to FLT_MIN it leaves every exponential at 1, as the smaller one would.
inline float scale_log2_of(float sm_scale) { return std::max(sm_scale * 1.4426950408889634f, FLT_MIN); }

// What a plan's words hold of a PARTIAL tile, for plans without them. KeyRun: of 32 W keys of key tile kt from word w0 on, what words are formed from
// (w0 is a multiple of W). words(): those of the query rows of a warp, of which this lane has row qi. desc, tilebits: the sequence's.
template <int W>
struct KeyRun {
  uint32_t kd[W], pre[W], ctx[W], ins[W];
  int j0;
  __device__ __forceinline__ KeyRun(const uint32_t* desc, const uint32_t* tilebits, int kt, int w0, int lane) : j0(kt * KD_TILE + w0 * 32) {
    const uint32_t* tb = tilebits + kt * 32 + w0;
#pragma unroll
    for (int w = 0; w < W; ++w) kd[w] = __ldcg(desc + j0 + w * 32 + lane);
    load(pre, tb + 4 * TB_PRE);
    load(ctx, tb + 4 * TB_CTX);
    load(ins, tb + 4 * TB_INS);
  }
  static __device__ __forceinline__ void load(uint32_t (&m)[W], const uint32_t* src) {
    if constexpr (W == 4) {
      const uint4 x = __ldcg(reinterpret_cast<const uint4*>(src));
      m[0] = x.x; m[1] = x.y; m[2] = x.z; m[3] = x.w;
    } else if constexpr (W == 2) {
      const uint2 x = __ldcg(reinterpret_cast<const uint2*>(src));
      m[0] = x.x; m[1] = x.y;
    } else {
      static_assert(W == 1, "1, 2 or 4 words");
      m[0] = __ldcg(src);
    }
  }
  __device__ __forceinline__ void words(uint32_t qd, int qi, uint32_t* m) const {
    query_row_mask<W>(qd, qi, j0, pre, ctx, ins, m);
    uint32_t any = 0u;
#pragma unroll
    for (int w = 0; w < W; ++w) any |= ins[w];
    add_same_span<W>(qd, any != 0u, kd, m);
  }
};
template <int W>
__device__ __forceinline__ void form_words(const uint32_t* desc, const uint32_t* tilebits, int qi, int kt, int w0, int lane, uint32_t* m) {
  const uint32_t qd = __ldcg(desc + qi);
  KeyRun<W>(desc, tilebits, kt, w0, lane).words(qd, qi, m);
}

// High words of the two descriptor kinds used here (layout, version, stride byte offset 1024);
// the low word carries the start address and the leading byte offset.
__device__ __forceinline__ uint32_t desc_hi_sw128() {
  return static_cast<uint32_t>(make_smem_desc(0, 0, 1024, KD_LAYOUT_SW128) >> 32);
}
// low word of a K-major tile descriptor at k-step 0 (leading byte offset field = 1)
__device__ __forceinline__ uint32_t desc_lo_kmajor(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }
// low word of an MN-major tile descriptor whose 64-wide MN blocks are 16 KB apart
__device__ __forceinline__ uint32_t desc_lo_mnmajor(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1024u << 16); }
// offset (in 16-byte units) of k-step kk inside a K-major tile built from [rows][64] blocks 16 KB apart
__device__ __forceinline__ constexpr uint32_t koff_kmajor(int kk) { return static_cast<uint32_t>((kk / 4) * 1024 + (kk % 4) * 2); }
// offset (16-byte units) of k-step kk (16 rows of 128 bytes) inside an MN-major tile
__device__ __forceinline__ constexpr uint32_t koff_mnmajor(int kk) { return static_cast<uint32_t>(kk * 128); }

__device__ __forceinline__ void mma_ss_split(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t hi,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "mov.b64 da, {%1, %3};\n"
      "mov.b64 db, {%2, %3};\n"
      "setp.ne.b32 p, %5, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n"
      "}\n"
      ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// MMA forms whose shared-memory descriptors are complete 64-bit values. The issuing thread forms
// them BEFORE it waits for the barriers of a unit, so that once the barriers have fired the MMAs go
// out back to back with no address arithmetic between them: that thread shares its scheduler with
// busy compute warps, and every dependent instruction in its path costs it 10-20 cycles.
__device__ __forceinline__ uint64_t desc64(uint32_t lo, uint32_t hi) { return (static_cast<uint64_t>(hi) << 32) | lo; }
// maximum of three floats in one instruction (sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <bool kAccumulate>
__device__ __forceinline__ void mma_ss64(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
template <bool kAccumulate>
__device__ __forceinline__ void mma_ts64(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
// accumulate flag known only at run time (first product into an accumulator)
__device__ __forceinline__ void mma_ts64_p(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_ts_split(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t hi,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 db;\n"
      "mov.b64 db, {%2, %3};\n"
      "setp.ne.b32 p, %5, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// MMA forms for a warp whose control flow is uniform: every lane calls them with warp-uniform operands and one elected
// lane issues. The operands then live in uniform registers, where the instruction wants them; issued from inside a
// "lane 0 only" branch each MMA first moves five values there. Measured on an idle SM: 22 cycles per issued MMA against
// 54 (and 75-90 beside busy compute warps), i.e. less than the 32-64 cycles the tensor pipe needs for it.
__device__ __forceinline__ void mma_ss_uniform(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  if (elect_one()) mma_ss_split(d_tmem, alo, blo, hi, idesc, accumulate);
}
__device__ __forceinline__ void mma_ts_uniform(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  if (elect_one()) mma_ts_split(d_tmem, a_tmem, blo, hi, idesc, accumulate);
}
__device__ __forceinline__ void commit_uniform(uint32_t bar) {
  if (elect_one()) mma_commit(bar);
}

// stores 32 fp32 accumulator values (scaled) as 16-bit elements to a row in global memory
template <bool kBf16>
__device__ __forceinline__ void store_row32(uint16_t* dst, const uint32_t (&r)[32], float f) {
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    uint4 v;
    v.x = pack2<kBf16>(__uint_as_float(r[j + 0]) * f, __uint_as_float(r[j + 1]) * f);
    v.y = pack2<kBf16>(__uint_as_float(r[j + 2]) * f, __uint_as_float(r[j + 3]) * f);
    v.z = pack2<kBf16>(__uint_as_float(r[j + 4]) * f, __uint_as_float(r[j + 5]) * f);
    v.w = pack2<kBf16>(__uint_as_float(r[j + 6]) * f, __uint_as_float(r[j + 7]) * f);
    *reinterpret_cast<uint4*>(dst + j) = v;
  }
}

template <bool kBf16>
__device__ __forceinline__ void store_row16(uint16_t* dst, const uint32_t (&r)[16], float f) {
#pragma unroll
  for (int j = 0; j < 16; j += 8) {
    uint4 v;
    v.x = pack2<kBf16>(__uint_as_float(r[j + 0]) * f, __uint_as_float(r[j + 1]) * f);
    v.y = pack2<kBf16>(__uint_as_float(r[j + 2]) * f, __uint_as_float(r[j + 3]) * f);
    v.z = pack2<kBf16>(__uint_as_float(r[j + 4]) * f, __uint_as_float(r[j + 5]) * f);
    v.w = pack2<kBf16>(__uint_as_float(r[j + 6]) * f, __uint_as_float(r[j + 7]) * f);
    *reinterpret_cast<uint4*>(dst + j) = v;
  }
}

// 32 (or 16) accumulator columns starting at column `col` of a row whose real width is d_real (a multiple
// of 16): the columns at or beyond d_real belong to the zero-filled part of a tile and are not stored.
template <bool kBf16>
__device__ __forceinline__ void store_row32_upto(uint16_t* dst, const uint32_t (&r)[32], float f, int col, int d_real) {
  if (col + 32 <= d_real) {
    store_row32<kBf16>(dst, r, f);
  } else if (col < d_real) {   // 16 columns left
#pragma unroll
    for (int j = 0; j < 16; j += 8) {
      uint4 v;
      v.x = pack2<kBf16>(__uint_as_float(r[j + 0]) * f, __uint_as_float(r[j + 1]) * f);
      v.y = pack2<kBf16>(__uint_as_float(r[j + 2]) * f, __uint_as_float(r[j + 3]) * f);
      v.z = pack2<kBf16>(__uint_as_float(r[j + 4]) * f, __uint_as_float(r[j + 5]) * f);
      v.w = pack2<kBf16>(__uint_as_float(r[j + 6]) * f, __uint_as_float(r[j + 7]) * f);
      *reinterpret_cast<uint4*>(dst + j) = v;
    }
  }
}
// The same columns of a float32 row. (Four lanes' 16-byte stores fill a line between them in L2.)
__device__ __forceinline__ void store_row32_f32_upto(float* dst, const uint32_t (&r)[32], float f, int col, int d_real) {
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    if (col + j < d_real)   // 16 columns at a time, as d_real
      *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(r[j]) * f, __uint_as_float(r[j + 1]) * f, __uint_as_float(r[j + 2]) * f, __uint_as_float(r[j + 3]) * f);
}
__device__ __forceinline__ void store_row16_f32_upto(float* dst, const uint32_t (&r)[16], float f, int col, int d_real) {
  if (col >= d_real) return;
#pragma unroll
  for (int j = 0; j < 16; j += 4)
    *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(r[j]) * f, __uint_as_float(r[j + 1]) * f, __uint_as_float(r[j + 2]) * f, __uint_as_float(r[j + 3]) * f);
}
template <bool kBf16>
__device__ __forceinline__ void store_row16_upto(uint16_t* dst, const uint32_t (&r)[16], float f, int col, int d_real) {
  if (col < d_real) store_row16<kBf16>(dst, r, f);
}

// SMs of the device that was current at the first call (the devices of a machine are alike: the library runs on sm_100 alone).
inline int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? v : 148;
  }();
  return n;
}

// Order of a launch's items (tiles of one (batch, head) pair): chunks of heads whose tensors share L2, inside a chunk rank by
// rank (longest lists first) and for a rank head by head. The chunks differ by one head at most: each begins with its longest
// items, and a small last one gets them when the SMs run out of work (hier 8 x 16 x 2048 x 64: backward 207 us, 198 with even
// chunks).
struct ItemOrder {
  int heads, big;   // (batch, head) pairs of a chunk; the first `big` chunks have one more
  __device__ __forceinline__ void decode(int idx, int per_head, int& bh, int& rank) const {
    const int in_big = big * (heads + 1) * per_head;
    const bool second = idx >= in_big;
    const int n = second ? heads : heads + 1, rest = second ? idx - in_big : idx;
    const int c = rest / (n * per_head), r = rest - c * n * per_head;
    rank = r / n;
    bh = (second ? big * (heads + 1) : 0) + c * n + (r - rank * n);
  }
  // As many (batch, head) pairs to a chunk as take l2_bytes, and enough of them that it holds two items per SM of 148. The number of
  // chunks is rounded down, so that a chunk takes up to twice as much.
  static ItemOrder make(int pairs, int per_head, double pair_bytes, double l2_bytes) {
    long long chunk = static_cast<long long>(std::min<double>(pairs, std::max(1.0, l2_bytes / pair_bytes)));
    chunk = std::min<long long>(pairs, std::max<long long>(chunk, (296 + per_head - 1) / per_head));
    const int n = static_cast<int>(pairs / chunk);
    ItemOrder o;
    o.heads = pairs / n;
    o.big = pairs % n;
    return o;
  }
};

// Raises a kernel's dynamic shared-memory limit, once per device (one instance per kernel): the attribute call
// costs about a microsecond of host time, which a small launch would pay every time.
struct SmemOptIn {
  std::atomic<uint64_t> done{0};   // bit d: set on device d
  template <typename Kernel>
  cudaError_t operator()(Kernel kern, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

// used while unwinding after an abort: lets a TMA copy that is already in flight land, with the limit of the other waits (a number of tests is
// no limit in time, for the hardware may suspend each of them)
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity) { mbar_wait_short(bar, parity); }

}  // namespace kd
