// Rules of the forward kernels that are plain index arithmetic, callable from host code as well.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define KD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define KD_HOST_DEVICE inline
#endif

namespace kd {

// The ring of Q tiles: loads are numbered over all items of a CTA, and load q lies in slot q % kSlots. A "full" barrier is waited for
// by parity, which is sound only for a warp that has seen every earlier phase of that barrier: to a warp that has missed one, the
// phase before the missed one looks like the awaited one, and it reads a tile that has not landed. A single issuing warp waits for
// every load, so one barrier per slot serves it. With an issuing warp per query tile, each waits for its own tiles only, and a slot
// changes hands between the two (with three slots, item k's tile 1 lies where tile 0 of item k - 1 was): then each slot has a
// barrier per query tile, all of whose phases belong to one warp. A barrier is armed again only when its slot has been
// released, that is by a warp that had waited for the load before.
template <int kSlots, int kWarps>
struct QRing {
  static_assert(kWarps == 1 || kWarps == 2, "issuing warps");
  static constexpr int SLOTS = kSlots, FULL = kSlots * kWarps;   // "full" barriers; "empty" ones: one per slot, which the producer alone waits for
  static KD_HOST_DEVICE int slot(int load) { return load % kSlots; }
  static KD_HOST_DEVICE int full(int load, int tile) { return slot(load) * kWarps + (kWarps == 2 ? tile : 0); }
  static KD_HOST_DEVICE uint32_t empty_parity(int load) { return static_cast<uint32_t>((load / kSlots) & 1) ^ 1u; }
};

// parities of a set of barriers, for a role that goes through all of their phases
struct PhaseBits {
  uint32_t next = 0u;   // bit j: parity of barrier j's next phase
  KD_HOST_DEVICE uint32_t take(int j) {
    const uint32_t p = (next >> j) & 1u;
    next ^= 1u << j;
    return p;
  }
  KD_HOST_DEVICE uint32_t last(int j) const { return ((next >> j) & 1u) ^ 1u; }   // of the phase taken last
};

using FwdWideQRing = QRing<3, 2>;   // head dims above 64 (shared memory has room for three tiles)
using FwdQRing = QRing<4, 1>;       // head dims up to 64

}  // namespace kd
