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

// A list entry: key tile | class for query tile 0 << 8 | class for query tile 1 << 10 (class 0: EMPTY).
KD_HOST_DEVICE uint32_t entry_class(uint32_t ent, int i) { return (ent >> (8 + 2 * i)) & 3u; }
// What is left of an entry in an item of query tile i alone: 0 where that tile does not need it.
KD_HOST_DEVICE uint32_t entry_of_tile(uint32_t ent, int i) { return entry_class(ent, i) != 0u ? ent & (i == 0 ? 0x3FFu : 0xCFFu) : 0u; }

// Head dims above 64: do the two tiles of a CTA's first item, of n entries with `first` ahead, begin half a unit apart? With lists of
// one or two entries they would compute their exponentials at the same time, with the special-function units idle before and after.
// Where only one tile begins with the entry there is nothing to take turns with, and the half unit would be lost (20 calls in a graph, items of
// one tile, us a call: causal 1 x 16 x 173 x 128 7.4 -> 6.9, no mask 1 x 16 x 256 x 128 7.6 -> 7.1, hierarchical 2 x 16 x 256 x 96 6.3 -> 5.9).
KD_HOST_DEVICE bool tiles_take_turns(uint32_t first, int n) { return n <= 2 && entry_class(first, 0) != 0u && entry_class(first, 1) != 0u; }

using FwdWideQRing = QRing<3, 2>;   // head dims above 64 (shared memory has room for three tiles)
using FwdQRing = QRing<4, 1>;       // head dims up to 64

}  // namespace kd
