// Host-side checks of the kernels' rules (fwd_rules.cuh, launch_rules.cuh). Built and run by tests/test_host_logic.py (host code only; no GPU needed).
//
// 1. A model of the Q tile hand-over in the kernel for head dims above 64 (attn_fwd.cuh, attn_fwd_wide.cu): the producer, two issuing warps that run ahead of each other, and copies that land in any order. Every product must read
// the tile it is meant for, landed, and no slot may be released or filled before that. Random schedules of random items, among
// them items whose tiles have no units, odd last tiles and lists of up to four entries. With one "full" barrier per slot, which a warp
// then does not see all phases of, the model must find the wrong product (the check of the model itself).
// 2. Entries of an item of one query tile, and which items' tiles begin half a unit apart.
// 3. Which calls have items of one query tile (launch_rules.cuh): never more items than SMs, and none beyond half of the SMs where the
//    lists are short.
// 4. Heads per CTA of the deterministic backward (launch_rules.cuh): one or two up to twelve tiles per SM, and two only where lists are short
//    or the tiles many.
#include <cstdio>
#include <cstdint>
#include <vector>
#include "../kerneldev_b200/csrc/fwd_rules.cuh"
#include "../kerneldev_b200/csrc/launch_rules.cuh"

using namespace kd;

static uint64_t rng_state = 1;
static uint32_t rnd(uint32_t n) {
  rng_state = rng_state * 6364136223846793005ull + 1442695040888963407ull;
  return static_cast<uint32_t>(rng_state >> 33) % n;
}

struct OneBarrierPerSlot {   // the mistake
  static constexpr int SLOTS = 3, FULL = 3;
  static int slot(int load) { return load % 3; }
  static int full(int load, int) { return load % 3; }
  static uint32_t empty_parity(int load) { return static_cast<uint32_t>((load / 3) & 1) ^ 1u; }
  static uint32_t wait_parity(PhaseBits&, int load, int) { return static_cast<uint32_t>((load / 3) & 1); }
};
struct AsBuilt : FwdWideQRing {
  static uint32_t wait_parity(PhaseBits& p, int load, int tile) { return p.take(full(load, tile)); }
};

struct Item { int ntile, n; bool own[2][4]; };   // query tiles, list entries, which of them are a tile's
enum Kind { WAIT, ARRIVE, LOAD, PRODUCT };
struct Op { Kind kind; int bar; uint32_t parity; int slot, tag; };
struct Bar {
  int count, pending, bytes = 0, phase = 0;
  explicit Bar(int c) : count(c), pending(c) {}
  bool settle() {
    if (pending < 0) return false;   // armed or released twice in a phase
    if (pending == 0 && bytes == 0) { ++phase; pending = count; }
    return true;
  }
};

template <typename R>
static const char* run(uint64_t seed) {   // nullptr: no fault
  rng_state = seed * 0x9E3779B97F4A7C15ull + 1;
  constexpr int KST = 2, NITEM = 2, N = 9;
  constexpr int QFULL = 0, QEMPTY = QFULL + R::FULL, KFULL = QEMPTY + R::SLOTS, KEMPTY = KFULL + KST, IFULL = KEMPTY + KST, IEMPTY = IFULL + NITEM,
                NBAR = IEMPTY + NITEM;
  std::vector<Bar> bars;
  for (int b = 0; b < NBAR; ++b) bars.emplace_back((b >= KEMPTY && b < IFULL) || b >= IEMPTY ? 2 : 1);
  std::vector<Op> prog[3];   // producer, issuers
  int q = 0, kv = 0, q_first[2] = {0, 0}, kv_first[2] = {0, 0};
  PhaseBits seen[2];
  for (int k = 0; k < N; ++k) {
    Item it;
    it.ntile = rnd(4) == 0 ? 1 : 2;
    it.n = static_cast<int>(rnd(5));
    const bool none[2] = {rnd(3) == 0, it.ntile == 1 || rnd(2) == 0};
    for (int e = 0; e < it.n; ++e) {
      for (int i = 0; i < 2; ++i) it.own[i][e] = !none[i] && rnd(3) != 0;
      if (!it.own[0][e] && !it.own[1][e]) it.own[0][e] = true;   // an entry is some tile's
    }
    const int slot = k % NITEM;
    const uint32_t item_parity = (k / NITEM) & 1;
    auto load_q = [&](int t) {
      prog[0].push_back({WAIT, QEMPTY + R::slot(q), R::empty_parity(q), 0, 0});
      prog[0].push_back({LOAD, QFULL + R::full(q, t), 0u, R::slot(q), 2 * k + t});
      ++q;
    };
    prog[0].push_back({WAIT, IEMPTY + slot, item_parity ^ 1u, 0, 0});
    prog[0].push_back({ARRIVE, IFULL + slot, 0u, 0, 0});
    load_q(0);
    for (int e = 0; e < it.n; ++e, ++kv) {
      prog[0].push_back({WAIT, KEMPTY + kv % KST, static_cast<uint32_t>((kv / KST) & 1) ^ 1u, 0, 0});
      prog[0].push_back({LOAD, KFULL + kv % KST, 0u, -1, 0});
      if (e == 0 && it.ntile == 2) load_q(1);
    }
    if (it.n == 0 && it.ntile == 2) load_q(1);
    for (int i = 0; i < 2; ++i) {
      std::vector<Op>& p = prog[1 + i];
      p.push_back({WAIT, IFULL + slot, item_parity, 0, 0});
      const int load = q_first[i] + i;
      int left = 0;
      for (int e = 0; e < it.n; ++e) left += it.own[i][e];
      if (i < it.ntile) {
        p.push_back({WAIT, QFULL + R::full(load, i), R::wait_parity(seen[i], load, i), 0, 0});
        p.push_back({PRODUCT, -1, 0u, R::slot(load), 2 * k + i});   // (also without units: the tile must be there before it is released)
        if (left == 0) p.push_back({ARRIVE, QEMPTY + R::slot(load), 0u, 0, 0});
      }
      q_first[i] += it.ntile;
      for (int e = 0; e < it.n; ++e, ++kv_first[i]) {
        p.push_back({WAIT, KFULL + kv_first[i] % KST, static_cast<uint32_t>((kv_first[i] / KST) & 1), 0, 0});
        if (it.own[i][e]) p.push_back({PRODUCT, -1, 0u, R::slot(load), 2 * k + i});
        p.push_back({ARRIVE, KEMPTY + kv_first[i] % KST, 0u, 0, 0});
        if (it.own[i][e] && --left == 0) p.push_back({ARRIVE, QEMPTY + R::slot(load), 0u, 0, 0});
      }
      p.push_back({ARRIVE, IEMPTY + slot, 0u, 0, 0});
    }
  }
  int in_slot[R::SLOTS];
  for (int& s : in_slot) s = -1;
  struct Copy { int bar, slot, tag; };
  std::vector<Copy> flying;
  size_t pc[3] = {0, 0, 0};
  const uint32_t land_weight = 1 + rnd(4), lag = rnd(3);   // how eagerly copies land, which role is held back
  for (;;) {
    int runnable[3], nr = 0;
    for (int r = 0; r < 3; ++r) {
      if (pc[r] == prog[r].size()) continue;
      const Op& op = prog[r][pc[r]];
      if (op.kind == WAIT && (static_cast<uint32_t>(bars[op.bar].phase) & 1u) == op.parity) continue;   // the phase in progress has it
      runnable[nr++] = r;
    }
    if (nr == 0 && flying.empty()) break;
    if (!flying.empty() && (nr == 0 || rnd(8) < land_weight)) {
      const int j = static_cast<int>(rnd(static_cast<uint32_t>(flying.size())));
      const Copy c = flying[j];
      flying.erase(flying.begin() + j);
      if (c.slot >= 0) in_slot[c.slot] = c.tag;
      --bars[c.bar].bytes;
      if (!bars[c.bar].settle()) return "barrier";
      continue;
    }
    int r = runnable[rnd(static_cast<uint32_t>(nr))];
    if (r == static_cast<int>(lag) && rnd(4) != 0) r = runnable[rnd(static_cast<uint32_t>(nr))];
    const Op& op = prog[r][pc[r]++];
    if (op.kind == ARRIVE) {
      --bars[op.bar].pending;
      if (!bars[op.bar].settle()) return "a barrier completed twice";
    } else if (op.kind == LOAD) {
      for (const Copy& c : flying)
        if (op.slot >= 0 && c.slot == op.slot) return "a slot is filled while a copy into it is under way";
      if (bars[op.bar].pending < 1) return "a barrier is armed twice in a phase";
      ++bars[op.bar].bytes;
      --bars[op.bar].pending;
      flying.push_back({op.bar, op.slot, op.tag});
      if (op.slot >= 0) in_slot[op.slot] = -1;
    } else if (op.kind == PRODUCT && in_slot[op.slot] != op.tag) {
      return "a product reads a tile that is not there";
    }
  }
  for (int r = 0; r < 3; ++r)
    if (pc[r] != prog[r].size()) return "nothing can go on";
  return nullptr;
}

static int list_rules() {   // mistakes
  int bad = 0;
  for (uint32_t kt = 0; kt < 128; ++kt)
    for (uint32_t c0 = 0; c0 < 3; ++c0)
      for (uint32_t c1 = 0; c1 < 3; ++c1) {
        const uint32_t ent = kt | (c0 << 8) | (c1 << 10), cls[2] = {c0, c1};
        for (int i = 0; i < 2; ++i) {
          const uint32_t one = entry_of_tile(ent, i);
          bad += cls[i] == 0u ? one != 0u : (one & 0xFFu) != kt || entry_class(one, i) != cls[i] || entry_class(one, 1 - i) != 0u;
          for (int n = 1; n <= 3; ++n) bad += tiles_take_turns(one, n);   // alone on its SM
        }
        for (int n = 1; n <= 3; ++n) bad += tiles_take_turns(ent, n) != (n <= 2 && c0 != 0u && c1 != 0u);
      }
  return bad;
}

static int split_rule() {   // mistakes
  int bad = 0;
  for (long long pairs = 1; pairs <= 400; ++pairs)
    for (int tiles = 1; tiles <= 128; ++tiles) {
      const long long items = 2 * pairs;
      const int split = split_pairs(pairs, tiles, 148);
      bad += split && (tiles == 1 || items > 148 || (tiles < 5 && items > 74));
      bad += !split && tiles > 1 && items <= (tiles < 5 ? 74 : 148);
    }
  return bad + split_pairs(1LL << 40, 128, 148);
}

int main() {
  int bad = list_rules() + split_rule(), found = 0;
  for (uint64_t seed = 1; seed <= 20000; ++seed) {
    const char* e = run<AsBuilt>(seed);
    if (e != nullptr && bad++ == 0) printf("seed %llu: %s\n", static_cast<unsigned long long>(seed), e);
    found += run<OneBarrierPerSlot>(seed) != nullptr;
  }
  printf("bad=%d, with one barrier per slot %d\n", bad, found);
  return bad == 0 && found > 0 ? 0 : 1;
}
