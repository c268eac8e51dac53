// Rules by which a launch divides its work: plain arithmetic on sizes and the number of SMs, callable from host code alone.
#pragma once

namespace kd {

// Forward: pairs of query tiles are split into items of one tile each (returns 1) where SMs would have nothing to do otherwise: two tiles'
// exponentials on one SM take turns at its special-function units. `tiles`: query tiles of a head. A CTA takes an SM, so
//  * with up to half as many items as SMs two launches of a stream still run side by side, the start of one under the end of the other;
//  * beyond that a launch waits for the SMs of the one before, which short lists do not make up for: lists have at most
//    `tiles` entries, and from five tiles on the halved item is the longer part;
//  * with more items than SMs some SMs have two items to others' one: unequal lists would still gain (causal, 80 pairs of T = 1000:
//    19.0 -> 15.5 us), equal ones lose (no mask: 20.6 -> 25.6), and the lists are on the device.
// Calls of a graph, pairs -> tiles, bf16 D = 64 (us, no mask | causal | hierarchical; head dim 128 has the same signs):
//   T = 256, 36 pairs  7.3 -> 5.6 | 6.9 -> 6.0 | 5.8 -> 4.9      74 pairs  7.5 -> 9.9 | 7.0 -> 9.3 | 5.9 -> 8.4
//   T = 500, 36 pairs 11.5 -> 9.0 | 10.5 -> 8.9 | 8.0 -> 7.7     60 pairs 11.6 -> 9.6 | 10.6 -> 9.2 | 8.1 -> 10.5
//   T = 600, 60 pairs  0.87 | 0.97 | 0.94 of the time            T = 700, 60 pairs 0.75 | 0.79 | 1.05
//   T = 1000, 72 pairs 19.6 -> 16.0 | 18.7 -> 14.9 | 11.8 -> 11.0   T = 4096, 64 pairs 49.0 -> 37.9 | 48.5 -> 37.4
// A call by itself gains in all of them or is level.
inline int split_pairs(long long pairs, int tiles, int sms) { return tiles > 1 && (4 * pairs <= sms || (tiles >= 5 && 2 * pairs <= sms)) ? 1 : 0; }

}  // namespace kd
