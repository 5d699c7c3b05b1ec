// Splitters of the flattening's tour (ptl_flatten.cu): the rule, and how far a walk goes.
#pragma once

#include "ptl_common.cuh"

namespace ptl {

// Events of the tour are enter(v) = 2v and exit(v) = 2v + 1.  One in 2^lg of each is a
// splitter, never both of one node, spread evenly over any run of consecutive node numbers
// (multiplicative hashing by the golden ratio: two events in a row are 0.62 apart).  Exits
// are among them so that a deep tree, which closes with a run of exits as long as it is
// deep, is cut too: with enters only, a path of 100,000 nodes was one walk of as many events
// (21.7 ms against 0.34 by pointer jumping over all events).
PTL_HD bool is_splitter(uint32_t event, uint32_t lg) { return ((event * 0x9E3779B1u) >> (32u - lg)) == 0; }
// A splitter per 32 events of a large tree, per 16 of a small one (whose walks are over
// sooner than the jumps between more splitters cost).
PTL_HD uint32_t splitter_lg(uint32_t n) { return n >= (1u << 20) ? 5u : 4u; }
PTL_HD uint32_t splitters_most(uint32_t n) {  // the hash's share, a quarter more, and the root's
    const uint32_t lg = splitter_lg(n);
    return (n >> (lg - 1u)) + (n >> (lg + 1u)) + 64u;
}
// Events of a walk before pointer jumping over all events takes over.  Node numbers that
// have nothing to do with the hash make one walk in 10^14 this long; a caller may number
// the nodes in any order, though, one that keeps the hash's nodes apart from the others
// among them.
PTL_HD uint32_t walk_most(uint32_t lg) { return 32u << lg; }

}  // namespace ptl
