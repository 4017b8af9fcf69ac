// How many node pairs of a traversal level one slot list can number, and how
// many are decided at once.
#pragma once
#include <algorithm>
#include <cstdint>

namespace d2g {

// A level's slot list names slot s of node pair w as 64 w + s; bit 30 marks an
// entry (k_ccd_level: all its edge-edge tests are clear; k_np_filter: only the
// whole distance decides it).  So one list numbers 2^24 node pairs.
constexpr int32_t kSlotMark = 1 << 30;
constexpr int32_t kMaxListPairs = kSlotMark / 64;

// Node pairs of a level of n decided at once.  A level that may give up its
// chunk does so before it passes the budget or a list's numbers; the level of a
// single body pair runs in ranges of this many: its list (256 bytes a node
// pair, x1.5 growth slack) within the budget, as far as 256 node pairs go.
constexpr int32_t kMinRangePairs = 256;
inline int32_t level_range(int32_t n, double budget) {
    const double fit = std::max((double)kMinRangePairs, budget / (1.5 * 256.0));
    return (int32_t)std::min({(double)n, (double)kMaxListPairs, fit});
}

}  // namespace d2g
