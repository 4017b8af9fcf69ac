// Small rules that both sides read and a host test can check: how many node
// pairs of a traversal level are decided at once, and the lanes of the solve's
// waves.
#pragma once
#include <algorithm>
#include <cstdint>

#include "d2g_math.cuh"

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

// The solve's normal loop on a block with n_tasks tasks (of four contacts) in
// `levels` waves: sixteen lanes a contact in the waves where it has one task, or
// eight (four a body side) throughout.  lanes: D2G_TUNE_SOLVE_LANES, 16 or 4
// for the one or the other, 0 for sixteen while a wave has hardly more than one
// task here: a single task's chain is then the interval's length (8 cubes: 61
// -> 60 us per iteration, 100 cubes on 16 blocks 164 -> 140).  With more tasks
// the loads ahead and the dealing of waves cost more than the few narrow waves
// give (27 cubes, 1.5 tasks a wave: 123 -> 129).
D2G_HD bool narrow_waves(int lanes, int n_tasks, int levels) {
    return lanes ? lanes == 16 : 4LL * n_tasks <= 5LL * levels;
}

}  // namespace d2g
