"""A traversal level of a single body pair larger than one slot list numbers,
or than its budget, is decided in ranges of node pairs.  On the CPU: the ranges
cover a level, and every slot number of a range decodes to its node pair and
slot beside the mark bit, at the sizes where 32-bit numbers would not.  On the
GPU: with the smallest budget every body pair runs alone and its wide levels in
ranges, with the results of whole levels."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "delta2_gb300", "csrc")

HARNESS = r"""
#include "d2g_limits.hpp"
#include <cstdio>
using namespace d2g;
int main() {
    const int sizes[] = {1, 255, 256, 257, 1000, (1 << 24) - 1, 1 << 24, (1 << 24) + 1, 3 << 23, 1 << 25, (1 << 25) + 1,
                         1 << 28};
    const double budgets[] = {1.0, 98304.0, 98688.0, 1e6, 5e10, 1e30};
    for (int n : sizes)
        for (double budget : budgets) {
            const int range = level_range(n, budget);
            if (range < 1 || range > n) return std::printf("range %d of %d\n", range, n), 1;
            if (range < n && range > kMinRangePairs && 64.0 * 4 * 1.5 * range > budget)
                return std::printf("range %d past the budget %g\n", range, budget), 1;
            if (range < n && range < kMinRangePairs) return std::printf("range %d\n", range), 1;
            long long covered = 0;
            for (int r0 = 0; r0 < n; r0 += range) covered += std::min(range, n - r0);
            if (covered != n) return std::printf("%lld of %d\n", covered, n), 1;
            for (int w : {0, range / 2, range - 1})  // as the kernels number and decode them
                for (int slot : {0, 31, 63})
                    for (int mark : {0, (int)kSlotMark}) {
                        const long long exact = 64LL * w + slot;
                        const int item = (int)exact | mark, id = item & ~kSlotMark;
                        if (exact >= kSlotMark || item < 0 || id >> 6 != w || (id & 63) != slot ||
                            (item & kSlotMark) != mark)
                            return std::printf("n %d: node pair %d slot %d\n", n, w, slot), 1;
                    }
        }
    return 0;
}
"""


def test_ranges_cover_a_level_and_number_its_slots(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "h"), str(tmp_path / "h.cpp")],
                   check=True)
    out = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "witnesses", "bounds off"])
def test_levels_in_ranges_match_whole_levels(gpu_required, form):
    import delta2_gb300 as D
    from delta2_gb300 import build as B
    from oracle import oracle as O
    B.build()
    s = D.make_scene(5, nx=2, ny=1, nz=1, spacing=1.1, speed_sigma=0.5, seed=3)
    pairs = D.broad_phase(s)
    mt = np.full(len(pairs), 0.02)
    ref, ref_off = O.ccd(s.copy(), pairs, mt)[:2]
    ctx = D.Context(0)
    try:
        ctx.set_ccd_witnesses(form == "witnesses")
        ctx.set_fp32_bounds(form != "bounds off")
        out = []
        for budget in (0, 1):
            ctx.set_level_budget(budget)
            ctx.set_scene(s.copy())
            c, off, cnt = ctx.compare_trees_full_continuous(pairs, mt)
            assert np.array_equal(off, ref_off), budget
            assert np.array_equal(c.view(np.uint64), ref.view(np.uint64)), budget
            c2, off2, cnt2 = ctx.compare_trees_full(pairs)
            out.append((cnt[:3].tolist(), c2.view(np.uint64).tolist(), off2.tolist(), cnt2[:2].tolist()))
        assert cnt[0] > 1000  # node pairs: levels wider than a range of 256
        assert out[0][1:] == out[1][1:]
        if form != "witnesses":  # (the second call skips node pairs the first one witnessed)
            assert out[0][0] == out[1][0]
    finally:
        ctx.close()
