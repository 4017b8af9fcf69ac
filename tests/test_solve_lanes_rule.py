"""The solve's rule for the lanes of its normal-impulse waves: the setting
forces either form whatever the waves' widths, and 0 leaves it to them (at most
five tasks of four contacts to four waves).  The harness compiles the library's
header for the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "delta2_gb300", "csrc")

HARNESS = r"""
#include "d2g_limits.hpp"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
    std::printf("%d\n", d2g::narrow_waves(atoi(argv[1]), atoi(argv[2]), atoi(argv[3])) ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def narrow(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("lanes")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", CSRC, "-o", str(d / "h"), str(d / "h.cpp")], check=True)
    return lambda *a: int(subprocess.run([str(d / "h")] + [str(x) for x in a], capture_output=True, text=True).stdout)


@pytest.mark.parametrize("tasks, levels, by_width", [
    (0, 1, 1), (1, 1, 1), (5, 4, 1), (6, 4, 0), (46, 46, 1), (135, 89, 0), (10 ** 9, 10 ** 9, 1), (2 * 10 ** 9, 1, 0)])
def test_setting_forces_the_form(narrow, tasks, levels, by_width):
    assert narrow(0, tasks, levels) == by_width
    assert narrow(16, tasks, levels) == 1
    assert narrow(4, tasks, levels) == 0
