"""The FP32 bound that leaves an edge-edge CCD test out (the gap along the
direction between the closest points at the start, at both ends of the motion)
against FP64 distances over the motion: an edge pair it leaves out never comes
within the limit, also where the direction's squared length underflows (edges
closer than 1e-20 m).  The harness compiles the library's header for the
host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "delta2_gb300", "csrc")

HARNESS = r"""
#include "d2g_prune.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace d2g;
static std::mt19937 g(1);
static float U(float a, float b) { return a + (b - a) * std::uniform_real_distribution<float>(0, 1)(g); }
static V3 d3(F3 a) { return mk(a.x, a.y, a.z); }
int main(int argc, char** argv) {
    const int kind = atoi(argv[1]);
    long out = 0, under = 0, bad = 0;
    for (long it = 0; it < 200000; it++) {
        const float s = kind == 0 ? U(.05f, 1) : (kind == 1 ? powf(10, U(-24, -18)) : powf(10, U(-16, -6)));
        const float q = kind == 0 ? U(0, 1) : s * powf(10, U(-8, 0)), lim = 0.02f;
        F3 p[2][4];
        for (int k = 0; k < 4; k++) p[0][k] = f3(U(-s, s), U(-s, s), U(-s, s));
        p[0][2] = f3(p[0][0].x + U(-q, q), p[0][0].y + U(-q, q), p[0][0].z + U(-q, q));
        const float m = it & 1 ? .2f : 0;
        const F3 v = f3(U(-m, m), U(-m, m), U(-m, m));
        for (int k = 0; k < 4; k++)
            p[1][k] = k < 2 ? p[0][k] : f3(p[0][k].x + v.x, p[0][k].y + v.y, p[0][k].z + v.z);
        float d2;
        const F3 d = seg_vector(p[0][0], p[0][1], p[0][2], p[0][3], d2);
        under += d2 == 0.f && fminf(dot3(d, p[0][2]), dot3(d, p[0][3])) > fmaxf(dot3(d, p[0][0]), dot3(d, p[0][1]));
        if (!edges_stay_apart(p, lim)) continue;
        out++;
        for (int k = 0; k <= 16; k++) {
            const double t = k / 16.0;
            V3 P, Q;
            V3 x[4];
            for (int j = 0; j < 4; j++) x[j] = lerp(d3(p[0][j]), d3(p[1][j]), t);
            if (edge_closest(x[0], x[1], x[2], x[3], P, Q) < lim - 1e-6) {
                bad++;
                break;
            }
        }
    }
    std::printf("left out %ld underflows %ld wrong %ld\n", out, under, bad);
    return bad != 0 || (kind == 0 && out < 1000) || (kind == 1 && under < 100);
}
"""


@pytest.mark.parametrize("kind", range(3), ids=["ordinary", "underflow", "tiny"])
def test_left_out_edge_pairs_stay_apart(tmp_path, kind):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "h"),
                    str(tmp_path / "h.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "h"), str(kind)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
