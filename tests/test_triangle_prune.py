"""The narrow phase's triangle distance with FP32 bounds (tri_tri_dist_below)
against the plain one: wherever the distance is below the limit, the same
bits of the distance and both points; elsewhere a distance that is not below
the limit.  Random triangles, and the forms that could fool a bound: parallel
faces and edges, shared vertices, slivers, needles, degenerate edges, a large
ground triangle, touching triangles; limits at the distance itself.  The
harness compiles the library's header for the host."""
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
#include <cstring>
#include <random>
using namespace d2g;
static std::mt19937_64 g(11);
static double U(double a, double b) { return a + (b - a) * std::uniform_real_distribution<double>(0, 1)(g); }
static V3 rv(double s) { return mk(U(-s, s), U(-s, s), U(-s, s)); }
static void shift(Tri& t, V3 o) { t.A = t.A + o, t.B = t.B + o, t.C = t.C + o; }
int main(int argc, char** argv) {
    const int kind = atoi(argv[1]);
    long bad = 0, below = 0;
    for (long it = 0; it < 30000; it++) {
        const double s = U(0, 1) < .3 ? U(.01, .05) : U(.1, .6);
        Tri a{rv(s), rv(s), rv(s)}, b{rv(s), rv(s), rv(s)};
        V3 off = rv(1.2 * s);
        if (kind == 1) b = a, off = mk(0, 0, U(0, .3));                             // parallel copies
        if (kind == 2) b = Tri{a.A, a.C, a.B}, off = rv(1e-3);                      // shared vertices
        if (kind == 3) a.C = a.A + (a.B - a.A) * U(0, 1) + rv(1e-4 * s);            // slivers
        if (kind == 4) a.C = a.B;                                                   // a degenerate edge
        if (kind == 5) {                                                            // axis-aligned faces
            a = Tri{mk(-.5, -.5, 0), mk(.5, -.5, 0), mk(.5, .5, 0)};
            b = Tri{mk(-.5, -.5, 0), mk(.5, .5, 0), mk(-.5, .5, 0)};
            off = mk(U(-1.2, 1.2), it & 1 ? U(-1, 1) : 0, U(0, .3));
        }
        if (kind == 6) b.B = b.A + (a.B - a.A);                                     // parallel edges
        if (kind == 7) {                                                            // a large ground triangle
            a.A = a.A * 300, a.B = a.B * 300, a.C = a.C * 300, a.A.z = a.B.z = a.C.z = 0;
            off = mk(U(-50, 50), U(-50, 50), U(0, .4));
        }
        if (kind == 8) b.A = a.A, off = mk(0, 0, 0);                                // touching
        if (kind == 9) b.B = b.A + (a.B - a.A) + rv(1e-7);                          // nearly parallel edges
        if (kind == 10) a.C = a.A + (a.B - a.A) * U(0, 1) + rv(1e-9 * s);           // needles
        const V3 w = it % 3 == 0 ? rv(1000) : (it % 3 == 1 ? rv(5) : mk(0, 0, 0));
        shift(b, off), shift(a, w), shift(b, w);
        V3 P, Q, P2, Q2;
        const double d = tri_tri_dist(a, b, P, Q);
        for (double lim : {0.25, 0.05, 1e9, d, d * (1 + 1e-15), d * (1 - 1e-15)}) {
            const double e = tri_tri_dist_below(a, b, lim, P2, Q2);
            bool ok = !(e < lim);
            if (d < lim) {
                below++;
                ok = !std::memcmp(&d, &e, 8) && !std::memcmp(&P, &P2, 24) && !std::memcmp(&Q, &Q2, 24);
            }
            if (!ok && bad++ < 5) std::printf("limit %.17g distance %.17g, bounded %.17g\n", lim, d, e);
        }
    }
    std::printf("below the limit %ld mismatches %ld\n", below, bad);
    return bad != 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("prune")
    (d / "prune.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-I", CSRC, "-o", str(d / "prune"),
                    str(d / "prune.cpp")], check=True)
    return str(d / "prune")


@pytest.mark.parametrize("kind", range(11))
def test_bounded_triangle_distance_matches_the_plain_one(harness, kind):
    out = subprocess.run([harness, str(kind)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout
