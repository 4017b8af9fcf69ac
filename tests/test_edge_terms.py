"""The shortened forms of the edge-edge test (edgeEdgeCCD) against the plain
ones, bit for bit: the Newton quantities at one scale instead of three, the
bisection's decisions from the cubic, closest points with shared reciprocals,
integer comparisons.  Random edges and motions at scales from 1e-160 to 1e150,
still and degenerate edges, coplanar ones, large coordinates, values at the
ends of the exponent range.  The harness compiles the library's header for the
host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "delta2_gb300", "csrc")

HARNESS = r"""
#include "d2g_geom.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace d2g;
static std::mt19937_64 g(5);
static double U(double a, double b) { return a + (b - a) * std::uniform_real_distribution<double>(0, 1)(g); }
static V3 rv(double s) { return mk(U(-s, s), U(-s, s), U(-s, s)); }
static bool same(double a, double b) { return m_bits(a) == m_bits(b) || (a != a && b != b); }
static bool same(V3 a, V3 b) { return same(a.x, b.x) && same(a.y, b.y) && same(a.z, b.z); }
static V3 constrain(V3 A, V3 B, V3 p) {
    const V3 ba = B - A;
    const double t = dot(p - A, ba) / dot(ba, ba);
    return lerp(A, B, t < 0 ? 0 : (t > 1 ? 1 : t));
}
static double closest(V3 SA, V3 SB, V3 EA, V3 EB, V3& P, V3& Q) {
    const V3 dc = EB - EA;
    const double l = dot(dc, dc);
    const V3 pA = SA - (dot(SA - EA, dc) / l) * dc, pB = SB - (dot(SB - EA, dc) / l) * dc, ba = pB - pA;
    double t = dot(EA - pA, ba) / dot(ba, ba);
    t = pA.x != pB.x || pA.y != pB.y || pA.z != pB.z ? t : 0.0;
    Q = constrain(EA, EB, lerp(SA, SB, t < 0 ? 0 : (t > 1 ? 1 : t)));
    P = constrain(SA, SB, Q);
    return norm(Q - P);
}
static double bisect(const Edge& aS, const Edge& aE, const Edge& bS, const Edge& bE, double d0, Ccd& r) {
    double lo = 0, hi = 1;
    for (int k = 0; k < 20; k++) {
        const double m = (lo + hi) / 2;
        const V3 aA = lerp(aS.A, aE.A, m), aB = lerp(aS.B, aE.B, m), bA = lerp(bS.A, bE.A, m), bB = lerp(bS.B, bE.B, m);
        const double d = dot(bB - aA, cross(aB - aA, bA - aA));
        if (fabs(d) < 1e-8) { lo = hi = m; break; }
        if (d0 * d < 0) hi = m; else lo = m;
    }
    r.toc = (lo + hi) / 2;
    return closest(lerp(aS.A, aE.A, r.toc), lerp(aS.B, aE.B, r.toc), lerp(bS.A, bE.A, r.toc), lerp(bS.B, bE.B, r.toc),
                   r.P, r.Q);
}
int main(int argc, char** argv) {
    const int kind = atoi(argv[1]);
    const double scales[] = {1.0, 1.0, 1e-3, 30.0, 1e-160, 1e150, 1e-4, 1e5};
    const double s = scales[kind], off = kind == 1 ? 50.0 : (kind == 6 ? 10.0 : 0.0);
    long bad = 0, bisected = 0;
    for (long it = 0; it < 40000; it++) {
        const V3 o = rv(off), da = rv(.3 * s), db = rv(.3 * s);
        Edge aS{o + rv(s), o + rv(s)}, bS{o + rv(s), o + rv(s)}, aE{aS.A + da, aS.B + da}, bE{bS.A + db, bS.B + db};
        if (it % 3 == 0) aE.B = aE.B + rv(.1 * s), bE.A = bE.A + rv(.1 * s);  // turning
        if (it % 7 == 0) aE = aS;                                             // still
        if (it % 11 == 0) bS.B = bS.A;                                        // a point
        if (it % 13 == 0) aS.A.z = aS.B.z = bS.A.z = bS.B.z = 0.0;            // coplanar
        if (it % 17 == 0) bS = aS;
        if (it % 5 == 0) aS.B = aS.A + mk(1, 0, 0) * s, bS.B = bS.A + mk(0, 1, 0) * s;
        const double t = it % 4 == 0 ? (it % 8 ? 0.0 : 1.0) : U(0, 1);
        const Edge at{lerp(aS.A, aE.A, t), lerp(aS.B, aE.B, t)}, bt{lerp(bS.A, bE.A, t), lerp(bS.B, bE.B, t)};
        V3 P, Q, P1, Q1, P2, Q2;
        EdgeDiv d;
        const double ref = closest(at.A, at.B, bt.A, bt.B, P, Q);
        bad += !same(ref, edge_closest(at.A, at.B, bt.A, bt.B, P1, Q1, d)) || !same(P, P1) || !same(Q, Q1);
        bad += !same(ref, edge_closest(at.A, at.B, bt.A, bt.B, P2, Q2)) || !same(P, P2) || !same(Q, Q2);
        double pa = edge_project(at.A, at.B, P), pb = edge_project(bt.A, bt.B, Q);
        bad += !same(pa, m_div_recip(dot(P - at.A, at.B - at.A), d.S, d.rS));
        if (it % 6 == 0) pa = it % 12 ? 0.0 : 1.0;
        if (it % 9 == 0) pb = it % 18 ? 1.0 : 4.9e-324;
        double x, y, x1, y1;
        ee_newton_terms_plain(aS, aE, bS, bE, pa, pb, t, x, y);
        ee_newton_terms(aS, aE, bS, bE, at, bt, pa, pb, t, x1, y1);
        bad += !same(x, x1) || !same(y, y1);
        const double d0 = ee_coplanarity(aS, bS);
        if (d0 * ee_coplanarity(aE, bE) < 0.0) {
            Ccd r0, r1;
            bad += !same(bisect(aS, aE, bS, bE, d0, r0), ee_bisect(aS, aE, bS, bE, d0, r1)) || !same(r0.toc, r1.toc) ||
                   !same(r0.P, r1.P) || !same(r0.Q, r1.Q);
            bisected++;
        }
    }
    const double inf = 1.0 / 0.0, nan = inf - inf, sp[] = {0.0, -0.0, 1.0, -1.0, 0.5, 1.0000000000000002, 4.9e-324,
                                                          -4.9e-324, inf, -inf, nan, -nan, 1e300};
    for (double u : sp) {
        bad += !same(clamp01(u), u < 0 ? 0.0 : (u > 1 ? 1.0 : u));
        for (double v : sp) bad += m_ne(u, v) != (u != v);
    }
    std::printf("bad %ld bisected %ld\n", bad, bisected);
    return bad != 0 || (kind < 4 && bisected < 100);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("edge_terms")
    (d / "h.cpp").write_text(HARNESS)
    exe = d / "h"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(d / "h.cpp"), "-o", str(exe)],
                   check=True)
    return str(exe)


@pytest.mark.parametrize("kind", range(8))
def test_shortened_edge_terms_match_plain(harness, kind):
    r = subprocess.run([harness, str(kind)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
