"""Triangles none of whose features has a distance: points, and coordinates
that are not finite; and triangles so far out that FP64 rounding at their place
shapes them.  The reference's triangle distance (comparison_dist.h:
12-189) is then what its comparisons leave, 0 with both points at the origin,
and so a hit.  The form with FP32 bounds gives the same (on the CPU, through a
harness that compiles the library's header), and so do the discrete narrow
phase's entry points, in leaf buckets and in the inner ones of a descent,
against the oracle (on the GPU)."""
import contextlib
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.small_scenes import SmallScene, state

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "delta2_gb300", "csrc")

HARNESS = r"""
#include "d2g_prune.cuh"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
using namespace d2g;
static std::mt19937_64 g(3);
static double U(double a, double b) { return a + (b - a) * std::uniform_real_distribution<double>(0, 1)(g); }
static V3 rv(double s) { return mk(U(-s, s), U(-s, s), U(-s, s)); }
static double& at(Tri& t, int k) { return (&(k < 3 ? t.A : (k < 6 ? t.B : t.C)).x)[k % 3]; }
int main(int argc, char** argv) {
    const int kind = atoi(argv[1]);
    long bad = 0, zero = 0;
    for (long it = 0; it < 20000; it++) {
        Tri a{rv(1), rv(1), rv(1)}, b{rv(1), rv(1), rv(1)};
        const V3 w = it % 3 ? rv(it % 3 == 1 ? 5 : 1000) : mk(0, 0, 0);
        Tri* t[2] = {&a, &b};
        for (int k = 0; k < 2; k++) {
            Tri& x = *t[k];
            if (kind == 2 || kind == k) x.B = x.C = x.A;                          // points: a, b, both
            if (kind == 3 && k == it % 2) at(x, it % 9) = NAN;                    // one coordinate
            if (kind == 4 && k == it % 2) at(x, it % 9) = it & 4 ? INFINITY : -INFINITY;
            if (kind == 5 && k == it % 2) x.A.y = x.B.y = x.C.y = NAN;            // a pose
            if (kind == 6 && k == it % 2) x.A = x.A * 1e-200, x.B = x.B * 1e-200, x.C = x.C * 1e-200;
            if (kind == 7 && k == it % 2) x.A = x.A * 1e160, x.B = x.B * 1e160, x.C = x.C * 1e160;
            if (kind == 8 && k == it % 2) x.B = x.A + rv(1e-17), x.C = x.A + rv(1e-17);
            const double size[] = {1, 1e-3, 1e-9, 1}, away[] = {1e14, 1e12, 1e7, 1e11};
            if (kind >= 9) x.A = x.A * size[kind - 9], x.B = x.B * size[kind - 9], x.C = x.C * size[kind - 9];
            V3 o = w;
            if (kind >= 9) o = mk(away[kind - 9], -0.3 * away[kind - 9], 0.7 * away[kind - 9]);
            x.A = x.A + o, x.B = x.B + o, x.C = x.C + o;
        }
        V3 P, Q, P2, Q2;
        const double d = tri_tri_dist(a, b, P, Q);
        for (double lim : {0.25, 3.0, 1e-6, d * (1 + 1e-9)}) {
            const double e = tri_tri_dist_below(a, b, lim, P2, Q2);
            bool ok = !(e < lim);
            if (d < lim) {
                zero += d == 0.0;
                ok = !std::memcmp(&d, &e, 8) && !std::memcmp(&P, &P2, 24) && !std::memcmp(&Q, &Q2, 24);
            }
            if (!ok && bad++ < 5) std::printf("limit %g distance %.17g, bounded %.17g\n", lim, d, e);
        }
    }
    std::printf("zero distances %ld mismatches %ld\n", zero, bad);
    return bad != 0 || (kind < 9 && zero == 0);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("degenerate")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-std=c++17", "-I", CSRC, "-o", str(d / "h"), str(d / "h.cpp")],
                   check=True)
    return str(d / "h")


@pytest.mark.parametrize("kind", range(13))
def test_bounded_distance_without_features_matches_the_plain_one(harness, kind):
    out = subprocess.run([harness, str(kind)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout


FLAT = [[0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0, 0.0]]
NAN_X = state(x=(np.nan, 0.2, 0.0))
INF_X = state(x=(0.0, np.inf, 0.0))


def _scene(inner, point, fut):
    """A triangle, and beside it a body whose triangle (inner: its root's, over
    a leaf that holds an ordinary one) is a point."""
    s = SmallScene()
    s.add_leaf_mesh(FLAT)
    s.add_leaf_mesh([list(point) * 3])
    tilt = TILTED if point[0] > 0.5 else state()
    s.add_body(0, 0.01, cur=tilt, fut=tilt)
    s.add_body(1, 0.01, cur=fut, fut=fut)
    sc = s.build().to_product()
    if inner:
        sc.mesh_node_off = np.array([0, 1, 3], np.int32)
        sc.nodes = np.array([[-1, 0, 0, 0], [2, 1, 1, 0], [-1, 0, 0, 1]], np.int32)
        sc.ntris = np.array([1, 1, 1], np.int32)
        near = np.array(FLAT, dtype=np.float64) + np.tile([0.0, 0.0, 0.012], 3)
        sc.tris = np.concatenate([sc.tris, np.zeros((1, 8, 9))])
        sc.tris[2, 0] = near
        sc.eps, sc.inner_eps = np.zeros((3, 8)), np.zeros((3, 8))
    return sc


# the point (outside the triangle's prism, so that nothing has a distance), the pose
CASES = {
    "near": ((-0.004, -0.004, 0.004), state()),
    "just beyond": ((-0.0204, 0.5, 0.0), state()),  # 0.4 mm past the limit of 20 mm
    "nan pose": ((0.1, 0.1, 0.005), NAN_X),
    "infinite pose": ((0.1, 0.1, 0.005), INF_X),
    "beside a face": ((0.9, 0.6, 0.1), state()),  # in the tilted triangle's box, 0.35 m off its plane
}
TILTED = state(q=(np.cos(np.pi / 8), np.sin(np.pi / 8), 0, 0))


@pytest.mark.gpu
@pytest.mark.parametrize("inner", [False, True], ids=["leaf", "inner"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_narrow_phase_entry_points_match_oracle(gpu_required, case, inner):
    import torch

    import delta2_gb300 as D
    from delta2_gb300 import build as B
    from oracle import oracle as O
    B.build()
    sc = _scene(inner, *CASES[case])
    pairs = np.array([[0, 1]], np.int32)
    ref, ref_off, ref_cnt = O.narrowphase(sc.copy(), pairs)
    assert len(ref) > 0
    with contextlib.closing(D.Context(0)) as ctx:
        ctx.set_scene(sc.copy())
        for bounds in (True, False):
            ctx.set_fp32_bounds(bounds)
            c, off, cnt = ctx.compare_trees_full(pairs)
            assert np.array_equal(off, ref_off), (bounds, len(c), len(ref))
            assert np.array_equal(c.view(np.uint64), ref.view(np.uint64)), bounds
            assert cnt[:2].tolist() == ref_cnt[:2].tolist()
        ctx.set_fp32_bounds(True)
        hits, used = ctx.find_contacts_bucket_comparison(0, 1, [[0, 1]])
        want, want_used = O.bucket_comparison(sc, 0, 1, [[0, 1]])
        assert used.tolist() == want_used.tolist() and len(want) > 0
        assert np.array_equal(hits.view(np.uint64), want.view(np.uint64))
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(sc, k))).cuda() for k in
         ("mesh_node_off", "nodes", "ntris", "tris", "eps", "inner_eps", "mesh", "fut", "geo_eps")}
    ds = D.DeviceScene(2, len(sc.ntris), t["mesh_node_off"].data_ptr(), t["nodes"].data_ptr(), t["ntris"].data_ptr(),
                       t["tris"].data_ptr(), t["eps"].data_ptr(), t["inner_eps"].data_ptr(), sc.n_bodies,
                       t["mesh"].data_ptr(), t["fut"].data_ptr(), t["geo_eps"].data_ptr())
    d_pairs = torch.from_numpy(pairs).cuda()
    out = torch.zeros((64, D.CONTACT_LEN), dtype=torch.float64, device="cuda")
    off = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    n = D.compare_trees_full_noalloc(ds, d_pairs.data_ptr(), 1, out.data_ptr(), 64, off.data_ptr())
    assert n == len(ref) and off.tolist() == ref_off.tolist()
    assert np.array_equal(out[:n].cpu().numpy().view(np.uint64), ref.view(np.uint64))
