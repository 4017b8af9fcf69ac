"""The CCD counters are the same in every run, and the modes that switch the
FP32 bounds and the certificates off, alone and together, give the oracle's
contacts."""
import itertools

import numpy as np
import pytest

import delta2_gb300 as D

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_required):
    from delta2_gb300 import build as B
    B.build()
    c = D.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("config, n, spacing", [(1, (3, 3, 3), 1.12), (2, (8, 8, 8), 1.23), (5, (2, 2, 2), 1.15)])
def test_counters_do_not_depend_on_timing(ctx, config, n, spacing):
    s = D.make_scene(config, nx=n[0], ny=n[1], nz=n[2], spacing=spacing, speed_sigma=2.0, seed=9)
    pairs = D.broad_phase(s)
    mt = np.full(len(pairs), 0.02)
    seen = set()
    for _ in range(12):
        ctx.set_scene(s.copy())
        ctx.ccd_stats(reset=True)
        ctx.compare_trees_full_continuous(pairs, mt, capacity=1 << 22)
        st = ctx.ccd_stats(reset=True)
        seen.add((st["ee_tests_cut"], st["newton_iters_saved"]))
    assert len(seen) == 1, seen
    cut, saved = seen.pop()
    assert 0 < cut <= saved <= 10 * cut


@pytest.mark.parametrize("config, n, spacing", [(1, (2, 2, 2), 1.12), (2, (2, 2, 1), 1.1), (5, (2, 1, 1), 1.1)])
def test_modes_match_oracle(ctx, config, n, spacing):
    from oracle import oracle as O
    s = D.make_scene(config, nx=n[0], ny=n[1], nz=n[2], spacing=spacing, speed_sigma=1.0, seed=5)
    pairs = D.broad_phase(s)
    mt = np.full(len(pairs), 0.02)
    ref, ref_off, _, ref_cnt = O.ccd(s.copy(), pairs, mt)
    assert len(ref) > 0
    try:
        for bounds, certificates in itertools.product((True, False), repeat=2):
            ctx.set_fp32_bounds(bounds)
            ctx.set_ccd_certificates(certificates)
            ctx.set_scene(s.copy())
            ctx.ccd_stats(reset=True)
            c, off, cnt = ctx.compare_trees_full_continuous(pairs, mt, capacity=1 << 22)
            mode = (bounds, certificates)
            assert np.array_equal(off, ref_off), mode
            assert np.array_equal(c.view(np.uint64), ref.view(np.uint64)), mode
            assert cnt[:3].tolist() == ref_cnt.tolist(), mode
            if not certificates:
                assert ctx.ccd_stats(reset=True)["ee_tests_cut"] == 0
    finally:
        ctx.set_fp32_bounds(True)
        ctx.set_ccd_certificates(True)
