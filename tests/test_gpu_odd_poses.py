"""Continuous and discrete queries of bodies whose orientation is not a unit quaternion: the
pose's linear part scales and shears, and the reference measures distances
after it, while a triangle's bounding sphere does not follow; a huge one gives
coordinates beyond FP32's range.  Contacts, offsets and futures against the
oracle, bit for bit."""
import numpy as np
import pytest

import delta2_gb300 as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_required):
    from delta2_gb300 import build as B
    B.build()
    c = D.Context(0)
    yield c
    c.close()


def ccd_against_oracle(ctx, s, pairs, mt):
    ref_s = s.copy()
    ref, ref_off, _, ref_cnt = O.ccd(ref_s, pairs, mt)
    gs = s.copy()
    ctx.set_scene(gs)
    c, off, cnt = ctx.compare_trees_full_continuous(pairs, mt, capacity=max(1024, 2 * len(ref)))
    assert off.tolist() == ref_off.tolist()
    assert np.array_equal(c.view(np.uint64), ref.view(np.uint64))
    assert cnt[:3].tolist() == ref_cnt.tolist()
    ctx.get_bodies(gs)
    touched = np.unique(pairs)
    same = gs.fut[touched].view(np.uint64) == ref_s.fut[touched].view(np.uint64)
    assert np.all(same | (np.isnan(gs.fut[touched]) & np.isnan(ref_s.fut[touched])))
    return len(ref)


@pytest.mark.parametrize("config", [1, 2])
@pytest.mark.parametrize("mt", [0.0, 0.02])
@pytest.mark.parametrize("form", [0.5, 0.9, 0.999, 1.0001, 1.1, "x 0", "w 0", "y 1e-300", "z 0.9"])
def test_continuous_queries_match_oracle(ctx, config, mt, form):
    total = 0
    for seed in range(4):
        s = D.make_scene(config, nx=2, ny=2, nz=1, spacing=1.05 if config == 1 else 0.95, speed_sigma=1.0, seed=seed)
        moving = np.flatnonzero(s.is_static == 0)
        b = moving[seed % len(moving)]
        if isinstance(form, str):
            comp, value = form.split()
            s.cur[b, 1 + "wxyz".index(comp)] = float(value)
        else:
            s.cur[b, 1:5] *= form
        pairs = D.broad_phase(D.make_scene(config, nx=2, ny=2, nz=1, spacing=0.9, speed_sigma=0.0, seed=seed))
        total += ccd_against_oracle(ctx, s, pairs, np.full(len(pairs), mt))
    assert total > 0


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("value", [1e15, 1e18, 1e19, 1e20, 1e22, 1e100])
def test_coordinates_beyond_fp32_match_oracle(ctx, value, seed):
    for comp in range(1, 5):
        s = D.make_scene(1, nx=2, ny=2, nz=1, spacing=1.2, speed_sigma=0.0, seed=seed)
        moving = np.flatnonzero(s.is_static == 0)
        s.cur[moving[seed], comp] = value
        pairs = D.broad_phase(D.make_scene(1, nx=2, ny=2, nz=1, spacing=1.0, speed_sigma=0.0, seed=seed))
        ccd_against_oracle(ctx, s, pairs, np.full(len(pairs), 0.02))


@pytest.mark.parametrize("config", [1, 2])
@pytest.mark.parametrize("scale", [0.5, 0.999, 1.0001, 1.1, 1.3, 2.0])
def test_discrete_queries_match_oracle(ctx, config, scale):
    total = 0
    for seed in range(4):
        s = D.make_scene(config, nx=2, ny=2, nz=1, spacing=1.3, speed_sigma=0.0, seed=seed)
        moving = np.flatnonzero(s.is_static == 0)
        s.cur[moving, 1:5] *= scale
        s.fut[...] = s.cur
        pairs = D.broad_phase(D.make_scene(config, nx=2, ny=2, nz=1, spacing=0.9, speed_sigma=0.0, seed=seed))
        ref, ref_off, ref_cnt = O.narrowphase(s.copy(), pairs)
        ctx.set_scene(s.copy())
        c, off, cnt = ctx.compare_trees_full(pairs, capacity=max(1024, 2 * len(ref)))
        assert off.tolist() == ref_off.tolist()
        assert np.array_equal(c.view(np.uint64), ref.view(np.uint64))
        assert cnt[:2].tolist() == ref_cnt[:2].tolist()
        total += len(ref)
    assert total > 0 or scale < 1.0  # (smaller bodies no longer touch)
