"""Child links outside the trees are refused before any traversal, also where
the first child's index is so large that the last one's overflows 32 bits."""
import numpy as np
import pytest

import delta2_gb300 as D

pytestmark = pytest.mark.gpu

LINKS = [(2 ** 31 - 1, 1), (2 ** 31 - 8, 8), (2 ** 31 - 2, 2), (3, 1), (2, 2), (-1, 1)]


def _scene(first, count):
    s = D.make_scene(1, nx=2, ny=1, nz=1, spacing=1.05, speed_sigma=0.0)
    s.mesh_node_off = np.array([0, 3], np.int32)
    s.mesh = np.zeros(s.n_bodies, np.int32)
    s.nodes = np.array([[first, count, 1, 0], [-1, 0, 0, 1], [-1, 0, 0, 1]], np.int32)
    s.ntris = np.ones(3, np.int32)
    s.tris = np.zeros((3, 8, 9))
    s.tris[:, 0] = [0, 0, 0, 1, 0, 0, 0, 1, 0]
    s.eps, s.inner_eps = np.zeros((3, 8)), np.zeros((3, 8))
    return s


@pytest.fixture(scope="module", autouse=True)
def built(gpu_required):
    from delta2_gb300 import build as B
    B.build()


@pytest.mark.parametrize("first, count", LINKS)
def test_context_refuses_links_outside_the_trees(first, count):
    ctx = D.Context(0)
    try:
        with pytest.raises(D.D2GError, match="invalid node 0"):
            ctx.set_scene(_scene(first, count))
        ctx.set_scene(_scene(1, 2))
    finally:
        ctx.close()


@pytest.mark.parametrize("first, count", LINKS)
def test_allocation_free_call_refuses_links_outside_the_trees(first, count):
    import torch
    s = _scene(first, count)
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(s, k))).cuda() for k in
         ("mesh_node_off", "nodes", "ntris", "tris", "eps", "inner_eps", "mesh", "fut", "geo_eps")}
    ds = D.DeviceScene(1, 3, t["mesh_node_off"].data_ptr(), t["nodes"].data_ptr(), t["ntris"].data_ptr(),
                       t["tris"].data_ptr(), t["eps"].data_ptr(), t["inner_eps"].data_ptr(), s.n_bodies,
                       t["mesh"].data_ptr(), t["fut"].data_ptr(), t["geo_eps"].data_ptr())
    pairs = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda")
    out = torch.zeros((64, D.CONTACT_LEN), dtype=torch.float64, device="cuda")
    off = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(D.D2GError, match="out of range"):
        D.compare_trees_full_noalloc(ds, pairs.data_ptr(), 1, out.data_ptr(), 64, off.data_ptr())
