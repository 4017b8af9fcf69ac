"""A tree file whose child links reach outside their mesh is refused, also
where the children's count overflows 32 bits."""
import numpy as np
import pytest

import delta2_gb300 as D


@pytest.mark.parametrize("first, count", [(1, 2 ** 31 - 1), (3, 2 ** 31 - 2), (4, 2), (1, 5), (5, 1)])
def test_tree_file_refuses_links_outside_the_mesh(tmp_path, first, count):
    s = D.make_scene(1, nx=1, ny=1, nz=1)
    s.mesh_node_off = np.array([0, 5], np.int32)
    s.nodes = np.array([[1, 4, 1, 0]] + [[-1, 0, 0, 1]] * 4, np.int32)
    s.ntris = np.ones(5, np.int32)
    s.tris = np.zeros((5, 8, 9))
    s.eps, s.inner_eps = np.zeros((5, 8)), np.zeros((5, 8))
    path = str(tmp_path / "t.d2g")
    D.save_trees(s, path)
    assert len(D.load_trees(path)["nodes"]) == 5
    s.nodes[0, :2] = first, count
    D.save_trees(s, path)
    with pytest.raises(D.D2GError, match="child link outside its mesh"):
        D.load_trees(path)
