"""Mesh grids (lsdem_mesh_grid) of more than 2^27 nodes.

The pruned search takes a warp, 32 threads, per node: thread numbers pass 32 bits at 2^27 nodes.
"""
import numpy as np
import pytest

from test_gpu_mesh_grid_paths import _cube

pytestmark = pytest.mark.gpu

H = 2.0 ** -12  # coordinates of nodes are exact


def test_more_than_2_27_nodes(lsdem):
    v, t = _cube(8 * H)  # +-32 spacings
    v = v + np.array([200.3, 210.7, 470.1]) * H
    n = 513
    sdf, size, _ = lsdem.mesh_grid(v, t, H, origin=np.zeros(3), size=(n, n, n))
    assert tuple(size) == (n, n, n)
    sdf = np.asarray(sdf).reshape(n, n, n)
    for z in (0, 480, n - 4):  # the planes from 510 on have indices past 2^27
        part, _, _ = lsdem.mesh_grid(v, t, H, origin=np.array([0.0, 0.0, z * H]), size=(n, n, 4))
        assert np.array_equal(sdf[z:z + 4], np.asarray(part).reshape(4, n, n)), z
    assert (sdf[480] < 0).any()
