"""Mesh grids (lsdem_mesh_grid) of more than 2^27 nodes, and on a device with little memory left.

The pruned search takes a warp, 32 threads, per node: thread numbers pass 32 bits at 2^27 nodes.
Its workspace is 33 bytes a node; where that does not fit, the path with 8 bytes a node takes the call.
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


def test_little_memory_left(lsdem):
    torch = pytest.importorskip("torch")
    v, t = _cube(16 * H)
    n = 384
    args = dict(origin=np.full(3, -0.5 * (n - 1) * H), size=(n, n, n))
    ref, _, _ = lsdem.mesh_grid(v, t, H, **args)
    free = torch.cuda.mem_get_info()[0]
    left = 16 * n ** 3 + (64 << 20)  # between the two paths' needs
    hold = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        sdf, _, _ = lsdem.mesh_grid(v, t, H, **args)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(np.abs(sdf), np.abs(ref))
    far = np.abs(ref) > 0.6 * H  # next to the surface the sign is down to rounding
    assert np.array_equal(np.asarray(sdf)[far], np.asarray(ref)[far])
