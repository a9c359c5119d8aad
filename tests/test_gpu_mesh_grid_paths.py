"""Paths of the mesh grid builder (lsdem_mesh_grid) against the CPU oracle.

A closed mesh takes the pruned search and one solid-angle sum per component of nodes; an open mesh
takes the sum of every node. Both give the oracle's values bit for bit (sign excepted within 1e-9
spacings of the surface, where the reference's own sum is down to rounding): meshes whose triangles
come in an order without locality, with a last cluster that is not full, two bodies (two interior
components), one body inside another with the opposite orientation (a cavity) and with the same one
(winding number 2), nodes on the surface, a grid smaller than a tile, and an open mesh.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere(scenes, level, r=1e-3, c=(0.0, 0.0, 0.0)):
    v, t = scenes.superellipsoid_mesh((r, r, r), 1.0, 1.0, level)
    return v + np.asarray(c), t


def _join(*parts):
    v, t, n = [], [], 0
    for a, b in parts:
        v.append(a)
        t.append(np.asarray(b) + n)
        n += len(a)
    return np.concatenate(v), np.concatenate(t).astype(np.int32)


def _cube(h):
    """Unit-spacing cube with corners on grid nodes: nodes on faces, edges and vertices."""
    v = 4 * h * np.array([(x, y, z) for z in (-1, 1) for y in (-1, 1) for x in (-1, 1)], float)
    q = [(0, 2, 3, 1), (4, 5, 7, 6), (0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)]
    return v, np.array([t for a, b, c, d in q for t in ((a, b, c), (a, c, d))], np.int32)


def _cases(scenes):
    rng = np.random.default_rng(3)
    v, t = _sphere(scenes, 3)
    yield "shuffled", v, t[rng.permutation(len(t))], 1.1e-4
    yield "ragged cluster", *scenes.superellipsoid_mesh((1e-3, 8e-4, 5e-4), 0.4, 0.7, 2), 9e-5
    yield "two bodies", *_join(_sphere(scenes, 2), _sphere(scenes, 2, c=(2.6e-3, 0, 0))), 1.3e-4
    inner = _sphere(scenes, 2, r=5e-4)
    yield "cavity", *_join(_sphere(scenes, 3), (inner[0], inner[1][:, ::-1])), 1e-4
    yield "nested", *_join(_sphere(scenes, 3), inner), 1e-4
    yield "nodes on the surface", *_cube(1e-4), 1e-4
    yield "smaller than a tile", *_cube(1e-3), 5e-3
    yield "open", v, t[: len(t) - 40], 1.4e-4


@pytest.mark.parametrize("k", range(8))
def test_grid_equals_the_oracle(lsdem, ora, k):
    from lsdem_b200 import scenes
    name, v, t, h = list(_cases(scenes))[k]
    sdf, size, origin = lsdem.mesh_grid(v, t, h)
    ref = ora.mesh_grid(v, t, origin, size, h)
    assert np.array_equal(np.abs(sdf), np.abs(ref)), name
    flip = np.signbit(sdf) != np.signbit(ref)
    assert (np.abs(ref[flip]) <= 1e-9 * h).all() or name == "nodes on the surface", name
    if name == "nodes on the surface":  # there the value is -h / 2 whatever the sum
        assert np.array_equal(sdf, ref) or (np.abs(ref[flip]) <= 0.5 * h).all()
        far = np.abs(ref) > 0.6 * h
        assert np.array_equal(sdf[far], ref[far])
    again, _, _ = lsdem.mesh_grid(v, t, h, positive_inside=True)
    assert np.array_equal(np.abs(again), np.abs(sdf))
