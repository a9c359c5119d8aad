"""Mesh grids with nodes on the mesh: a finely meshed box whose faces lie on planes of nodes.

A node within rounding of the surface takes the solid angles' sum in the triangles' order, as the reference
does. Its sign decides -1e-17 from 1e-17; with thousands of such nodes the sum must not take a closed mesh longer
than every node's sum takes the same mesh with a hole.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(k, half=1.0):
    """Box of k x k quads a face, vertices shared, the first three corners of a cell towards the inside last."""
    at, tris = {}, []

    def vertex(ax, lev, a, b):
        q = [0, 0, 0]
        q[ax], q[(ax + 1) % 3], q[(ax + 2) % 3] = lev, a, b
        return at.setdefault(tuple(q), len(at))

    for ax in range(3):
        for lev in (0, k):
            for i in range(k):
                for j in range(k):
                    a, b, c, d = (vertex(ax, lev, *p) for p in ((i, j), (i + 1, j), (i + 1, j + 1), (i, j + 1)))
                    t = [(a, b, c), (a, c, d)]
                    tris += t if lev else [u[::-1] for u in t]
    return np.array(list(at), float) * (2.0 * half / k) - half, np.array(tris, np.int32)


@pytest.mark.parametrize("scale", [1.0, 1.0 + 1e-16 * 3, 1.0 + 1e-9])
def test_values_of_nodes_on_faces(lsdem, ora, scale):
    h = 2.0 / 12
    v, t = _box(7)
    v = v * scale
    sdf, size, origin = lsdem.mesh_grid(v, t, h)
    ref = ora.mesh_grid(v, t, origin, size, h)
    assert (np.abs(ref) < 1e-8).sum() + (np.abs(ref) == 0.5 * h).sum() > 500
    assert np.array_equal(np.abs(sdf), np.abs(ref))
    off = np.abs(ref) > 1e-12  # below, the last bit of a sum of solid angles decides the sign
    assert np.array_equal(sdf[off], ref[off])


def test_time_of_nodes_on_faces(lsdem):
    v, t = _box(60)
    h = 2.0 / 40

    def best(t):
        ts = []
        for _ in range(4):
            t0 = time.perf_counter()
            lsdem.mesh_grid(v, t, h)
            ts.append(time.perf_counter() - t0)
        return min(ts)

    closed, hole = best(t), best(t[:-1])
    assert closed < hole, (closed, hole)
