"""The candidate search's wall part at the edges of its blocks, against the search of every step.

A small system's walls are tested in blocks of their own (128 particles each) behind the pairs' blocks (32
each); from 47,360 particles (148 SMs x 10 warps x 32) on, in the pairs' blocks. A layer of touching ellipsoids
cuts a floor: every step's numbers of candidate pairs, the wall and particle contacts and the state equal
the run that sorts and walks afresh every step.
"""
import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu


def _run(lsdem, scenes, n, prec, lists):
    rng = np.random.default_rng(n)
    shp = scenes.make_ellipsoid((5e-3, 4e-3, 3e-3), 16, 300)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    m = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    L = (m + 1) * 9e-3
    pos = np.stack([(i % m + 0.9) * 9e-3, (i // m + 0.9) * 9e-3, np.full(n, 2.9e-3)], 1)
    pos[:, :2] += rng.uniform(-3e-4, 3e-4, size=(n, 2))
    sv = lsdem.Solver()
    sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
    sv.add_particles(np.full(n, sid), pos, scenes.random_quaternions(rng, n), 1.0 / mp["mass"],
                     np.tile(mp["inv_inertia"], (n, 1)), 1e5, 8e4, 0.5, 0.6, angvel=rng.normal(0.0, 20.0, size=(n, 3)))
    f = scenes.make_plane_wall((L, L))
    sv.add_wall(f["verts"], f["sdf"], f["size"], f["origin"], f["spacing"], [0.5 * L, 0.5 * L, 0.0], [1.0, 0, 0, 0], 0.5, 0.6)
    sv.set_precision(prec)
    sv.set_neighbour_lists(lists)
    sv.initialize(np.zeros(3), np.array([L, L, 0.05]), np.array([0.0, 0.0, -9.81]))
    sv.set_record_contacts(True)
    per = []
    for _ in range(3):
        sv.step(2e-6, 1)
        s = sv.step_stats()
        per.append((s["pairs_particle"], s["pairs_wall"], s["contacts"]))
    out = per, sv.contacts(lsdem.CONTACT_WALL), sv.contacts(lsdem.CONTACT_PARTICLE), sv.state()
    sv.close()
    return out


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 47_359, 47_360])
def test_walls_of_a_small_system(lsdem, n, prec):
    from lsdem_b200 import scenes
    a = _run(lsdem, scenes, n, prec, True)
    b = _run(lsdem, scenes, n, prec, False)
    assert a[0] == b[0] and a[0][0][1] == n and len(a[1]["node"]) > 0  # every body is near the floor
    for ca, cb in ((a[1], b[1]), (a[2], b[2])):
        oa, ob = canon(ca), canon(cb)
        for k in ("node", "partner"):
            assert np.array_equal(np.asarray(ca[k])[oa], np.asarray(cb[k])[ob]), k
    for k in ("pos", "vel", "angvel", "quat"):
        # only the order of the FP64 force sums differs
        assert np.abs(a[3][k] - b[3][k]).max() <= 1e-11 * max(np.abs(b[3][k]).max(), 1e-30), k
