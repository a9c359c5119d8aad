"""Lists of bodies that several lanes share in the rebuild, against the search of every step.

Up to 8 lanes walk a body's cells where the bodies do not fill the grid's threads; a lane's buffer of found bodies fills up, and is
emptied several times, in a crowd of small bodies about a large one. Sizes on both sides of each number of lanes, and the
order of the found pairs through the contacts of every step.
"""
import numpy as np
import pytest

from test_gpu_crossings import AXES, _compare

pytestmark = pytest.mark.gpu


def _run(lsdem, scenes, n, periodic, lists):
    rng = np.random.default_rng(n)
    shp = scenes.make_ellipsoid(AXES, 16, 60)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    sv = lsdem.Solver()
    sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
    scale = np.where(rng.random(n) < 0.02, 1.0, rng.uniform(0.25, 0.35, n))
    side = max(0.03, (n * 1.1e-8) ** (1.0 / 3.0))  # dozens of bodies within reach of a small one, hundreds of a large one
    pos = rng.random((n, 3)) * side
    sv.add_particles(np.full(n, sid), pos, scenes.random_quaternions(rng, n), 1.0 / (mp["mass"] * scale ** 3),
                     mp["inv_inertia"][None] / scale[:, None] ** 5, 1.0, 0.8, 0.5, 0.6, scale=scale,
                     vel=rng.normal(0.0, 5.0, size=(n, 3)))
    sv.set_capacity(pp=512, wall=1, ghost=512, contacts=1 << 23)
    sv.set_periodic(periodic)
    sv.set_neighbour_lists(lists)
    sv.initialize(np.zeros(3), np.full(3, side), np.zeros(3))
    sv.set_record_contacts(True)
    per = []
    for _ in range(4):
        sv.step(1e-6, 1)
        per.append((0, 0, sv.step_stats()["contacts"]))
    out = per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state()
    sv.close()
    return out


@pytest.mark.parametrize("periodic", [0, 7])
@pytest.mark.parametrize("n", [32, 64, 65, 129, 257, 1_000, 9_472, 9_473, 18_945, 37_889])
def test_shared_bodies(lsdem, n, periodic):
    from lsdem_b200 import scenes
    a, b = (_run(lsdem, scenes, n, periodic, lists) for lists in (True, False))
    assert a[0][-1][2] > 0 or n < 257
    _compare(a, b)
