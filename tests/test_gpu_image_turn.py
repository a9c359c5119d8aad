"""Image list of a body whose solid reaches beyond its nodes.

A body's bounding radius is its nodes' (0.5 mm here). A node near one of its images is tested by cell window
and grid, with no bounding sphere, so that the whole solid counts there (an ellipsoid of 7, 3, 3 mm). It turns in place beside a
sphere across the face: 0.3 mm apart at first, more than the list's 0.8 margin, and touching while 0.5 mm from the centre has
moved by less than the rebuild's bound. Every step equals the run without lists.
"""
import numpy as np
import pytest

from test_gpu_crossings import _compare

pytestmark = pytest.mark.gpu

MM = 1e-3


def _run(lsdem, scenes, periodic, prec, lists):
    T = [scenes.make_ellipsoid((7 * MM, 3 * MM, 3 * MM), 32, 300), scenes.make_ellipsoid((2 * MM,) * 3, 16, 600)]
    T[0]["nodes"] = 0.25 * T[1]["nodes"]
    mp = [lsdem.mass_properties(t["sdf"], t["size"], t["origin"], t["spacing"], 2500.0) for t in T]
    sv = lsdem.Solver()
    ids = np.array([sv.add_shape(t["nodes"], t["sdf"], t["size"], t["origin"], t["spacing"]) for t in T])
    L, gap, c, s = 81 * MM, 0.3 * MM, np.cos(np.pi / 4), np.sin(np.pi / 4)
    # the ellipsoid turned by 135 degrees: the normal (c, s) of its frame is -x; its support point there
    h = np.hypot(7 * MM * c, 3 * MM * s)
    p = np.array([(7 * MM) ** 2 * c, (3 * MM) ** 2 * s]) / h
    p = np.array([-c * p[0] - s * p[1], s * p[0] - c * p[1]])
    pos = np.array([[L + 1 * MM + p[0] - 2 * MM - gap, 40 * MM + p[1], 40 * MM], [1 * MM, 40 * MM, 40 * MM]])
    quat = np.array([[1.0, 0, 0, 0], [np.cos(3 * np.pi / 8), 0, 0, np.sin(3 * np.pi / 8)]])
    k = [1, 0]
    sv.add_particles(ids[k], pos, quat, np.array([1.0 / mp[i]["mass"] for i in k]), np.array([mp[i]["inv_inertia"] for i in k]),
                     1e5, 8e4, 0.5, 0.6, vel=np.zeros((2, 3)), angvel=np.array([[0.0, 0, 0], [0, 0, 5e3]]))
    sv.set_capacity(pp=64, wall=1, ghost=64, contacts=1 << 16)
    sv.set_precision(prec)
    sv.set_periodic(periodic)
    sv.set_neighbour_lists(lists)
    sv.initialize(np.zeros(3), np.full(3, L), np.zeros(3))
    sv.set_record_contacts(True)
    per = []
    for _ in range(14):  # 0.01 rad a step; 0.16 rad move a point 0.5 mm off by the bound, 0.08 mm
        sv.step(2e-6, 1)
        st = sv.step_stats()
        per.append((0, 0, st["contacts"]))  # numbers of candidates may differ: the walk keeps pairs the build drops
    out = per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state(), sv.num(9)
    sv.close()
    return out


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("periodic", [1, 7])
def test_solid_beyond_the_nodes(lsdem, periodic, prec):
    from lsdem_b200 import scenes
    a, b = (_run(lsdem, scenes, periodic, prec, lists) for lists in (True, False))
    assert b[0][0][2] == 0 and b[0][-1][2] > 0
    _compare(a, b)
