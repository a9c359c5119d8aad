"""Lists at the crossing of a periodic face by, or beside, a body outside the domain along another axis.

A body outside the domain owns pairs (its cell is clamped) and is no one's partner, so the pair of an outside body and one
inside exists when the outside one has the smaller index. The two of a scene touch across a face; one of them, or both, cross it
in the third of twelve steps and nothing else sets off a rebuild, so that the steps after the crossing live on what
that rebuild listed. Every step equals the run without lists.

Where many bodies cross at once, their pairs are left to the next step's rebuild.
"""
import time

import numpy as np
import pytest

from test_gpu_crossings import AXES, _compare

pytestmark = pytest.mark.gpu

L, H = 81e-3, 60e-3  # wide: 8 radii are 40 mm, the grids reach 11 mm
EPS = 2.5e-6         # before the face, at 1e-6 a step
NEAR = 2e-3


def _pair(case):
    """Positions and velocities; the ellipsoids (5, 4, 3 mm) overlap by about 0.1 mm once both are on one side."""
    up, down = H + 1e-3, H - 4.75e-3
    fast, rest = [0.5, 0.0, 0.0], [0.0, 0.0, 0.0]
    y = 30e-3
    return {
        "outside crosses": ([[L - EPS, y, up], [NEAR, y, down]], [fast, rest]),
        "outside crosses back": ([[EPS, y, up], [L - NEAR, y, down]], [[-0.5, 0.0, 0.0], rest]),
        "inside crosses": ([[NEAR, y, up], [L - EPS, y, down]], [rest, fast]),
        "both cross": ([[L - EPS, y, up], [L - EPS, y, down]], [fast, fast]),
        "outside crosses an edge": ([[L - EPS, L - EPS, up], [NEAR, 1e-3, down]], [[0.5, 0.5, 0.0], rest]),
        "below": ([[L - EPS, y, -1e-3], [NEAR, y, 4.75e-3]], [fast, rest]),
        # the outside body has the larger index: no pair
        "inside owns": ([[NEAR, y, down], [L - EPS, y, up]], [rest, fast]),
    }[case]


def _run(lsdem, scenes, pos, vel, prec, lists):
    shp = scenes.make_ellipsoid(AXES, 16, 300)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    sv = lsdem.Solver()
    sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
    n = len(pos)
    sv.add_particles(np.full(n, sid), pos, np.tile([1.0, 0, 0, 0], (n, 1)), 1.0 / mp["mass"], np.tile(mp["inv_inertia"], (n, 1)),
                     1e5, 8e4, 0.5, 0.6, vel=vel, angvel=np.zeros((n, 3)))
    sv.set_capacity(pp=64, wall=1, ghost=64, contacts=1 << 18)  # no growth, which rebuilds
    sv.set_precision(prec)
    sv.set_periodic(3)
    sv.set_neighbour_lists(lists)
    sv.initialize(np.zeros(3), np.array([L, L, H]), np.zeros(3))
    sv.set_record_contacts(True)
    per = []
    for _ in range(12):
        sv.step(2e-6, 1)
        s = sv.step_stats()
        per.append((s["pairs_particle"], s["pairs_ghost"], s["contacts"]))
    out = per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state(), sv.num(9)
    sv.close()
    return out


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("others", [0, 98])  # more bodies in no cell, far off (64: where images are sorted again)
@pytest.mark.parametrize("case", ["outside crosses", "outside crosses back", "inside crosses", "both cross",
                                  "outside crosses an edge", "below", "inside owns"])
def test_pair_with_a_body_outside(lsdem, case, others, prec):
    from lsdem_b200 import scenes
    pos, vel = (np.array(v) for v in _pair(case))
    i = np.arange(others)
    far = np.stack([5e-3 + 11e-3 * (i % 7), 5e-3 + 11e-3 * (i // 7 % 7), H + 30e-3 + 11e-3 * (i // 49)], 1).reshape(-1, 3)
    pos, vel = np.concatenate([pos, far]), np.concatenate([vel, np.zeros(far.shape)])
    a, b = (_run(lsdem, scenes, pos, vel, prec, lists) for lists in (True, False))
    assert a[4] <= 3  # the first step's, the crossing's and at most one that the contact's motion sets off
    assert (b[0][-1][0] > 0 and b[0][-1][2] > 0) or case == "inside owns"
    _compare(a, b)


@pytest.mark.parametrize("n", [3_000, 4_500, 60_000])  # 3,000 are looked up (below 2^24 pairs), the others not
def test_all_bodies_cross_at_once(lsdem, n):
    """Bodies handed over a domain's length off, some of them touching, across faces among them."""
    from lsdem_b200 import scenes
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    a = 9.8e-3
    pos = np.stack([i % m, (i // m) % m, i // (m * m)], 1) * a + rng.uniform(0.0, 1e-3, size=(n, 3))
    side = m * a
    shp = scenes.make_ellipsoid(AXES, 16, 100)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    out, took = {}, {True: [], False: []}
    for lists in (True, True, True, False):  # the shortest of three: an allocation can stall on a shared host
        sv = lsdem.Solver()
        sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
        sv.add_particles(np.full(n, sid), pos + [side, 0, -side], scenes.random_quaternions(np.random.default_rng(1), n),
                         1.0 / mp["mass"], np.tile(mp["inv_inertia"], (n, 1)), 1e5, 8e4, 0.5, 0.6, vel=np.zeros((n, 3)))
        sv.set_capacity(pp=64, wall=1, ghost=64, contacts=1 << 21)
        sv.set_periodic(7)
        sv.set_neighbour_lists(lists)
        sv.initialize(np.zeros(3), np.full(3, side), np.zeros(3))
        sv.set_record_contacts(True)
        per = []
        t0 = time.perf_counter()
        for _ in range(4):
            sv.step(1e-7, 1)
            st = sv.step_stats()
            per.append((0, 0, st["contacts"]))
        took[lists].append(time.perf_counter() - t0)
        out[lists] = (per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state())
        sv.close()
    _compare(out[True], out[False])
    assert out[True][0][-1][2] > 0
    assert min(took[True]) < 5 * min(took[False]) + 0.1, took


@pytest.mark.parametrize("n, outside", [(700, 63), (700, 64), (700, 65), (700, 699), (300, 257), (5_000, 1_200)])
def test_order_of_bodies_in_no_cell(lsdem, n, outside):
    """Bodies outside in any order among the others: listed in index order by chunks of a block each (above 64 of them)."""
    from lsdem_b200 import scenes
    rng = np.random.default_rng(n + outside)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    p = rng.permutation(m ** 3)
    i = np.arange(n)
    a = 9e-3
    pos = (np.stack([i % m, (i // m) % m, i // (m * m)], 1) + 0.5) * a + rng.uniform(-2e-4, 2e-4, size=(n, 3))
    z = np.sort(pos[:, 2])
    cut = 0.5 * (z[n - outside - 1] + z[n - outside])
    pos = pos[np.argsort(p[:n])]
    shp = scenes.make_ellipsoid(AXES, 16, 200)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    out = []
    for lists in (True, False):
        sv = lsdem.Solver()
        sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
        sv.add_particles(np.full(n, sid), pos, scenes.random_quaternions(np.random.default_rng(2), n), 1.0 / mp["mass"],
                         np.tile(mp["inv_inertia"], (n, 1)), 1e5, 8e4, 0.5, 0.6,
                         vel=np.random.default_rng(3).normal(0.0, 2.0, size=(n, 3)))
        sv.set_capacity(pp=64, wall=1, ghost=64, contacts=1 << 20)
        sv.set_periodic(3)
        sv.set_neighbour_lists(lists)
        sv.initialize(np.array([0.0, 0.0, -0.01]), np.array([m * a, m * a, cut]), np.zeros(3))
        sv.set_record_contacts(True)
        per = []
        for _ in range(8):
            sv.step(2e-6, 1)
            per.append((0, 0, sv.step_stats()["contacts"]))
        h = sv.hash()
        key = h["key"]
        assert np.array_equal(h["sorted_idx"], np.argsort(key, kind="stable"))
        out.append((per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state()))
        sv.close()
    assert abs((key < 0).sum() - outside) <= 12  # some move through the upper face
    _compare(*out)
