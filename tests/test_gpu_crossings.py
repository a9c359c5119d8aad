"""Neighbour and image lists against the search of every step, where their dispatch branches.

* Bodies crossing periodic faces, edges and corners while they touch others across them: in domains wide
  enough for the lists to take a crossing body at its next position (more than 8 bounding radii and the
  images' reach), in narrow ones, with few and with many bodies outside the domain (images searched
  in the particle sort, or in a second one). Every step's numbers of candidate pairs (particles,
  images) and contacts and the final contacts and state equal the run that sorts, walks and images
  afresh every step.
* The three splits of the candidate search (8, 32 and 128 particles a warp) and their ragged ends.
"""
import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu

AXES = (5e-3, 4e-3, 3e-3)


def _solver(lsdem, scenes, pos, vel, lo, hi, periodic, prec, lists, seed):
    rng = np.random.default_rng(seed)
    shp = scenes.make_ellipsoid(AXES, 16, 300)
    mp = lsdem.mass_properties(shp["sdf"], shp["size"], shp["origin"], shp["spacing"], 2500.0)
    sv = lsdem.Solver()
    sid = sv.add_shape(shp["nodes"], shp["sdf"], shp["size"], shp["origin"], shp["spacing"])
    n = len(pos)
    quat = scenes.random_quaternions(rng, n)
    sv.add_particles(np.full(n, sid), pos, quat, 1.0 / mp["mass"], np.tile(mp["inv_inertia"], (n, 1)), 1e5, 8e4, 0.5, 0.6,
                     vel=vel, angvel=rng.normal(0.0, 20.0, size=(n, 3)))
    sv.set_capacity(pp=64, wall=1, ghost=64, contacts=1 << 20)  # no growth, which rebuilds
    sv.set_precision(prec)
    sv.set_periodic(periodic)
    sv.set_neighbour_lists(lists)
    sv.initialize(lo, hi, np.zeros(3))
    return sv


def _run(lsdem, scenes, *scene, steps, **kw):
    sv = _solver(lsdem, scenes, *scene, **kw)
    sv.set_record_contacts(True)
    per = []
    for _ in range(steps):
        sv.step(2e-6, 1)
        s = sv.step_stats()
        per.append((s["pairs_particle"], s["pairs_ghost"], s["contacts"]))
    out = per, sv.contacts(lsdem.CONTACT_PARTICLE), sv.contacts(lsdem.CONTACT_GHOST), sv.state(), sv.num(9)
    sv.close()
    return out


def _compare(a, b):
    assert a[0] == b[0]
    for ca, cb in ((a[1], b[1]), (a[2], b[2])):
        keys = ("node", "partner", "image")
        oa, ob = canon(ca, keys), canon(cb, keys)
        for k in keys:
            assert np.array_equal(np.asarray(ca[k])[oa], np.asarray(cb[k])[ob]), k
    for k in ("pos", "vel", "angvel", "quat"):
        # only the order of the FP64 force sums differs
        assert np.abs(a[3][k] - b[3][k]).max() <= 1e-11 * max(np.abs(b[3][k]).max(), 1e-30), k


def _lattice(m, a, seed, vmax):
    """m^3 bodies, a layer of them on each lower face, moving so that bodies cross in every step."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3) * a
    pos = g + rng.uniform(-2e-5, 2e-5, size=g.shape)
    return pos % (m * a), rng.uniform(-vmax, vmax, size=g.shape), m * a


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("periodic", [1, 2, 4, 3, 7])
@pytest.mark.parametrize("m", [4, 9])  # 36 mm: narrow; 81 mm: wide (8 radii are 40 mm, the grids reach 11 mm)
def test_bodies_crossing_faces(lsdem, m, periodic, prec):
    from lsdem_b200 import scenes
    pos, vel, L = _lattice(m, 9e-3, 10 * m + periodic, 2.0)
    scene = (pos, vel, np.zeros(3), np.full(3, L), periodic, prec)
    a = _run(lsdem, scenes, *scene, lists=True, seed=1, steps=40)
    b = _run(lsdem, scenes, *scene, lists=False, seed=1, steps=40)
    _compare(a, b)
    assert max(s[1] for s in a[0]) > 0 and a[0][-1][2] > 0  # image pairs and contacts were there
    assert a[4] > 5  # crossings set off rebuilds


@pytest.mark.parametrize("above", [1, 3])  # layers above the domain: 81 and 243 bodies in no cell
def test_bodies_outside_the_domain(lsdem, above):
    from lsdem_b200 import scenes
    pos, vel, L = _lattice(9, 9e-3, 5 + above, 2.0)
    pos[:, 2] += 4e-3  # no layer on the lower face, the top ones beyond the upper
    hi = np.array([L, L, L - 9e-3 * above])
    scene = (pos, vel, np.zeros(3), hi, 3, 0)
    _compare(_run(lsdem, scenes, *scene, lists=True, seed=2, steps=25),
             _run(lsdem, scenes, *scene, lists=False, seed=2, steps=25))


@pytest.mark.parametrize("n", [1, 7, 33, 23_681, 47_361, 189_441])
def test_candidate_splits(lsdem, n):
    from lsdem_b200 import scenes
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    pos = (np.stack([i % m, (i // m) % m, i // (m * m)], 1) + 0.6 + rng.uniform(-0.05, 0.05, size=(n, 3))) * 9e-3
    scene = (pos, np.zeros((n, 3)), np.zeros(3), np.full(3, (m + 1) * 9e-3), 0, 2)
    _compare(_run(lsdem, scenes, *scene, lists=True, seed=3, steps=2), _run(lsdem, scenes, *scene, lists=False, seed=3, steps=2))
