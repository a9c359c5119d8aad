"""Pairs with many contacts: cubes pressed together by their faces, at rest and sliding.

Hundreds of nodes of a pair touch, so that a warp of the contact pass takes a few pairs only and each pair fills several
rounds of its lanes. Sliding layers change the set of touching nodes in every step: a contact's spring is then at another rank
of the pair's old segment, or in none. Lists, springs and forces against the CPU oracle, step by step.
"""
import numpy as np
import pytest

from helpers import history_from_gpu
from test_gpu_parity import _capture, _close, _compare_lists, _oracle_from

pytestmark = pytest.mark.gpu


def _solver(lsdem, scenes, nodes, speed, prec, loose):
    s = 2e-3
    T = scenes.make_from_sdf(scenes.rounded_box_sdf([s] * 3, 0.2e-3), np.array([s] * 3), 24, nodes)
    mp = lsdem.mass_properties(T["sdf"], T["size"], T["origin"], T["spacing"], 2500.0)
    sv = lsdem.Solver()
    sid = sv.add_shape(T["nodes"], T["sdf"], T["size"], T["origin"], T["spacing"])
    i = np.arange(8)
    pos = (np.stack([i % 2, i // 2 % 2, i // 4], 1) + 0.5) * (2 * s * 0.99)
    far = np.stack([6e-3 * np.arange(loose) + 0.02, np.zeros(loose), np.zeros(loose)], 1)  # pairs with a few nodes, or none
    far[1::2, 0] -= 2.05e-3
    pos = np.concatenate([pos, far])
    n = len(pos)
    vel = np.zeros((n, 3))
    vel[:8, 0] = np.where(i // 4 == 1, speed, 0.0)
    vel[:8, 1] = np.where(i // 4 == 1, 0.5 * speed, 0.0)
    quat = np.tile([1.0, 0, 0, 0], (n, 1))
    quat[8:] = scenes.random_quaternions(np.random.default_rng(3), loose)
    sv.add_particles(np.full(n, sid), pos, quat, 1.0 / mp["mass"], np.tile(mp["inv_inertia"], (n, 1)), 1e3, 8e2, 0.5, 0.6, vel=vel)
    sv.set_precision(prec)
    sv.set_record_contacts(True)
    lo, hi = pos.min(0) - 0.02, pos.max(0) + 0.02
    sv.initialize(lo, hi, np.zeros(3))
    return sv, {"min": lo, "max": hi, "gravity": np.zeros(3)}


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("nodes, speed, loose", [(1000, 0.0, 0), (1000, 60.0, 40), (4000, 60.0, 0), (4000, 400.0, 40)])
def test_faces_pressed_together(lsdem, nodes, speed, loose, prec):
    from lsdem_b200 import scenes
    sv, sc = _solver(lsdem, scenes, nodes, speed, prec, loose)
    dt = 1e-6
    prev, changed = None, 0
    for _ in range(4):
        box, hook = _capture(sv)
        sv.step(dt, 1, hook=hook)
        sim = _oracle_from(sv, lsdem, box, sc)
        n_tot = sim.nodes.total
        if prev is not None:
            sim.old["pp"] = history_from_gpu(prev, n_tot)
        sim.detect_all()
        c = sv.contacts(lsdem.CONTACT_PARTICLE, geometry=True)
        assert len(c["node"]) > nodes / 2
        og, oo = _compare_lists(c, sim.last["pp"], n_tot, "particle")
        sim.forces(dt)
        s_scale = max(np.abs(sim.last["pp"]["spring"]).max(), 1e-300)
        assert _close(c["spring"][og], sim.last["pp"]["spring"][oo], rtol=1e-7, scale=s_scale)
        assert _close(box["force"], sim.F, rtol=1e-7, scale=np.abs(sim.F).max())
        assert _close(box["torque"], sim.T, rtol=1e-7, scale=np.abs(sim.T).max())
        if prev is not None:
            changed += len(np.setxor1d(prev["node"], c["node"]))
        prev = c
    assert changed > 0 or speed < 60.0
    sv.close()
