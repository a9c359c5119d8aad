"""Network queues of the learned form: one set where images come from the image list, a second one where they are
searched in every step, and the same contacts whichever way the lists are switched on the way.

A set has at least 2^20 pending nodes and twice as many rows of 32 bytes: above 64 MB.
"""
import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu


def _solver(lsdem, lists):
    from lsdem_b200 import scenes
    T = scenes.unit_templates(n_grid=24, n_nodes=400)[:1]
    sc = scenes.polydisperse_periodic(lsdem, n=600, box=0.1 * (600 / 1e5) ** (1.0 / 3.0), seed=5, templates=T, n_grid=24,
                                      n_nodes=400)
    scenes.resolve_deep_overlaps(lsdem, sc)
    sv = lsdem.Solver()
    scenes.load_polydisperse(sv, sc)
    sv.set_precision(2)
    sv.set_neighbour_lists(lists)
    sv.initialize(sc["min"], sc["max"], sc["gravity"])
    sv.train_learned_sdf(iterations=200, batch=4096, samples=1 << 14)
    sv.set_learned_sdf(True)
    return sv


def _first_step_bytes(lsdem, torch, lists):
    sv = _solver(lsdem, lists)
    before = torch.cuda.mem_get_info()[0]
    sv.step(2e-7, 1)
    after = torch.cuda.mem_get_info()[0]
    sv.close()
    return before - after


def test_one_set_of_queues_with_the_image_list(lsdem):
    torch = pytest.importorskip("torch")
    _first_step_bytes(lsdem, torch, True)  # module load and the like
    on, off = (_first_step_bytes(lsdem, torch, lists) for lists in (True, False))
    assert on >= 64 << 20
    assert on <= off - (64 << 20), (on, off)


def test_lists_switched_between_steps(lsdem):
    out = []
    for order in ((True, False, True), (False, False, False)):
        sv = _solver(lsdem, order[0])
        sv.set_record_contacts(True)
        per = []
        for lists in order:
            sv.set_neighbour_lists(lists)
            sv.step(2e-7, 4)
            c = sv.contacts(lsdem.CONTACT_GHOST)
            o = canon(c, ("node", "partner", "image"))
            per.append([np.asarray(c[k])[o] for k in ("node", "partner", "image")] + [sv.step_stats()["contacts"]])
        out.append(per)
        sv.close()
    for a, b in zip(*out):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    assert len(out[0][-1][0]) > 0
