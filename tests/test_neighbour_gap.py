"""What the lists' rebuild may drop, and for how long (CPU).

k_rebuild drops a pair when one of two directions shows its bodies 0.8 skin apart, and the lists serve until a body's
|m| + 2 |dq| r passes 0.4 skin (m its move, dq the difference of its quaternion from the build's, r the radius of its points
that count). Restated here in float32 as the kernels round it. Pairs at the nearest distance at which the build drops
them are moved and turned towards each other up to the bound: no node of the one may be in the other. With a smaller gap,
or with the turn left out of the bound, some are.
"""
import functools

import numpy as np
import pytest

import support_restate as sr
from support_restate import f32
from test_separation_directions import (_dot_f, _fma, _matrices, _phi, _rot_f, _sup_f, _templates, _torus, solid_corners,
                                        solid_support)

SKIN = 0.1  # in largest bounding radii


templates = functools.lru_cache(_templates)


def _tables(t):
    if "tables" not in t:
        t["tables"] = _make_tables(t)
    return t["tables"]


def _make_tables(t):
    c, nodes = solid_corners(t), np.asarray(t["nodes"])
    W = sr.vertex_dirs().reshape(-1, 3)
    h = solid_support(c, W)
    return {"n": sr.vertex_table(nodes), "s": sr.round_up32(h).reshape(6, sr.M + 1, sr.M + 1),
            "r": sr.round_up32([np.linalg.norm(c[0], axis=1).max()])[0],
            "t": (h / np.linalg.norm(W, axis=1)).max() * 1.0071, "nodes": nodes, "nr": np.linalg.norm(nodes, axis=1).max()}


def _separated(ta, tb, xa, qa, sa, xb, qb, sb, gap, dirs=2):
    """pair_separated<dirs>(..., gap) over arrays of pairs: (dropped, direction, B's support point in the world)."""
    pa, pb = xa.astype(f32), xb.astype(f32)
    qa, qb, sa, sb = (v.astype(f32) for v in (qa, qb, sa, sb))
    d = [pb[k] - pa[k] for k in range(3)]
    D2 = _dot_f(d, d)
    D = np.sqrt(D2)
    Di = f32(1.0) / D
    n1 = (np.abs(pa[0]) + np.abs(pa[1]) + np.abs(pa[2])) + (np.abs(pb[0]) + np.abs(pb[1]) + np.abs(pb[2]))
    rho = (sa * f32(ta["nr"])).astype(f32) + sb * tb["r"]
    eps = f32(4e-7) * (n1 + D) * Di + f32(8e-6)
    slack = gap.astype(f32) + _fma(eps, rho, _fma(np.full_like(D, 1e-6), n1, f32(1e-5) * D))
    s = [x * Di for x in d]
    done, out, at = np.zeros(len(D), bool), np.zeros((3, len(D)), f32), np.zeros((3, len(D)), f32)
    for _ in range(dirs):
        hA, gA = _sup_f(ta["n"], np.array(_rot_f(s, qa[0], -qa[1], -qa[2], -qa[3])))
        hB, gB = _sup_f(tb["s"], np.array(_rot_f([-x for x in s], qb[0], -qb[1], -qb[2], -qb[3])))
        sd, need = _dot_f(s, d), ((sa * hA + sb * hB) + slack) * f32(1.0 + 1e-5)
        wA, wB = _rot_f(gA, *qa), _rot_f(gB, *qb)
        hit = ~done & (need < sd)
        out[:, hit], at[:, hit] = np.array(s)[:, hit], np.array(wB)[:, hit]
        done |= hit
        dl = [_fma(sb, wB[a], _fma(-sa, wA[a], d[a])) for a in range(3)]
        c = (f32(1.75) * (need - sd)) / _dot_f(dl, dl)
        s = [_fma(c, dl[a], s[a]) for a in range(3)]
        i = f32(1.0) / np.sqrt(_dot_f(s, s))
        s = [x * i for x in s]
    return done, out.astype(np.float64), at.astype(np.float64)


def _turn(q, point, to, move, r):
    """q turned about the centre so that point moves towards `to`, by the angle whose 2 |dq| r is `move`."""
    axis = np.cross(point.T, to.T)
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    half = 2.0 * np.arcsin(0.25 * move / r)  # |dq| = 2 sin(angle / 4)
    a = np.concatenate([np.cos(half)[None], (axis * np.sin(half)[:, None]).T])
    w, x, y, z = a
    W, X, Y, Z = q
    return np.array([w * W - x * X - y * Y - z * Z, w * X + x * W + y * Z - z * Y, w * Y - x * Z + y * W + z * X,
                     w * Z + x * Y - y * X + z * W])


def _inside(A, B, xa, qa, sa, xb, qb, sb, r):
    """Pairs with a node of A at phi <= 0 of B and within r of B's centre."""
    w = np.einsum("nij,kj->nki", _matrices(qa), A["nodes"]) * sa[:, None, None] + (xa - xb).T[:, None]
    p = np.einsum("nji,nkj->nki", _matrices(qb), w) / sb[:, None, None]
    g = (p - B["origin"]) / B["spacing"]
    ok = ((g >= 0) & (g < np.asarray(B["size"]) - 1)).all(-1) & (np.linalg.norm(w, axis=-1) <= r[:, None])
    hit = np.zeros(ok.shape, bool)
    hit[ok] = _phi(B, p[ok]) <= 0
    return hit.any(1)


def _hits(A, B, seed, offset, gap=0.8, move=0.4, turns=(0.0, 0.5, 1.0), extra=0.0, solid=False):
    """Pairs found touching after moves within the bound (extra: turned beyond it by so many skins)."""
    rng = np.random.default_rng(seed)
    n = 100
    ta, tb = _tables(A), _tables(B)
    qa, qb = (q / np.linalg.norm(q, axis=0) for q in rng.normal(size=(2, 4, n)))
    sa, sb = 2e-3 * np.exp(0.25 * rng.standard_normal((2, n)))
    ra, rb = sa * ta["nr"], sb * tb["nr"]
    turn_b = sb * max(tb["nr"], tb["t"]) if solid else rb
    skin = SKIN * np.maximum(ra, rb)
    u = rng.normal(size=(3, n))
    u /= np.linalg.norm(u, axis=0)
    xa = offset + rng.uniform(0.0, 0.05, size=(3, n))
    lo, hi = np.zeros(n), 1.5 * (ra + sb * tb["r"]) + skin
    g = gap * skin * (1.0 + 1e-5)
    for _ in range(30):  # nearest distance at which the build drops the pair
        mid = 0.5 * (lo + hi)
        drop = _separated(ta, tb, xa, qa, sa, xa + mid * u, qb, sb, g)[0]
        lo, hi = np.where(drop, lo, mid), np.where(drop, mid, hi)
    xb = xa + hi * u
    drop, s, pb = _separated(ta, tb, xa, qa, sa, xb, qb, sb, g)
    assert drop.all()
    na = np.einsum("nij,kj->nki", _matrices(qa), A["nodes"])
    na = na[np.arange(n), np.einsum("nki,in->nk", na, s).argmax(1)].T
    out = 0
    for f in turns:  # share of the bound that is turn
        t = (f * move + extra) * skin * (1.0 - 2e-6)
        m = (1.0 - f) * move * skin * (1.0 - 2e-6)
        ya, yb = xa + m * s, xb - m * s
        out += int(_inside(A, B, ya, _turn(qa, na, s, t, ra), sa, yb, _turn(qb, pb, -s, t, turn_b), sb,
                           np.full(n, np.inf) if solid else rb).sum())
    return out


@functools.lru_cache
def _cases():
    T = templates()[:4]
    return [(a, b) for a in T for b in T] + [(T[0], dict(_torus(), nodes=0.9 * np.asarray(T[1]["nodes"])))]


@pytest.mark.parametrize("offset", (0.0, 3.0))
@pytest.mark.parametrize("solid", (False, True))
def test_dropped_pairs_stay_apart_up_to_the_rebuild(offset, solid):
    """Of another body (nodes within the bounding radius) and of an image (its whole solid)."""
    assert sum(_hits(a, b, k, offset, solid=solid) for k, (a, b) in enumerate(_cases())) == 0


def test_an_image_with_a_solid_beyond_its_nodes():
    T = templates()
    few = {**{k: v for k, v in T[0].items() if k != "tables"}, "nodes": 0.2 * np.asarray(T[0]["nodes"])}
    assert _hits(T[1], few, 3, 0.0, solid=True) == 0
    # counted at the nodes' radius, its turn brings it into contact
    tb = _tables(few)
    assert _hits(T[1], few, 3, 0.0, solid=True, extra=0.4 * (tb["t"] / tb["nr"] - 1.0)) > 0


def test_the_gap_and_the_turn_are_needed():
    T = templates()[:4]
    assert sum(_hits(a, b, 1, 0.0, gap=0.5) for a in T for b in T) > 0
    assert sum(_hits(a, b, 1, 0.0, turns=(0.0,), extra=0.4) for a in T for b in T) > 0


@pytest.mark.parametrize("k", range(7))
def test_the_solids_radius(k):
    """sup_t: at least the distance of any point with phi <= 0, and within 2 % of a convex distance's."""
    t = templates()[k]
    rng = np.random.default_rng(k)
    p = np.asarray(t["origin"]) + rng.random((200_000, 3)) * (np.asarray(t["size"]) - 1) * t["spacing"]
    r = np.linalg.norm(p[_phi(t, p) <= 0], axis=1).max()
    W = sr.vertex_dirs().reshape(-1, 3)
    bound = (solid_support(solid_corners(t), W) / np.linalg.norm(W, axis=1)).max() * 1.0071
    assert r <= bound
    if k == 0:  # the ellipsoid's longest semi-axis
        assert bound <= 0.5 * 1.02
