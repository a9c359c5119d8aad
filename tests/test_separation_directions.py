"""The separation test's solid table and its search for a separating direction (CPU).

Restated in numpy: the table of the solid (k_support_vertices: over the corners c of the grid
cells that phi changes sign on, the smallest over a few l of max(w . c - l |w| phi_c)) and the
directions pair_separated tries, in float32 with each operation rounded as the kernel rounds it.
Checked in FP64: no point with phi <= 0 projects beyond the table's values, for signed distances
of convex bodies, of a torus (not convex) and for a grid that is no distance; and every pair the
FP32 search drops is separated along the direction it found.
"""
import numpy as np
import pytest

import support_restate as sr
from support_restate import f32

SUP_L = (0.0, 0.5, 0.7, 0.85, 1.0, 1.2, 1.5, 2.5)
DIRS = 5


def solid_corners(t):
    """(points, phi) of the corners of every cell with both signs of phi, or on the boundary with phi <= 0."""
    gx, gy, gz = (int(v) for v in t["size"])
    phi = np.asarray(t["sdf"], np.float64).reshape(gz, gy, gx)
    corner = [(slice(z, gz - 1 + z), slice(y, gy - 1 + y), slice(x, gx - 1 + x)) for z in (0, 1) for y in (0, 1)
              for x in (0, 1)]
    c = np.stack([phi[s] for s in corner], -1)
    tol = 1e-12 * np.abs(c).max(-1)
    edge = np.ones(c.shape[:-1], bool)
    edge[1:-1, 1:-1, 1:-1] = False
    cell = (c.min(-1) <= tol) & ((c.max(-1) >= -tol) | edge)
    m = np.zeros(phi.shape, bool)
    for s in corner:
        m[s] |= cell
    z, y, x = np.nonzero(m)
    return np.asarray(t["origin"]) + t["spacing"] * np.stack([x, y, z], 1), phi[m]


def solid_support(corners, W):
    p, phi = corners
    lw = np.linalg.norm(W, axis=1)[:, None]
    r, big = np.linalg.norm(p, axis=1).max(), np.abs(phi).max()
    wp = W @ p.T
    return np.min([(wp - l * lw * phi).max(1) + 1e-11 * lw[:, 0] * (r + l * big) for l in SUP_L], axis=0)


def _torus(n=32):
    h = 2.4 / (n - 5)
    size = np.array([n, n, n], np.int32)
    origin = -0.5 * (n - 1) * h * np.ones(3)
    from lsdem_b200 import scenes
    p = scenes.grid_points(size, origin, h)
    sdf = np.hypot(np.hypot(p[:, 0], p[:, 1]) - 0.8, p[:, 2]) - 0.3
    return {"sdf": sdf, "size": size, "origin": origin, "spacing": h}


def _templates():
    from conftest import load_package
    load_package()
    from lsdem_b200 import scenes
    T = scenes.unit_templates(n_grid=16, n_nodes=200)
    return T + [scenes.make_superellipsoid((0.5, 0.4, 0.3), 0.5, 0.8, 24, 300), _torus(),
                # scaled field: |grad phi| = 3, and the whole grid inside the solid
                dict(T[0], sdf=3.0 * T[0]["sdf"]), dict(T[0], sdf=np.full(16 ** 3, -0.1))]


def _phi(t, p):
    nx, ny, nz = (int(v) for v in t["size"])
    g = (p - t["origin"]) / t["spacing"]
    i = np.minimum(np.floor(g).astype(int), [nx - 2, ny - 2, nz - 2])
    f = g - i
    out = 0.0
    for k in range(8):
        o = (k & 1, (k >> 1) & 1, k >> 2)
        w = np.prod([f[:, a] if o[a] else 1 - f[:, a] for a in range(3)], axis=0)
        out = out + w * t["sdf"][i[:, 0] + o[0] + nx * (i[:, 1] + o[1] + ny * (i[:, 2] + o[2]))]
    return out


@pytest.mark.parametrize("k", range(8))
def test_no_point_of_the_solid_projects_beyond_the_table(k):
    t = _templates()[k]
    rng = np.random.default_rng(k)
    ext = (np.asarray(t["size"]) - 1) * t["spacing"]
    p = np.asarray(t["origin"]) + rng.random((200_000, 3)) * ext
    p = p[_phi(t, p) <= 0]
    assert len(p) > 1000
    W = sr.vertex_dirs().reshape(-1, 3)[:: 7]
    h = solid_support(solid_corners(t), W)
    assert ((W @ p.T).max(1) <= h).all()


def test_a_convex_distance_is_bounded_by_the_body_itself():
    """l = 1 on the signed distance of an ellipsoid: never beyond the ellipsoid, whose support is |R u|."""
    t = _templates()[0]
    W = sr.vertex_dirs().reshape(-1, 3)
    h = solid_support(solid_corners(t), W)
    body = np.linalg.norm(W * np.array([0.5, 0.4, 0.3]), axis=1)
    assert (h <= body * (1 + 1e-9) + 1e-9).all()  # the bisection behind the grid's values ends at 1e-12


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f32)


def _rot_f(v, w, a, b, c):
    two = f32(2.0)
    tx, ty, tz = two * _fma(b, v[2], -(c * v[1])), two * _fma(c, v[0], -(a * v[2])), two * _fma(a, v[1], -(b * v[0]))
    return (_fma(w, tx, v[0]) + _fma(b, tz, -(c * ty)), _fma(w, ty, v[1]) + _fma(c, tx, -(a * tz)),
            _fma(w, tz, v[2]) + _fma(a, ty, -(b * tx)))


def _dot_f(a, b):
    return _fma(a[0], b[0], _fma(a[1], b[1], a[2] * b[2]))


def _sup_f(tab, u):
    """Bound and gradient for direction arrays u, one table."""
    M, half = sr.M, f32(0.5 * sr.M)
    a = np.abs(u)
    ax = np.where((a[0] >= a[1]) & (a[0] >= a[2]), 0, np.where(a[1] >= a[2], 1, 2))
    at = np.arange(len(ax))
    um, p, q = u[ax, at], u[(ax + 1) % 3, at], u[(ax + 2) % 3, at]
    f, m = 2 * ax + (um < 0), np.abs(um)
    r = (f32(1.0) / m).astype(f32)
    p, q = p * r, q * r
    x, y = (p + f32(1.0)) * half, (q + f32(1.0)) * half
    i, j = np.clip(np.floor(x).astype(int), 0, M - 1), np.clip(np.floor(y).astype(int), 0, M - 1)
    s, t = np.clip(x - i.astype(f32), f32(0), f32(1)), np.clip(y - j.astype(f32), f32(0), f32(1))
    c0, c1, c2, c3 = tab[f, j, i], tab[f, j, i + 1], tab[f, j + 1, i], tab[f, j + 1, i + 1]
    low = s + t <= f32(1.0)
    ds, dt = np.where(low, c1 - c0, c3 - c2), np.where(low, c2 - c0, c3 - c1)
    v = np.where(low, _fma(s, ds, _fma(t, dt, c0)), _fma(s - f32(1), ds, _fma(t - f32(1), dt, c3)))
    gp, gq = ds * half, dt * half
    g0 = _fma(-gp, p, _fma(-gq, q, v))
    g = np.zeros((3, len(ax)), f32)
    g[ax, at], g[(ax + 1) % 3, at], g[(ax + 2) % 3, at] = np.where(f & 1, -g0, g0), gp, gq
    return m * v, g


def _search(tab, pa, ra, qa, sa, pb, qb, sb):
    """pair_separated over arrays of pairs of one template pair: (dropped, direction)."""
    d = [pb[k] - pa[k] for k in range(3)]
    D2 = _dot_f(d, d)
    D = np.sqrt(D2)
    Di = f32(1.0) / D
    n1 = (np.abs(pa[0]) + np.abs(pa[1]) + np.abs(pa[2])) + (np.abs(pb[0]) + np.abs(pb[1]) + np.abs(pb[2]))
    rho = ra + sb * tab["r"]
    eps = f32(4e-7) * (n1 + D) * Di + f32(8e-6)
    slack = _fma(eps, rho, _fma(np.full_like(D, 1e-6), n1, f32(1e-5) * D))
    s = [x * Di for x in d]
    done, out = np.zeros(len(D), bool), np.zeros((3, len(D)), f32)
    live = np.ones(len(D), bool)
    for k in range(DIRS):
        hA, gA = _sup_f(tab["n"], np.array(_rot_f(s, qa[0], -qa[1], -qa[2], -qa[3])))
        hB, gB = _sup_f(tab["s"], np.array(_rot_f([-x for x in s], qb[0], -qb[1], -qb[2], -qb[3])))
        hA, hB = sa * hA, sb * hB
        sd, need = _dot_f(s, d), ((hA + hB) + slack) * f32(1.0 + 1e-5)
        hit = live & (need < sd)
        out[:, hit] = np.array(s)[:, hit]
        done |= hit
        live &= ~hit
        wA, wB = _rot_f(gA, *qa), _rot_f(gB, *qb)
        dl = [_fma(sb, wB[a], _fma(-sa, wA[a], d[a])) for a in range(3)]
        dd = _dot_f(dl, dl)
        live &= dd > f32(1e-10) * D2
        with np.errstate(all="ignore"):
            c = (f32(1.75) * (need - sd)) / dd
            s = [_fma(c, dl[a], s[a]) for a in range(3)]
            i = f32(1.0) / np.sqrt(_dot_f(s, s))
        s = [np.where(live, x * i, f32(0.57735)) for x in s]
    return done, out


def _matrices(q):
    w, x, y, z = q
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


@pytest.mark.parametrize("offset", (0.0, 3.0))
def test_dropped_pairs_are_separated_along_the_direction_found(offset):
    T = _templates()[:4]
    rng = np.random.default_rng(int(offset))
    found = centre = wrong = 0
    for ta in T:
        for tb in T:
            n = 800
            corners, nodes = solid_corners(tb), np.asarray(ta["nodes"])
            W = sr.vertex_dirs().reshape(-1, 3)
            tab = {"n": sr.vertex_table(nodes), "s": sr.round_up32(solid_support(corners, W)).reshape(6, sr.M + 1, sr.M + 1),
                   "r": sr.round_up32([np.linalg.norm(corners[0], axis=1).max()])[0]}
            qa, qb = (q / np.linalg.norm(q, axis=0) for q in rng.normal(size=(2, 4, n)))
            sa, sb = 2e-3 * np.exp(0.25 * rng.standard_normal((2, n)))
            u = rng.normal(size=(3, n))
            u /= np.linalg.norm(u, axis=0)
            ra = sa * np.linalg.norm(nodes, axis=1).max()
            D = (ra + sb * np.linalg.norm(corners[0], axis=1).max()) * rng.uniform(0.5, 1.0, n)
            xa = offset + rng.uniform(0.0, 0.05, size=(3, n))
            xb = xa + D * u
            done, s = _search(tab, xa.astype(f32), ra.astype(f32), qa.astype(f32), sa.astype(f32), xb.astype(f32),
                              qb.astype(f32), sb.astype(f32))
            s = s.astype(np.float64)
            # exact: A's nodes and the bound of B's solid along the very direction
            la = np.einsum("nji,jn->ni", _matrices(qa), s)
            lb = -np.einsum("nji,jn->ni", _matrices(qb), s)
            i = np.nonzero(done)[0]
            reach = sa[i] * (la[i] @ nodes.T).max(1) + sb[i] * solid_support(corners, lb[i])
            wrong += int((reach >= (s * (xb - xa)).sum(0)[i]).sum())
            found += len(i)
            centre += int((np.abs((s * u).sum(0)[i]) > 1 - 1e-6).sum())
    assert wrong == 0
    assert found > 1.1 * centre > 0  # other directions than the line of centres are found, too
