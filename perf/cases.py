"""Measured cases: what users of the library have it do, through its public Python API.

Time stepping is the product: a case builds a scene with add_shape / add_particles / add_wall /
add_bond, initializes a solver in one arithmetic form, and a pass is one Solver.step call of the
stated number of steps. Its outputs are the particles' state arrays on the device, where an
external-force hook or a reader finds them. The other case kind is a level-set grid of a triangle
mesh (mesh_grid), which every program builds for each of its shapes before it can step.

Scenes are synthetic and seeded, in the families of the library's own benchmark configurations:
ellipsoids falling on a floor; polydisperse bodies in a triply periodic box; superquadrics settling
in a box periodic in x and y; a rotating drum; a bonded lattice under a moving wall; and a dense bed
in which every body touches its neighbours.
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "lsdem2.0_b200"

FORMS = {"fp64": 0, "fp16": 1, "bf16": 2, "learned": 2}
STATE = (("force", 3), ("torque", 3), ("vel", 3), ("angvel", 3), ("pos", 3), ("quat", 4))
DRAG = 1e-3  # kg/s, the external force of the hooked cases: -DRAG * velocity


def _lib():
    if "lsdem_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("lsdem_b200", _PKG / "__init__.py",
                                                      submodule_search_locations=[str(_PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["lsdem_b200"] = mod
        spec.loader.exec_module(mod)
    from lsdem_b200 import scenes
    return sys.modules["lsdem_b200"], scenes


# ---------------------------------------------------------------------------
# The cases

def listed():
    return [
        # the smallest call: a program that couples to the solver step by step, with a force of
        # its own added in the hook of every step
        {"name": "falling-150-hook", "scene": "falling", "n": 150, "form": "fp64", "steps": 1, "hook": True},
        # the tutorial-sized run: 2,000 ellipsoids landing on a floor
        {"name": "falling-2000", "scene": "falling", "n": 2000, "form": "fp64", "steps": 64, "hook": False},
        # polydisperse gas with seven image sets: the 16-bit screens' configuration, at full size ...
        {"name": "polydisperse-100k-bf16", "scene": "polydisperse", "n": 100_000, "form": "bf16", "steps": 16,
         "hook": False},
        # ... and at a small odd size in the other 16-bit format
        {"name": "polydisperse-9973-fp16", "scene": "polydisperse", "n": 9_973, "form": "fp16", "steps": 16,
         "hook": False},
        # bonded solid compressed by a wall: the force is the bonds'
        {"name": "bonded-12k-fp64", "scene": "bonded", "n": 12_000, "form": "fp64", "steps": 16, "hook": False},
        # rotating drum: one curved wall that every body near it is tested against
        {"name": "drum-60k-bf16", "scene": "drum", "n": 60_000, "form": "bf16", "steps": 16, "hook": False},
        # the benchmark's configuration at its full size, in the fastest form
        {"name": "settling-2M-bf16", "scene": "settling", "n": 2_000_000, "form": "bf16", "steps": 16, "hook": False},
        # the same physics with the network screen
        {"name": "settling-300k-learned", "scene": "settling", "n": 299_997, "form": "learned", "steps": 16,
         "hook": False},
        # and in the plain form, the reference's arithmetic
        {"name": "settling-300k-fp64", "scene": "settling", "n": 299_997, "form": "fp64", "steps": 16, "hook": False},
        # a settled bed: contacts everywhere, spring history carried from step to step
        {"name": "bed-100k-bf16", "scene": "bed", "n": 100_000, "form": "bf16", "steps": 16, "hook": False},
        {"name": "bed-20011-fp64", "scene": "bed", "n": 20_011, "form": "fp64", "steps": 16, "hook": False},
        # grid of one benchmark shape from its 20,480-triangle mesh
        {"name": "grid-20480-triangles", "scene": "grid", "level": 5, "n_grid": 48},
    ]


# sizes a scene is drawn from (the largest at most what a listed case has) and its forms
_RANGES = {
    "falling": (100, 4_000, ("fp64", "fp64", "bf16")),
    "polydisperse": (2_000, 100_000, ("fp64", "fp16", "bf16")),
    "bonded": (1_000, 12_000, ("fp64", "bf16")),
    "drum": (5_000, 60_000, ("fp64", "bf16")),
    "settling": (10_000, 1_000_000, ("fp64", "bf16", "bf16", "learned")),
    "bed": (2_000, 100_000, ("fp64", "bf16", "fp16")),
}


def draw(rng):
    kind = rng.choice(["falling", "polydisperse", "bonded", "drum", "settling", "settling", "bed", "grid"])
    if kind == "grid":
        return {"scene": "grid", "level": rng.choice([2, 3, 4, 5]), "n_grid": rng.randint(20, 48)}
    lo, hi, forms = _RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1
    hook = kind == "falling" and rng.random() < 0.5
    return {"scene": kind, "n": n, "form": rng.choice(forms), "steps": 1 if hook else rng.randint(4, 16), "hook": hook}


# ---------------------------------------------------------------------------
# Shapes: fixed families, built once per process

_shapes = {}


def _unit_density(lsdem, T):
    out = []
    for t in T:
        mp = lsdem.mass_properties(t["sdf"], t["size"], t["origin"], t["spacing"], 1.0)
        c = mp["centroid"]
        nodes = t["nodes"] - c
        out.append({"nodes": nodes, "sdf": t["sdf"], "size": t["size"], "origin": t["origin"] - c,
                    "spacing": t["spacing"], "mass": mp["mass"], "inv_inertia": mp["inv_inertia"],
                    "bound": float(np.max(np.linalg.norm(nodes, axis=1)))})
    return out


def _templates(kind):
    """Templates (frame at the centroid, mass and inertia at density 1) of a scene family."""
    kind = "settling" if kind == "drum" else kind
    if kind in _shapes:
        return _shapes[kind]
    lsdem, scenes = _lib()
    if kind == "falling":  # semi-axes 5, 4, 3 mm, 32^3 grid, 1,000 nodes
        T = [scenes.make_ellipsoid((5e-3, 4e-3, 3e-3), 32, 1000)]
    elif kind in ("bonded", "bed"):  # semi-axes 2, 1.6, 1.2 mm
        T = [scenes.make_ellipsoid((2e-3, 1.6e-3, 1.2e-3), 32, 1000)]
    elif kind == "polydisperse":  # bounding diameter 1; 48^3 grids, 2,000 nodes
        hs = 0.5 / 3 ** 0.25
        s = 1.0 / (math.sqrt(3.0) * 0.8 + 0.2)
        v, f = scenes.superellipsoid_mesh((hs, hs, hs), 0.5, 0.5, 4)
        T = [scenes.make_ellipsoid(np.array([0.5, 0.4, 0.3]), 48, 2000),
             scenes.make_mesh_template(lsdem, v, f, 2 * hs / 43, nodes=scenes.superellipsoid_nodes((hs, hs, hs), 0.5, 0.5, 2000)),
             scenes.make_from_sdf(scenes.rounded_box_sdf([s / 2] * 3, 0.1 * s), np.array([s / 2] * 3), 48, 2000),
             scenes.make_from_sdf(scenes.capsule_sdf(0.25, 0.25), np.array([0.25, 0.25, 0.5]), 48, 2000)]
    else:  # 16 superquadrics, exponents 2-6, semi-axes 1-2.5 mm, 48-node grids, 1,500 nodes
        T = scenes.superquadric_templates(lsdem, np.random.default_rng(scenes.seed_for(4)), 16, (2.0, 6.0),
                                          (1e-3, 2.5e-3), 48, 1500, level=4)
    _shapes[kind] = _unit_density(lsdem, T)
    return _shapes[kind]


# ---------------------------------------------------------------------------
# Scenes

_tiles = {}


def _packing(kind, n):
    """About n bodies packed at random without deep overlaps in a box that is periodic in every axis: (k, m, tile), k
    copies per axis of a tile of m bodies. The tile is random sequential addition of spheres smaller than the bodies'
    bounding spheres; bodies that reach deeper into a neighbour than 1 % of its radius are then shrunk until none does,
    so that neighbours of all distances are met, touching ones among them, and none is thrown apart."""
    lsdem, scenes = _lib()
    kind = "settling" if kind == "drum" else kind
    k = max(1, round((n / 16_000) ** (1.0 / 3.0)))
    m = max(64, round(n / k ** 3))
    if (kind, m) in _tiles:
        return k, m, _tiles[kind, m]
    rng = np.random.default_rng([len(kind), m])
    T = _templates(kind)
    shape = rng.integers(0, len(T), size=m).astype(np.int32)
    bound = np.array([t["bound"] for t in T])[shape]
    if kind == "polydisperse":  # log-normal bounding diameters, median 2 mm
        scale = 2e-3 * np.exp(0.25 * rng.standard_normal(m))
        L, exclusion = (m * 1.15e-8) ** (1.0 / 3.0), 0.8
    else:
        scale = np.ones(m)
        L, exclusion = (np.array([t["mass"] for t in T])[shape].sum() / 0.25) ** (1.0 / 3.0), 0.85
    order = np.argsort(-bound * scale, kind="stable")
    pos = np.empty((m, 3))
    pos[order] = lsdem.pack_rsa((exclusion * bound * scale)[order], np.zeros(3), np.full(3, L), periodic=True, seed=m,
                                max_tries=20000)
    quat = scenes.random_quaternions(rng, m)
    for _ in range(20):
        depth, b = _overlaps(T, shape, scale, pos, quat, L)
        bad = np.unique(b[depth > 0.01 * (bound * scale)[b]])
        if not len(bad):
            break
        scale[bad] *= 0.95
    _tiles[kind, m] = {"shape": shape, "scale": scale, "pos": pos, "quat": quat, "L": L}
    return k, m, _tiles[kind, m]


def _overlaps(T, shape, scale, pos, quat, L):
    """Deepest node of the one in the other's level set (minus its value, at least 0) for every pair of bodies of a
    periodic box whose bounding spheres meet, and the other body."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)
    r = np.array([t["bound"] for t in T])[shape] * scale
    X, R = t64(pos), t64(r)
    A, B = [], []
    for i in torch.arange(len(pos), device=dev).split(1024):
        d = X[i][:, None] - X[None]
        d = d - L * torch.round(d / L)
        a, b = torch.nonzero((d ** 2).sum(-1) < (R[i][:, None] + R[None]) ** 2, as_tuple=True)
        A.append(i[a])
        B.append(b)
    A, B = torch.cat(A), torch.cat(B)
    keep = A != B
    A, B = A[keep], B[keep]
    depth = torch.zeros(len(A), dtype=torch.float64, device=dev)
    Q, S, kind = t64(quat), t64(scale), torch.as_tensor(shape, device=dev)
    for sa, ta in enumerate(T):
        nodes = t64(ta["nodes"])
        for sb, tb in enumerate(T):
            sdf = t64(tb["sdf"])
            for p in torch.nonzero((kind[A] == sa) & (kind[B] == sb)).flatten().split(2048):
                a, b = A[p], B[p]
                d = X[a] - X[b]
                d = d - L * torch.round(d / L)
                w = _rot(Q[a][:, None], nodes[None] * S[a][:, None, None]) + d[:, None]
                g = (_rot_inv(Q[b][:, None], w) / S[b][:, None, None] - t64(tb["origin"])) / tb["spacing"]
                phi, _ = _trilinear(g, tb["size"], sdf)
                depth[p] = (-phi.amin(1)).clamp(min=0) * S[b]
    return depth.cpu().numpy(), B.cpu().numpy()


def _block(rng, kind, n):
    """The packing as one block, seen from another side and shifted for each rng: positions, orientations, shapes,
    scales, sides."""
    _, scenes = _lib()
    k, m, t = _packing(kind, n)
    L, K = t["L"], k * t["L"]
    c = np.stack(np.meshgrid(*(np.arange(k),) * 3, indexing="ij"), -1).reshape(-1, 1, 3) * L
    pos = (t["pos"][None] + c).reshape(-1, 3)
    quat = np.tile(t["quat"], (k ** 3, 1))
    # a turn by 120 degrees about the cube's diagonal, once, twice or not at all, permutes the axes
    for _ in range(int(rng.integers(0, 3))):
        pos = pos[:, [2, 0, 1]]
        a, b = np.array([0.5, 0.5, 0.5, 0.5]), quat
        quat = np.concatenate([(a[0] * b[:, :1] - b[:, 1:] @ a[1:, None]),
                               a[0] * b[:, 1:] + b[:, :1] * a[1:] + np.cross(np.broadcast_to(a[1:], (len(b), 3)), b[:, 1:])], 1)
    pos = (pos + rng.uniform(0, K, size=3)) % K
    p = rng.permutation(len(pos))
    return pos[p], quat[p], np.tile(t["shape"], k ** 3)[p], np.tile(t["scale"], k ** 3)[p], K


def _lattice(rng, dims, n, spacing, jitter):
    """n of the dims[0] x dims[1] x dims[2] lattice sites (x fastest), each moved by up to jitter x spacing per axis."""
    i = np.arange(n)
    p = np.stack([i % dims[0], (i // dims[0]) % dims[1], i // (dims[0] * dims[1])], 1) + 0.5
    return (p + rng.uniform(-jitter, jitter, size=p.shape)) * spacing


def _material(T, shape, scale, density=2500.0):
    m = np.array([t["mass"] for t in T])[shape]
    inertia = np.array([t["inv_inertia"] for t in T])[shape]
    return 1.0 / (density * m * scale ** 3), inertia / (density * scale[:, None] ** 5)


def _scene(case, seed):
    """The scene's arrays, in the layout scenes.load_polydisperse takes."""
    lsdem, scenes = _lib()
    rng = np.random.default_rng([seed, case["n"]])
    kind, n = case["scene"], case["n"]
    T = _templates(kind)
    shape, scale, quat = np.zeros(n, np.int32), np.ones(n), scenes.random_quaternions(rng, n)
    vel = np.zeros((n, 3))
    walls, bonds, periodic, grav, dt = [], None, 0, -9.81, 5e-7
    lo = np.zeros(3)
    if kind == "falling":  # layers above the floor, the lowest already touching it here and there
        a = 9.9e-3
        side = max(3, int(round((4.0 * n) ** (1.0 / 3.0))))
        pos = _lattice(rng, (side, side), n, a, 0.005)
        pos[:, 2] += 4.95e-3 - 0.5 * a
        hi = np.array([side * a, side * a, pos[:, 2].max() + 0.1])
        vel = rng.normal(0.0, 0.05, size=(n, 3))
        walls = [scenes.plane_wall(side * a, [0.5 * hi[0], 0.5 * hi[1], 0.0])]
        dt = 1e-6
    elif kind == "polydisperse":
        pos, quat, shape, scale, K = _block(rng, kind, n)
        hi = np.full(3, K)
        vel = rng.normal(0.0, 0.1, size=pos.shape)
        periodic, grav = 7, 0.0
    elif kind == "settling":  # a cube: the packing without the bodies that reach through the floor or the ceiling
        pos, quat, shape, scale, K = _block(rng, kind, n)
        b = max(t["bound"] for t in T)
        # the same count for every seed: the bodies nearest to mid-height
        i = np.sort(np.argsort(np.abs(pos[:, 2] - 0.5 * K), kind="stable")[:int(len(pos) * (1.0 - 2.0 * b / K))])
        pos, quat, shape, scale = pos[i], quat[i], shape[i], scale[i]
        hi = np.full(3, K)
        vel = rng.normal(0.0, 0.02, size=pos.shape)
        periodic = 3
        walls = [scenes.plane_wall(K, [0.5 * K, 0.5 * K, 0.0]), scenes.plane_wall(K, [0.5 * K, 0.5 * K, K], up=False)]
    elif kind == "drum":  # lower two thirds of a closed drum of radius R and length 2 R about x, 30 rpm
        pos, quat, shape, scale, K = _block(rng, kind, int(1.9 * n))
        R, b = 0.5 * K, max(t["bound"] for t in T)
        pos -= R
        inside = (np.abs(pos[:, 0]) < R - 0.8 * b) & (np.hypot(pos[:, 1], pos[:, 2]) < R - 0.8 * b)
        i = np.nonzero(inside)[0]
        i = np.sort(i[np.argsort(pos[i, 2], kind="stable")[:n]])
        pos, quat, shape, scale = pos[i], quat[i], shape[i], scale[i]
        vel = np.zeros(pos.shape)
        w = scenes.drum_wall(R, 2 * R, R / 50)
        w.update(pos=np.zeros(3), quat=np.array([1.0, 0, 0, 0]), angvel=np.array([math.pi, 0, 0]))
        walls = [w]
        lo, hi = -np.full(3, R), np.full(3, R)
    else:  # bonded, bed: aligned ellipsoids on the HCP lattice mapped to their axes
        ax = np.array([2e-3, 1.6e-3, 1.2e-3])
        # contact spacing x (1 + gap): open for the bonded solid, 0.2 % compressed for the bed
        r = 0.5 * (1.05 if kind == "bonded" else 0.998)
        dx, dy, dz = 2 * r, math.sqrt(3.0) * r, math.sqrt(8.0 / 3.0) * r
        side = n ** (1.0 / 3.0)
        nx = max(2, int(round(side)))
        ny = 2 * max(1, int(round(0.5 * side)))
        nz = 2 * max(1, int(math.ceil(n / (2 * nx * ny))))
        i = np.arange(nx * ny * nz)
        ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
        u = np.stack([ix * dx + r * (iy % 2) + r * (iz % 2), iy * dy + (r / math.sqrt(3.0)) * (iz % 2), iz * dz], 1)
        period = np.array([nx * dx, ny * dy, nz * dz])
        quat = np.tile([1.0, 0, 0, 0], (n, 1))
        if kind == "bed":  # periodic in all axes: compressed alike from all sides, at rest but for a shake
            u = u[:n] + r + 1e-4 * rng.uniform(-1, 1, size=(n, 3))
            pos, hi = (u % period) * (2 * ax), period * 2 * ax
            vel = rng.normal(0.0, 2e-3, size=(n, 3))
            periodic, grav, dt = 7, 0.0, 2e-7
        else:
            d = rng.normal(size=(n, 3))
            d *= (rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(d, axis=1))[:, None]
            i, j = _lattice_neighbours(ix[:n], iy[:n], iz[:n], nx, ny, u)
            pos = (u[:n] + 0.02 * d) * (2 * ax) + 1.05 * ax
            lo, hi = -np.array([8e-3, 8e-3, 0.0]), pos.max(0) + ax * 1.05 + 8e-3
            top = pos[:, 2].max() + 1.05 * ax[2]
            ext = float(max(hi[0], hi[1]))
            walls = [scenes.plane_wall(ext, [0.5 * hi[0], 0.5 * hi[1], 0.0]),
                     dict(scenes.plane_wall(ext, [0.5 * hi[0], 0.5 * hi[1], top], up=False), vel=np.array([0, 0, -0.1]))]
            v = pos[i] - pos[j]
            L = np.linalg.norm(v, axis=1)
            k = len(i)
            bonds = {"master": i, "slave": j, "point": 0.5 * (pos[i] + pos[j]), "normal": v / L[:, None], "length": L,
                     "radius": np.full(k, float(np.prod(ax) ** (1.0 / 3.0))), "youngs": 1e8, "poisson": 0.3,
                     "tensile": 1e6 * np.exp(0.3 * rng.standard_normal(k)),
                     "cohesion": 1e6 * np.exp(0.3 * rng.standard_normal(k)), "mu": 0.0}
            dt = 2e-7
    inv_mass, inv_inertia = _material(T, shape, scale)
    return {"templates": T, "shape": shape, "scale": scale, "pos": pos, "quat": quat, "vel": vel, "inv_mass": inv_mass,
            "inv_inertia": inv_inertia, "kn": 1e5, "ks": 0.8e5, "mu": 0.5, "e": 0.6, "dt": dt, "min": lo, "max": hi,
            "gravity": np.array([0.0, 0.0, grav]), "periodic": periodic, "walls": walls, "bonds": bonds}


def _lattice_neighbours(ix, iy, iz, nx, ny, u):
    """Pairs (i < j) of HCP sites at contact distance, from the sites within one row and layer."""
    n = len(ix)
    at = np.arange(n)
    out = []
    for dz in (0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                x, y = ix + dx, iy + dy
                j = at + dx + nx * dy + nx * ny * dz
                ok = (j > at) & (j < n) & (x >= 0) & (x < nx) & (y >= 0) & (y < ny)
                i0, j0 = at[ok], j[ok]
                near = np.linalg.norm(u[i0] - u[j0], axis=1) < 1.1
                out.append((i0[near], j0[near]))
    return np.concatenate([o[0] for o in out]).astype(np.int32), np.concatenate([o[1] for o in out]).astype(np.int32)


def _mesh(case, seed):
    lsdem, scenes = _lib()
    rng = np.random.default_rng([seed, case["level"], case["n_grid"]])
    # the exponents vary, the semi-axes do not, so that every seed's grid has the same size
    ax = (2.5e-3, 1.9e-3, 1.4e-3)
    ee, en = rng.uniform(1.0 / 3.0, 1.0, size=2)
    v, f = scenes.superellipsoid_mesh(ax, float(ee), float(en), case["level"])
    return v, f, 2.0 * ax[0] / (case["n_grid"] - 5.5)


# ---------------------------------------------------------------------------
# Preparation and the measured pass

class _DeviceArray:
    """A solver's device buffer for torch, keeping the solver alive."""

    def __init__(self, solver, ptr, n, k):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (n, k), "typestr": "<f8", "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def prepare(case, seed):
    lsdem, scenes = _lib()
    if case["scene"] == "grid":
        v, f, h = _mesh(case, seed)
        return {"mesh": (v, f, h), "lsdem": lsdem}
    sc = _scene(case, seed)
    sv = lsdem.Solver(device=0)
    scenes.load_polydisperse(sv, sc)
    sv.set_precision(FORMS[case["form"]])
    sv.initialize(sc["min"], sc["max"], sc["gravity"])
    if case["form"] == "learned":
        sv.set_learned_training(clip_lo=-0.1, clip_hi=0.3, near_fraction=0.8)
        sv.train_learned_sdf(iterations=1500, batch=4096, samples=1 << 15, lr=1e-2)
        sv.set_learned_sdf(True)
    ptr = sv.device_pointers()
    n = len(sc["pos"])
    out = {k: torch.as_tensor(_DeviceArray(sv, ptr[k], n, w), device="cuda") for k, w in STATE}

    def drag(_t):
        out["force"].add_(out["vel"], alpha=-DRAG)

    return {"solver": sv, "dt": sc["dt"], "steps": case["steps"], "hook": drag if case["hook"] else None, "out": out}


def run(state):
    if "mesh" in state:
        v, f, h = state["mesh"]
        sdf, _size, _origin = state["lsdem"].mesh_grid(v, f, h)
        return {"sdf": sdf}
    state["solver"].step(state["dt"], state["steps"], hook=state["hook"])
    return state["out"]


def work(case):
    """Bytes: per particle and step, pose, velocities, force and torque read and written once and the constants
    read (448 B); per bond its frames, constants and state (450 B). The grid: mesh read, values written."""
    if case["scene"] == "grid":
        t = 20 * 4 ** case["level"]
        n = 0.6 * case["n_grid"] ** 3
        # per node: one triangle's distance and solid angle, and a search over the others
        return {"bytes": 36.0 * t + 8 * n, "flops": n * (250 + 60 * math.log2(t))}
    n, k = case["n"], case["steps"]
    bonds = 5.7 * n if case["scene"] == "bonded" else 0
    contacts = {"bed": 6.0, "falling": 0.2}.get(case["scene"], 0.05) * n
    return {"bytes": k * (448.0 * n + 450.0 * bonds + 64.0 * contacts), "flops": k * (350.0 * n + 600.0 * bonds + 400.0 * contacts)}


# ---------------------------------------------------------------------------
# The same outputs in plain 64-bit torch

def exact(case, seed):
    if case["scene"] == "grid":
        return {"sdf": _exact_grid(*_mesh(case, seed))}
    if case["scene"] != "falling":
        return None
    return _exact_falling(_scene(case, seed), case["steps"], case["hook"])


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _closest(p, a, b, c):
    """Closest point to p on each triangle (a, b, c), by the Voronoi regions of its vertices, edges and face."""
    ab, ac, bc = b - a, c - a, c - b
    d1, d2 = _dot(ab, p - a), _dot(ac, p - a)
    d3, d4 = _dot(ab, p - b), _dot(ac, p - b)
    d5, d6 = _dot(ab, p - c), _dot(ac, p - c)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    den = 1.0 / (va + vb + vc)
    x = a + ab * (vb * den)[..., None] + ac * (vc * den)[..., None]
    for hit, at in (((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0), b + bc * ((d4 - d3) / ((d4 - d3) + (d5 - d6)))[..., None]),
                    ((vb <= 0) & (d2 >= 0) & (d6 <= 0), a + ac * (d2 / (d2 - d6))[..., None]),
                    ((d6 >= 0) & (d5 <= d6), c.expand_as(x)),
                    ((vc <= 0) & (d1 >= 0) & (d3 <= 0), a + ab * (d1 / (d1 - d3))[..., None]),
                    ((d3 >= 0) & (d4 <= d3), b.expand_as(x)), ((d1 <= 0) & (d2 <= 0), a.expand_as(x))):
        x = torch.where(hit[..., None], at, x)
    return x


def _exact_grid(v, f, h):
    """Signed distance to the closed mesh at the nodes of its padded, snapped box."""
    pad = 2 * h
    lo, hi = h * np.floor((v.min(0) - pad) / h), h * np.ceil((v.max(0) + pad) / h)
    nx, ny, nz = (int(math.floor(d / h + 0.5)) + 1 for d in hi - lo)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    i = torch.arange(nx * ny * nz, device=dev)
    ijk = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1).double()
    P = torch.as_tensor(lo, device=dev) + ijk * h
    tri = torch.as_tensor(v[np.asarray(f)], device=dev)
    a, b, c = (tri[None, :, k] for k in range(3))
    out = []
    for p in P.split(max(1, 4_000_000 // len(tri))):
        p = p[:, None]
        d2 = ((p - _closest(p, a, b, c)) ** 2).sum(-1).min(1).values
        r0, r1, r2 = a - p, b - p, c - p
        l0, l1, l2 = (r.norm(dim=-1) for r in (r0, r1, r2))
        den = l0 * l1 * l2 + _dot(r0, r1) * l2 + _dot(r1, r2) * l0 + _dot(r2, r0) * l1
        angle = 2.0 * torch.atan2(_dot(r0, _cross(r1, r2)), den).sum(1)
        out.append(torch.where(angle.abs() > 2.0 * math.pi, -1.0, 1.0) * d2.sqrt())
    return torch.cat(out).cpu().numpy()


def _rot(q, v):
    t = 2.0 * _cross(q[..., 1:].expand(v.shape), v)
    return v + q[..., :1] * t + _cross(q[..., 1:].expand(v.shape), t)


def _rot_inv(q, v):
    return _rot(torch.cat([q[..., :1], -q[..., 1:]], -1), v)


def _trilinear(g, size, sdf):
    """phi and its gradient (x weight of the y and z differences truncated, the reference's rule) at grid points g;
    +1 where g is outside the grid."""
    nx, ny, nz = (int(s) for s in size)
    i = torch.floor(g)
    lim = torch.tensor([nx - 1, ny - 1, nz - 1], device=g.device)
    ok = ((i >= 0) & (i < lim)).all(-1)
    f = g - i
    i = torch.where(ok[..., None], i, torch.zeros_like(i)).long()
    b = i[..., 0] + nx * (i[..., 1] + ny * i[..., 2])
    c = [sdf[b + (k & 1) + nx * ((k >> 1) & 1) + nx * ny * (k >> 2)] for k in range(8)]
    x, y, z = f[..., 0], f[..., 1], f[..., 2]
    phi = sum(c[k] * (x if k & 1 else 1 - x) * (y if k & 2 else 1 - y) * (z if k & 4 else 1 - z) for k in range(8))
    gx = (c[1] - c[0]) * (1 - y) * (1 - z) + (c[3] - c[2]) * y * (1 - z) + (c[5] - c[4]) * (1 - y) * z + (c[7] - c[6]) * y * z
    gy = (c[2] - c[0]) * (1 - z) + (c[6] - c[4]) * z
    gz = (c[4] - c[0]) * (1 - y) + (c[6] - c[2]) * y
    return torch.where(ok, phi, torch.ones_like(phi)), torch.stack([gx, gy, gz], -1)


def _exact_falling(sc, steps, hook):
    """Ellipsoids on a floor: the step in 64 bits (half kick, drift, node-in-grid detection, linear spring and dashpot
    with tangential history, second half kick)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)
    T, W = sc["templates"][0], sc["walls"][0]
    nodes, n, dt, M = t64(T["nodes"]), len(sc["pos"]), sc["dt"], len(T["nodes"])
    x, v, q = t64(sc["pos"]), t64(sc["vel"]), t64(sc["quat"])
    q = q / q.norm(dim=1, keepdim=True)
    w, im, grav = torch.zeros_like(x), t64(sc["inv_mass"])[:, None], t64(sc["gravity"])
    I = t64(sc["inv_inertia"])
    I = torch.stack([I[:, [0, 3, 4]], I[:, [3, 1, 5]], I[:, [4, 5, 2]]], 1)
    F, N = torch.zeros_like(x), torch.zeros_like(x)
    eye = torch.eye(3, device=dev, dtype=torch.float64)
    kn, ks, mu, e = sc["kn"], sc["ks"], sc["mu"], sc["e"]
    f32 = lambda s: float(np.sqrt(np.float32(s)))
    diss = -math.log(e) / f32(math.log(e) ** 2 + math.pi ** 2)
    keys, springs = torch.empty(0, dtype=torch.long, device=dev), torch.empty(0, 3, dtype=torch.float64, device=dev)

    def spin():  # angular acceleration
        R = torch.stack([_rot(q, eye[k].expand(n, 3)) for k in range(3)], 2)
        return (R @ I @ R.transpose(1, 2) @ N[..., None])[..., 0]

    for _ in range(steps):
        v = v + (F * im + grav) * (0.5 * dt)
        w = w + spin() * (0.5 * dt)
        x = x + dt * v
        h = w * (0.5 * dt)
        q = q + torch.cat([-_dot(q[:, 1:], h)[:, None], q[:, :1] * h + _cross(h, q[:, 1:])], 1)
        q = q / q.norm(dim=1, keepdim=True)
        F, N = torch.zeros_like(x), torch.zeros_like(x)
        hits = []
        near = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist") <= 2 * T["bound"] * (1 + 1e-9)
        A, B = torch.nonzero(torch.triu(near, 1), as_tuple=True)
        inside = ((x >= t64(sc["min"])) & (x < t64(sc["max"]))).all(1)
        A, B = A[inside[B]], B[inside[B]]
        for A_, B_, xo, qo, tmpl in ((A, B, x[B], q[B], T),
                                     (torch.arange(n, device=dev), None, t64(W["pos"])[None], t64(W["quat"])[None], W)):
            if len(A_) == 0:
                continue
            p = _rot(q[A_][:, None], nodes[None].expand(len(A_), M, 3)) + x[A_][:, None]
            l = _rot_inv(qo[:, None], p - xo[:, None])
            g = (l - t64(tmpl["origin"])) / tmpl["spacing"]
            phi, grad = _trilinear(g, tmpl["size"], t64(tmpl["sdf"]))
            k, m = torch.nonzero(phi <= 0, as_tuple=True)
            if len(k) == 0:
                continue
            wall = B_ is None
            a, b = A_[k], (None if wall else B_[k])
            qb = qo.expand(len(A_), 4)[k]
            nrm = _rot(qb, grad[k, m])
            nrm = nrm / nrm.norm(dim=1, keepdim=True)
            ov = -phi[k, m][:, None]
            hits.append((a, b, m, p[k, m] + 0.5 * ov * nrm, nrm, ov))
        new_keys, new_springs = [], []
        for a, b, m, pc, nrm, ov in hits:
            wall = b is None
            key = (a * M + m) * (n + 1) + (n if wall else b)
            s = torch.zeros(len(key), 3, dtype=torch.float64, device=dev)
            if len(keys):
                at = torch.searchsorted(keys, key).clamp(max=len(keys) - 1)
                s = torch.where((keys[at] == key)[:, None], springs[at], s)
            vc = v[a] + _cross(w[a], pc - x[a])
            if not wall:
                vc = vc - v[b] - _cross(w[b], pc - x[b])
            c_kn, c_ks = (kn, ks) if wall else (0.5 * kn, 0.5 * ks)
            mass = 1.0 / (im[a] if wall else im[a] + im[b])
            root = lambda z: torch.sqrt(z.float()).double()
            cn, cs = 2 * diss * root(mass * c_kn), 2 * diss * root(mass * c_ks)
            vn = _dot(vc, nrm)[:, None] * nrm
            vs = vc - vn
            fn = c_kn * ov * nrm - cn * vn
            pr = s - _dot(s, nrm)[:, None] * nrm
            ln = pr.norm(dim=1, keepdim=True)
            pr = torch.where(ln > 1e-20, pr * (s.norm(dim=1, keepdim=True) / ln.clamp(min=1e-300)), pr)
            s = pr + vs * dt
            fs = -c_ks * s - cs * vs
            afs, afn = fs.norm(dim=1, keepdim=True), fn.norm(dim=1, keepdim=True)
            slip = (afs > 1e-20) & (afs > mu * afn)
            fs = torch.where(slip, fs * (mu * afn / afs.clamp(min=1e-300)), fs)
            s = torch.where(slip, -(fs + cs * vs) / c_ks, s)
            on = ov > 0
            s = torch.where(on, s, torch.zeros_like(s))
            f = torch.where(on, fn - c_ks * s - cs * vs, torch.zeros_like(s))
            F.index_add_(0, a, f)
            N.index_add_(0, a, _cross(pc - x[a], f))
            if not wall:
                F.index_add_(0, b, -f)
                N.index_add_(0, b, _cross(pc - x[b], -f))
            new_keys.append(key)
            new_springs.append(s)
        if new_keys:
            keys, order = torch.sort(torch.cat(new_keys))
            springs = torch.cat(new_springs)[order]
        else:
            keys, springs = keys[:0], springs[:0]
        if hook:
            F = F - DRAG * v
        v = v + (F * im + grav) * (0.5 * dt)
        w = w + spin() * (0.5 * dt)
    return {"force": F, "torque": N, "vel": v, "angvel": w, "pos": x, "quat": q}
