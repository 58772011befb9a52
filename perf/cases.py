"""The framework's work as cases that can be timed: one frame of a simulation through the
public Python facades (VBDPhysics for tet meshes, VBDClothSimulationFramework for cloth).

A frame is what a caller that owns the simulation state does per step: hand positions and
velocities to the handle, run the step, read both back (the twist, whose boundary moves with
the handle's clock, continues its own state instead). Scenes are the synthetic ones of
gaia_gb300.scenes at the sizes of the tests and the benchmark.
"""
import json
import math
import os
import shutil
import tempfile
import atexit

import numpy as np
import torch

from gaia_gb300 import VBDClothSimulationFramework, VBDPhysics, scenes

_CASES = [
    # the smallest scene of the tests (a 6^3 cube above the ground, the reference's default
    # contact detection on, default precision): launches and latency
    {"name": "drop_6_contact_mixed", "kind": "drop", "n": 6, "iterations": 10, "precision": "mixed", "contact": True},
    # the plain drop benchmark: 10^3 lattice, greedy coloring, no contact detection
    {"name": "drop_10_greedy_fp32", "kind": "drop", "n": 10, "iterations": 20, "precision": "fp32", "contact": False,
     "coloring": "greedy"},
    # the plain FP64 engine on a cube with an odd side
    {"name": "drop_13_fp64", "kind": "drop", "n": 13, "iterations": 20, "precision": "fp64", "contact": False},
    # four bodies meeting at test size (vertex-face contact, CCD and DCD live), default precision
    {"name": "cluster_contact_mixed", "kind": "cluster", "iterations": 30, "precision": "mixed"},
    # batches of independent cubes of uneven size (the benchmark's sides 4..24): a small and a large one
    {"name": "batch_24_mixed", "kind": "batch", "scenes": 24, "iterations": 20, "precision": "mixed"},
    {"name": "batch_200_fp32", "kind": "batch", "scenes": 200, "iterations": 20, "precision": "fp32"},
    # the twist: an odd mid-sized lattice in the default precision, and the benchmark's headline
    {"name": "twist_47_mixed", "kind": "twist", "n": 47, "iterations": 50, "precision": "mixed"},
    {"name": "twist_100_fp32", "kind": "twist", "n": 100, "iterations": 50, "precision": "fp32"},
    # the collision-heavy drop of the benchmark
    {"name": "collide_32_fp32", "kind": "collide", "objects": 32, "iterations": 30, "precision": "fp32"},
    # cloth over a sphere with self-contact: an odd small one, the benchmark's, and contact detection alone
    {"name": "cloth_33", "kind": "cloth", "n": 33, "iterations": 20, "precision": "fp32"},
    {"name": "cloth_512", "kind": "cloth", "n": 512, "iterations": 20, "precision": "fp32"},
    {"name": "detect_200", "kind": "detect", "n": 200, "precision": "fp32"},
]


def listed():
    return [dict(c) for c in _CASES]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop", "drop", "batch", "twist", "collide", "cloth", "detect"])
    prec = rng.choice(["mixed", "mixed", "fp32", "fp32", "dfhi"])
    if kind == "drop":
        if rng.random() < 0.25:
            return {"kind": kind, "n": rng.randint(5, 14), "iterations": rng.randint(10, 20), "precision": "fp64",
                    "contact": False}
        contact = rng.random() < 0.4
        return {"kind": kind, "n": _log_int(rng, 4, 40), "iterations": rng.randint(10, 30), "precision": prec,
                "contact": contact, "coloring": rng.choice(["tool", "greedy"])}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 6, 200), "iterations": rng.randint(10, 20), "precision": prec}
    if kind == "twist":
        return {"kind": kind, "n": _log_int(rng, 24, 80), "iterations": rng.randint(20, 50), "precision": prec}
    if kind == "collide":
        return {"kind": kind, "objects": _log_int(rng, 4, 32), "iterations": rng.randint(10, 30),
                "precision": rng.choice(["mixed", "fp32"])}
    if kind == "cloth":
        return {"kind": kind, "n": _log_int(rng, 20, 250), "iterations": rng.randint(8, 20),
                "precision": rng.choice(["fp32", "fp32", "mixed"])}
    return {"kind": kind, "n": _log_int(rng, 32, 300), "precision": "fp32"}


# ---- scenes on disk (what a user has: Models.json, Parameters.json, meshes, colorings) ----
_ROOT = None
_FILES = {}


def _key(case):
    return json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)


def _scene(case):
    """(Models.json, Parameters.json) of the case, written once per process."""
    global _ROOT
    key = _key(case)
    if key in _FILES:
        return _FILES[key]
    if _ROOT is None:
        _ROOT = tempfile.mkdtemp(prefix="gaia_cases_")
        atexit.register(shutil.rmtree, _ROOT, True)
    d = os.path.join(_ROOT, "s%d" % len(_FILES))
    os.makedirs(d)
    it, prec, kind = case.get("iterations", 20), case["precision"], case["kind"]
    if kind == "drop":
        f = scenes.drop_cube(d, n=case["n"], iterations=it, precision=prec, height=0.002,
                             coloring=case.get("coloring", "tool"),
                             collision=None if case["contact"] else scenes.NO_CONTACT)
    elif kind == "cluster":
        f = scenes.contact_cluster(d, iterations=it, precision=prec)
    elif kind == "batch":
        f = scenes.batch_cubes(d, n_scenes=case["scenes"], iterations=it, precision=prec)
    elif kind == "twist":
        f = scenes.twist_cube(d, n=case["n"], iterations=it, precision=prec, omega=0.25)
    elif kind == "collide":
        f = scenes.collision_drop(d, n_objects=case["objects"], iterations=it, precision=prec)
    else:
        f = scenes.cloth_on_sphere(d, n=case["n"], iterations=it, precision=prec, gap=0.001)
    _FILES[key] = f
    return f


def _models(case):
    with open(_scene(case)[0]) as f:
        return json.load(f)["Models"]


def _params(case):
    with open(_scene(case)[1]) as f:
        return json.load(f)


def _read_t(path):
    """Vertices (float32, as the file gives them) and tets of a .t file."""
    with open(path) as f:
        text = f.read()
    cut = text.find("Tet ")
    v = np.array(text[:cut].replace("Vertex", " ").split(), np.float64).reshape(-1, 4)[:, 1:]
    t = np.array(text[cut:].replace("Tet", " ").split(), np.int64).reshape(-1, 5)[:, 1:]
    return v.astype(np.float32), t


_MESH = {}


def _rest(model):
    """Rest positions (float32, rotated and translated as the file's model says) and tets."""
    if model["path"] not in _MESH:
        if len(_MESH) > 40:
            _MESH.clear()
        _MESH[model["path"]] = _read_t(model["path"])
    X, T = _MESH[model["path"]]
    r = np.asarray(model["rotation"], np.float64)
    a = np.linalg.norm(r)
    if a > 0:
        k, c, s = r / a, math.cos(a), math.sin(a)
        K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
        R = c * np.eye(3) + s * K + (1 - c) * np.outer(k, k)
        X = (X.astype(np.float64) @ R.T).astype(np.float32)
    return X + np.asarray(model["translation"], np.float32), T


def _state(case, seed):
    """Positions and velocities (float32, all meshes) of a frame in mid-simulation, from the
    rest positions of the scene files: each body a little deformed, moving and spinning."""
    rng = np.random.Generator(np.random.PCG64([seed, 77]))
    if case["kind"] in ("cloth", "detect"):
        n = case["n"]
        X = _read_obj(_models(case)[0]["path"])
        i, j = np.arange(n * n) % n, np.arange(n * n) // n
        ph = rng.uniform(0, 2 * math.pi, 4)
        fold = 4e-3 * (np.sin(2 * math.pi * 5 * i / n + ph[0]) + np.sin(2 * math.pi * 4 * j / n + ph[1]))
        X[:, 1] += fold + 8e-3 + rng.uniform(-2e-4, 2e-4, len(X))
        V = rng.uniform(-0.02, 0.02, X.shape)
        V[:, 1] -= 0.5
        return X, V
    xs, vs = [], []
    rests = [_rest(m)[0].astype(np.float64) for m in _models(case)]
    for m, X in zip(_models(case), rests):
        c = X.mean(0)
        A = rng.uniform(-0.01, 0.01, (3, 3))
        if case["kind"] == "twist":
            A *= 0.02
        x = X + (X - c) @ A.T + rng.uniform(-2e-5, 2e-5, X.shape)
        w = rng.uniform(-1, 1, 3) * (0.0 if case["kind"] == "twist" else 1.0)
        v = np.cross(w, X - c) + rng.uniform(-1e-3, 1e-3, X.shape)
        if case["kind"] in ("drop", "batch"):
            x[:, 1] -= x[:, 1].min() + rng.uniform(0, 5e-4)  # the lowest vertices in the ground
            v += np.array([rng.uniform(-0.3, 0.3), -0.5, rng.uniform(-0.3, 0.3)])
        elif case["kind"] == "cluster":
            if xs:  # each body falls on the one below within the step
                x[:, 1] += xs[-1][:, 1].max() + 1e-3 - x[:, 1].min()
            v[:, 1] -= 2.0 * len(xs)
        elif case["kind"] == "collide":
            v[:, 1] -= 0.2
            # a ball (odd) whose nearest neighbour is a cube has come close to it and touches it
            near = np.argsort([np.linalg.norm(q.mean(0) - c) - np.ptp(q, 0).max() / 2 for q in rests])
            k = int([j for j in near if j != len(xs)][0])
            if len(xs) % 2 and k % 2 == 0:
                u = (rests[k].mean(0) - c) / np.linalg.norm(rests[k].mean(0) - c)
                x += (((rests[k] - c) @ u).min() - ((x - c) @ u).max() - 1e-3) * u
                v += 0.6 * u
        if case["kind"] == "twist":
            v = np.zeros_like(x)
            x[m["fixedPoints"]] = X[m["fixedPoints"]]
        xs.append(x)
        vs.append(v)
    return np.concatenate(xs).astype(np.float32), np.concatenate(vs).astype(np.float32)


def _read_obj(path):
    with open(path) as f:
        return np.array([ln.split()[1:4] for ln in f if ln.startswith("v ")], np.float64)


class _State:
    pass


def prepare(case, seed):
    mp, pp = _scene(case)
    s = _State()
    s.kind = case["kind"]
    x, v = _state(case, seed)
    if s.kind in ("cloth", "detect"):
        s.sim = VBDClothSimulationFramework()
        s.sim.loadRunningparameters(mp, pp)
        s.sim.initialize()
        s.x, s.v = x, v
        return s
    s.sim = VBDPhysics()
    s.sim.loadRunningparameters(mp, pp)
    s.sim.initialize()
    n = len(x)
    s.x, s.v = (torch.from_numpy(a).contiguous().pin_memory() for a in (x, v))
    s.xo, s.vo = (torch.empty(n, 3, dtype=torch.float32).pin_memory() for _ in range(2))
    if s.kind == "twist":
        s.sim.set_state_f32(s.x.data_ptr(), s.v.data_ptr())
        s.sim.synchronize()
    return s


def run(s):
    sim = s.sim
    if s.kind == "detect":
        sim.setPositions(0, s.x)
        sim.applyCollisionDetection()
        vf, fv, ee = sim.minDistances(0)
        return {"bounds": sim.conservativeBounds(0), "vf": vf, "fv": fv, "ee": ee}
    if s.kind == "cloth":
        sim.setPositions(0, s.x)
        sim.setVelocities(0, s.v)
        sim.runStep(1)
        return {"x": sim.positions(0).astype(np.float32), "v": sim.velocities(0).astype(np.float32)}
    if s.kind != "twist":
        sim.set_state_f32(s.x.data_ptr(), s.v.data_ptr())
    sim.runStep(1)
    sim.get_positions_f32(s.xo.data_ptr())
    sim.get_velocities_f32(s.vo.data_ptr())
    return {"x": s.xo, "v": s.vo}


def _counts(case):
    """(vertices, tets or faces) of all meshes."""
    if case["kind"] in ("cloth", "detect"):
        n = case["n"]
        return n * n, 2 * (n - 1) ** 2
    nv = nt = 0
    for m in _models(case):
        X, T = _rest(m)
        nv += len(X)
        nt += len(T)
    return nv, nt


def work(case):
    """State in and out and the mesh once (a vertex's rest position and mass, a tet's vertices
    and inverse rest shape, a face's likewise); per iteration and vertex-tet incidence the
    element force and 3x3 Hessian (about 150 operations), per vertex the 3x3 solve."""
    nv, nt = _counts(case)
    b = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "detect":
        # positions and faces in, the distances out; per vertex and per edge (3 nv) about 30
        # candidate pairs of a closest-point test of about 100 operations
        return {"bytes": nv * 12 + nt * 12 + (2 * nv + nt + 3 * nv) * 4, "flops": 4 * nv * 30 * 100}
    it = case["iterations"]
    if case["kind"] == "cloth":
        # per vertex 6 membrane faces and about 45 active contact pairs of 200 operations
        return {"bytes": nv * 48 + nt * (12 + 20), "flops": it * nv * (6 * 150 + 45 * 200)}
    return {"bytes": nv * (24 + 24 + 16) + nt * (16 + 9 * b), "flops": it * (4 * nt * 150 + nv * 100)}


# ---- the step in 64 bits ---------------------------------------------------------------
def _colors(m):
    """Vertex lists of a model's colors, largest first (equal sizes in the file's order)."""
    with open(m["verticesColoringCategoriesPath"]) as f:
        c = json.load(f)
    return sorted((np.asarray(x, np.int64) for x in c), key=lambda a: -len(a))


def exact(case, seed):
    """One VBD step (block Gauss-Seidel over the colors) in float64 for the scenes without
    contact between bodies; contact sets and cloth have no plain restatement here."""
    if case["kind"] not in ("drop", "batch", "twist") or case.get("contact"):
        return None
    dev = "cuda"
    F = torch.float64
    P = _params(case)
    p = P["PhysicsParams"]
    dt = p["timeStep"] / p["numSubsteps"]
    g = torch.tensor(p["gravity"], dtype=F, device=dev)
    lo, hi = (torch.tensor(b, dtype=F, device=dev) for b in p["worldBounds"])
    x_np, v_np = _state(case, seed)
    rests, tets, mus, lmbds, masses, fixed, steps = [], [], [], [], [], [], {}
    off = 0
    for m in _models(case):
        X, T = _rest(m)
        rests.append(X.astype(np.float64))
        tets.append(T + off)
        mus.append(np.full(len(T), m["miu"]))
        lmbds.append(np.full(len(T), m["lmbd"]))
        fx = np.zeros(len(X), bool)
        fx[m["fixedPoints"]] = True
        fixed.append(fx)
        masses.append(np.full(len(T), m["density"]))
        # a model's colors, largest first, go to the merged steps with the fewest vertices so far
        free = list(range(len(_colors(m))))
        for c in _colors(m):
            k = min(free, key=lambda q: (sum(map(len, steps.get(q, []))), free.index(q)))
            free.remove(k)
            steps.setdefault(k, []).append(c + off)
        off += len(X)
    cat = lambda a, t=F: torch.as_tensor(np.concatenate(a), dtype=t, device=dev)  # noqa: E731
    X, T, mu, lm, rho = cat(rests), cat(tets, torch.long), cat(mus), cat(lmbds), cat(masses)
    fx = cat(fixed, torch.bool)
    nv = len(X)
    for d in P.get("Deformers", []):
        fx[torch.as_tensor(d["selectedVertices"][0], device=dev)] = True
    Dm = torch.stack([X[T[:, k]] - X[T[:, 0]] for k in (1, 2, 3)], 2)
    Di = torch.linalg.inv(Dm)
    A = torch.linalg.det(Dm) / 6
    mass = torch.zeros(nv, dtype=F, device=dev)
    for k in range(4):
        mass.index_add_(0, T[:, k], 0.25 * A * rho)
    rows = torch.cat([-Di.sum(1, keepdim=True), Di], 1)  # dF/dx row of each of the 4 vertices
    del Dm
    x = torch.as_tensor(x_np, dtype=F, device=dev)
    v = torch.as_tensor(v_np, dtype=F, device=dev)
    x0 = x.clone()
    v = v + dt * g
    v[fx] = 0
    y = x + dt * v
    x = y.clone()
    for d in P.get("Deformers", []):
        sel = torch.as_tensor(d["selectedVertices"][0], device=dev)
        th = dt * d["angularVelocity"]
        ax = torch.tensor(d["axis"], dtype=F, device=dev)
        op = X[sel] - torch.tensor(d["center"], dtype=F, device=dev)
        root = (op @ ax)[:, None] * ax
        q = X[sel] - root
        x[sel] = root + q * math.cos(th) + torch.linalg.cross(ax.expand_as(q), q) * math.sin(th) \
            + (q @ ax)[:, None] * ax * (1 - math.cos(th))
    # incidences (tet, local vertex) by vertex
    iv = T.reshape(-1)
    order = torch.argsort(iv, stable=True)
    ptr = torch.zeros(nv + 1, dtype=torch.long, device=dev)
    ptr[1:] = torch.cumsum(torch.bincount(iv, minlength=nv), 0)
    mub, epsU, kb = p["boundaryFrictionDynamic"], p["boundaryFrictionEpsV"] * dt, p["boundaryCollisionStiffness"]
    plan = []
    for k in sorted(steps):
        c = torch.as_tensor(np.concatenate(steps[k]), device=dev)
        c = c[~fx[c]]
        cnt = ptr[c + 1] - ptr[c]
        own = torch.repeat_interleave(torch.arange(len(c), device=dev), cnt)
        at = order[torch.arange(len(own), device=dev) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
                   + torch.repeat_interleave(ptr[c], cnt)]
        t, l = at // 4, at % 4
        plan.append((c, own, t, rows[t, l]))
    eye = torch.eye(3, dtype=F, device=dev)
    chunk = 1 << 20  # incidences evaluated at a time
    for _ in range(p["iterations"]):
        for c, own, t, mo in plan:
            f = torch.zeros(len(c), 3, dtype=F, device=dev)
            H = torch.zeros(len(c), 9, dtype=F, device=dev)
            for b in range(0, len(own), chunk):
                tt, o, r = t[b:b + chunk], own[b:b + chunk], mo[b:b + chunk]
                Tt = T[tt]
                Fm = torch.eye(3, dtype=F, device=dev) + torch.einsum("nkr,nkc->nrc", x[Tt] - X[Tt], rows[tt])
                cof = torch.stack([torch.linalg.cross(Fm[:, 1], Fm[:, 2]), torch.linalg.cross(Fm[:, 2], Fm[:, 0]),
                                   torch.linalg.cross(Fm[:, 0], Fm[:, 1])], 1)
                J = (Fm[:, 0] * cof[:, 0]).sum(1)
                ge = torch.einsum("nrc,nc->nr", cof, r)
                a = 1 + mu[tt] / lm[tt]
                fe = -A[tt, None] * (mu[tt, None] * torch.einsum("nrc,nc->nr", Fm, r)
                                     + (lm[tt] * (J - a))[:, None] * ge)
                He = (A[tt] * lm[tt])[:, None, None] * ge[:, :, None] * ge[:, None, :] \
                    + (A[tt] * mu[tt] * (r * r).sum(1))[:, None, None] * eye
                f.index_add_(0, o, fe)
                H.index_add_(0, o, He.reshape(-1, 9))
            H = H.reshape(-1, 3, 3)
            w = mass[c] / (dt * dt)
            xc, dx = x[c], x[c] - x0[c]
            f = f + w[:, None] * (y[c] - xc)
            H = H + w[:, None, None] * eye
            if p["usePlaneGround"]:
                for d in range(3):
                    below, above = lo[d] - xc[:, d], xc[:, d] - hi[d]
                    pen = torch.where(below > 0, below, torch.where(above > 0, above, torch.zeros_like(below)))
                    hit = (pen > 0).to(F)
                    f[:, d] += torch.where(below > 0, pen, -pen) * kb
                    H[:, d, d] += hit * kb
                    a1, a2 = (d + 1) % 3, (d + 2) % 3
                    un = torch.sqrt(dx[:, a1] ** 2 + dx[:, a2] ** 2)
                    f1 = torch.where(un > epsU, 1 / un.clamp_min(1e-300), (-un / epsU + 2) / epsU)
                    s = torch.where(un > 0, mub * pen * kb * f1, torch.zeros_like(un))
                    for q in (a1, a2):
                        f[:, q] -= s * dx[:, q]
                        H[:, q, q] += s
            step = torch.linalg.solve(H, f[:, :, None])[:, :, 0]
            still = (f * f).sum(1) <= 1e-10
            step[still] = 0
            x[c] = xc + p["stepSize"] * step
    v = (x - x0) / dt
    vm = torch.linalg.norm(v, dim=1)
    v[vm <= 1e-6] = 0
    v[fx] = 0
    return {"x": x.cpu(), "v": v.cpu()}
