"""The one-ring form of the vertex block: vertices with many neighbours (lists cut into
segments), lists around the lane counts, and tets of negative rest volume, against the FP64
oracle in every schedule."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(n, flip):
    """A hub joined to a ring of n vertices and two poles: 2 n tets at the hub, which has
    n + 2 neighbours. flip: every second tet's vertices are ordered to a negative volume."""
    a = 2 * np.pi * np.arange(n) / n
    rng = np.random.Generator(np.random.PCG64(n))
    ring = np.stack([np.cos(a), 0.1 * np.sin(3 * a), np.sin(a)], 1) * 0.05
    X = np.concatenate([[[0, 0, 0], [0, 0.05, 0], [0, -0.05, 0]], ring]) + rng.uniform(-1e-4, 1e-4, (n + 3, 3))
    T = []
    for k in range(n):
        i, j = 3 + k, 3 + (k + 1) % n
        T += [[0, i, 1, j], [0, i, j, 2]]
    T = np.array(T, np.int32)
    d = X[T[:, 1:]] - X[T[:, :1]]
    neg = np.einsum("ij,ij->i", d[:, 0], np.cross(d[:, 1], d[:, 2])) < 0
    want = np.zeros(len(T), bool)
    if flip:
        want[::2] = True
    sw = neg != want
    T[sw, 2], T[sw, 3] = T[sw, 3].copy(), T[sw, 2].copy()
    return X, T


def _scene(d, n, flip, precision, **over):
    from gaia_gb300 import scenes

    X, T = _fan(n, flip)
    tp, cp = scenes._write_mesh(str(d), "fan", X, T, coloring="greedy")
    models = [scenes.model_entry(tp, cp, fixedPoints=[3], initialVelocity=[0.1, 0.0, 0.05])]
    params = scenes.physics_params(1.0 / 300.0, 8, precision=precision, ground_y=-0.05)
    mp, pp = scenes._write_json(str(d), models, params, collision=scenes.NO_CONTACT)
    return mp, scenes.set_precision(pp, precision, **over)


# rel. error bounds: FP64 is a rearrangement of the same sums (1e-9, as the other parity
# tests); FP32-compute modes at the FP32 parity bound (1e-5). The hub's block sums up to 800
# incidences. Negative volumes give a negative mass, so only the force block is compared there.
@pytest.mark.parametrize("n", [4, 30, 126, 127, 200, 400])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-5)])
@pytest.mark.parametrize("sweep", ["merged", "scenes", "cluster", "grid"])
def test_hub_of_many_tets(tmp_path, gaia_lib, oracle_lib, n, precision, tol, sweep):
    from gaia_gb300 import VBDPhysics
    from oracle import oracle as orc
    from oracle import scene_io

    mp, pp = _scene(tmp_path, n, False, precision, sweepMode=sweep)
    phys = VBDPhysics()
    phys.loadRunningparameters(mp, pp)
    phys.initialize()
    o = orc.OracleScene(scene_io.load_scene(mp, pp), precision=64, nthreads=2)
    x0 = phys.positions(0)
    phys.runStep(5)
    o.step(5)
    x, xo = phys.positions(0), o.positions(0)
    st = phys.stats()
    phys.close()
    assert st["failed_solves"] == 0 and st["device_timeouts"] == 0
    assert np.linalg.norm(x - xo) <= tol * np.linalg.norm(xo - x0)


@pytest.mark.parametrize("n", [5, 200])
def test_force_and_hessian_with_negative_volumes(tmp_path, gaia_lib, n):
    """The hub's force and Hessian of a deformed fan against the dense sum over its tets."""
    from gaia_gb300 import VBDPhysics

    mp, pp = _scene(tmp_path, n, True, "fp64")
    with open(mp) as f:
        m = json.load(f)["Models"][0]
    phys = VBDPhysics()
    phys.loadRunningparameters(mp, pp)
    phys.initialize()
    T = _fan(n, True)[1]
    X = phys.positions(0)  # the rest positions as the mesh file gives them
    rng = np.random.Generator(np.random.PCG64(3))
    x = X + rng.uniform(-2e-3, 2e-3, X.shape)
    phys.setPositions(0, x)
    x = phys.positions(0)
    f, H = phys.vertexForceHessian(0, 0, False)
    dm, vol, mass = phys.restShape(0)
    phys.close()
    assert (vol < 0).sum() >= n // 2
    fr, Hr = np.zeros(3), np.zeros((3, 3))
    for t in range(len(T)):
        D = dm[t].reshape(3, 3).T
        rows = np.concatenate([-D.sum(0, keepdims=True), D])
        F = np.eye(3) + (x[T[t]] - X[T[t]]).T @ rows
        g = np.linalg.det(F) * np.linalg.inv(F).T @ rows[0]
        a = 1 + m["miu"] / m["lmbd"]
        fr -= vol[t] * (m["miu"] * F @ rows[0] + m["lmbd"] * (np.linalg.det(F) - a) * g)
        Hr += vol[t] * (m["lmbd"] * np.outer(g, g) + m["miu"] * rows[0] @ rows[0] * np.eye(3))
    # the inertia term's part: the probe's inertia target is the rest position at time zero
    w = mass[0] * 300.0 ** 2
    fr += w * (X[0] - x[0])
    Hr += w * np.eye(3)
    # the summands are up to mu A |m| each; the sums cancel, so the bound is relative to them
    scale = np.abs(vol).sum() * m["miu"] / 0.05 * 10
    assert np.abs(f - fr).max() <= 1e-9 * max(scale, np.abs(fr).max())
    assert np.abs(H - Hr).max() <= 1e-9 * np.abs(Hr).max()
