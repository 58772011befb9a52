"""The FP32-compute force of rotated and flattened one-rings: no further from the FP64 engine's
than the same sum written per tet with the stored rows of dF/dx (P = mu (G - Cg) + lambda dJ
cof F from the entries of G = F - I), evaluated in float32 on the same state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rotation(axis, angle):
    k = np.asarray(axis, float) / np.linalg.norm(axis)
    K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
    return np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K


def _mesh(flat, seed):
    """Tets of random points (the badly shaped ones left out), flattened across a slanted axis."""
    from scipy.spatial import Delaunay

    rng = np.random.Generator(np.random.PCG64(seed))
    X = rng.uniform(-0.1, 0.1, (300, 3))
    T = Delaunay(X).simplices.astype(np.int32)
    D = X[T[:, 1:]] - X[T[:, :1]]
    edges = np.concatenate([D, D[:, 1:] - D[:, :1], D[:, 2:] - D[:, 1:2]], 1)
    vol = np.linalg.det(D)
    T = T[np.abs(vol) > 0.03 * np.linalg.norm(edges, axis=2).max(1) ** 3]
    used, T = np.unique(T, return_inverse=True)
    X, T = X[used], T.reshape(-1, 4).astype(np.int32)
    Q = _rotation([1.0, 2.0, -1.0], 0.7)
    X = ((X @ Q.T) * [1.0, 1.0, flat]) @ Q
    neg = np.linalg.det(X[T[:, 1:]] - X[T[:, :1]]) < 0
    T[neg, 2], T[neg, 3] = T[neg, 3].copy(), T[neg, 2].copy()
    return X, T


def _row_form(u, T, rows, vol, mu, lm):
    """Elastic force of every vertex in float32 from float32 rows of dF/dx."""
    F = np.float32
    m = rows.astype(F)
    f = np.zeros((len(u), 3), F)
    for o in range(4):
        oth = [j for j in range(4) if j != o]
        G = np.zeros((len(T), 3, 3), F)
        for j in oth:
            e = u[T[:, j]] - u[T[:, o]]
            G += e[:, :, None] * m[:, j, None, :]
        mo = -((m[:, oth[0]] + m[:, oth[1]]) + m[:, oth[2]])
        g = [[G[:, r, c] for c in range(3)] for r in range(3)]
        one = F(1)
        C = np.empty_like(G)
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3
            C[:, i, i] = (g[j][j] + g[k][k]) + (g[j][j] * g[k][k] - g[j][k] * g[k][j])
            C[:, i, j] = g[j][k] * g[k][i] - g[j][i] * (one + g[k][k])
            C[:, i, k] = g[j][i] * g[k][j] - (one + g[j][j]) * g[k][i]
        dJ = ((g[0][0] * (one + C[:, 0, 0]) + g[0][1] * C[:, 0, 1]) + g[0][2] * C[:, 0, 2]) + C[:, 0, 0]

        def times(M):
            return (M[:, :, 0] * mo[:, :1] + M[:, :, 1] * mo[:, 1:2]) + M[:, :, 2] * mo[:, 2:]

        cm = times(C)
        A = vol.astype(F)[:, None]
        fe = -((A * F(mu)) * (times(G) - cm) + (A * F(lm)) * dJ[:, None] * (mo + cm))
        np.add.at(f, T[:, o], fe)  # in tet order, one after another
    return f


# The bound is the row form itself: the error of a vertex's step (the FP64 block solved for the
# force error), averaged over the mesh, may not be larger.
@pytest.mark.parametrize("lanes", [4, 32])
@pytest.mark.parametrize("flat,angle", [(1.0, 0.3), (1.0, 2.0), (0.2, 0.3), (0.1, 2.0), (0.02, 1.0)])
def test_force_of_rotated_flat_rings(tmp_path, gaia_lib, flat, angle, lanes):
    from gaia_gb300 import VBDPhysics, scenes

    X, T = _mesh(flat, 5)
    tp, cp = scenes._write_mesh(str(tmp_path), "ring", X, T, coloring="greedy")
    model = scenes.model_entry(tp, cp, E=1e6, nu=0.45, density=1e-6)
    params = scenes.physics_params(1.0 / 300.0, 4, precision="fp64", ground_y=-50.0)
    mp, pp = scenes._write_json(str(tmp_path), [model], params, collision=scenes.NO_CONTACT)
    rng = np.random.Generator(np.random.PCG64(9))
    out, step = {}, {}
    for precision in ("fp64", "mixed", "fp32", "dfhi"):
        phys = VBDPhysics()
        phys.loadRunningparameters(mp, scenes.set_precision(pp, precision, out_path="%s.%s.json" % (pp, precision),
                                                            autotune=False, lanesPerVertex=lanes,
                                                            smallColorVertices=0))
        phys.initialize()
        if precision == "fp64":
            rest = phys.positions(0)
            x = rest @ _rotation([0.3, -1.0, 0.5], angle).T
            x = x + (x - x.mean(0)) @ rng.uniform(-1e-3, 1e-3, (3, 3)).T
            u = (x - rest).astype(np.float32)  # a displacement that every mode holds exactly
            dm, vol, _ = phys.restShape(0)
        phys.setPositions(0, rest + u.astype(float))
        fh = [phys.vertexForceHessian(0, v, False) for v in range(len(rest))]
        phys.close()
        out[precision] = np.array([f for f, _ in fh])
        if precision == "fp64":
            H = np.array([h for _, h in fh])
    D = np.swapaxes(np.asarray(dm).reshape(-1, 3, 3), 1, 2)
    rows = np.concatenate([-D.sum(1, keepdims=True), D], 1)
    mu, lm = model["miu"], model["lmbd"]
    out["rows"] = _row_form(u, T, rows, np.asarray(vol), mu, lm).astype(float)
    for k in ("mixed", "fp32", "dfhi", "rows"):
        step[k] = np.linalg.norm(np.linalg.solve(H, (out[k] - out["fp64"])[:, :, None])[:, :, 0], axis=1)
    print(f"flat {flat} angle {angle} lanes {lanes}:", {k: "%.3f" % (v.mean() / step["rows"].mean()) for k, v in step.items()})
    for k in ("mixed", "fp32", "dfhi"):
        assert step[k].mean() <= step["rows"].mean(), k
