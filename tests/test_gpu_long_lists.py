"""Vertices with long neighbour lists beside ordinary ones: solved a warp per vertex, the
others as without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(d, precision, rings, side=9, **over):
    """A lattice cube and, beside it, one fan per entry of rings (a hub of ring + 2 neighbours)."""
    from gaia_gb300 import scenes
    from test_gpu_one_ring import _fan

    d.mkdir(exist_ok=True)
    X, T = scenes.lattice_cube((side,) * 3, 0.01, (0.0, 0.0, 0.0))[:2]
    models = []
    for k, (X, T) in enumerate([(X, T)] + [_fan(n, False) for n in rings]):
        tp, cp = scenes._write_mesh(str(d), f"m{k}", X + [0.3 * k, 0.06, 0.0], T, coloring="greedy")
        models.append(scenes.model_entry(tp, cp, initialVelocity=[0.1, -0.4, 0.05]))
    params = scenes.physics_params(1.0 / 300.0, 10, precision=precision, ground_y=0.05)
    mp, pp = scenes._write_json(str(d), models, params, collision=scenes.NO_CONTACT)
    return mp, scenes.set_precision(pp, precision, **over)


def _open(mp, pp):
    from gaia_gb300 import VBDPhysics

    phys = VBDPhysics()
    phys.loadRunningparameters(mp, pp)
    phys.initialize()
    return phys


# rings of 40, 100 (more than 32 and 64 neighbours) and 200 (several segments); FP64 and FP32
# parity bounds as in the other parity tests. blockSize 64 and 128: warps of both kinds of list
# share the staging areas.
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-5), ("fp32", 1e-5)])
@pytest.mark.parametrize("sweep,lanes,variant", [("merged", 4, 0), ("merged", 8, 4), ("merged", 2, 6), ("merged", 4, 1),
                                                 ("merged", 4, 7), ("merged", 32, 0), ("scenes", 4, -1),
                                                 ("scenes", 16, -1), ("grid", 2, -1), ("grid", 8, -1),
                                                 ("cluster", 4, -1), ("cluster", 32, -1)])
def test_hubs_beside_a_lattice(tmp_path, gaia_lib, oracle_lib, precision, tol, sweep, lanes, variant):
    from oracle import oracle as orc
    from oracle import scene_io

    mp, pp = _scene(tmp_path / "s", precision, [40, 100, 200], sweepMode=sweep, lanesPerVertex=lanes,
                    blockSize=64 if lanes == 8 else 128, solveVariant=variant, autotune=False, smallColorVertices=0)
    phys = _open(mp, pp)
    o = orc.OracleScene(scene_io.load_scene(mp, pp), precision=64, nthreads=2)
    x0 = [phys.positions(m) for m in range(4)]
    phys.runStep(6)
    o.step(6)
    st = phys.stats()
    assert st["failed_solves"] == 0 and st["device_timeouts"] == 0
    for m in range(4):
        x, xo = phys.positions(m), o.positions(m)
        assert np.linalg.norm(x - xo) <= tol * np.linalg.norm(xo - x0[m]), m
    f, H = phys.vertexForceHessian(3, 0, False)
    assert np.isfinite(f).all() and np.linalg.eigvalsh(H)[0] > 0
    phys.close()


def test_one_hub_does_not_slow_a_large_scene(tmp_path, gaia_lib):
    """A 40^3 lattice at four lanes per vertex with and without one hub of 202 neighbours: the
    hub adds a launch to its color, two to three microseconds of about ten per color."""
    ms = []
    for rings in ([], [200]):
        mp, pp = _scene(tmp_path / f"s{len(rings)}", "fp32", rings, side=40, sweepMode="merged", lanesPerVertex=4,
                        blockSize=128, solveVariant=0, autotune=False, smallColorVertices=0)
        phys = _open(mp, pp)
        phys.runStep(3)
        phys.synchronize()
        ms.append(min(phys.run_steps_timed(5, False)[0] for _ in range(5)))
        phys.close()
    print("40^3 with and without a hub:", ms)
    assert ms[1] <= 1.5 * ms[0]
