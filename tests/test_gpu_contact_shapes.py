"""Contact terms in every solve kernel: lanes per vertex, kernel variants, programmatic launches,
the accelerator and repeated detection (whose snapshots alternate), against the FP64 oracle; and
the world-box test at its margin."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ITERATIONS = 10


@pytest.fixture(scope="module")
def cluster(tmp_path_factory, gaia_lib):
    """Two cubes and two balls colliding in a column, and the oracle's end state per setting."""
    from gaia_gb300 import scenes
    from oracle import oracle as orc
    from oracle import scene_io

    d = tmp_path_factory.mktemp("cluster")
    mp, pp = scenes.contact_cluster(str(d), precision="fp64", iterations=ITERATIONS)
    nm = len(json.load(open(mp))["Models"])
    ends = {}

    def end(**over):
        key = json.dumps(over, sort_keys=True)
        if key not in ends:
            p = scenes.set_precision(pp, "fp64", out_path="%s.o%d.json" % (pp, len(ends)), **over)
            o = orc.OracleScene(scene_io.load_scene(mp, p), precision=64, nthreads=0)
            x0 = np.concatenate([o.positions(m) for m in range(nm)])
            rows = 0
            for _ in range(20):
                o.step(1)
                rows += len(o.contacts())
            assert rows > 50
            ends[key] = (x0, np.concatenate([o.positions(m) for m in range(nm)]))
        return ends[key]

    return mp, pp, nm, end


def _run(cluster, precision, name, **over):
    from gaia_gb300 import VBDPhysics, scenes

    mp, pp, nm, _ = cluster
    phys = VBDPhysics()
    phys.loadRunningparameters(mp, scenes.set_precision(pp, precision, out_path=f"{pp}.{name}.json", autotune=False,
                                                        smallColorVertices=0, blockSize=128, **over))
    phys.initialize()
    phys.runStep(20)
    x = np.concatenate([phys.positions(m) for m in range(nm)])
    st = phys.stats()
    phys.close()
    assert st["device_timeouts"] == 0 and st["nonfinite_solves"] == 0
    return x


# FP64 1e-8 and FP32 compute 1e-4, the bounds of the other contact trajectories
SHAPES = [("mixed", L, v) for L in (2, 4, 8, 16, 32) for v in (0, 1, 4, 6, 7)] + \
         [("fp64", L, v) for L in (2, 4, 8, 16, 32) for v in (0, 4)] + [("fp32", L, 0) for L in (2, 8, 32)]


@pytest.mark.parametrize("precision,lanes,variant", SHAPES)
def test_every_shape(cluster, precision, lanes, variant):
    x0, xo = cluster[3]()
    x = [_run(cluster, precision, "s", lanesPerVertex=lanes, solveVariant=variant, usePDL=pdl) for pdl in (True, False)]
    np.testing.assert_array_equal(x[0], x[1])
    rel = np.linalg.norm(x[0] - xo) / np.linalg.norm(xo - x0)
    assert rel <= (1e-8 if precision == "fp64" else 1e-4), rel


# detections at every iteration, every second and every third: after odd and even iterations
@pytest.mark.parametrize("every", [1, 2, 3])
@pytest.mark.parametrize("accelerator", [False, True])
@pytest.mark.parametrize("lanes", [4, 32])
def test_repeated_detection_and_accelerator(cluster, every, accelerator, lanes):
    over = {"intermediateCollisionIterations": every}
    if accelerator:
        over.update(useAccelerator=True, acceleratorRho=0.9)
    x0, xo = cluster[3](**over)
    x = _run(cluster, "fp64", "r", lanesPerVertex=lanes, solveVariant=0, **over)
    rel = np.linalg.norm(x - xo) / np.linalg.norm(xo - x0)
    assert rel <= 1e-8, rel


# Distances that each mode's state holds beside a wall at 0.375: FP32 two units in the last
# place of the wall, the others far below one.
@pytest.mark.parametrize("precision,delta", [("fp64", 1e-14), ("mixed", 1e-9), ("dfhi", 1e-9), ("fp32", 6e-8)])
@pytest.mark.parametrize("frames", [True, False])
def test_wall_at_its_margin(tmp_path, gaia_lib, precision, delta, frames):
    """The stiffness of the world box enters exactly where the vertex is past the wall."""
    from gaia_gb300 import VBDPhysics, scenes

    big = 1e30
    X, T = scenes.lattice_cube((3, 3, 3), 0.125, (0.375, 0.375, 0.375))[:2]
    tp, cp = scenes._write_mesh(str(tmp_path), "cube", X, T, coloring="greedy")

    def open_(bounds, plane=True):
        params = scenes.physics_params(1.0 / 300.0, 2, precision=precision, worldBounds=bounds, usePlaneGround=plane)
        mp, pp = scenes._write_json(str(tmp_path), [scenes.model_entry(tp, cp)], params, collision=scenes.NO_CONTACT)
        phys = VBDPhysics()
        phys.loadRunningparameters(mp, scenes.set_precision(pp, precision, autotune=False, meshFrames=frames))
        phys.initialize()
        return phys, params["boundaryCollisionStiffness"]

    wall = 0.375  # the rest position of vertex 0, on all three axes
    lo_box, hi_box = [[wall] * 3, [big] * 3], [[-big] * 3, [wall] * 3]
    free = open_([[-1e300] * 3, [1e300] * 3])[0]
    none = open_(lo_box, plane=False)[0]
    for bounds, side in ((lo_box, 1.0), (hi_box, -1.0)):
        phys, kb = open_(bounds)
        for d in range(3):
            for past in (-1.0, 0.0, 1.0):
                x = phys.positions(0)
                x[0] = wall + side * 1e-3
                x[0, d] = wall - side * past * delta
                H = []
                for p in (phys, free, none):
                    p.setPositions(0, x)
                    f, h = p.vertexForceHessian(0, 0, False)
                    assert np.isfinite(f).all() and np.isfinite(h).all()
                    H.append(h)
                want = np.zeros((3, 3))
                want[d, d] = kb if past > 0 else 0.0
                np.testing.assert_array_equal(H[1], H[2])
                np.testing.assert_allclose(H[0] - H[2], want, rtol=0, atol=1e-6 * np.abs(H[2]).max())
        phys.close()
    free.close()
    none.close()
