"""What is reported of a launch is what runs: lanes per vertex, threads and variant where the
requested ones do not fit a block's shared memory."""
import pytest

pytestmark = pytest.mark.gpu


def _open(mp, pp, **over):
    from gaia_gb300 import VBDPhysics, scenes

    phys = VBDPhysics()
    phys.loadRunningparameters(mp, scenes.set_precision(pp, "mixed", out_path=pp + ".e.json", autotune=False,
                                                        smallColorVertices=0, **over))
    phys.initialize()
    return phys


def _fan(d, n):
    from gaia_gb300 import scenes
    from test_gpu_one_ring import _fan as fan

    X, T = fan(n, False)
    tp, cp = scenes._write_mesh(str(d), "fan", X, T, coloring="greedy")
    mp, pp = scenes._write_json(str(d), [scenes.model_entry(tp, cp)], scenes.physics_params(1.0 / 300.0, 4, precision="mixed"),
                                collision=scenes.NO_CONTACT)
    return mp, pp


def test_lanes_that_do_not_fit(tmp_path, gaia_lib):
    """62 neighbours of 48 bytes at two lanes per vertex are 372 KB a block of 256 threads, at
    four 186 KB."""
    mp, pp = _fan(tmp_path, 60)
    phys = _open(mp, pp, sweepMode="merged", lanesPerVertex=2, blockSize=256, solveVariant=0)
    phys.runStep(1)
    phys.synchronize()
    lanes = [c["lanes"] for c in phys.colorConfigs()]
    assert 4 in lanes and set(lanes) <= {2, 4}, lanes
    phys.close()


def test_variant_that_does_not_fit(tmp_path, gaia_lib):
    mp, pp = _fan(tmp_path, 60)
    phys = _open(mp, pp, sweepMode="merged", lanesPerVertex=2, blockSize=256, solveVariant=7)
    phys.runStep(1)
    phys.synchronize()
    shapes = {(c["lanes"], c["variant"]) for c in phys.colorConfigs()}
    assert shapes <= {(2, 7), (4, 0)} and (4, 0) in shapes, shapes
    phys.close()


@pytest.mark.parametrize("sweep", ["scenes", "grid"])
def test_sweep_lanes_that_do_not_fit(tmp_path, gaia_lib, sweep):
    mp, pp = _fan(tmp_path, 60)
    phys = _open(mp, pp, sweepMode=sweep, lanesPerVertex=2, blockSize=256)
    phys.runStep(1)
    phys.synchronize()
    assert phys.stats()["lanes_per_vertex"] == 4
    phys.close()


def test_a_wide_launch_of_long_lists(tmp_path, gaia_lib):
    """A color of long lists only takes a warp per vertex whatever was asked for."""
    mp, pp = _fan(tmp_path, 200)
    phys = _open(mp, pp, sweepMode="merged", lanesPerVertex=4, blockSize=128, solveVariant=0)
    assert sorted({c["lanes"] for c in phys.colorConfigs()}) == [4, 32]
    phys.close()
