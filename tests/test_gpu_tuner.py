"""The autotuner's picks in the step: as fast as the best of the uniform shapes, on colors of
a thousand vertices."""
import pytest

pytestmark = pytest.mark.gpu


def _step_ms(mp, pp, **over):
    from gaia_gb300 import VBDPhysics, scenes

    phys = VBDPhysics()
    phys.loadRunningparameters(mp, scenes.set_precision(pp, over.pop("precision"), out_path=pp + ".t.json", sweepMode="merged",
                                                        **over))
    phys.initialize()
    ms = []
    for _ in range(6):
        phys.reset()
        phys.runStep(12)  # into the ground
        ms.append(phys.run_steps_timed(3, False)[0] / 3)
    phys.close()
    return min(ms)


# Bounds: the pick may lose 10% to the best uniform shape (the spread of one shape over handles is
# 2-3%). A warp per vertex, the pick before for colors of up to 1024 vertices, loses 20-27% there.
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_pick_is_near_the_best_uniform_shape(tmp_path, gaia_lib, precision):
    from gaia_gb300 import scenes

    mp, pp = scenes.drop_cube(str(tmp_path), n=16, iterations=20, precision=precision, height=0.001,
                              collision=scenes.NO_CONTACT)
    fixed = {L: _step_ms(mp, pp, precision=precision, lanesPerVertex=L, blockSize=128, solveVariant=0, autotune=False,
                         smallColorVertices=0) for L in (2, 4, 8, 16, 32)}
    picked = _step_ms(mp, pp, precision=precision)
    print(precision, "picked %.3f ms" % picked, {k: "%.3f" % v for k, v in fixed.items()})
    assert picked <= 1.1 * min(fixed.values())
