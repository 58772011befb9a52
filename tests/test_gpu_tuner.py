"""The autotuner's picks in the step: as fast as the best of the uniform shapes, on colors of
several hundred vertices and with bodies in contact."""
import pytest

pytestmark = pytest.mark.gpu


def _step_ms(mp, pp, x=None, **over):
    from gaia_gb300 import VBDPhysics, scenes

    phys = VBDPhysics()
    phys.loadRunningparameters(mp, scenes.set_precision(pp, over.pop("precision"), out_path=pp + ".t.json", sweepMode="merged",
                                                        **over))
    phys.initialize()
    ms = []
    for _ in range(6):
        phys.reset()
        phys.runStep(12)  # into the ground, or into contact
        ms.append(phys.run_steps_timed(3, False)[0] / 3)
    phys.close()
    return min(ms)


# Bounds: the pick may lose 10% to the best uniform shape (the spread of one shape over handles is
# 2-3%). A warp per vertex, the pick before for colors of up to 1024 vertices, loses 20-27% at
# 1024 vertices per color; two lanes in FP64 with contact 50%.
@pytest.mark.parametrize("scene,precision", [("drop16", "fp32"), ("drop16", "mixed"), ("stack", "fp64")])
def test_pick_is_near_the_best_uniform_shape(tmp_path, gaia_lib, scene, precision):
    from gaia_gb300 import scenes

    if scene == "stack":
        mp, pp = scenes.stack_drop(str(tmp_path), n_lower=16, n_upper=14, spacing=0.01, gap=0.002, speed=1.0,
                                   precision=precision)
    else:
        mp, pp = scenes.drop_cube(str(tmp_path), n=16, iterations=20, precision=precision, height=0.001,
                                  collision=scenes.NO_CONTACT)
    fixed = {L: _step_ms(mp, pp, precision=precision, lanesPerVertex=L, blockSize=128, solveVariant=0, autotune=False,
                         smallColorVertices=0) for L in (2, 4, 8, 16, 32)}
    picked = _step_ms(mp, pp, precision=precision)
    print(scene, precision, "picked %.3f ms" % picked, {k: "%.3f" % v for k, v in fixed.items()})
    assert picked <= 1.1 * min(fixed.values())
