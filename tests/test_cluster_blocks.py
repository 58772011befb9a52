"""Blocks of the cluster sweep where the staging areas do not fit beside the scene: fewer
threads, always whole warps."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_smaller_blocks_are_whole_warps(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text("""
#include <cstdio>
#include "launch_shape.hpp"
int main() {
    for (int b = 64; b <= 256; b += 32)
        for (int c = b;;) {
            const int n = gaia::smaller_block(c);
            std::printf("%d %d\\n", c, n);
            if (n == c) break;
            c = n;
        }
}
""")
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", os.path.join(ROOT, "gaia_gb300", "csrc"), str(src),
                    "-o", exe], check=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert {r[0] for r in rows} >= set(range(64, 257, 32))
    for c, n in rows:
        assert n % 32 == 0 and 64 <= n <= max(64, c // 2)


def _fan_and_tets(n_ring, n_tets):
    """A hub with n_ring + 2 neighbours (long lists: large staging areas) and separate tets
    (many states, few incidences: a cluster's block holds the states only)."""
    from test_gpu_one_ring import _fan

    X, T = _fan(n_ring, False)
    rng = np.random.Generator(np.random.PCG64(1))
    c = np.stack(np.meshgrid(*[np.arange(12)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n_tets] * 0.02 + [0.2, 0.0, 0.2]
    tet = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]) * 0.01
    Y = (c[:, None] + tet + rng.uniform(-1e-4, 1e-4, (n_tets, 4, 3))).reshape(-1, 3)
    T = np.concatenate([T, len(X) + np.arange(4 * n_tets).reshape(-1, 4)])
    X = np.concatenate([X, Y])
    at = rng.permutation(len(X))  # the fan's vertices spread over the blocks of a cluster
    out = np.empty_like(X)
    out[at] = X
    return out, at[T].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("block", [96, 160, 224])
def test_cluster_block_beside_a_large_scene(tmp_path, gaia_lib, block):
    """6001 states of 32 bytes leave about 36 KB for the staging of 128 neighbours per vertex:
    224 threads at a warp per vertex need 43 KB, so the launch takes fewer; 160 and 96 fit."""
    from gaia_gb300 import VBDPhysics, scenes

    X, T = _fan_and_tets(126, 1468)
    tp, cp = scenes._write_mesh(str(tmp_path), "fan", X, T, coloring="greedy")
    models = [scenes.model_entry(tp, cp, initialVelocity=[0.1, 0.0, 0.05])]
    params = scenes.physics_params(1.0 / 300.0, 8, precision="mixed", ground_y=-0.05)
    mp, pp = scenes._write_json(str(tmp_path), models, params, collision=scenes.NO_CONTACT)
    common = dict(lanesPerVertex=32, blockSize=block, autotune=False, smallColorVertices=0, solveVariant=0)
    x = {}
    for mode, extra in (("merged", {}), ("cluster", {"clusterSize": 16})):
        phys = VBDPhysics()
        phys.loadRunningparameters(mp, scenes.set_precision(pp, "mixed", out_path="%s.%s.json" % (pp, mode), sweepMode=mode,
                                                            **common, **extra))
        phys.initialize()
        phys.runStep(3)
        x[mode] = phys.positions(0)
        st = phys.stats()
        phys.close()
        assert st["sweep_mode"] == {"merged": 0, "cluster": 2}[mode]
    np.testing.assert_array_equal(x["merged"], x["cluster"])


@pytest.mark.gpu
@pytest.mark.parametrize("cluster,fits", [(4, False), (8, True)])
def test_autotuner_times_the_cluster_sizes_that_can_be_asked_for(tmp_path, gaia_lib, cluster, fits):
    """A 9^3 cube in FP64: 4 blocks are past the mode's limit of states and incidences per block,
    8 are not, for the explicit mode and for the autotuner alike."""
    from gaia_gb300 import VBDPhysics, scenes
    from gaia_gb300._lib import GaiaError

    X, T = scenes.lattice_cube((9, 9, 9), 0.01)[:2]
    tp, cp = scenes._write_mesh(str(tmp_path), "cube", X, T)
    mp, pp = scenes._write_json(str(tmp_path), [scenes.model_entry(tp, cp)],
                                scenes.physics_params(1.0 / 300.0, 4, precision="fp64"), collision=scenes.NO_CONTACT)
    timed = {}
    for mode in ("cluster", "auto"):
        phys = VBDPhysics()
        phys.loadRunningparameters(mp, scenes.set_precision(pp, "fp64", out_path="%s.%s.json" % (pp, mode), sweepMode=mode,
                                                            clusterSize=cluster))
        try:
            phys.initialize()
            timed[mode] = mode == "cluster" or phys.stats()["sweep_ms_cluster"] > 0
        except GaiaError:
            timed[mode] = False
        phys.close()
    assert timed == {"cluster": fits, "auto": fits}
