"""The per-vertex probe keeps nothing on the host for the vertices it was asked about."""
import ctypes

import pytest


class _Info(ctypes.Structure):
    _fields_ = [(k, ctypes.c_size_t) for k in ("arena", "ordblks", "smblks", "hblks", "hblkhd", "usmblks", "fsmblks",
                                               "uordblks", "fordblks", "keepcost")]


def _in_use():
    f = ctypes.CDLL(None).mallinfo2
    f.restype = _Info
    return f().uordblks


@pytest.mark.gpu
def test_probing_many_vertices_keeps_no_host_memory(tmp_path, gaia_lib):
    from gaia_gb300 import VBDPhysics, scenes

    mp, pp = scenes.drop_cube(str(tmp_path), n=24, iterations=2, precision="fp32", collision=scenes.NO_CONTACT)
    phys = VBDPhysics()
    phys.loadRunningparameters(mp, scenes.set_precision(pp, "fp32", autotune=False))
    phys.initialize()
    for v in range(500):
        phys.vertexForceHessian(0, v)
    before = _in_use()
    for v in range(500, 24 ** 3):
        phys.vertexForceHessian(0, v)
    grown = _in_use() - before
    phys.close()
    # an entry per vertex would be 13,324 tree nodes of 56 bytes and more
    assert grown < 400 * 1024, grown
