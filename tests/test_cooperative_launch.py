"""What the one-launch forms do where their cooperative launch is not made as asked for."""
import numpy as np
import pytest

from npbench_gb300 import _lib
from oracle import cref


def test_kinds_of_launch_are_checked():
    lib = _lib.load()
    assert lib.npbgb_selftest_launch(-1) == _lib.NPBGB_ERR_ARG
    assert lib.npbgb_selftest_launch(0) == _lib.NPBGB_OK


def _jacobi_2d(A, B, tsteps, how):
    """The one-launch form's fields, and the library's launches."""
    import torch

    from npbench_gb300 import autotune, stencils
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    was, old = autotune.enabled(), _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, 2)
    autotune.disable()
    try:
        n0 = _lib.launches()
        _lib.check(_lib.load().npbgb_selftest_launch(how), "selftest_launch")
        stencils.jacobi_2d_kernel(tsteps, dA, dB)
        torch.cuda.synchronize()
        _lib.device_status()
        return dA.cpu().numpy(), dB.cpu().numpy(), _lib.launches() - n0
    finally:
        _lib.load().npbgb_selftest_launch(0)
        _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, old)
        if was:
            autotune.enable()


# One cluster of bands; several; rows and threads that do not divide evenly; three columns.
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", [(40, 50), (120, 130), (451, 477), (700, 3)])
def test_bands_without_their_clusters(dtype, shape):
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal(shape).astype(dtype), rng.random(shape).astype(dtype)
    a, b, launches = _jacobi_2d(A, B, 9, _lib.NPBGB_LAUNCH_UNCLUSTERED)
    cref.jacobi_2d_kernel(9, A, B)
    assert launches == 1
    assert a.tobytes() == A.tobytes() and b.tobytes() == B.tobytes()
