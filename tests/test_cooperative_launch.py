"""What the one-launch forms do where their cooperative launch is not made as asked for."""
import numpy as np
import pytest

from npbench_gb300 import _lib
from oracle import cref


def test_kinds_of_launch_are_checked():
    lib = _lib.load()
    assert lib.npbgb_selftest_launch(-1) == _lib.NPBGB_ERR_ARG
    assert lib.npbgb_selftest_launch(0) == _lib.NPBGB_OK


def _jacobi_2d(A, B, tsteps, how, bands=2):
    """The fields, and the library's launches."""
    import torch

    from npbench_gb300 import autotune, stencils
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    was, old = autotune.enabled(), _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, bands)
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


# Each of these ran before it had a one-launch form, and runs where that one is refused.
@pytest.mark.gpu
@pytest.mark.parametrize("dtype, shape, bands", [(np.float32, (120, 130), 1), (np.float64, (120, 130), 2),
                                                 (np.float64, (301, 481), 1)])
def test_jacobi_2d_where_the_launch_is_refused(dtype, shape, bands):
    rng = np.random.default_rng(4)
    A, B = rng.random(shape).astype(dtype), rng.random(shape).astype(dtype)
    a, b, launches = _jacobi_2d(A, B, 20, _lib.NPBGB_LAUNCH_REFUSED, bands)
    cref.jacobi_2d_kernel(20, A, B)
    assert launches == 38
    assert a.tobytes() == A.tobytes() and b.tobytes() == B.tobytes()
    assert _jacobi_2d(A, B, 20, 0, bands)[2] == 1  # the next launch is made as always


@pytest.mark.gpu
def test_jacobi_1d_where_the_launch_is_refused():
    import torch

    from npbench_gb300 import stencils
    rng = np.random.default_rng(5)
    A, B = rng.random(5000).astype(np.float32), rng.random(5000).astype(np.float32)
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    n0 = _lib.launches()
    _lib.check(_lib.load().npbgb_selftest_launch(_lib.NPBGB_LAUNCH_REFUSED), "selftest_launch")
    stencils.jacobi_1d_kernel(100, dA, dB)
    _lib.device_status()
    assert _lib.launches() - n0 > 1
    cref.jacobi_1d_kernel(100, A, B)
    assert dA.cpu().numpy().tobytes() == A.tobytes() and dB.cpu().numpy().tobytes() == B.tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("flow", ["cavity", "channel"])
def test_flows_where_the_launch_is_refused(flow):
    import torch

    from npbench_gb300 import stencils
    ny, nx = 40, 33
    rng = np.random.default_rng(6)
    u, v, p = (1e-4 * rng.random((ny, nx)) for _ in range(3))
    dx, dy, dt = 2 / (nx - 1), 2 / (ny - 1), 1e-4

    def run():
        d = [torch.from_numpy(x).cuda() for x in (u, v, p)]
        n0, n = _lib.launches(), None
        if flow == "cavity":
            stencils.cavity_flow(nx, ny, 4, 7, d[0], d[1], dt, dx, dy, d[2], 1.0, 0.1)
        else:
            n = stencils.channel_flow(7, d[0], d[1], dt, dx, dy, d[2], 1.0, 0.1, 1e-6)
        _lib.device_status()
        assert _lib.launches() - n0 == 1
        return [x.cpu().numpy().tobytes() for x in d] + [n]

    want = run()
    _lib.check(_lib.load().npbgb_selftest_launch(_lib.NPBGB_LAUNCH_REFUSED), "selftest_launch")
    assert run() == want
