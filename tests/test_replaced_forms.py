"""Forms that the defaults have left to some sizes, workspaces and settings only, against the
oracle, and the launches that tell which form ran."""
import ctypes

import numpy as np
import pytest

from npbench_gb300 import _lib
from oracle import cref

pytestmark = pytest.mark.gpu


@pytest.fixture
def settings():
    """Sets knobs for one test."""
    old = {}

    def put(key, value):
        was = _lib.set_config(key, value)
        old.setdefault(key, was)

    yield put
    for key, value in old.items():
        _lib.set_config(key, value)


# Staged through shared memory by plain loads; the TMA ring.
@pytest.mark.parametrize("form", ["plain", "ring"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (9, 40, 36), (5, 37, 46), (12, 10, 34), (66, 130, 200)])
def test_binary32_heat_staged(form, shape, settings):
    import torch
    from conftest import bits_equal
    from npbench_gb300 import autotune, stencils
    if form == "plain":
        settings(_lib.NPBGB_CFG_HEAT_TMA, 0)
        settings(_lib.NPBGB_CFG_HEAT_ROWS, 1)
    else:
        settings(_lib.NPBGB_CFG_HEAT_STAGES, 8)
    A = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    B = A.copy()
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    was = autotune.enabled()
    autotune.disable()
    try:
        stencils.heat_3d_kernel(5, dA, dB)
    finally:
        if was:
            autotune.enable()
    _lib.device_status()
    cref.heat_3d_kernel(5, A, B)
    assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)


# Segments of 148 points and more in one launch; one point too many for halos of 32; too few
# steps.
@pytest.mark.parametrize("n, tsteps, one", [(4, 64, True), (150, 64, True), (32000, 76, True), (59698, 64, False),
                                            (32000, 63, False)])
def test_binary32_jacobi_1d_launches(n, tsteps, one):
    import torch

    from npbench_gb300 import stencils
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 152:
        n = n * sms // 152
    A, B = (torch.rand(n, device="cuda") for _ in range(2))
    n0 = _lib.launches()
    stencils.jacobi_1d_kernel(tsteps, A, B)
    _lib.device_status()
    assert (_lib.launches() - n0 == 1) == one


def test_settings_put_back_leave_the_default_form(settings):
    import torch

    from npbench_gb300 import stencils
    A, B = (torch.rand(32000, device="cuda") for _ in range(2))
    for key, other in ((_lib.NPBGB_CFG_JACOBI1D_CTAS, 2), (_lib.NPBGB_CFG_JACOBI1D_DEPTH, 16)):
        old = _lib.get_config(key)
        for value, one in ((other, False), (old, True)):
            settings(key, value)
            n0 = _lib.launches()
            stencils.jacobi_1d_kernel(100, A, B)
            _lib.device_status()
            assert (_lib.launches() - n0 == 1) == one


def _round_up(n):
    return -(-n // 256) * 256


def _flow_fields(ny, nx):
    rng = np.random.default_rng(ny * nx)
    u, v, p = (1e-5 * rng.random((ny, nx)) for _ in range(3))
    return u, v, p, 2 / (nx - 1), 2 / (ny - 1), .1 / ((nx - 1) * (ny - 1))


def _channel_oracle(nit, u, v, dt, dx, dy, p, F, limit):
    """The reference's loop, cut at `limit` steps."""
    import oracle.stencils_np as onp
    steps, udiff, k = 0, 1.0, onp.cfd_constants(dt, dx, dy, 1.0)
    while udiff > .001 and steps < limit:
        un, vn, b = u.copy(), v.copy(), np.zeros_like(u)
        onp._chan_build_up_b(b, 1.0, u, v, k)
        onp._chan_pressure(nit, p, b, k)
        onp._chan_velocity(u, v, un, vn, p, dt, dx, dy, 0.1, F * dt, k)
        u[0, :] = u[-1, :] = v[0, :] = v[-1, :] = 0
        udiff = (np.sum(u) - np.sum(un)) / np.sum(u)
        steps += 1
    return steps if udiff <= .001 else -steps


def _channel(shape, nit, limit, nbytes=None):
    import torch
    from conftest import bits_equal
    ny, nx = shape
    u, v, p, dx, dy, dt = _flow_fields(ny, nx)
    d = [torch.from_numpy(x.copy()).cuda() for x in (u, v, p)]
    n = int(_lib.load().npbgb_channel_flow_workspace_bytes(ny, nx)) if nbytes is None else nbytes
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    steps = ctypes.c_int64(0)
    _lib.check(_lib.load().npbgb_channel_flow(
        d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), ny, nx, nit, dt, dx, dy, 1.0, 0.1, 1.0, limit, _lib.NPBGB_F64,
        ws.data_ptr(), n, ctypes.byref(steps), torch.cuda.current_stream().cuda_stream), "channel_flow")
    _lib.device_status()
    assert steps.value == _channel_oracle(nit, u, v, dt, dx, dy, p, 1.0, limit)
    assert all(bits_equal(x.cpu().numpy(), y) for x, y in zip(d, (u, v, p)))


# More than 1024 columns; bands of more values than shared memory holds.
@pytest.mark.parametrize("shape", [(6, 1025), (20, 1100), (1300, 700), (155, 1024)])
@pytest.mark.parametrize("nit", [0, 5])
def test_channel_in_global_memory(shape, nit):
    _channel(shape, nit, 3)


def test_channel_with_the_smaller_workspace():
    ny, nx = 60, 33
    mail = 3 * _round_up(58 * 4 * nx * 16)  # 58 bands, one row each
    assert mail > 4 * _round_up(ny * nx * 8)  # its own part of the workspace
    _channel((ny, nx), 5, 3, int(_lib.load().npbgb_channel_flow_workspace_bytes(ny, nx)) - mail)


def test_cavity_with_the_smaller_workspace():
    import torch
    from conftest import bits_equal
    ny, nx = 60, 33
    u, v, p, dx, dy, dt = _flow_fields(ny, nx)
    d = [torch.from_numpy(x.copy()).cuda() for x in (u, v, p)]
    n = 4 * _round_up(ny * nx * 8) + 256  # four fields and the band counters
    assert n < int(_lib.load().npbgb_cavity_flow_workspace_bytes(ny, nx))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().npbgb_cavity_flow(
        d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), ny, nx, 4, 6, dt, dx, dy, 1.0, 0.1, _lib.NPBGB_F64,
        ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream), "cavity_flow")
    _lib.device_status()
    cref.cavity_flow(nx, ny, 4, 6, u, v, dt, dx, dy, p, 1.0, 0.1)
    assert all(bits_equal(x.cpu().numpy(), y) for x, y in zip(d, (u, v, p)))
