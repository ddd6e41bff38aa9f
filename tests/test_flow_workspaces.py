"""The flows through the C ABI on the workspaces that callers may pass: any that is aligned for
doubles, and one that only the band form's fields fit."""
import numpy as np
import pytest

from npbench_gb300 import _lib

pytestmark = pytest.mark.gpu

CASES = [(40, 33), (101, 64), (330, 31), (25, 513)]


def _fields(ny, nx):
    rng = np.random.default_rng(ny)
    u, v, p = (1e-4 * rng.random((ny, nx)) for _ in range(3))
    return u, v, p, 2 / (nx - 1), 2 / (ny - 1), .1 / ((nx - 1) * (ny - 1))


def _cavity(shape, offset, nbytes=None):
    """The fields of three steps with a workspace `offset` bytes past an aligned address."""
    import torch
    ny, nx = shape
    u, v, p, dx, dy, dt = _fields(ny, nx)
    d = [torch.from_numpy(x).cuda() for x in (u, v, p)]
    n = int(_lib.load().npbgb_cavity_flow_workspace_bytes(ny, nx)) if nbytes is None else nbytes
    ws = torch.full((n + offset,), 0x5a, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 256 == 0
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().npbgb_cavity_flow(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), ny, nx, 3, 7, dt, dx, dy,
                                             1.0, 0.1, _lib.NPBGB_F64, ws.data_ptr() + offset, n, st), "cavity_flow")
    _lib.device_status()
    return [x.cpu().numpy() for x in d]


def _channel(shape, offset, nbytes=None):
    """The fields and steps of a run of at most four steps, likewise."""
    import ctypes

    import torch
    ny, nx = shape
    u, v, p, dx, dy, dt = _fields(ny, nx)
    d = [torch.from_numpy(x).cuda() for x in (u, v, p)]
    n = int(_lib.load().npbgb_channel_flow_workspace_bytes(ny, nx)) if nbytes is None else nbytes
    ws = torch.full((n + offset,), 0x5a, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 256 == 0
    st, steps = torch.cuda.current_stream().cuda_stream, ctypes.c_int64(0)
    _lib.check(_lib.load().npbgb_channel_flow(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), ny, nx, 7, dt, dx, dy,
                                              1.0, 0.1, 1.0, 4, _lib.NPBGB_F64, ws.data_ptr() + offset, n,
                                              ctypes.byref(steps), st), "channel_flow")
    _lib.device_status()
    return [x.cpu().numpy() for x in d] + [np.array([float(steps.value)])]


def _equal(x, y):
    return all(a.tobytes() == b.tobytes() for a, b in zip(x, y))


@pytest.mark.parametrize("shape", CASES)
@pytest.mark.parametrize("flow", [_cavity, _channel])
def test_a_workspace_aligned_for_doubles(flow, shape):
    assert _equal(flow(shape, 8), flow(shape, 0))
    assert _equal(flow(shape, 24), flow(shape, 0))
