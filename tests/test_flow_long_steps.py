"""Channel flow with a step of more pressure iterations than a wait's two seconds hold."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


def test_a_step_may_take_longer_than_a_wait():
    import torch
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    ny, nx, nit = 5, 6, 4_000_000  # three bands, at least 0.7 us a sweep
    rng = np.random.default_rng(8)
    u, v, p = 1e-3 + 1e-4 * rng.random((ny, nx)), 1e-4 * rng.random((ny, nx)), rng.random((ny, nx))
    u[0] = u[-1] = v[0] = v[-1] = 0.0
    dx, dy, dt = 2 / (nx - 1), 2 / (ny - 1), 1e-4
    d = [torch.from_numpy(x.copy()).cuda() for x in (u, v, p)]
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e[0].record()
    got = stencils.channel_flow(nit, d[0], d[1], dt, dx, dy, d[2], 1.0, 0.1, 0.0)
    e[1].record()
    _lib.device_status()
    want = cref.channel_flow(nit, u, v, dt, dx, dy, p, 1.0, 0.1, 0.0)
    assert e[0].elapsed_time(e[1]) > 2000.0  # or this test shows nothing
    assert got == want
    for x, y in zip(d, (u, v, p)):
        assert bits_equal(x.cpu().numpy(), y)
