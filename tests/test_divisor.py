"""Division by a loop constant (npbench_gb300/csrc/divisor.cuh) equals IEEE division, checked on
the CPU against its own (tests/divisor_check.cpp), and the flows built on it equal the oracle at
the sizes where their bands, threads and columns end."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_division_by_a_constant_is_correctly_rounded(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "divisor_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "divisor_check.cpp")], check=True)
    r = subprocess.run([exe, "2000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


def _fields(ny, nx, seed):
    rng = np.random.default_rng(seed)
    u, v, p = (1e-3 * rng.standard_normal((ny, nx)) for _ in range(3))
    p[rng.random((ny, nx)) < 0.3] = 0.0
    return u, v, p, 2 / (nx - 1), 2 / (ny - 1), .1 / ((nx - 1) * (ny - 1))


# One row per band and several; 1, 2 and 4 columns per thread with ragged ends; the
# smallest interior; a grid whose bands do not fit in shared memory (last).
SHAPES = [(3, 3), (4, 5), (60, 33), (101, 64), (154, 65), (330, 31), (40, 255), (30, 257), (25, 513),
          (12, 1024), (1300, 700)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("nit", [0, 1, 6])
def test_cavity_bands(shape, nit):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    from oracle import cref
    u, v, p, dx, dy, dt = _fields(*shape, seed=3)
    d = [torch.from_numpy(x.copy()).cuda() for x in (u, v, p)]
    stencils.cavity_flow(shape[1], shape[0], 3, nit, d[0], d[1], dt, dx, dy, d[2], 1.0, 0.1)
    cref.cavity_flow(shape[1], shape[0], 3, nit, u, v, dt, dx, dy, p, 1.0, 0.1)
    _lib.device_status()
    for x, y in zip(d, (u, v, p)):
        assert bits_equal(x.cpu().numpy(), y)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES[:-1] + [(5, 2), (153, 40)])
@pytest.mark.parametrize("nit,limit", [(0, 5), (1, 1), (6, 4), (3, 1000)])
def test_channel_bands(shape, nit, limit):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    from oracle import cref
    u, v, p, dx, dy, dt = _fields(*shape, seed=4)
    u, v = 1e-4 * np.abs(u), 1e-4 * v
    F = 1.0 if limit < 1000 else 1e-4  # the last case settles within the bound
    d = [torch.from_numpy(x.copy()).cuda() for x in (u, v, p)]
    try:
        got = stencils.channel_flow(nit, d[0], d[1], dt, dx, dy, d[2], 1.0, 0.1, F, max_steps=limit)
    except RuntimeError:
        got = -limit
    # the reference's own loop has no bound: the oracle's is cut at the same step
    import oracle.stencils_np as onp
    steps, udiff, k = 0, 1.0, onp.cfd_constants(dt, dx, dy, 1.0)
    with np.errstate(all="ignore"):
        while udiff > .001 and steps < limit:
            un, vn, b = u.copy(), v.copy(), np.zeros_like(u)
            onp._chan_build_up_b(b, 1.0, u, v, k)
            onp._chan_pressure(nit, p, b, k)
            onp._chan_velocity(u, v, un, vn, p, dt, dx, dy, 0.1, F * dt, k)
            u[0, :] = u[-1, :] = v[0, :] = v[-1, :] = 0
            udiff = (np.sum(u) - np.sum(un)) / np.sum(u)
            steps += 1
    assert abs(got) == steps and (got < 0) == (udiff > .001)
    _lib.device_status()
    for x, y in zip(d, (u, v, p)):
        assert bits_equal(x.cpu().numpy(), y)
