"""Exactness of the binary32-limb form of binary64 addition (npbench_gb300/csrc/fxl.cuh).

The header the CUDA kernels include is compiled for the CPU and checked bit for
bit against IEEE binary64 arithmetic (tests/fxl_check.cpp); on a GPU the kernels
built on it are checked against the oracle where their tiles and ranges end.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_limbs_match_ieee_binary64(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "fxl_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "fxl_check.cpp")], check=True)
    r = subprocess.run([exe, "3000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


def _awkward(shape, seed):
    """U[0,1) with values the limbs refuse or treat apart: zeros, tiny, exact powers of
    two, a constant block, numbers of one and more, negatives, inf and NaN."""
    rng = np.random.default_rng(seed)
    A = rng.random(shape)
    f = A.reshape(-1)
    n = f.size
    f[: n // 9] = 0.5
    for value, share in ((0.0, 30), (2.0 ** -7, 40), (1 - 2.0 ** -53, 40), (5e-324, 200),
                         (2.0 ** -7 - 2.0 ** -60, 150), (1.0, 150), (-0.25, 200), (-0.0, 150),
                         (3e200, 400), (np.inf, 900), (np.nan, 900)):
        f[rng.integers(0, n, n // share)] = value
    return A


# Tiles are 8 or 16 rows by 32 columns, chunks 1 plane or more: one past, exactly
# and one short of them, and the smallest grid with an interior.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 10, 34), (9, 9, 33), (6, 18, 66), (5, 19, 35),
                                   (40, 50, 67), (310, 60, 200)])
@pytest.mark.parametrize("chunk", [0, 1, 4])
def test_heat_limbs_at_tile_edges(shape, chunk):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    from oracle import cref
    old = _lib.set_config(_lib.NPBGB_CFG_HEAT_CHUNK, chunk)
    try:
        for A in (np.random.default_rng(1).random(shape), _awkward(shape, 2)):
            B = A[::-1].copy()
            dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
            stencils.heat_3d_kernel(4, dA, dB)
            with np.errstate(all="ignore"):
                cref.heat_3d_kernel(4, A, B)
            assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)
    finally:
        _lib.set_config(_lib.NPBGB_CFG_HEAT_CHUNK, old)


# The frame follows the values: NPBench's own initial field, scaled fields, fields whose
# planes differ by large factors, values beyond any frame; one and two pairs a thread.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(5, 19, 35), (40, 50, 67), (310, 60, 200)])
@pytest.mark.parametrize("values", ["npbench", "3e3", "2e-13", "steps", "1e200", "awkward"])
def test_heat_limbs_follow_the_values(shape, values):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import stencils
    from oracle import cref
    rng = np.random.default_rng(3)
    if values == "npbench":
        i, j, k = np.indices(shape)
        A = (i + j + (shape[2] - k)) * 10 / shape[2]
    elif values == "steps":
        A = rng.random(shape) * 10.0 ** rng.integers(-40, 40, (shape[0], 1, 1))
    elif values == "awkward":
        A = _awkward(shape, 4) * 512
    else:
        A = (0.1 + rng.random(shape)) * float(values)
    B = A[::-1].copy()
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    stencils.heat_3d_kernel(4, dA, dB)
    cref.heat_3d_kernel(4, A, B)
    assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)


# Jacobi-2D in limbs, one launch per half-sweep: strips of 30 columns, four to a CTA, two
# row ranges of which the second may be one short; fields in and out of the frame.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 3), (4, 32), (5, 33), (9, 122), (34, 123), (65, 62)])
@pytest.mark.parametrize("values", ["unit", "npbench", "awkward", "signed", "hot_wall", "steps"])
def test_jacobi_limbs_at_strip_edges(shape, values):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    from oracle import cref
    rng = np.random.default_rng(7)
    A = rng.random(shape)
    if values == "npbench":
        i, j = np.indices(shape)
        A = i * (j + 2) / shape[0]
    elif values == "awkward":
        A = _awkward(shape, 5)
    elif values == "signed":
        A = rng.standard_normal(shape)
    elif values == "hot_wall":
        A = np.zeros(shape)
        A[0] = 100.0
    elif values == "steps":
        A = A * 10.0 ** rng.integers(-40, 40, (shape[0], 1))
    B = A[::-1].copy()
    old = [(k, _lib.set_config(k, v)) for k, v in ((_lib.NPBGB_CFG_JACOBI_BANDS, 0),
                                                   (_lib.NPBGB_CFG_JACOBI_CHUNK, 0))]
    try:
        for chunk in (0, 1, 5):
            _lib.set_config(_lib.NPBGB_CFG_JACOBI_CHUNK, chunk)
            a, b = A.copy(), B.copy()
            dA, dB = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
            stencils.jacobi_2d_kernel(6, dA, dB)
            with np.errstate(all="ignore"):
                cref.jacobi_2d_kernel(6, a, b)
            assert bits_equal(dA.cpu().numpy(), a) and bits_equal(dB.cpu().numpy(), b)
    finally:
        for k, v in old:
            _lib.set_config(k, v)


# Large grids, whose warps are CTAs of their own: an odd number of rows and of strips, the
# last strip of one column.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1301, 1263), (4003, 453)])
@pytest.mark.parametrize("values", ["unit", "npbench", "signed"])
def test_jacobi_limbs_on_large_grids(shape, values):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import bits_equal
    from npbench_gb300 import stencils
    from oracle import cref
    rng = np.random.default_rng(9)
    i, j = np.indices(shape)
    A = (rng.random(shape) if values == "unit" else rng.standard_normal(shape) if values == "signed"
         else i * (j + 2) / shape[0])
    B = A[::-1].copy()
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    stencils.jacobi_2d_kernel(3, dA, dB)
    cref.jacobi_2d_kernel(3, A, B)
    assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)
