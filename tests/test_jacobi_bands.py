"""Jacobi-2D with the time loop in one launch, at the edges of its split: columns a
thread, bands a cluster, pairs a thread, odd rows."""
import numpy as np
import pytest

from oracle import cref

gpu = pytest.mark.gpu


def _run(A, B, tsteps, bands):
    import torch

    from npbench_gb300 import _lib, stencils
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    old = _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, bands)
    try:
        n0 = _lib.launches()
        stencils.jacobi_2d_kernel(tsteps, dA, dB)
        torch.cuda.synchronize()
        _lib.device_status()
        return dA.cpu().numpy(), dB.cpu().numpy(), _lib.launches() - n0
    finally:
        _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, old)


def _same(x, y):
    w = np.uint64 if x.dtype == np.float64 else np.uint32
    return bool(np.all((x.view(w) == y.view(w)) | (np.isnan(x) & np.isnan(y))))


# (rows, columns): 3 and 4 interior rows (a lone second row or none); 64 and 65 (16 bands of two
# pairs, one cluster and one more band); 449 (bands of three pairs); widths on both sides of the
# columns that 1, 2 or 3 (binary64) and 2, 4 or 8 (binary32) a thread cover.
_SHAPES = [(5, 34), (6, 3), (66, 97), (67, 97), (451, 66)]
_WIDE = {np.float64: (481, 482, 961, 962, 1057), np.float32: (1025, 1026, 2049, 2050, 4096)}


@gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("case", range(10))
@pytest.mark.parametrize("values", ["unit", "ramp", "special"])
def test_bands_equal_the_oracle(dtype, case, values):
    from npbench_gb300 import autotune
    shape = _SHAPES[case] if case < 5 else (23, _WIDE[dtype][case - 5])
    rng = np.random.default_rng(case)
    A, B = rng.random(shape).astype(dtype), rng.random(shape).astype(dtype)
    if values == "ramp":  # NPBench's own initial field
        i, j = np.indices(shape)
        A, B = (i * (j + 2) / shape[0]).astype(dtype), (i * (j + 3) / shape[0]).astype(dtype)
    if values == "special":
        at = lambda n: (rng.integers(0, shape[0], n), rng.integers(0, shape[1], n))  # noqa: E731
        for v in (0.0, -0.0, np.nan, np.inf, 2.0 ** -7, np.finfo(dtype).tiny, -0.3, 0.5):
            A[at(3)], B[at(3)] = v, v
    rA, rB = A.copy(), B.copy()
    cref.jacobi_2d_kernel(5, rA, rB)
    was = autotune.enabled()
    autotune.disable()
    try:
        a, b, launches = _run(A, B, 5, 2)
        assert launches == 1
        assert _same(a, rA) and _same(b, rB)
        a, b, launches = _run(A, B, 5, 0)
        assert launches == 8
        assert _same(a, rA) and _same(b, rB)
    finally:
        if was:
            autotune.enable()


@gpu
@pytest.mark.parametrize("dtype, shape, launches", [
    (np.float32, (40, 50), 1), (np.float32, (300, 2049), 1), (np.float32, (300, 2050), 30),
    (np.float32, (700, 2050), 1), (np.float64, (300, 481), 1), (np.float64, (300, 482), 30),
    (np.float64, (700, 481), 30)])
def test_the_default_takes_bands_where_they_are_faster(dtype, shape, launches):
    from npbench_gb300 import autotune
    rng = np.random.default_rng(1)
    A, B = rng.random(shape).astype(dtype), rng.random(shape).astype(dtype)
    was = autotune.enabled()
    autotune.disable()
    try:
        a, b, n = _run(A, B, 16, 1)
        assert n == launches
        ra, rb, _ = _run(A, B, 16, 0)
        assert _same(a, ra) and _same(b, rb)
    finally:
        if was:
            autotune.enable()
