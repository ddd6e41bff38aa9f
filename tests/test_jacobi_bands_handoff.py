"""Jacobi-2D with the time loop in one launch against the chained launches over many
half-sweeps: every halo row taken whole, by the lanes that poll for other clusters' rows
(one element a lane to sixteen) and through cluster shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Two clusters and several; pairs with and without a second row (bands of 3, 4, 5 and 6 rows).
@pytest.mark.parametrize("dtype, shape", [
    (np.float64, (69, 33)), (np.float64, (301, 479)), (np.float64, (460, 300)), (np.float64, (203, 1056)),
    (np.float32, (69, 33)), (np.float32, (301, 1025)), (np.float32, (575, 1409)), (np.float32, (700, 1600)),
    (np.float32, (450, 2049)), (np.float32, (690, 4096))])
def test_bands_equal_chained_launches(dtype, shape):
    import torch

    from npbench_gb300 import _lib, autotune, stencils
    gen = torch.Generator(device="cuda")
    gen.manual_seed(shape[0])
    dt = torch.float64 if dtype == np.float64 else torch.float32
    A = torch.rand(shape, generator=gen, device="cuda", dtype=dt)
    B = torch.rand(shape, generator=gen, device="cuda", dtype=dt)
    was, old = autotune.enabled(), _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, 0)
    autotune.disable()
    try:
        want = A.clone(), B.clone()
        stencils.jacobi_2d_kernel(301, *want)
        _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, 2)
        for _ in range(4):
            got, n0 = (A.clone(), B.clone()), _lib.launches()
            stencils.jacobi_2d_kernel(301, *got)
            _lib.device_status()
            assert _lib.launches() - n0 == 1
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    finally:
        _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, old)
        if was:
            autotune.enable()


# On both sides of the line for grids whose threads take eight columns.
@pytest.mark.parametrize("shape, tsteps, one", [
    ((600, 2300), 16, False), ((700, 2300), 16, True), ((750, 2500), 19, False), ((750, 2500), 20, True),
    ((750, 3300), 40, False), ((1000, 3300), 20, True), ((900, 4096), 40, False), ((1200, 4096), 20, True)])
def test_wide_grids_of_few_rows_keep_chained_launches(shape, tsteps, one):
    import torch

    from npbench_gb300 import _lib, autotune, stencils
    A, B = (torch.rand(shape, device="cuda") for _ in range(2))
    was = autotune.enabled()
    autotune.disable()
    try:
        results = []
        for bands in (1, 0):
            old = _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, bands)
            got, n0 = (A.clone(), B.clone()), _lib.launches()
            stencils.jacobi_2d_kernel(tsteps, *got)
            _lib.device_status()
            _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, old)
            results.append((got, _lib.launches() - n0))
    finally:
        if was:
            autotune.enable()
    assert results[0][1] == (1 if one else 2 * (tsteps - 1)) and results[1][1] == 2 * (tsteps - 1)
    assert all(torch.equal(x, y) for x, y in zip(results[0][0], results[1][0]))
