"""Binary64 Jacobi-2D in chained launches on fields that no frame of binary32 limbs holds:
strips that take hardware binary64 throughout, against the oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


def _field(values, shape):
    rng = np.random.default_rng(9)
    A = rng.standard_normal(shape)
    if values == "specials":
        for v in (0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.3e-308, 1.7e308, 2.0 ** -1000, -(2.0 ** 980)):
            A.reshape(-1)[rng.integers(0, A.size, 2)] = v
    elif values == "subnormal":  # sums on both sides of the smallest normal number
        A *= 2.0 ** -1021
    elif values == "huge":  # sums that overflow and products that do not
        A *= 2.0 ** 1021
    elif values == "signed and zero":  # strips of zeros next to strips of signed values
        A[:, shape[1] // 3: shape[1] // 2] = 0.0
        A[:, : shape[1] // 4] = -0.0
    return A


# Strips of 30 columns: a part of one, one, a column more; two rows a warp and more.
@pytest.mark.parametrize("values", ["signed", "specials", "subnormal", "huge", "signed and zero"])
@pytest.mark.parametrize("shape", [(5, 12), (9, 32), (10, 33), (300, 700), (1203, 901)])
def test_refused_strips_equal_the_oracle(values, shape):
    import torch
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    A = _field(values, shape)
    B = A[::-1].copy()
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    old = _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, 0)
    try:
        stencils.jacobi_2d_kernel(4, dA, dB)
    finally:
        _lib.set_config(_lib.NPBGB_CFG_JACOBI_BANDS, old)
    with np.errstate(all="ignore"):
        cref.jacobi_2d_kernel(4, A, B)
    assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)
