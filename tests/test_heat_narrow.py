"""Binary32 Heat-3D on large arrays with short rows, on both sides of the line between strips of
30 columns and TMA's of 32, against the oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


# 110 MB in both arrays, just below and above; rows that TMA cannot copy; an address that it
# cannot; rows that 30 columns suit better.
@pytest.mark.parametrize("shape, first", [((500, 429, 64), 0), ((500, 430, 64), 0), ((430, 500, 65), 0),
                                          ((500, 430, 64), 1), ((340, 500, 96), 0), ((380, 500, 80), 0)])
def test_equal_to_the_oracle(shape, first):
    import torch
    from conftest import bits_equal
    from npbench_gb300 import _lib, autotune, stencils
    A = np.random.default_rng(7).standard_normal(shape).astype(np.float32)
    B = A[::-1].copy()
    dA, dB = (torch.empty(A.size + first, dtype=torch.float32, device="cuda")[first:].view(shape) for _ in range(2))
    dA.copy_(torch.from_numpy(A))
    dB.copy_(torch.from_numpy(B))
    was = autotune.enabled()
    autotune.disable()
    try:
        stencils.heat_3d_kernel(3, dA, dB)
    finally:
        if was:
            autotune.enable()
    _lib.device_status()
    cref.heat_3d_kernel(3, A, B)
    assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)
