"""Binary32 Heat-3D streamed by rows, at the edges of its strips of 30 columns, blocks of
six rows (four to a CTA) and chunks of planes, against the oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 5, 32), (5, 8, 33), (6, 9, 62), (12, 25, 63), (7, 26, 64),
                                   (9, 27, 92), (41, 50, 31)])
@pytest.mark.parametrize("chunk", [0, 1, 4])
def test_rows_equal_the_oracle(shape, chunk):
    import torch
    from conftest import bits_equal
    from npbench_gb300 import _lib, stencils
    rng = np.random.default_rng(2)
    plain = rng.random(shape).astype(np.float32)
    special = rng.standard_normal(shape).astype(np.float32)
    for v in (0.0, -0.0, np.inf, np.nan, 3e38, 1e-45):
        special.reshape(-1)[rng.integers(0, special.size, 2)] = v
    old = _lib.set_config(_lib.NPBGB_CFG_HEAT_CHUNK, chunk)
    try:
        for A in (plain, special):
            A, B = A.copy(), A[::-1].copy()
            # an odd first element: no more than 4-byte alignment
            dA = torch.empty(A.size + 1, dtype=torch.float32, device="cuda")[1:].view(shape)
            dB = torch.empty(A.size + 3, dtype=torch.float32, device="cuda")[3:].view(shape)
            dA.copy_(torch.from_numpy(A))
            dB.copy_(torch.from_numpy(B))
            stencils.heat_3d_kernel(4, dA, dB)
            with np.errstate(all="ignore"):
                cref.heat_3d_kernel(4, A, B)
            assert bits_equal(dA.cpu().numpy(), A) and bits_equal(dB.cpu().numpy(), B)
    finally:
        _lib.set_config(_lib.NPBGB_CFG_HEAT_CHUNK, old)
