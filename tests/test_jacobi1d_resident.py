"""Binary32 Jacobi-1D in one launch, at the edges of its segments and rounds, against the
oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


# One segment of 148 points filled, short of it and one past it; a last segment of one point;
# segments of more than 148 (halos of 120 and of 36 points) and one point too many for halos
# of 32 on 152 SMs.  Half-sweeps that end inside, at and past a round.
@pytest.mark.parametrize("n", [3, 4, 149, 150, 151, 297, 299, 22500, 32000, 58000, 59700])
@pytest.mark.parametrize("tsteps", [64, 75, 76, 150])
def test_resident_equals_the_oracle(n, tsteps):
    import torch

    from npbench_gb300 import _lib, stencils
    rng = np.random.default_rng(n)
    A, B = rng.random(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    for v in (0.0, -0.0, np.inf, np.nan, 1e-45):
        A[rng.integers(0, n)] = v
    if n % 2:
        A, B = B, A
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    stencils.jacobi_1d_kernel(tsteps, dA, dB)
    _lib.device_status()
    with np.errstate(all="ignore"):
        cref.jacobi_1d_kernel(tsteps, A, B)
    for x, y in ((dA.cpu().numpy(), A), (dB.cpu().numpy(), B)):
        assert np.all((x.view(np.uint32) == y.view(np.uint32)) | (np.isnan(x) & np.isnan(y)))
