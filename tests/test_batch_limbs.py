"""Stepped batches of Jacobi-2D grids in limbs: units of one strip by a few rows, whose
rows shrink as grids finish, against the oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


def _same(x, y):
    w = np.uint64 if x.dtype == np.float64 else np.uint32
    return bool(np.all((x.view(w) == y.view(w)) | (np.isnan(x) & np.isnan(y))))


# Widths around one and four strips of 30 and 32 columns and a tile's eight units; one
# large grid that finishes first, so that the rows per unit change three times.
_GRIDS = [((3, 3), 9), ((4, 32), 7), ((9, 33), 12), ((34, 62), 5), ((65, 63), 12), ((70, 122), 8),
          ((130, 242), 6), ((700, 900), 2), ((1500, 1700), 2)]


@pytest.mark.parametrize("values", ["unit", "ramp", "signed"])
@pytest.mark.parametrize("rows, emulation", [(0, 1), (5, 1), (0, 0)])
def test_stepped_units_equal_the_oracle(values, rows, emulation):
    import torch

    from npbench_gb300 import _lib
    from npbench_gb300.batch import Batch
    rng = np.random.default_rng(11)
    host = []
    for n, (shape, steps) in enumerate(_GRIDS):
        dt = np.float32 if n % 3 == 2 else np.float64
        if values == "ramp":
            i, j = np.indices(shape)
            A = (i * (j + 2) / shape[0]).astype(dt)
        else:
            A = (rng.random(shape) if values == "unit" else rng.standard_normal(shape)).astype(dt)
        host.append((A, A[::-1].copy(), steps))
    dev = [(torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda(), t) for A, B, t in host]
    with Batch(dev, band_rows=rows, mode="stepped") as b:  # planned in limbs
        old = _lib.set_config(_lib.NPBGB_CFG_F64_EMULATION, emulation)
        try:
            b.launch()
            torch.cuda.synchronize()
        finally:
            _lib.set_config(_lib.NPBGB_CFG_F64_EMULATION, old)
    for (A, B, t), (dA, dB, _) in zip(host, dev):
        with np.errstate(all="ignore"):
            cref.jacobi_2d_kernel(t, A, B)
        assert _same(dA.cpu().numpy(), A) and _same(dB.cpu().numpy(), B), (A.shape, t)
