"""Vertical advection (few columns and many) where neighbouring levels of u are equal, opposite zeros, infinite or
NaN: the product that one level hands to the next, against the oracle."""
import numpy as np
import pytest

from oracle import cref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 5, 2), (4, 3, 3), (3, 4, 8), (5, 7, 13), (2, 33, 40), (139, 141, 4), (140, 141, 8)])
@pytest.mark.parametrize("values", ["few", "zeros", "special"])
def test_products_handed_on(shape, values):
    import torch
    from conftest import bits_equal

    from npbench_gb300 import stencils
    I, J, K = shape
    rng = np.random.default_rng(I * K)
    r = lambda *s: rng.random(s)  # noqa: E731
    us, w, up, ut = r(I, J, K), r(I + 1, J, K) - 0.5, r(I, J, K), r(I, J, K)
    choices = {"few": (0.25, 0.5, -0.5), "zeros": (0.0, -0.0, 0.5),
               "special": (0.25, 0.25, np.inf, -np.inf, np.nan, 5e-324, 0.0, -0.0)}[values]
    u = rng.choice(np.array(choices), size=shape)
    if values == "zeros":
        up, ut, us = up * 0.0, ut * -0.0, us * 0.0
        w[::2] = -0.0
    dev = [torch.from_numpy(x.copy()).cuda() for x in (us, u, w, up, ut)]
    stencils.vadv(*dev, 3.0 / 20.0)
    with np.errstate(all="ignore"):
        cref.vadv(us, u, w, up, ut, 3.0 / 20.0)
    assert bits_equal(dev[0].cpu().numpy(), us)
