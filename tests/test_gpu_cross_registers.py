"""The cross products of the finest levels, kept in registers (5 and 9 operands
a channel; the VJP also 13): statistics, variances and gradients with and without
masks against the FP64 oracle, at a level of fewer pixels than a CTA's step and
at one of many ranges."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,J,B,masked", [(4, 1, 1, False), (8, 2, 2, True), (16, 3, 2, False), (32, 3, 1, True)])
def test_cross_products_match_the_oracle(nside, J, B, masked):
    import stl_b200
    rng = np.random.default_rng(17 * nside + J)
    n = 12 * nside * nside
    x = np.exp(rng.standard_normal((B, 2, n)) - 0.5)
    e = stl_b200.NativeEngine(nside, J, batch=B, dtype="float64", cross=True)
    o = O.OracleEngine(nside, J, batch=B, channels=2, cross_only=True)
    if masked:
        m = (rng.random((3, n)) < 0.6).astype(np.float64)
        e.set_masks(m)
        o.set_masks(m)
    v, var = e.forward(x, moments=True)
    r, rvar = o.forward(x, moments=True)
    # FP64 sums over at most 12 nside^2 pixels in another order
    assert np.max(np.abs(v - r)) <= 1e-12 * np.max(np.abs(r))
    assert np.max(np.abs(var - rvar)) <= 1e-11 * np.max(np.abs(rvar))
    cot = rng.standard_normal(r.shape) + 1j * rng.standard_normal(r.shape)
    g, gr = e.vjp(cot), o.vjp(cot).reshape(x.shape)
    # rn(z) has a gradient ~ |z|^-1/2, which magnifies the last bits where |z| is small
    assert np.max(np.abs(g - gr)) <= 1e-9 * np.max(np.abs(gr))
    np.testing.assert_array_equal(e.forward(x)[0], v)  # without variances: the same sums
    e.close()
