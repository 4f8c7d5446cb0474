"""The full-sky wavelets in the grid layout (levels of nside 16 and more): the
statistics and their gradient against the FP64 oracle where the layout can go
wrong -- nside 16, every tile of which reaches across face edges and vertices
(displacements of 5 cells), the first FP32 level above nside 32, and batches whose
row counts give a CTA one or two groups of 1, 2 or 4 rows; both kernel sizes.  Each
level is in the layout its size calls for."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,J,batch,dtype,kernel", [
    (16, 1, 1, "float64", 5), (16, 2, 3, "float64", 5), (32, 2, 2, "float64", 5), (16, 2, 2, "float64", 3),
    (64, 1, 1, "float32", 5), (64, 2, 2, "float32", 5), (64, 1, 3, "float32", 5), (64, 2, 4, "float32", 5),
    (64, 1, 8, "float32", 5), (64, 2, 4, "float32", 3)])
def test_grid_wavelets_match_the_oracle(nside, J, batch, dtype, kernel):
    import stl_b200
    rng = np.random.default_rng(1000 * nside + 10 * batch + J)
    x = np.exp(rng.standard_normal((batch, 12 * nside * nside)) - 0.5)
    e = stl_b200.NativeEngine(nside, J, batch=batch, dtype=dtype, kernel=kernel)
    o = O.OracleEngine(nside, J, batch=batch, kernel=kernel)
    v, r = e.forward(x)[0], o.forward(x)
    for d, op in enumerate(e.info()["operators"]):  # not the layout that a level falls back to
        assert op["layout"] == ("grid" if nside >> d >= 16 else "coloured"), (d, op)
    # FP64: sums of 44 products in another order; FP32: the 1e-6 criterion of the
    # statistics relative to the largest of their family, and for a gradient
    # value two chains of at most 44 and 8 rounded products: 52 * 2^-24 = 3.1e-6 of
    # its largest terms
    family = np.array([c["family"] for c in e.plan])
    for f in np.unique(family):
        a, b = v[:, family == f], r[:, family == f]
        assert np.max(np.abs(a - b)) <= (1e-12 if dtype == "float64" else 1e-6) * np.max(np.abs(b)), f
    cot = rng.standard_normal(v.shape) + 1j * rng.standard_normal(v.shape)
    g, gr = e.vjp(cot), o.vjp(cot)
    assert np.max(np.abs(g - gr)) <= (1e-11 if dtype == "float64" else 3.1e-6) * np.max(np.abs(gr))
    again = stl_b200.NativeEngine(nside, J, batch=batch, dtype=dtype, kernel=kernel, autotune=False)
    np.testing.assert_array_equal(again.forward(x)[0], v)  # whatever the tile heights
    np.testing.assert_array_equal(again.vjp(cot), g)
    e.close()
    again.close()


@pytest.mark.parametrize("kernel,dtype", [(3, "float32"), (5, "float32"), (3, "float64"), (5, "float64")])
def test_every_level_from_nside_16_on_has_the_grid_layout(kernel, dtype):
    import stl_b200
    e = stl_b200.NativeEngine(1024, 8, dtype=dtype, kernel=kernel, autotune=False)
    e.prepare()
    assert [o["layout"] for o in e.info()["operators"]] == ["grid"] * 7 + ["coloured"]
    e.close()
