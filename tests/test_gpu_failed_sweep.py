"""A sweep that failed (its error flag set, here from outside, as a wait that ran out
sets it) raises, and the caller's gradient array is left as it was: for the
small pinned buffer, one and several pinned chunks, FP32 widened on the host, and
device tensors.  The next call works again."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Flag:
    """The engine's error flag as a CUDA array of one int32."""

    def __init__(self, engine):
        address = C.c_uint64()
        assert engine._lib.stlp_error_flag(engine._handle, C.byref(address)) == 0
        self.__cuda_array_interface__ = dict(shape=(1,), typestr="<i4", data=(address.value, False), version=2)


@pytest.mark.parametrize("nside,batch,dtype", [
    (16, 1, "float64"), (256, 1, "float64"), (512, 2, "float64"), (64, 1, "float32"), (512, 4, "float32")])
def test_a_failed_reverse_sweep_leaves_the_gradient(nside, batch, dtype):
    import stl_b200
    import torch
    rng = np.random.default_rng(nside)
    x = rng.standard_normal((batch, 12 * nside * nside))
    e = stl_b200.NativeEngine(nside, 2, batch=batch, dtype=dtype)
    v, _ = e.forward(x)
    flag = torch.as_tensor(Flag(e), device="cuda")

    def fail():
        flag.fill_(1)
        torch.cuda.synchronize()

    want = e.vjp(v).copy()
    out = np.full(want.shape, 7.0)
    fail()
    with pytest.raises(RuntimeError, match="timed out in the reverse sweep"):
        e.vjp(v, out=out)
    assert (out == 7.0).all()
    np.testing.assert_array_equal(e.vjp(v, out=out), want)
    for kind in (torch.float32, torch.float64):
        dev = torch.full(want.shape, 7.0, dtype=kind, device="cuda")
        fail()
        with pytest.raises(RuntimeError, match="timed out in the reverse sweep"):
            e.vjp_tensor(v, dev)
        assert bool((dev == 7.0).all())
        e.vjp_tensor(v, dev)
        np.testing.assert_array_equal(dev.cpu().numpy(), want.astype(dev.cpu().numpy().dtype))
    fail()
    with pytest.raises(RuntimeError, match="timed out in the forward sweep"):
        e.forward(x)
    np.testing.assert_array_equal(e.forward(x)[0], v)
    e.close()
