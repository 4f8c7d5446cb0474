"""Patches gathered from memory of their own while they are copied
(stlp_patch_forward_parts): the same statistics, bit for bit, as the packed
vector's, where parts end inside and across the copy threads' ranges and the pinned
chunks (32 MB); other dtypes and strides are converted first; a non-finite value
in any part is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,radii", [(64, [9.0, 25.0, 3.0, 14.0, 30.0, 1.5]),  # one small pinned buffer
                                         (512, [13.0 + 0.37 * i for i in range(48)])])  # two pinned chunks
def test_parts_equal_the_packed_patches(nside, radii):
    import stl_b200
    rng = np.random.default_rng(nside)
    centres = rng.standard_normal((len(radii), 3))
    pe = stl_b200.PatchEngine(nside, 2, dtype="float32", autotune=False)
    ids = pe.select(centres, np.array(radii))
    patches = [rng.standard_normal(i.size) for i in ids]
    packed = np.concatenate(patches)
    assert (packed.nbytes > 32 << 20) == (nside == 512)
    v, _ = pe.forward(patches, moments=False, generation=1)
    p = stl_b200._ptr
    again = np.empty_like(v)
    assert pe._lib.stlp_patch_forward(pe._handle, p(packed), packed.size, 2, False, p(again.view(np.float64)), None) == 0
    np.testing.assert_array_equal(again, v)
    mixed = [x.astype(np.float32) if i % 2 else np.repeat(x, 2)[::2] for i, x in enumerate(patches)]
    same = [np.asarray(x, np.float64).copy() for x in mixed]
    np.testing.assert_array_equal(pe.forward(mixed, moments=False)[0], pe.forward(same, moments=False)[0])
    for i in (0, len(ids) - 1):
        bad = list(patches)
        bad[i] = patches[i].copy()
        bad[i][-1] = np.inf
        with pytest.raises(ValueError):
            pe.forward(bad, moments=False)
    with pytest.raises(ValueError):
        pe.forward([x[:-1] for x in patches], moments=False)
    pe.close()


def test_statistics_may_overwrite_the_patches():
    """``out`` in the patches' own memory: the discs of a later engine group are read
    after the statistics of an earlier one were written."""
    import stl_b200
    rng = np.random.default_rng(5)
    pe = stl_b200.PatchEngine(32, 2, autotune=False, group_pixels=1)  # a group a disc
    ids = pe.select(rng.standard_normal((3, 3)), 40.0)
    assert sum(i.size for i in ids) > 2 * 3 * pe.ncoeff
    buf = rng.standard_normal(sum(i.size for i in ids))
    patches = np.split(buf, np.cumsum([i.size for i in ids])[:-1])
    want = pe.forward([p.copy() for p in patches], moments=False)[0]
    out = buf[-2 * want.size:].view(np.complex128).reshape(want.shape)  # the last patch among it
    got = pe.forward(patches, moments=False, out=out)[0]
    assert got is out
    np.testing.assert_array_equal(got, want)
    pe.close()
