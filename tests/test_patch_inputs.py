"""The patches a disc engine is given, checked against its selection (no device
needed: the selection is set by hand, or made by a stand-in for the library)."""
import threading

import numpy as np
import pytest

import stl_b200


def selected(sizes):
    pe = stl_b200.PatchEngine.__new__(stl_b200.PatchEngine)
    pe._handle = None
    pe.ids = [np.arange(n) for n in sizes]
    pe._sizes = np.array(sizes, np.uintp)
    return pe


def test_patches_must_be_vectors_of_their_discs_size():
    pe = selected([1, 3])
    ok = np.arange(3.0)
    for scalar in (2.0, np.float64(2.0), np.array(2.0), np.array([[2.0]])):  # a disc of one pixel takes a vector of one
        with pytest.raises(ValueError, match="patch 0 has shape"):
            pe._parts([scalar, ok])
    for bad in (np.arange(4.0), ok[:2], ok[None], np.float64(1.0)):
        with pytest.raises(ValueError, match="patch 1 has shape"):
            pe._parts([[2.0], bad])
    with pytest.raises(ValueError, match="1 patches given for 2"):
        pe._parts([ok])


def test_patches_are_converted_to_contiguous_doubles():
    pe = selected([1, 3])
    for given in (np.arange(3, dtype=np.float32), np.arange(6.0)[::2] / 2, [0, 1, 2], np.arange(3.0)):
        flat, addresses = pe._parts([[7], given])
        assert all(m.dtype == np.float64 and m.flags.c_contiguous for m in flat)
        assert [a for a in addresses] == [m.ctypes.data for m in flat]
        np.testing.assert_array_equal(flat[1], [0.0, 1.0, 2.0])


def test_a_selection_that_fails_leaves_ids_and_sizes_of_one_selection():
    class Library:
        fail = False

        def stlp_patch_select(self, handle, vectors, n, radius, core, counts):
            for i in range(n):
                counts[i] = 5
            return 0

        def stlp_patch_ids(self, handle, i, out):
            return 0

        def stlp_patch_core_pixels(self, handle, out):
            return int(self.fail)

    pe = selected([])
    pe._mutex, pe._handle, pe._lib = threading.RLock(), 1, Library()
    pe._selection, pe.levels, pe._native, pe.nside = None, 2, np.zeros(3, np.int64), 16
    pe.close = lambda: None
    pe.select(np.eye(3)[:2], 10.0)
    assert len(pe.ids) == pe._sizes.size == pe._cuts.size == 2
    pe._lib.fail = True
    with pytest.raises((RuntimeError, ValueError)):
        pe.select(np.eye(3), 20.0)
    assert len(pe.ids) == pe._sizes.size == pe._cuts.size == 2 and pe._selection is None
