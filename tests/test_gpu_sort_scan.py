"""The device sort where its digit scan changes rounds: a round covers 2048 tiles of
4096 keys, so rows that end with the round, one key past it, and within its
last tile, against the stable total order of the oracle."""
import numpy as np
import pytest

import terms as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047 * 4096 + 5, 2048 * 4096, 2048 * 4096 + 1])
def test_sort_across_a_scan_round(n):
    import torch
    import stl_b200
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32).astype(np.float64)  # with ties
    x[:: 1000] = -0.0
    t = stl_b200.Terms(sort=n)
    perm = t.sort(torch.tensor(x, device="cuda")).cpu().numpy().astype(np.int64)
    np.testing.assert_array_equal(perm, T.sort_positions(x))
    t.close()
