"""Ordered solves on both sides of 18 anchors (4,608 rows), up to which the second
tile lists are what the priority lists leave of all tiles.

The data has far groups, so that the priority lists' order matters, and copies of
one row; neighbours are compared with a k-d tree's, by their f64 distances (the
lists are exact, so these are the same real numbers, summed in two orders: 1e-12
relative, and 0 for copies).
"""

from __future__ import annotations

import numpy as np
import pytest
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 1281, 4351, 4352, 4607, 4608, 4609, 8448])
@pytest.mark.parametrize("k", [2, 15, 40])
def test_few_anchors(built_library, n, k):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    rng = np.random.default_rng(n)
    x = (rng.integers(0, 5, n)[:, None] * 40.0 + rng.normal(size=(n, 4))).astype(np.float32)
    x[n // 2 : n // 2 + 8] = x[0]
    idx, _ = _scrust.knn(x, k, "auto")
    assert idx.max() < n and not np.any(idx == np.arange(n, dtype=np.uint32)[:, None])
    want, _ = cKDTree(x.astype(np.float64)).query(x.astype(np.float64), k + 1)
    got = np.sqrt(((x[:, None].astype(np.float64) - x[idx].astype(np.float64)) ** 2).sum(2))
    np.testing.assert_allclose(got, want[:, 1:], rtol=1e-12)
