"""Ordered solves at row-block counts on both sides of where the one-block sort
of the work order changes its width, and past its largest (8,192 blocks).

A row block left out of the order leaves rows unwritten; the neighbours of
sampled rows are compared with a k-d tree's, by their f64 distances (the lists
are exact, so these are the same real numbers, summed in two orders: 1e-12).
"""

from __future__ import annotations

import numpy as np
import pytest
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


@pytest.mark.parametrize("blocks", [9, 32, 33, 1024, 1025, 2049, 4097, 8193])
def test_every_row_block_is_solved(scrust, blocks):
    n, k = 256 * blocks - 100, 5
    rng = np.random.default_rng(blocks)
    x = rng.uniform(-100.0, 100.0, size=(n, 3)).astype(np.float32)
    idx, dist = scrust.knn(x, k, "auto")
    assert idx.max() < n and not np.any(idx == np.arange(n, dtype=np.uint32)[:, None])
    assert np.all(np.diff(dist, axis=1) >= 0)
    rows = np.unique(np.concatenate([rng.integers(0, n, 3000), [0, n - 1]]))
    want, _ = cKDTree(x.astype(np.float64)).query(x[rows].astype(np.float64), k + 1)
    d64 = np.sqrt(((x[rows, None].astype(np.float64) - x[idx[rows]].astype(np.float64)) ** 2).sum(2))
    np.testing.assert_allclose(d64, want[:, 1:], rtol=1e-12)
