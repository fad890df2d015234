"""Queries at counts that cut the atlas into few, many (more than 16, so that a
lane of the merge holds four lists and the rerank walks its lists in groups of
32) and the most column segments, for the register top-16 and top-32 and k = 1.

Neighbours are compared with a k-d tree's, by their f64 distances (the lists are
exact, so these are the same real numbers, summed in two orders: 1e-12 relative).
"""

from __future__ import annotations

import numpy as np
import pytest
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu


def points(n: int, seed: int) -> np.ndarray:
    return np.random.default_rng(seed).uniform(-100.0, 100.0, size=(n, 4)).astype(np.float32)


@pytest.mark.parametrize("cells", [8_500, 16_700, 120_000])
@pytest.mark.parametrize("k", [1, 2, 16, 17, 32])
def test_queries(built_library, cells, k):
    from mrustsc_gb300 import _scrust, serving

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    atlas = points(cells, cells)
    tree = cKDTree(atlas.astype(np.float64))
    server = serving.Server(atlas, k)
    try:
        for q in (1, 40, 300, 1500, 2600, 5000):
            query = points(q, q)
            idx, _, _, _ = server.query(query)
            want = tree.query(query.astype(np.float64), k)[0].reshape(q, k)
            got = np.sqrt(((query[:, None].astype(np.float64) - atlas[idx].astype(np.float64)) ** 2).sum(2))
            np.testing.assert_allclose(got, want, rtol=1e-12)
    finally:
        server.close()
