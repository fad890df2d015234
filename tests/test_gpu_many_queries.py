"""One request of more query groups than a grid's second dimension has blocks
(65,535 groups of 64).

Neighbours are compared with a k-d tree's, by their f64 distances (the lists are
exact, so these are the same real numbers, summed in two orders: 1e-12 relative)."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu


def test_a_request_of_four_million_queries(built_library):
    from mrustsc_gb300 import _scrust, serving

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    k, groups = 2, 65_535
    r = np.random.default_rng(0)
    atlas = r.uniform(-100.0, 100.0, size=(20_000, 4)).astype(np.float32)
    query = r.uniform(-100.0, 100.0, size=(64 * groups + 1000, 4)).astype(np.float32)
    with serving.Server(atlas, k) as server:
        idx, dist, (indptr, _, _), _ = server.query(query)
    assert len(indptr) == len(query) + 1
    rows = np.concatenate([r.choice(64 * groups, 5000, replace=False), np.arange(64 * groups, len(query))])
    q = query[rows].astype(np.float64)
    want = cKDTree(atlas.astype(np.float64)).query(q, k)[0]
    got = np.sqrt(((q[:, None] - atlas[idx[rows]].astype(np.float64)) ** 2).sum(2))
    np.testing.assert_allclose(got, want, rtol=1e-12)
    np.testing.assert_allclose(dist[rows], want, rtol=1e-6)
