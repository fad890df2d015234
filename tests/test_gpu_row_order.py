"""Rows put in the order of their anchors by one block (up to 8,192 rows) and by
the general sort above it, at the sizes where the block's groups change and
with one and two digits of anchors (an atlas of up to 128 anchors, of more).

A row lost or doubled by the order leaves another row's answer or none in its
place; neighbours are compared with a k-d tree's, by their f64 distances (the
lists are exact, so these are the same real numbers, summed in two orders:
1e-12 relative).
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


def points(n: int, seed: int) -> np.ndarray:
    return np.random.default_rng(seed).uniform(-100.0, 100.0, size=(n, 3)).astype(np.float32)


def check(query: np.ndarray, rows: np.ndarray, idx: np.ndarray, own: bool) -> None:
    k = idx.shape[1]
    want, _ = cKDTree(rows.astype(np.float64)).query(query.astype(np.float64), k + own)
    got = np.sqrt(((query[:, None].astype(np.float64) - rows[idx].astype(np.float64)) ** 2).sum(2))
    np.testing.assert_allclose(got, want[:, own:], rtol=1e-12)


@pytest.mark.parametrize("n", [1024, 1025, 1055, 2048, 2049, 4096, 4097, 8192, 8193])
def test_rows_of_a_solve(scrust, n):
    x = points(n, n)
    idx, _ = scrust.knn(x, 6, "auto")
    assert not np.any(idx == np.arange(n, dtype=np.uint32)[:, None])
    check(x, x, idx, True)


@pytest.mark.parametrize("cells", [20_000, 32_768, 33_100, 300_000])
def test_rows_of_a_query(built_library, cells):
    from mrustsc_gb300 import serving

    atlas = points(cells, cells)
    server = serving.Server(atlas, 6)
    try:
        for q in (1, 2, 33, 1024, 1025, 4097, 8192, 8193):
            query = points(q, q)
            idx, _, _, _ = server.query(query)
            check(query, atlas, idx, False)
    finally:
        server.close()
