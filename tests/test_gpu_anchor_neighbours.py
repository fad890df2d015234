"""Ordered solves whose anchors have many equal distances between them: more
candidates for an anchor's nearest than its sort holds (256), which go through
the lists in every lane, and anchors all at one point.  The neighbours have to
be the plain form's, and every row solved.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


# Rows on the corners of a cube: n / 256 anchors, an eighth of them at each
# corner (n = 150,000: 73 at distance 0, 220 at the next).
@pytest.mark.parametrize("n", [2304, 20_000, 150_000])
@pytest.mark.parametrize("corners", [1, 8])
def test_anchors_at_equal_distances(scrust, n, corners):
    rng = np.random.default_rng(n)
    cube = np.array([[(c >> b) & 1 for b in range(3)] for c in range(corners)], np.float32) * 4
    x = np.concatenate([cube[np.arange(n) % corners], np.zeros((n, 5), np.float32)], 1)
    spread = rng.permutation(n)[: n // 2]
    x[spread, 3:] = rng.standard_normal((len(spread), 5)).astype(np.float32) * 0.5
    x[spread] += 0.01
    rows = spread[rng.integers(0, len(spread), 200)]
    keep = np.unique(np.concatenate([spread, rng.permutation(n)[:200]]))
    y = x[keep]  # few duplicates: lists need not overflow
    idx, dist = scrust.knn(y, 6, "auto", form="tensor", ordering="on")
    at = np.searchsorted(keep, rows)
    d = ((y[at, None].astype(np.float64) - y[None].astype(np.float64)) ** 2).sum(2) if len(y) < 20_000 else None
    if d is None:
        pi, pd = scrust.knn(y, 6, "auto", form="plain")
        np.testing.assert_array_equal(idx, pi)
        np.testing.assert_array_equal(dist, pd)
        return
    d[np.arange(len(at)), at] = np.inf
    np.testing.assert_allclose(dist[at], np.sqrt(np.sort(d, 1)[:, :6]), rtol=1e-6, atol=1e-6)
