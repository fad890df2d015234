"""The exact fallback on both sides of the number of columns up to which a row
is a block's and from which it is a cluster's, and at the smallest solves, against
the oracle's FP64 neighbours."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crowded(n, d, seed):
    """A third of the rows copies of a few points, up to 1,500 of each: more
    than a row's lists hold, fewer than the 4,096 the fallback takes."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, d)).astype(np.float32)
    points = rng.standard_normal((max(1, n // 4500), d)).astype(np.float32)
    who = rng.permutation(n)[: n // 3]
    x[who] = points[rng.integers(0, len(points), len(who))]
    return x


@pytest.mark.parametrize("n,k", [(300, 5), (2500, 15), (2500, 40), (32_768, 15), (32_769, 15), (32_769, 40)])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_rows_past_their_lists(built_library, oracle, n, k, metric):
    from mrustsc_gb300 import _scrust

    x = crowded(n, 12, n + k)
    idx, _ = _scrust.knn(x, k, "auto", metric=metric, form="tensor")
    np.testing.assert_array_equal(idx, oracle.knn_fp64(x, k, metric=metric)[0])
