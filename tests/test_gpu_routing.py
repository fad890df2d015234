"""Queries routed to an ordered atlas, and ordered self solves, on data whose
cells are small: more clusters than a 256-row block's segments or home cells
hold, clusters of fewer rows than k, copies past the entries a row holds,
queries far from every cell, top-k widths on both sides of 1, 16 and 32, batch
sizes that leave one, few and many column segments."""

from __future__ import annotations

import numpy as np
import pytest

from mrustsc_gb300 import serving

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


def tiny_clusters(n, d, per, seed):
    """n rows in clusters of `per`, far apart."""
    g = np.random.default_rng(seed)
    centres = g.uniform(-20, 20, size=(-(-n // per), d))
    x = centres[np.arange(n) // per] + g.normal(size=(n, d)) * 0.3
    return np.ascontiguousarray(x[g.permutation(n)], dtype=np.float32)


@pytest.mark.parametrize("per", [3, 12, 40, 200])
@pytest.mark.parametrize("k", [1, 15, 31])
def test_self_solve_of_tiny_clusters(scrust, oracle, per, k):
    x = tiny_clusters(6000, 8, per, per + k)
    idx, _ = scrust.knn(x, k, "auto", form="tensor", ordering="on")
    np.testing.assert_array_equal(idx, oracle.knn_fp64(x, k)[0])


@pytest.mark.parametrize("k", [1, 2, 16, 17, 32])
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
def test_queries_on_tiny_clusters(scrust, oracle, k, precision):
    g = np.random.default_rng(k)
    atlas = tiny_clusters(9000, 12, 25, 5)
    atlas[100:400] = atlas[100]  # copies: more than a row's entries hold
    with serving.Server(atlas, k, precision=precision) as server:
        for q in (1, 5, 257, 1500):
            x = atlas[g.integers(0, len(atlas), q)] + g.normal(size=(q, 12)).astype(np.float32) * 0.1
            x[0] = atlas[100]
            if q > 4:
                x[1] = 300.0  # far from every cell
                x[2] = 0.0
            x = np.ascontiguousarray(x, dtype=np.float32)
            idx, dist, _, _ = server.query(x)
            oi, od = oracle.knn_fp64_cross(x, atlas, k)
            np.testing.assert_array_equal(idx, oi)
            assert np.all(np.abs(dist.astype(np.float64) - od) <= 1e-6 * od)
