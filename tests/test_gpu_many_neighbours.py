"""Ordered solves of more than 32 neighbours: thresholds from the top-32 of a
row's two or four lists, one collect pass, and the rerank of four entries a
lane.  Sizes where the lists are short (one, two and three tiles, a last tile
of a few rows), k on both sides of 32, 40, 64 and at 128, data without
structure, copies past what the lists and the four entries hold, tie groups
of mirror pairs, both metrics, the graph and the plain form's results."""

from __future__ import annotations

import numpy as np
import pytest

import refdata
from mrustsc_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


def ordered(scrust, x, k, **kw):
    return scrust.knn(x, k, "auto", form="tensor", ordering="on", **kw)


@pytest.mark.parametrize("n", [200, 257, 300, 600, 1024, 3001])
@pytest.mark.parametrize("k", [33, 40, 41, 64, 65, 100, 128])
def test_matches_fp64(scrust, oracle, n, k):
    x = synthetic.mixture(n, 20, clusters=4, dup_frac=0.01, near_dup_frac=0.01, seed=n + k)
    idx, dist = ordered(scrust, x, k)
    oi, od = oracle.knn_fp64(x, k)[:2]
    np.testing.assert_array_equal(idx, oi)
    assert np.all(np.abs(dist.astype(np.float64) - od) <= 1e-6 * od)


@pytest.mark.parametrize("k", [50, 90])
def test_without_structure(scrust, oracle, k):
    x = refdata.random_embedding(4000, 12, 3)
    idx, _ = ordered(scrust, x, k)
    np.testing.assert_array_equal(idx, oracle.knn_fp64(x, k)[0])


@pytest.mark.parametrize("copies", [45, 130, 400])
def test_copies_around_the_entries_a_row_holds(scrust, oracle, copies):
    x = synthetic.mixture(2500, 16, clusters=5, dup_frac=0.0, seed=4)
    x[700:700 + copies] = x[700]
    idx, dist = ordered(scrust, x, 48)
    oi, od = oracle.knn_fp64(x, 48)[:2]
    np.testing.assert_array_equal(idx, oi)
    assert np.count_nonzero(dist[700] == 0) == min(48, copies - 1)


@pytest.mark.parametrize("k", [34, 70])
def test_tie_groups_match_the_plain_form(scrust, k):
    """Mirror pairs and triple copies on a 1/16 lattice, as exact ties."""
    g = np.random.default_rng(31)
    x = (g.integers(-32, 32, size=(1500, 4)) / 16.0).astype(np.float32)
    for r in range(40):
        e = (g.integers(1, 4, size=4) / 64.0).astype(np.float32)
        x[200 + 2 * r] = x[r] + e
        x[201 + 2 * r] = x[r] - e
    for r in range(40, 80):
        x[400 + 3 * (r - 40):403 + 3 * (r - 40)] = x[r] + np.float32(1.0 / 32.0)
    for metric in ("euclidean", "cosine"):
        y = x + np.float32(3.0) if metric == "cosine" else x
        idx, dist = ordered(scrust, y, k, metric=metric)
        pidx, pdist = scrust.knn(y, k, "auto", form="plain", metric=metric)
        np.testing.assert_array_equal(idx, pidx)
        np.testing.assert_array_equal(dist, pdist)


def test_graph_of_many_neighbours_matches_the_oracle(scrust, oracle):
    x = synthetic.mixture(2500, 30, clusters=5, dup_frac=0.01, seed=8)
    idx, dist, conn = scrust.neighbors_graph(x, 70)
    ref = oracle.connectivities(idx, dist)
    np.testing.assert_array_equal(conn[0], ref[0])
    np.testing.assert_array_equal(conn[1], ref[1])
    np.testing.assert_allclose(conn[2], ref[2], atol=1e-5, rtol=0)
