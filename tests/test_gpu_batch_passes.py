"""Batches by two passes against single solves of the plain form, bit for bit.

Sample sizes around the neighbour count, the columns that give every minimum of
a first tile (8 k and 4 k), a tile's halves and tiles; duplicated rows past a
list's 256 entries, which take the exact fallback.
"""

from __future__ import annotations

import numpy as np
import pytest

from mrustsc_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


def check(scrust, samples, k, **kw):
    out = scrust.knn_batch(samples, k, "auto", **kw)
    for x, (idx, dist) in zip(samples, out):
        pi, pd = scrust.knn(x, k, "auto", form="plain", **kw)
        np.testing.assert_array_equal(idx, pi)
        np.testing.assert_array_equal(dist, pd)


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 32, 33])
@pytest.mark.parametrize("d", [3, 61])
def test_sample_sizes(scrust, k, d):
    sizes = [k + 1, k + 2, 4 * k + 1, 8 * k, 8 * k + 1, 16 * k, 127, 128, 129, 255, 256, 257, 511, 769, 4097, 5000]
    rng = np.random.default_rng(k * 100 + d)
    samples = [rng.standard_normal((max(n, k + 1), d)).astype(np.float32) for n in sizes]
    check(scrust, samples, k)


def test_duplicates_past_a_list(scrust):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((1500, 20)).astype(np.float32)
    x[100:900] = x[99]
    y = synthetic.mixture(600, 20, clusters=3, dup_frac=0.5, seed=1)
    check(scrust, [x, y, x[:300]], 12)


def test_cosine(scrust):
    rng = np.random.default_rng(6)
    check(scrust, [rng.standard_normal((n, 30)).astype(np.float32) for n in (40, 300, 2100)], 20, metric="cosine")
