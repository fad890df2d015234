"""The exact fallback of rows whose lists overflow, a cluster of blocks a row,
against the plain form, bit for bit: more such rows than clusters, solves whose
columns do not divide among a cluster's blocks (and batches, where a row's
columns are its own sample), both metrics, and tie groups across the blocks'
shares.
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


def crowded(n, d, seed):
    """Half of the rows within rounding of a few points: more than a list holds."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, d)).astype(np.float32)
    points = rng.standard_normal((3, d)).astype(np.float32)
    who = rng.permutation(n)[: n // 2]
    x[who] = points[rng.integers(0, 3, len(who))]
    near = who[: len(who) // 2]
    x[near] *= (1 + rng.uniform(-2e-7, 2e-7, (len(near), 1))).astype(np.float32)
    return x


def same(a, b):
    for u, v in zip(a, b):
        np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("n", [2501, 4103, 9000])
@pytest.mark.parametrize("k", [3, 20, 50])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_self_solves(scrust, n, k, metric):
    x = crowded(n, 12, n + k)
    same(scrust.knn(x, k, "auto", metric=metric, form="tensor", ordering="on"),
         scrust.knn(x, k, "auto", metric=metric, form="plain"))


def test_batches(scrust):
    samples = [crowded(n, 12, n) for n in (1801, 2600, 1203)]
    for x, got in zip(samples, scrust.knn_batch(samples, 15, "auto")):
        same(got, scrust.knn(x, 15, "auto", form="plain"))
