"""Cosine distances bit for bit: the f32 rounding of the FP64 form with its sums
in the rows' order, whether the value came from f32 pairs or from f64.

Sizes: both sides of a multiple of eight dimensions, of the widest rows that
have padded copies (128), of the register rerank (32 neighbours) and of a block
of 64 normalised rows; rows from 1e-20 to 1e25 in scale (whose products leave
the range of the pairs), duplicates and near duplicates (whose distances lie at
or below the pairs' error).
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


def rows(n, d, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, d)) * np.linspace(1.0, 3.0, d)
    x[: n // 4] = x[: n // 4, :] * 1e-3 + rng.standard_normal(d) * 5  # a tight cone
    x[n // 3] = x[n // 3 + 1]
    x[n // 3 + 2] = x[n // 3 + 1] * (1 + 1e-7)
    x[n // 2 : n // 2 + 5] *= 1e-20
    x[n // 2 + 5 : n // 2 + 9] *= 1e16
    x[n // 2 + 9, 0] = 1e-39 if d > 1 else 1.0
    return x.astype(np.float32)


def fp64_distances(x, idx, of=None):
    """1 - x.y / (|x| |y|) in f64, every sum in coordinate order, rounded to f32."""
    x = x.astype(np.float64)
    n2 = np.zeros(len(x))
    for t in range(x.shape[1]):
        n2 = n2 + x[:, t] * x[:, t]
    norm = np.sqrt(n2)
    dot = np.zeros(idx.shape)
    for t in range(x.shape[1]):
        dot = dot + x[:, t][:, None] * x[idx, t]
    return (1.0 - dot / (norm[:, None] * norm[idx])).astype(np.float32)


@pytest.mark.parametrize("n,d", [(70, 1), (129, 7), (300, 8), (2049, 50), (2500, 64), (2200, 125), (400, 128), (400, 129)])
@pytest.mark.parametrize("k", [3, 32, 40])
@pytest.mark.parametrize("form", ["auto", "plain"])
def test_distances_are_the_fp64_forms(scrust, n, d, k, form):
    x = rows(n, d, n + d)
    idx, dist = scrust.knn(x, k, "auto", metric="cosine", form=form)
    np.testing.assert_array_equal(dist, fp64_distances(x, idx))


def test_distances_of_a_batch(scrust):
    samples = [rows(n, 30, n) for n in (100, 257, 1000)]
    for x, (idx, dist) in zip(samples, scrust.knn_batch(samples, 12, "auto", metric="cosine")):
        np.testing.assert_array_equal(dist, fp64_distances(x, idx))
