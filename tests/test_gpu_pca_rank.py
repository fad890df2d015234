"""PCA asked for more components than the matrix has, at and around its rank.

A component past the rank stands on what the f32 products leave of the data
there, but it is a component all the same: its loadings have unit norm and are
orthogonal to the others' as far as the Gram of the projection resolves them.

The bounds: the projection's rows b_a past the rank r are of one size, those
before it larger, and an eigenvector past the rank weighs the rows before it by
no more than the ratio, so that the Gram's rounding (chains of 32 f32 products,
34 * 2^-24 of every entry) changes the product of two eigenvectors by at most
34 * 2^-24 (w + r)^2 of the size of the eigenvalues there, w = r + 4 + 20 the
sketch's width: 4e-3 for r = 10.  The first four eigenvalues past the rank lie
within a factor of ten of that size: 0.04 on a squared norm, doubled for the
products themselves."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [3, 5, 10])
@pytest.mark.parametrize("zero_center", [True, False])
def test_loadings_past_the_rank_are_orthonormal(built_library, rank, zero_center):
    from mrustsc_gb300 import _scrust

    r = np.random.default_rng(rank)
    x = (np.abs(r.normal(size=(2000, rank))) @ np.abs(r.normal(size=(rank, 200)))).astype(np.float32)
    m = sp.csr_matrix(x)
    res = _scrust.pca(m.indptr.astype(np.uint32), m.indices.astype(np.uint32), m.data, 200, rank + 4, zero_center, 0,
                      "auto")
    components = res["components"].astype(np.float64)
    np.testing.assert_allclose(components @ components.T, np.eye(rank + 4), atol=0.08)
    # The scores past the rank: what f32 products of 200 terms leave of the first.
    size = np.linalg.norm(res["embedding"].astype(np.float64), axis=0)
    assert np.all(size[rank:] <= 200 * 2.0 ** -24 * size[0])


def with_constant_columns(n, g):
    x = np.random.default_rng(n * g).random((n, g))
    x[:, ::2] = 3.0
    return x


def two_kinds_of_rows(n, g):
    x = np.zeros((n, g))
    x[: n // 2] = 1.0
    return x


@pytest.mark.parametrize("make", [with_constant_columns, two_kinds_of_rows])
@pytest.mark.parametrize("n,g", [(20, 50), (33, 33), (300, 40), (150, 300)])
@pytest.mark.parametrize("zero_center", [True, False])
def test_loadings_of_nothing_are_small(built_library, make, n, g, zero_center):
    """All components of matrices of low rank: where f32 resolves nothing of a
    component its loadings are zero; else their error is at most what it could
    resolve, the component's own size 1, so that no norm passes 2."""
    from mrustsc_gb300 import _lib, _scrust

    m = sp.csr_matrix(make(n, g).astype(np.float32))
    nc = min(n, g, 40)
    try:
        res = _scrust.pca(m.indptr.astype(np.uint32), m.indices.astype(np.uint32), m.data, g, nc, zero_center, 0, "auto")
    except _lib.ScrustError as e:
        assert "did not converge" in str(e) and make is two_kinds_of_rows  # refused, as it was
        return
    assert np.isfinite(res["components"]).all() and np.isfinite(res["embedding"]).all()
    assert np.linalg.norm(res["components"].astype(np.float64), axis=1).max() <= 2.0
    assert np.all(res["explained_variance"] >= 0)
