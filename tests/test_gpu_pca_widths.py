"""PCA at sketch widths around its kernels' tiles (32-column slabs, four-column
groups, odd and even numbers of rotated columns, the widest sketch) and rows
and genes of 0, 1, 31, 32, 33 and many entries, against the FP64 PCA.

A planted spectrum whose singular values fall by 0.8 a component: what the
power iterations leave of the leading components beyond the sketch is below
f32 rounding, so a leading variance carries the rounding of f32 products
alone.  Each of the ~5 products it passes through sums up to 700 terms in f32,
whose relative error in norm is at most 700 * 2^-24 = 4.2e-5 and of a variance
twice that; 4e-4 bounds five of them."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import pca_oracle

pytestmark = pytest.mark.gpu


def planted(n, g, rank):
    r = np.random.default_rng(n + g)
    left = np.linalg.qr(r.normal(size=(n, rank)))[0]
    right = np.linalg.qr(r.normal(size=(g, rank)))[0]
    x = (left * (200.0 * 0.8 ** np.arange(rank))) @ right.T
    x += r.normal(size=(n, g)) * 1e-3
    x[np.abs(x) < 0.02] = 0.0  # some sparsity
    for row, keep in ((3, 0), (4, 1), (5, 31), (6, 32), (7, 33)):
        x[row, keep:] = 0.0
    for col, keep in ((2, 0), (3, 1), (4, 31), (5, 32), (6, 33)):
        x[keep:, col] = 0.0
    return x.astype(np.float32)


@pytest.mark.parametrize("n,g,nc", [(700, 300, 1), (700, 300, 8), (700, 300, 9), (700, 300, 40), (300, 700, 41),
                                    (700, 300, 72), (700, 300, 73), (700, 300, 104), (90, 33, 20), (40, 64, 30)])
@pytest.mark.parametrize("zero_center", [True, False])
def test_leading_components_match_the_exact_pca(built_library, n, g, nc, zero_center):
    from mrustsc_gb300 import _scrust

    x = planted(n, g, 30)
    m = sp.csr_matrix(x)
    res = _scrust.pca(m.indptr.astype(np.uint32), m.indices.astype(np.uint32), m.data.astype(np.float32), g, nc,
                      zero_center, 0, "auto")
    lead = min(nc, 5)
    emb, comps, var, ratio = pca_oracle.exact_pca(x.astype(np.float64), lead, zero_center=zero_center)
    np.testing.assert_allclose(res["explained_variance"][:lead], var[:lead], rtol=4e-4)
    np.testing.assert_allclose(res["explained_variance_ratio"][:lead], ratio[:lead], rtol=4e-4)
    for c in range(lead):
        assert pca_oracle.correlation(res["embedding"][:, c], emb[:, c]) >= 0.9999
        assert pca_oracle.correlation(res["components"][c], comps[c]) >= 0.9999
    gram = res["components"][:lead].astype(np.float64) @ res["components"][:lead].T
    assert np.abs(gram - np.eye(lead)).max() <= 4e-4
    assert np.all(np.diff(res["explained_variance"].astype(np.float64)) <= 1e-6 * res["explained_variance"][0])


def test_a_rank_deficient_matrix_has_no_variance_past_its_rank(built_library):
    from mrustsc_gb300 import _scrust

    r = np.random.default_rng(5)
    x = (r.normal(size=(200, 3)) @ r.normal(size=(3, 60))).astype(np.float32)
    m = sp.csr_matrix(x)
    res = _scrust.pca(m.indptr.astype(np.uint32), m.indices.astype(np.uint32), m.data.astype(np.float32), 60, 8, True,
                      0, "auto")
    var = res["explained_variance"]
    assert np.isfinite(res["embedding"]).all() and np.isfinite(res["components"]).all()
    assert np.all(var[3:] <= 1e-6 * var[0]) and np.all(var[:3] > 1e-2 * var[0])
