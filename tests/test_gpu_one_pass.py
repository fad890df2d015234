"""pp.neighbors in one call against kNN and connectivities called one after the
other, on rows that the kNN cannot rank as well.

The arrays have to be the same bits: both ways take the same kNN, and the union
of a graph of distinct ids is formed in the same order by either path.
"""

from __future__ import annotations

import numpy as np
import pytest

from mrustsc_gb300 import pp
from mrustsc_gb300.anndata_lite import AnnData

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


class TwoCalls:
    """The core without its one-call form."""

    def __init__(self, core):
        self.knn, self.connectivities = core.knn, core.connectivities


def both(monkeypatch, scrust, x, n_neighbors, metric):
    out = []
    for core in (scrust, TwoCalls(scrust)):
        monkeypatch.setattr(pp, "_extension", lambda: core)
        adata = AnnData(obsm={"X_pca": x})
        try:
            pp.neighbors(adata, n_neighbors=n_neighbors, metric=metric)
        except ValueError as e:
            out.append(str(e))
            continue
        out.append([a for key in ("distances", "connectivities")
                    for m in (adata.obsp[key],) for a in (m.indptr, m.indices, m.data)])
    return out


# Two to 40 neighbours (the general union from 33 on), and graphs on both sides
# of the size from which the download goes range by range (4 Mi entries).
@pytest.mark.parametrize("n,d,k", [(3, 4, 3), (400, 10, 2), (2638, 50, 15), (30011, 20, 33), (3000, 20, 40),
                                   (140001, 8, 31)])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_one_call_is_two_calls(monkeypatch, scrust, n, d, k, metric):
    x = np.random.default_rng(n + k).standard_normal((n, d)).astype(np.float32)
    if n > 1000:
        x[7:300] = x[7]  # ties at zero
    one, two = both(monkeypatch, scrust, x, k, metric)
    for a, b in zip(one, two):
        assert a.dtype == b.dtype
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("bad", [1e30, -3e38])
def test_overflowing_rows(monkeypatch, scrust, bad):
    x = np.random.default_rng(0).standard_normal((500, 12)).astype(np.float32)
    x[11, 3] = bad
    x[200] = bad
    one, two = both(monkeypatch, scrust, x, 10, "euclidean")
    assert type(one) is type(two)
    if isinstance(one, str):
        assert one == two
    else:
        for a, b in zip(one, two):
            np.testing.assert_array_equal(a, b)
