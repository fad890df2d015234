"""Rows that the kNN cannot rank: more than 4,096 cells equidistant from one
cell.  Every entry point reports them as such, and the call after it is as good
as any."""

from __future__ import annotations

import numpy as np
import pytest

from mrustsc_gb300 import pp, synthetic
from mrustsc_gb300.anndata_lite import AnnData

pytestmark = pytest.mark.gpu

N, D = 5000, 20  # identical cells
MESSAGE = "more than 4096 cells are equidistant"


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


def identical() -> np.ndarray:
    return np.ones((N, D), np.float32)


def good(n: int) -> AnnData:
    return AnnData(obsm={"X_pca": synthetic.mixture(n, D, clusters=6, dup_frac=0.01, seed=n)})


@pytest.mark.parametrize("n_neighbors", [16, 41])
def test_the_graph_of_host_arrays(scrust, n_neighbors):
    first = good(9000)  # leaves ids past N in the workspace
    pp.neighbors(first, n_neighbors=n_neighbors)
    with pytest.raises(RuntimeError, match=MESSAGE):
        pp.neighbors(AnnData(obsm={"X_pca": identical()}), n_neighbors=n_neighbors)
    again = good(9000)
    pp.neighbors(again, n_neighbors=n_neighbors)
    for key in ("distances", "connectivities"):
        for a, b in zip((first.obsp[key].indices, first.obsp[key].data), (again.obsp[key].indices, again.obsp[key].data)):
            np.testing.assert_array_equal(a, b)
