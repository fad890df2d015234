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


def device_graph(x, k, form, prefill=0):
    """The device graph call; ids prefilled with `prefill`.  (ids, the status
    of the synchronise that follows)"""
    import ctypes

    torch = pytest.importorskip("torch")
    from mrustsc_gb300 import _lib

    L, ctx, st = _lib.lib(), _lib.context(0), _lib.Status()
    n, d = x.shape
    dx = torch.from_numpy(x).cuda()
    idx = torch.full((n, k), prefill, dtype=torch.int32, device="cuda")
    dist = torch.zeros((n, k), device="cuda")
    torch.cuda.synchronize()
    out = ctypes.c_void_p()
    _lib.check(L.scrust_cuda_neighbors_graph_device(ctx, dx.data_ptr(), n, d, k, ctypes.byref(_lib.options(form=form)),
                                                    idx.data_ptr(), dist.data_ptr(), ctypes.byref(out),
                                                    ctypes.byref(st)), st)
    code = L.scrust_cuda_synchronize(ctx, ctypes.byref(st))
    L.scrust_csr_free(out)
    return idx.cpu().numpy(), code, st.message.decode()


def assert_first_others(ids: np.ndarray, k: int):
    """Every row holds the first k ids other than its own."""
    rows = np.arange(len(ids))[:, None]
    t = np.arange(k)[None, :]
    np.testing.assert_array_equal(ids, t + (t >= rows))


@pytest.mark.parametrize("k", [15, 40])
def test_the_graph_of_device_arrays(scrust, k):
    ids, code, message = device_graph(identical(), k, "auto", prefill=N - 1)
    assert code and MESSAGE in message
    assert_first_others(ids, k)
    ids, code, message = device_graph(good(9000).obsm["X_pca"], k, "auto")
    assert code == 0, message


@pytest.mark.parametrize("form", ["plain", "tensor"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e30, -3e38])
@pytest.mark.parametrize("n,k", [(300, 5), (3000, 15), (3000, 40)])
def test_rows_that_are_no_numbers(scrust, form, bad, n, k):
    """Whatever the status, every row's ids are distinct others of its own."""
    x = np.random.default_rng(n).standard_normal((n, 20)).astype(np.float32)
    x[n // 2, 3] = bad
    ids, code, message = device_graph(x, k, form, prefill=n - 1)
    assert code == 0 or "inconsistent candidate set" in message
    assert ids.min() >= 0 and ids.max() < n
    assert not np.any(ids == np.arange(n)[:, None])
    assert np.all(np.diff(np.sort(ids, axis=1), axis=1) > 0)


def test_a_batch_with_such_a_sample(scrust):
    samples = [good(700).obsm["X_pca"], identical(), good(400).obsm["X_pca"]]
    want = scrust.knn_batch([samples[0], samples[2]], 15, "auto")
    with pytest.raises(RuntimeError, match=MESSAGE):
        scrust.neighbors_graph_batch(samples, 15, "auto")
    again = scrust.knn_batch([samples[0], samples[2]], 15, "auto")
    for (a, b), (c, d) in zip(want, again):
        np.testing.assert_array_equal(a, c)
        np.testing.assert_array_equal(b, d)
