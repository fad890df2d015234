"""The tensor form with two operand blocks per row (62 to 125 dimensions,
ordered solves of 2048 cells or more): the edges of the range, top-k widths on
both sides of 1, 16, 32 and 40, both operand types and metrics, sizes on and off
the tiles, against the FP64 oracle; and where it ends, the plain form."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from mrustsc_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(built_library):
    from mrustsc_gb300 import _lib, _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _lib


def solve(lib, x, k, **kw):
    """(ids, distances, sweep tiles, message) of one kNN call."""
    L = lib.lib()
    ctx = lib.context(0)
    st = lib.Status()
    n, d = x.shape
    opts = lib.options(**kw)
    idx = np.empty((n, k), np.uint32)
    dist = np.empty((n, k), np.float32)
    cnt = (ctypes.c_uint64 * 16)()
    L.scrust_cuda_kernel_stats(ctx, 1, cnt, 16)
    rc = L.scrust_cuda_knn(ctx, lib.ptr(x), n, d, k, ctypes.byref(opts), lib.ptr(idx), lib.ptr(dist), ctypes.byref(st))
    L.scrust_cuda_kernel_stats(ctx, 0, cnt, 16)
    lib.check(rc, st)
    return idx, dist, int(cnt[8]), st.message.decode()


def check(oracle, x, k, idx, dist, metric):
    """Ids equal to the FP64 kNN's, distances within 1e-6 relative (the FP32
    difference form is within (d / 4 + 4) 2^-24 = 2.1e-6 of d^2 at d = 125, so
    1.1e-6 of d; members of tie groups and cosine rows carry the FP64 value)."""
    oi, od = (oracle.knn_fp64(x, k) if metric == "euclidean" else oracle.knn_cosine_fp64(x, k))[:2]
    np.testing.assert_array_equal(idx, oi)
    bar = 1.2e-6 * np.abs(od) + (1e-7 if metric == "cosine" else 0.0)
    assert np.all(np.abs(dist.astype(np.float64) - od) <= bar)


@pytest.mark.parametrize("n,d,k", [(2048, 62, 15), (2049, 64, 16), (2303, 100, 17), (3000, 125, 32), (2500, 100, 1),
                                   (2500, 90, 2), (2600, 65, 33), (2700, 125, 41), (2048, 70, 64), (2400, 80, 65),
                                   (2100, 125, 128)])
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
def test_wide_rows_match_fp64(lib, oracle, n, d, k, precision):
    x = synthetic.mixture(n, d, clusters=6, dup_frac=0.01, near_dup_frac=0.01, seed=n + d + k)
    idx, dist, tiles, message = solve(lib, x, k, precision=precision)
    assert tiles > 0 and message == ""
    check(oracle, x, k, idx, dist, "euclidean")


def test_wide_rows_without_structure(lib, oracle):
    """Balls that prune nothing: every tile in both lists."""
    x = np.random.default_rng(3).normal(size=(2600, 110)).astype(np.float32)
    idx, dist, tiles, _ = solve(lib, x, 20)
    assert tiles > 0
    check(oracle, x, 20, idx, dist, "euclidean")


@pytest.mark.parametrize("d,k", [(62, 10), (125, 30)])
def test_wide_cosine_matches_the_plain_form(lib, d, k):
    x = synthetic.mixture(2300, d, clusters=6, dup_frac=0.01, seed=d)
    idx, dist, tiles, _ = solve(lib, x, k, metric="cosine")
    pidx, pdist, ptiles, _ = solve(lib, x, k, metric="cosine", form="plain")
    assert tiles > 0 and ptiles == 0
    np.testing.assert_array_equal(idx, pidx)
    np.testing.assert_array_equal(dist, pdist)


@pytest.mark.parametrize("n,d,kw", [(2047, 100, {}), (2300, 126, {}), (2300, 100, {"ordering": "off"}),
                                    (2300, 100, {"segments": 2}), (2300, 100, {"mode": "reference_snap"})])
def test_outside_its_range_the_plain_form_runs(lib, n, d, kw):
    x = synthetic.mixture(n, d, clusters=4, dup_frac=0.01, seed=5)
    _, _, tiles, message = solve(lib, x, 15, form="tensor", **kw)
    assert tiles == 0 and "ran the plain form" in message
    _, _, tiles, message = solve(lib, x, 15, **kw)
    assert tiles == 0 and message == ""
