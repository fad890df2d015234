"""Several contexts in one process on the GPU."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from mrustsc_gb300 import synthetic

pytestmark = pytest.mark.gpu


def test_a_small_solve_on_one_context_leaves_the_limits_of_another(built_library, oracle):
    """The ordering's kernels take shared memory by the number of rows, and
    the limit is the kernel's, not the context's: a context that solved a
    large set still solves one after another context solved a small set."""
    from mrustsc_gb300 import _lib

    L = _lib.lib()
    st = _lib.Status()
    opts = _lib.options(form="tensor", ordering="on")
    contexts = [L.scrust_cuda_context_create(0, ctypes.byref(st)) for _ in range(2)]
    assert all(contexts)
    try:
        for ctx, n in ((contexts[0], 9000), (contexts[1], 1100), (contexts[0], 8000)):
            x = synthetic.mixture(n, 20, clusters=6, dup_frac=0.01, seed=n)
            idx = np.empty((n, 10), np.uint32)
            dist = np.empty((n, 10), np.float32)
            _lib.check(L.scrust_cuda_knn(ctx, _lib.ptr(x), n, 20, 10, ctypes.byref(opts), _lib.ptr(idx),
                                         _lib.ptr(dist), ctypes.byref(st)), st)
            np.testing.assert_array_equal(idx, oracle.knn_fp64(x, 10)[0])
    finally:
        for ctx in contexts:
            L.scrust_cuda_context_destroy(ctx)
