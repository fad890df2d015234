"""Batch plans between other calls on their context that grow its workspace:
every launch gives what the first one gave."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from mrustsc_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

D = 20


class View:
    """A device array of the plan's, for torch."""

    def __init__(self, ptr, count, typestr):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


class Plan:
    def __init__(self, ctx, sizes, k, metric="euclidean", list_capacity=0):
        import torch

        self.torch, self.ctx, self.k, self.L, self.st = torch, ctx, k, _lib.lib(), _lib.Status()
        x = np.concatenate([synthetic.mixture(n, D, clusters=5, dup_frac=0.01, seed=n) for n in sizes])
        self.n = len(x)
        self.x = torch.from_numpy(x).cuda()
        self.idx = torch.empty((self.n, k), dtype=torch.int32, device="cuda")
        self.dist = torch.empty((self.n, k), device="cuda")
        offsets = np.zeros(len(sizes) + 1, np.uint64)
        offsets[1:] = np.cumsum(sizes)
        torch.cuda.synchronize()
        opts = _lib.options(form="tensor", metric=metric, list_capacity=list_capacity)
        self.p = self.L.scrust_cuda_batch_plan_create_graphs(ctx, _lib.ptr(offsets), len(sizes), D, k,
                                                             ctypes.byref(opts), self.x.data_ptr(),
                                                             self.idx.data_ptr(), self.dist.data_ptr(),
                                                             ctypes.byref(self.st))
        assert self.p, self.st.message.decode()

    def launch(self):
        self.idx.zero_()
        self.dist.zero_()
        self.torch.cuda.synchronize()
        _lib.check(self.L.scrust_cuda_batch_plan_launch(self.p, ctypes.byref(self.st)), self.st)
        _lib.check(self.L.scrust_cuda_synchronize(self.ctx, ctypes.byref(self.st)), self.st)
        ip, ix, vl = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
        self.L.scrust_cuda_batch_plan_graph(self.p, ctypes.byref(ip), ctypes.byref(ix), ctypes.byref(vl))
        grab = lambda p, count, kind: self.torch.as_tensor(View(p.value, count, kind), device="cuda").cpu().numpy()
        indptr = grab(ip, self.n + 1, "<i4")
        return [self.idx.cpu().numpy(), self.dist.cpu().numpy(), indptr, grab(ix, int(indptr[-1]), "<i4"),
                grab(vl, int(indptr[-1]), "<f4")]

    def close(self):
        self.L.scrust_cuda_batch_plan_destroy(self.p)


def same(a, b):
    for u, v in zip(a, b):
        np.testing.assert_array_equal(u, v)


def solve(ctx, n, k, metric):
    L, st = _lib.lib(), _lib.Status()
    x = synthetic.mixture(n, D, clusters=20, dup_frac=0.01, seed=n)
    idx, dist, out = np.empty((n, k), np.uint32), np.empty((n, k), np.float32), ctypes.c_void_p()
    opts = _lib.options(metric=metric)
    _lib.check(L.scrust_cuda_neighbors_graph(ctx, _lib.ptr(x), n, D, k, ctypes.byref(opts), _lib.ptr(idx),
                                             _lib.ptr(dist), ctypes.byref(out), ctypes.byref(st)), st)
    L.scrust_csr_free(out)


# Two passes, lists of a given capacity and more neighbours than either; a
# context of its own, so that nothing has grown the workspace before.
@pytest.mark.parametrize("k,capacity", [(15, 0), (15, 128), (40, 0)])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_launches_between_larger_calls(built_library, k, capacity, metric):
    pytest.importorskip("torch")
    L, st = _lib.lib(), _lib.Status()
    ctx = L.scrust_cuda_context_create(0, ctypes.byref(st))
    assert ctx, st.message.decode()
    plans = []
    try:
        plans.append(Plan(ctx, [300, 1500, 700], k, metric, capacity))
        first = plans[0].launch()
        same(first, plans[0].launch())
        solve(ctx, 30_000, 60, metric)  # every slot of a solve, the top-K's above 40 neighbours too
        same(first, plans[0].launch())
        plans.append(Plan(ctx, [9000, 20_000, 400, 12_000], k, metric, capacity))
        second = plans[1].launch()
        same(first, plans[0].launch())
        same(second, plans[1].launch())
        solve(ctx, 90_000, 128, metric)
        same(second, plans[1].launch())
        same(first, plans[0].launch())
    finally:
        for p in plans:
            p.close()
        L.scrust_cuda_context_destroy(ctx)


def test_kernel_counters_switched_off_after_the_capture(built_library):
    pytest.importorskip("torch")
    L, st = _lib.lib(), _lib.Status()
    ctx = L.scrust_cuda_context_create(0, ctypes.byref(st))
    assert ctx, st.message.decode()
    try:
        words = (ctypes.c_uint64 * 16)()
        L.scrust_cuda_kernel_stats(ctx, 1, None, 0)
        plan = Plan(ctx, [400, 900], 15)
        first = plan.launch()
        L.scrust_cuda_kernel_stats(ctx, 0, words, 16)  # frees the counters
        same(first, plan.launch())
        plan.close()
    finally:
        L.scrust_cuda_context_destroy(ctx)
