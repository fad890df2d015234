"""The UMAP epoch kernels at the sizes where their splits can go wrong: cells
without edges, degrees around the group and block sizes, a hub whose edges and
draws pass several chunks and windows, a last partial block, asymmetric rows,
one to sixteen components, and sample rates from none to many.

The oracle is one epoch's moves restated here one edge after another in f32
with the powers in f64: every weight is 1, so no edge fires in epoch 0 and
every edge in epoch 1.  A move's coefficient carries the rounding of a squared
distance of `dim` terms (dim + 2 roundings), two powers (CUDA states 4 ulp for
powf) and four more operations, under 32 half-ulps in all for dim <= 16; sums
run in the same order on both sides, so they differ by the moves' differences
and at most one ulp of the partial sum per addition.  That is the tolerance,
taken cell by cell."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1
GOLDEN = 0x9E3779B97F4A7C15
INIT_SALT = 0x5CA1AB1E0DDBA11
F = np.float32


class Tau:
    """TauRng (crates/scrust-core/src/umap.rs:174-201)."""

    def __init__(self, seed):
        words = []
        for _ in range(3):
            seed = (seed + GOLDEN) & M64
            z = seed
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            words.append((z ^ (z >> 31)) & 0xFFFFFFFF)
        self.s = [words[0] | 0x2, words[1] | 0x8, words[2] | 0x10]

    def next(self):
        m = 0xFFFFFFFF
        a, b, c = self.s
        a = (((a & 4294967294) << 12) & m) ^ ((((a << 13) & m) ^ a) >> 19)
        b = (((b & 4294967288) << 4) & m) ^ ((((b << 2) & m) ^ b) >> 25)
        c = (((c & 4294967280) << 17) & m) ^ ((((c << 3) & m) ^ c) >> 11)
        self.s = [a, b, c]
        return a ^ b ^ c


def initial(n, dim, seed):
    y = np.empty((n, dim), np.float32)
    for v in range(n):
        t = Tau(seed ^ ((v * GOLDEN) & M64) ^ INIT_SALT)
        for c in range(dim):
            u = F(t.next()) / F(4294967296.0)
            y[v, c] = (u * F(2.0) - F(1.0)) * F(10.0)
    lo, hi = y.min(0), y.max(0)
    return (F(10.0) * (y - lo)) / (hi - lo)


def clip(v):
    return np.minimum(np.maximum(v, F(-4.0)), F(4.0))


def sq(diff):
    s = F(0.0)
    for v in diff:
        s = s + v * v
    return s


def second_epoch(indptr, indices, y, a, b, neg_rate, alpha, seed):
    """(layout, tolerance) after the epoch in which every edge fires once."""
    n, dim = y.shape
    own = np.zeros_like(y)
    size = np.zeros((n, dim))   # sum of |move|
    bend = np.zeros((n, dim))   # sum of |partial sum| (one ulp of each)
    tmove = np.zeros((len(indices), dim), np.float32)
    n_neg = int((1.0 - 1.0 / neg_rate) / (1.0 / neg_rate)) if neg_rate else 0

    def add(h, mv):
        own[h] = own[h] + mv
        size[h] += np.abs(mv)
        bend[h] += np.abs(own[h])

    for h in range(n):
        t = Tau(seed ^ ((h * GOLDEN) & M64))
        for e in range(indptr[h], indptr[h + 1]):
            diff = y[h] - y[indices[e]]
            dist = sq(diff)
            coef = F(0.0)
            if dist > 0:
                coef = (F(-2.0) * a * b * F(float(dist) ** float(b - F(1.0)))) / (a * F(float(dist) ** float(b)) + F(1.0))
            tmove[e] = clip(coef * diff) * alpha
            add(h, tmove[e])
            for _ in range(n_neg):
                j = t.next() % n
                if j == h:
                    continue
                diff = y[h] - y[j]
                dist = sq(diff)
                if dist <= 0:
                    continue
                cr = (F(2.0) * b) / ((F(0.001) + dist) * (a * F(float(dist) ** float(b)) + F(1.0)))
                add(h, clip(cr * diff) * alpha)
    for e in np.argsort(indices, kind="stable"):
        add(indices[e], -tmove[e])
    return y + own, 32 * 2.0**-24 * size + 2.0**-23 * bend + 2.0**-23 * (np.abs(y) + np.abs(own))


def graph(n, hub):
    """Rows of 0, 1, 7, 8, 9, 31, 33 and `hub` edges among ordinary ones."""
    g = np.random.default_rng(n + hub)
    special = {0: hub, 1: 0, 5: 1, 6: 7, 7: 8, 8: 9, 20: 31, 31: 0, 32: 33, n - 1: 12}
    indptr, indices = [0], []
    for h in range(n):
        deg = special.get(h, int(g.integers(2, 20)))
        indices.extend(np.sort(g.choice(np.delete(np.arange(n), h), deg, replace=False)).tolist())
        indptr.append(len(indices))
    return np.array(indptr, np.uint32), np.array(indices, np.uint32)


@pytest.mark.parametrize("n,hub,dim,neg_rate", [(70, 60, 2, 5), (97, 90, 2, 40), (64, 60, 3, 5), (65, 60, 1, 5),
                                                (70, 60, 5, 12), (50, 45, 16, 7), (70, 60, 2, 0), (70, 60, 2, 1),
                                                (1300, 1250, 2, 2)])
def test_one_firing_epoch_matches_the_restatement(built_library, oracle, n, hub, dim, neg_rate):
    from mrustsc_gb300 import _scrust

    indptr, indices = graph(n, hub)
    values = np.ones(len(indices), np.float32)
    seed = 11
    y = _scrust.umap(indptr, indices, values, n, dim, 2, 0.5, 1.0, 1.0, neg_rate, seed, "auto")
    a, b = oracle.fit_ab_params(0.5, 1.0)
    ref, tol = second_epoch(indptr.astype(np.int64), indices.astype(np.int64), initial(n, dim, seed), F(a), F(b),
                            neg_rate, F(1.0), seed)
    assert np.isfinite(y).all()
    worst = np.abs(y.astype(np.float64) - ref) / tol
    assert worst.max() <= 1.0, worst.max()
