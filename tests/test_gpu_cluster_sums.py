"""Clustering with weights whose sums are exact as integers against the same
graph on the f64 path.

Two more nodes joined by an edge of 2^-100 leave the total and every other
node's strength as they were, but no longer let a level's weights be taken as
integers; every decision about the other nodes reads the same values, so their
Leiden partition has to be the same, whichever path formed the sums.  (Louvain's
need not be: its coarser levels number their nodes by community id, where the
pair's comes before the ids reserved for nodes that leave a community, and the
rounds a node is active in go by its number.)
"""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


def graph(n, degree, hubs, seed):
    """Planted groups of 50, `degree` edges a node, and hubs of given degrees."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), degree)
    near = (i // 50) * 50 + rng.integers(0, 50, i.size)
    j = np.where(rng.random(i.size) < 0.8, np.minimum(near, n - 1), rng.integers(0, n, i.size))
    for h, count in enumerate(hubs):
        i = np.concatenate([i, np.full(count, h)])
        j = np.concatenate([j, rng.permutation(n - len(hubs))[:count] + len(hubs)])
    w = rng.uniform(2.0 ** -10, 1.0, i.size).astype(np.float32)
    m = sp.coo_matrix((w, (i, j)), shape=(n, n)).tocsr().astype(np.float32)
    m.sort_indices()
    return m


def with_tiny_pair(m):
    n = m.shape[0]
    t = np.float32(2.0 ** -100)
    pair = sp.csr_matrix((np.array([t, t], np.float32), np.array([1, 0]), np.array([0, 1, 2])), shape=(2, 2))
    out = sp.block_diag([m, pair], format="csr").astype(np.float32)
    assert out.shape == (n + 2, n + 2) and out.data.min() == t
    return out


def args(m):
    return m.indptr.astype(np.uint32), m.indices.astype(np.uint32), m.data.astype(np.float32), m.shape[1]


def first_seen(labels):
    _, first, inverse = np.unique(labels, return_index=True, return_inverse=True)
    return np.argsort(np.argsort(first))[inverse]


# Rows of 2 entries; rows about 64 entries, where the small kernel ends; hubs of
# more entries than a block reads at once; and of more communities than the
# table holds (those hubs do not move on either path).
@pytest.mark.parametrize("n,degree,hubs", [(33, 1, ()), (1000, 15, (40, 64)), (1000, 32, (500,)), (5001, 8, (2049, 4000, 257))])
@pytest.mark.parametrize("resolution", [1.0, 30.0])
def test_integer_sums_decide_as_f64_sums(scrust, n, degree, hubs, resolution):
    m = graph(n, degree, hubs, seed=n + degree)
    t = with_tiny_pair(m)
    a, b = (np.asarray(scrust.leiden(*args(g), resolution, 2, 7, "auto")[0]) for g in (m, t))
    assert b[n] == b[n + 1] and not np.any(b[:n] == b[n])
    np.testing.assert_array_equal(first_seen(a), first_seen(b[:n]))


def test_repeat_calls_share_the_workspace(scrust):
    """Larger, smaller and larger graphs again, through one context's blocks."""
    graphs = [graph(n, 15, (), seed=n) for n in (500, 20000, 31, 7000)]
    first = [np.asarray(scrust.leiden(*args(m), 1.0, 2, 0, "auto")[0]) for m in graphs]
    for _ in range(2):
        for m, want in zip(graphs[::-1], first[::-1]):
            np.testing.assert_array_equal(np.asarray(scrust.leiden(*args(m), 1.0, 2, 0, "auto")[0]), want)
