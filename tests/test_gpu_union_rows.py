"""The union of rows of every length class against the general union of the
same neighbour lists, bit for bit: rows of at most 32, 64 and 128 entries in
all (sorted in one, two and four registers) and of more (sorted in memory).

Gaussian data of many dimensions has hubs, so that in-degrees run from none to
hundreds; the test checks that each class occurs.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


@pytest.mark.parametrize("k,classes", [(2, (32, 64, 128)), (15, (32, 64, 128, 10 ** 9)), (16, (32, 64, 128, 10 ** 9)),
                                       (31, (64, 128, 10 ** 9)), (32, (64, 128, 10 ** 9))])
def test_rows_of_every_length(scrust, k, classes):
    n, d = 6000, 60
    rng = np.random.default_rng(k)
    x = rng.standard_normal((n, d)).astype(np.float32)
    x[: n // 3] *= 0.7  # towards the centre: hubs
    idx, dist, one = scrust.neighbors_graph(x, k)
    total = k + np.bincount(idx.ravel(), minlength=n)
    low = 0
    for high in classes:
        assert np.any((total > low) & (total <= high)), (low, high)
        low = high
    for a, b in zip(one[:3], scrust.connectivities(idx, dist)[:3]):
        np.testing.assert_array_equal(a, b)
