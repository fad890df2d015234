"""smooth_knn at the sizes where its staging changes, and on rows whose offsets
leave the range of its branch-free division, against the oracle.

The tolerance is that of the other comparisons of sigma with the oracle: the
bisection stops within 1e-5 of its target, and the device's and the host's expf
differ by an ulp on some terms, which can move that stop by one step (both
stops lie in the band: 5e-5 relative).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA_RTOL = 5e-5


@pytest.fixture(scope="module")
def scrust(built_library):
    from mrustsc_gb300 import _scrust

    assert _scrust.gpu_available(), "these tests need an sm_103a GPU"
    return _scrust


# 64 | 65: rows a block; 128 | 129: staged or read from memory; row counts one
# past a block.
@pytest.mark.parametrize("n,k", [(1, 1), (129, 2), (65, 15), (300, 31), (129, 64), (65, 65), (129, 128), (65, 129),
                                 (40, 300)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 59, 1e22, 2.0 ** -30, 1e-25])
def test_rows_match_the_oracle(scrust, oracle, n, k, scale):
    rng = np.random.default_rng(n * 1000 + k)
    dist = np.sort(rng.gamma(2.0, 1.5, size=(n, k)), axis=1)
    dist[::3] *= scale
    dist[1::4, : k // 2] = 0.0          # leading zeros
    dist[2::7] = dist[2::7, :1]         # every neighbour at one distance
    dist = dist.astype(np.float32)
    s_gpu, r_gpu = scrust.smooth_knn_distances(dist)
    s_ref, r_ref = oracle.smooth_knn(dist)
    np.testing.assert_array_equal(r_gpu, r_ref)
    np.testing.assert_allclose(s_gpu, s_ref, rtol=SIGMA_RTOL)
