"""The service under a tight memory budget: a batch of few queries takes no
more column segments, and so no more lists, than the budget has room for, and
its results do not depend on how many those are."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def served(budget, atlas, query, k):
    """(results, device bytes that the request's workspaces took)"""
    import torch

    from mrustsc_gb300 import serving

    with serving.Server(atlas, k, budget_bytes=budget, slots=1) as server:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        idx, dist, csr, _ = server.query(query)
        return [idx, dist, *csr], before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("k", [1, 15, 32])
def test_lists_fit_the_budget(built_library, k):
    pytest.importorskip("torch")
    r = np.random.default_rng(k)
    atlas = r.uniform(-100.0, 100.0, size=(20_000, 4)).astype(np.float32)  # some 10 MiB resident
    query = r.uniform(-100.0, 100.0, size=(300, 4)).astype(np.float32)
    budget = 64 * MIB
    roomy, wide = served(0, atlas, query, k)
    tight, narrow = served(budget, atlas, query, k)
    for a, b in zip(roomy, tight):
        np.testing.assert_array_equal(a, b)
    # The 79 tiles in 40 segments of two: 512 padded rows of 80 lists of 384
    # slots of 8 bytes.  Under the budget, plus what 45 other workspaces of a
    # request this small take at 2 MiB each.
    assert wide >= 512 * 80 * 384 * 8
    assert narrow <= budget + 45 * 2 * MIB
