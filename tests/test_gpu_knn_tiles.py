"""The k-NN top buffer and the enclosing radius at the edges of their tiles
(32 queries, 64 candidates, 32-dimension chunks, k up to 64), bit for bit
against the edge kernel's squared distances of all pairs: the same FP32 chain,
so no tolerance."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _all_pairs(x):
    """(n, n) squared distances of the direct edge kernel, infinite on the diagonal."""
    from flashph_b200.rips import enumerate_edges
    n = x.shape[0]
    i, j, d = enumerate_edges(x, float("inf"), screen=False)
    m = torch.full((n, n), float("inf"), device=x.device)
    m[i.long(), j.long()] = d
    m[j.long(), i.long()] = d
    return m


@pytest.mark.parametrize("n,d", [(2, 1), (33, 3), (64, 31), (65, 32), (129, 33), (257, 2), (500, 70), (1031, 10)])
@pytest.mark.parametrize("ties", [False, True])
def test_tiles_match_the_edge_kernel(n, d, ties):
    from flashph_b200 import enclosing_radius
    from flashph_b200.threshold import knn_kth_distance
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 3, (n, d)) if ties else rng.standard_normal((n, d))
    x = torch.from_numpy(x.astype(np.float32)).cuda()
    m = _all_pairs(x)
    order = m.sort(dim=1).values
    for k in (1, 20, 63, 64):
        if k <= n - 1:
            got = knn_kth_distance(x, k)
            assert torch.equal(got.view(torch.int32), order[:, k - 1].sqrt().view(torch.int32)), k
    far = m.fill_diagonal_(0.0).amax(dim=1)
    assert enclosing_radius(x) == float(far.sqrt().min())


def test_fewer_finite_distances_than_k():
    """Points at infinity and NaN coordinates: their distances are never among the k smallest."""
    from flashph_b200.threshold import knn_kth_distance
    x = torch.randn(100, 4, generator=torch.Generator().manual_seed(1)).cuda()
    x[::3] = float("inf")
    x[1, 2] = float("nan")
    got = knn_kth_distance(x, 64)
    near = knn_kth_distance(x, 20)
    assert torch.isinf(got[0]) and torch.isinf(got[1]) and torch.isfinite(got[2])
    live = torch.ones(100, dtype=torch.bool, device="cuda")
    live[::3] = False
    live[1] = False
    assert torch.equal(near[live], knn_kth_distance(x[live].contiguous(), 20))
