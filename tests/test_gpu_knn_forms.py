"""Both forms of the k-NN scan bit for bit against the edge kernel's squared
distances of all pairs (the same FP32 chain, so no tolerance): the top buffer at
the edges of its tiles (32 queries, 128 candidates, chunks of 12 dimensions) and
of its two sizes (k up to 32 and up to 64), over enough tiles for every cut
(after the 1st, 4th, 16th and 64th, and of a full buffer), and the radix select
beyond k = 64, at the edges of its own (64 candidates, 32 dimensions)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sorted_distances(x):
    from flashph_b200.rips import enumerate_edges
    n = x.shape[0]
    i, j, d = enumerate_edges(x, float("inf"), screen=False)
    m = torch.full((n, n), float("inf"), device=x.device)
    m[i.long(), j.long()] = d
    m[j.long(), i.long()] = d
    return m.sort(dim=1).values.sqrt()


def _check(x, ks):
    from flashph_b200.batch import auto_threshold_batch
    from flashph_b200.threshold import auto_threshold, knn_kth_distance
    order = _sorted_distances(x)
    for k in ks:
        if k <= x.shape[0] - 1:
            got = knn_kth_distance(x, k)
            assert torch.equal(got.view(torch.int32), order[:, k - 1].contiguous().view(torch.int32)), k
            assert auto_threshold_batch([x[:40], x], k)[1] == auto_threshold(x, k)


@pytest.mark.parametrize("n,d", [
    (127, 12), (128, 13), (129, 24), (255, 25), (256, 11), (160, 12), (1100, 36), (2300, 5)])
@pytest.mark.parametrize("ties", [False, True])
def test_top_buffer(n, d, ties):
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 3, (n, d)) if ties else rng.standard_normal((n, d))
    _check(torch.from_numpy(x.astype(np.float32)).cuda(), (1, 31, 32, 33, 64))


# a line in order and in reverse: for the queries at one end every tile is
# nearer than the one before, so that it fills the buffer
@pytest.mark.parametrize("d", [1, 13])
@pytest.mark.parametrize("step", [-1.0, 1.0])
def test_every_tile_nearer(d, step):
    n = 66 * 128 + 5
    x = np.zeros((n, d), dtype=np.float32)
    x[:, d // 2] = step * np.arange(n)
    x += 0.01 * np.random.default_rng(d).standard_normal((n, d)).astype(np.float32)
    _check(torch.from_numpy(x).cuda(), (20, 32, 33, 64))


@pytest.mark.parametrize("n,d", [(66, 3), (128, 31), (129, 32), (193, 33), (1031, 10), (500, 70)])
@pytest.mark.parametrize("ties", [False, True])
def test_radix_select(n, d, ties):
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 3, (n, d)) if ties else rng.standard_normal((n, d))
    _check(torch.from_numpy(x.astype(np.float32)).cuda(), (65, 100, n // 2, n - 1))
