"""Adjacency rows of more than 16,384 entries in which one neighbour occurs many
times: a few by a thread (32), more by a warp (4096) and by the block, against a
stable argsort."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [
    [20000], [31, 32, 33, 34, 17000], [4095, 4096, 4097, 4098, 33], [1] * 9000 + [33] * 300 + [5000] * 3, [300000, 2, 70000]])
@pytest.mark.parametrize("far", [0, 70000])
def test_repeated_neighbours(copies, far):
    """Vertex 0 joined to vertex k + 1 (the odd ones ``far`` beyond) copies[k]
    times, in random order and direction, with self-loops of vertex 0."""
    from flashph_b200.rips import vertex_csr
    rng = np.random.default_rng(sum(copies) + far)
    dst = np.repeat(np.arange(len(copies)) + 1 + far * (np.arange(len(copies)) % 2), copies)
    dst = rng.permutation(np.concatenate([dst, np.zeros(50, dst.dtype)]))
    n, flip = int(dst.max()) + 1, rng.random(len(dst)) < 0.5
    ei, ej = np.where(flip, dst, 0).astype(np.int32), np.where(flip, 0, dst).astype(np.int32)
    ptr, idx, rank = vertex_csr(torch.from_numpy(ei).cuda(), torch.from_numpy(ej).cuda(), n)
    src = np.stack([ei, ej], 1).reshape(-1).astype(np.int64)
    to = np.stack([ej, ei], 1).reshape(-1).astype(np.int64)
    o = np.argsort(src * n + to, kind="stable")
    assert np.array_equal(ptr.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]))
    assert np.array_equal(idx.cpu().numpy(), to[o])
    assert np.array_equal(rank.cpu().numpy(), o // 2)
