"""The adjacency at the edges of its row sorts (8, 32, 64 to 1024 and 16,384 entries,
longer rows counted by ranges of 32,768 neighbours) and of the choice between
counting and the radix sort, against a stable argsort: repeated edges keep
their rank order, a self-loop is in its row twice."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _hub_rows(lengths, n, rng):
    """Edges giving vertex k a row of at least lengths[k] different neighbours, in random order and direction."""
    src = np.concatenate([np.full(m, k) for k, m in enumerate(lengths)])
    dst = np.concatenate([len(lengths) + rng.permutation(n - len(lengths))[:m] for m in lengths])
    flip = rng.random(len(src)) < 0.5
    at = rng.permutation(len(src))
    return np.where(flip, dst, src)[at].astype(np.int32), np.where(flip, src, dst)[at].astype(np.int32)


@pytest.mark.parametrize("kind,n,E", [
    ("rows", 40000, [1, 7, 8, 9, 31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 16383, 16384, 16385, 39000]),
    ("rows", 100003, [70000, 70000]), ("random", 5000, 24575), ("random", 5000, 24576), ("random", 40, 30000),
    ("random", 3, 60000), ("random", 3000000, 30000), ("random", 300, 400000), ("random", 3000, 500000), ("random", 250000, 400000)])
def test_adjacency_rows(kind, n, E):
    from flashph_b200.rips import vertex_csr
    rng = np.random.default_rng(n)
    if kind == "rows":
        ei, ej = _hub_rows(E, n, rng)
        E = len(ei)
    else:  # repeated pairs and self-loops among them
        ei, ej = rng.integers(0, n, E).astype(np.int32), rng.integers(0, n, E).astype(np.int32)
        ej[::41] = ei[::41]
        ei[1::50], ej[1::50] = ei[0], ej[0]
    ptr, idx, rank = vertex_csr(torch.from_numpy(ei).cuda(), torch.from_numpy(ej).cuda(), n)
    src = np.stack([ei, ej], 1).reshape(-1).astype(np.int64)
    dst = np.stack([ej, ei], 1).reshape(-1).astype(np.int64)
    o = np.argsort(src * n + dst, kind="stable")
    assert np.array_equal(ptr.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]))
    assert np.array_equal(idx.cpu().numpy(), dst[o])
    assert np.array_equal(rank.cpu().numpy(), o // 2)
