"""Exact triangle totals over degree-ordered words against a sparse matrix
product, at the edges of the words (64 vertices), of the words' summary (2048)
and of the vertex range, with hubs, and per cloud in a batch."""

import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")
scipy_sparse = pytest.importorskip("scipy.sparse")
pytestmark = pytest.mark.gpu


def _total(ei, ej, n):
    a = scipy_sparse.coo_matrix((np.ones(len(ei), np.int64), (ei, ej)), shape=(n, n)).tocsr()
    a = a + a.T
    return int((a @ a).multiply(a).sum()) // 6


def _edges(n, E, kind, rng):
    ei, ej = rng.integers(0, n, E), rng.integers(0, n, E)
    if kind == "hubs":  # a few vertices meet nearly all edges
        ei = np.where(rng.random(E) < 0.7, rng.integers(0, min(n, 9), E), ei)
    if kind == "core":  # one dense part in a sparse rest
        ei, ej = np.where(rng.random(E) < 0.6, ei % min(n, 300), ei), np.where(rng.random(E) < 0.6, ej % min(n, 300), ej)
    keep = ei != ej
    lo, hi = np.minimum(ei, ej)[keep], np.maximum(ei, ej)[keep]
    key = np.unique(lo.astype(np.int64) * n + hi)
    key = rng.permutation(key)
    return (key // n).astype(np.int32), (key % n).astype(np.int32)


@pytest.mark.parametrize("n,E,kind", [
    (3, 30, "any"), (63, 900, "any"), (64, 4000, "any"), (65, 4000, "any"), (700, 60000, "any"),
    (2048, 90000, "hubs"), (2049, 90000, "core"), (4097, 60000, "hubs"), (30000, 400000, "core"),
    (227329, 500000, "core"), (1638400, 700000, "core")])
def test_total_from_edges(n, E, kind):
    from flashph_b200 import _lib as L
    rng = np.random.default_rng(n + E)
    ei, ej = _edges(n, E, kind, rng)
    di, dj = torch.from_numpy(ei).cuda(), torch.from_numpy(ej).cuda()
    nb = L.query("ph_triangles_total_edges_workspace_bytes", len(ei), n)
    ws = L.workspace(nb, di.device)
    tot = torch.full((1,), 7, dtype=torch.int64, device="cuda")
    L.call("ph_triangles_total_edges", di.data_ptr(), dj.data_ptr(), len(ei), n, tot.data_ptr(), ws.data_ptr(), nb,
           L.stream_handle(di.device))
    assert int(tot.item()) == _total(ei, ej, n)


def test_batch_totals_per_cloud():
    """Clouds over and under the limit, those counted exactly and those that
    cannot be over it, in an order that mixes them: the totals of the errors."""
    from flashph_b200.batch import rips_persistence_batch
    rng = np.random.default_rng(11)
    sizes, ts, limit = [500, 90, 301, 2, 640, 64, 450], [1.2, 9.0, 9.0, 1.0, 0.9, 0.5, 1.5], 40000
    clouds = [rng.standard_normal((n, 3)).astype(np.float32) for n in sizes]
    got = rips_persistence_batch([torch.from_numpy(c).cuda() for c in clouds], ts, [1] * len(sizes), max_triangles=limit)
    over = 0
    for c, t, g in zip(clouds, ts, got):
        d = np.zeros((len(c), len(c)), np.float32)
        x = c.astype(np.float64)
        d = ((x[:, None] - x[None]) ** 2).sum(-1)
        ei, ej = np.nonzero(np.triu(d < t * t, 1))
        want = _total(ei, ej, len(c))
        if want > limit:
            over += 1
            assert isinstance(g, ValueError) and int(re.search(r"count (\d+)", str(g)).group(1)) == want
        else:
            assert not isinstance(g, Exception)
    assert 0 < over < len(sizes)
