"""Exact triangle totals from edges that are given more than once: each counts
once, and a vertex may have more half-edges than there are vertices."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
scipy_sparse = pytest.importorskip("scipy.sparse")
pytestmark = pytest.mark.gpu


def _total(ei, ej, n):
    a = scipy_sparse.coo_matrix((np.ones(len(ei), np.int64), (ei, ej)), shape=(n, n)).tocsr()
    a = ((a + a.T) > 0).astype(np.int64)
    return int((a @ a).multiply(a).sum()) // 6


# every edge several times, one edge very often, rows at the edges of the
# 64-vertex words and of their summary (2048 vertices)
@pytest.mark.parametrize("n,edges,copies,often", [
    (3, 3, 1, 40), (4, 6, 5, 0), (64, 700, 3, 9000), (65, 1500, 30, 100), (2048, 20000, 2, 70000),
    (2113, 30000, 1, 30000), (40000, 200000, 3, 1)])
def test_repeated_edges_count_once(n, edges, copies, often):
    from flashph_b200 import _lib as L
    rng = np.random.default_rng(n)
    key = np.unique(rng.integers(0, n, (edges * 8, 2)), axis=0)
    key = rng.permutation(key[key[:, 0] < key[:, 1]])[:edges]
    key = np.concatenate([key] * copies + [key[:1]] * often)
    ei, ej = np.ascontiguousarray(rng.permutation(key).T.astype(np.int32))
    di, dj = torch.from_numpy(ei.copy()).cuda(), torch.from_numpy(ej.copy()).cuda()
    nb = L.query("ph_triangles_total_edges_workspace_bytes", len(ei), n)
    ws = L.workspace(nb, di.device)
    for _ in range(2):
        tot = torch.full((1,), 7, dtype=torch.int64, device="cuda")
        L.call("ph_triangles_total_edges", di.data_ptr(), dj.data_ptr(), len(ei), n, tot.data_ptr(), ws.data_ptr(), nb,
               L.stream_handle(di.device))
        assert int(tot.item()) == _total(ei, ej, n)
