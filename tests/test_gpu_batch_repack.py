"""A batch over its simplex budget is packed again by what its clouds take of
the budget (rows of the H1 reduction, and for H2 the stored triangles and the
tetrahedra), so that it splits into no more parts than that asks for."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2])
def test_parts_by_the_budget(monkeypatch, dim):
    from flashph_b200 import batch as B
    rng = np.random.default_rng(dim)
    x = [torch.from_numpy(rng.standard_normal((n, 4)).astype(np.float32)).cuda() for n in range(60, 72)]
    dev = x[0].device
    whole = B.rips_persistence_batch(x, 99.0, dim)
    monkeypatch.setattr(B, "_BATCH_SIMPLICES", 1)
    with pytest.raises(B._Split) as e:
        B._native_chunk(x, [99.0] * 12, [dim] * 12, dev, 10 ** 7, 10 ** 7)
    for p, count in zip(x, e.value.counts):
        n = p.shape[0]
        if dim == 1:  # every pair is an edge: few of the triangles are rows
            assert 0 < count < math.comb(n, 3) / 4
        else:
            assert math.comb(n, 3) < count < 1.5 * math.comb(n, 3)  # the tetrahedra are not counted yet
    calls = []
    real = B._native_chunk

    def counted(pts, *a):
        calls.append(len(pts))
        return real(pts, *a)

    monkeypatch.setattr(B, "_native_chunk", counted)
    need = sum(e.value.counts) if dim == 1 else sum(math.comb(p.shape[0], 3) + math.comb(p.shape[0], 4) for p in x)
    monkeypatch.setattr(B, "_BATCH_SIMPLICES", need * 2 // 5)
    got = B.rips_persistence_batch(x, 99.0, dim)
    # the whole, three or four parts; H2 may split once by the rows and triangles and again by the tetrahedra
    assert calls[0] == 12 and len(calls) <= (5 if dim == 1 else 9)
    for a, b in zip(got, whole):
        for u, v in zip(a, b):
            assert torch.equal(u.view(torch.int32), v.view(torch.int32))
