"""The exact totals of a batch's clouds over the triangle limit, whose bitmaps
count words from the cloud's first vertex on: clouds at the edges of the words
(64 vertices) and of their summary (2048), at odd places in the union, against
the single call's errors; and a batch in which no cloud can be over the limit."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,limit", [
    ([2113, 37, 65, 640, 2048, 64, 2049], 4000), ([5, 64, 3, 129], 30), ([63, 64, 65], 50_000)])
def test_totals_per_cloud(sizes, limit):
    from flashph_b200.batch import rips_persistence_batch
    from flashph_b200.persistence import _compute_native
    rng = np.random.default_rng(sum(sizes))
    x = [torch.from_numpy(rng.standard_normal((n, 3)).astype(np.float32)).cuda() for n in sizes]
    ts = [9.0 if n < 100 else 0.7 for n in sizes]
    got = rips_persistence_batch(x, ts, 1, max_triangles=limit)
    over = 0
    for p, t, g in zip(x, ts, got):
        try:
            want = _compute_native(p, t, 1, p.device, max_triangles=limit)
        except ValueError as e:
            over += 1
            assert isinstance(g, ValueError) and str(g) == str(e)
            continue
        for a, b in zip(g, want):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert over == (0 if limit == 50_000 else sum(n > 6 for n in sizes))
