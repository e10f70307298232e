"""The screen's candidate queues: recomputed by all warps between items, within
an item where it alone fills one, and at a change of clouds; rows read by one,
two or four floats, by the dimension and the place of the first point. Edges
equal the direct kernel's to the bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _edges(x, t, screen):
    from flashph_b200.rips import enumerate_edges
    i, j, d = enumerate_edges(x, t, screen=screen)
    o = torch.argsort(i.long() * x.shape[0] + j.long())
    return i[o], j[o], d[o].view(torch.int32)


# d + 4 up to 16, 64, 160 and 256 (two row blocks an item, one, one column
# block); the share of pairs sets how often queues fill (256 a warp; an item
# has 2048 pairs a warp and row block, or 1024)
@pytest.mark.parametrize("d", [9, 10, 12, 58, 60, 61, 101, 150, 156, 250, 252])
@pytest.mark.parametrize("share", [0.003, 0.05, 0.6])
def test_queues(d, share):
    n = 1900
    g = torch.Generator().manual_seed(d)
    base = torch.randn(4 + n * d, generator=g).cuda()
    at = d % 4  # the first point's place, in floats
    x = base[at:at + n * d].view(n, d)
    s = torch.cdist(x[:300].double(), x.double()).flatten()
    t = float(s.kthvalue(max(1, int(share * s.numel()))).values)
    for u, v in zip(_edges(x, t, True), _edges(x, t, False)):
        assert torch.equal(u, v)


def test_clouds_of_all_alignments(monkeypatch):
    """A union in which the clouds' first points lie at every place modulo four
    floats, dense clouds after sparse ones (queues are emptied at the change)."""
    from flashph_b200 import rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    rng = np.random.default_rng(5)
    x = [torch.from_numpy(rng.standard_normal((n, d)).astype(np.float32)).cuda()
         for n, d in [(301, 9), (500, 12), (257, 11), (700, 60), (129, 10), (640, 61), (300, 60), (33, 14), (800, 52)]]
    ts = [1.5, 4.0, 2.0, 10.0, 3.0, 9.5, 10.5, 9.0, 9.0]
    want = [rips_persistence(p, t, max_dim=0)[0] for p, t in zip(x, ts)]
    for screen in ("on", "off"):
        monkeypatch.setenv("FLASHPH_EDGE_SCREEN", screen)
        for g, w in zip(rips_persistence_batch(x, ts, 0), want):
            assert torch.equal(g[0].view(torch.int32), w.view(torch.int32))
