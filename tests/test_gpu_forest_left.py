"""A batch's forest where blocks leave clouds to the grid: dense clouds of several
components among sparse ones, the same diagrams as in calls of their own."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _parts(sizes, d, rng, lattice=False):
    """Dense parts far from each other, in one cloud of mixed order."""
    x = [(rng.integers(0, 5, (n, d)) if lattice else rng.standard_normal((n, d))) + 1000.0 * k
         for k, n in enumerate(sizes)]
    return torch.from_numpy(rng.permutation(np.concatenate(x)).astype(np.float32)).cuda()


# one, two and three clouds of more than an eighth of the edges and 2^19 of them,
# with ties, single points apart, and a connected one that a block finishes
@pytest.mark.parametrize("big", [
    [([1200, 1200], False)], [([900, 1, 800], False), ([1700, 2], True)],
    [([700, 700, 700], True), ([1500], False), ([800, 640, 1], False)]])
def test_clouds_left_to_the_grid(big):
    from flashph_b200 import rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    rng = np.random.default_rng(len(big))
    x = [torch.from_numpy(rng.standard_normal((1000 + 7 * k, 3)).astype(np.float32)).cuda() for k in range(8)]
    ts = [0.2] * len(x)
    for k, (sizes, lattice) in enumerate(big):
        at = 3 * k
        x.insert(at, _parts(sizes, 3, rng, lattice))
        ts.insert(at, 60.0)
    got = rips_persistence_batch(x, ts, 0)
    for p, t, g in zip(x, ts, got):
        want = rips_persistence(p, t, max_dim=0)[0]
        assert torch.equal(g[0].view(torch.int32), want.view(torch.int32))
