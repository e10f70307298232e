"""Links longer than a group's list, and cofacet rows longer than the sorts'
shared memory: two hubs joined to many points that are far from each other,
so that the hubs' edge (the longest) has every point in its link and a row of
the reduction for almost each."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from golden_util import sorted_rows

pytestmark = pytest.mark.gpu

T = 1.405


def _hubs(points: int, pairs: int, seed: int, cluster: int = 0):
    """Hubs at -+0.7 along one axis (1.4 apart, 1.22-1.24 from the points);
    points at distance 1-1.02 along an axis each (at least 1.414 apart), the
    last ``pairs`` of them two to an axis (joined before the hubs are); far away,
    a cluster of points all joined to one another."""
    rng = np.random.default_rng(seed)
    axis = np.arange(points)
    axis[points - pairs:] = points - pairs + np.arange(pairs) // 2
    x = np.zeros((points + 2, int(axis.max()) + 2), dtype=np.float32)
    x[np.arange(points), axis] = rng.uniform(1.0, 1.02, points)
    x[points:, -1] = (-0.7, 0.7)
    far = 0.05 * rng.standard_normal((cluster, x.shape[1])).astype(np.float32) / np.sqrt(x.shape[1])
    far[:, -1] += 30.0
    x = np.concatenate([x, far])
    return x[rng.permutation(len(x))]


def _bits(a):
    return np.asarray(a, dtype=np.float32).view(np.uint32)


# The groups' lists hold 192 vertices in sparse graphs and 768 in dense ones
# (the cluster makes the graph dense on average): links around each length,
# tails beyond it with joined pairs on both sides, a row for the block's sort
@pytest.mark.parametrize("points,pairs,cluster", [
    (191, 0, 0), (192, 2, 0), (193, 100, 0), (450, 400, 0), (767, 0, 220), (768, 2, 220), (769, 300, 220),
    (1300, 700, 260)])
def test_long_link_matches_oracle(points, pairs, cluster):
    from flashph_b200 import rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    x = _hubs(points, pairs, points + pairs, cluster)
    dim = 1 if cluster else 2
    ref = oracle.run(x, T, dim, fused=True)
    got = [d.cpu().numpy() for d in rips_persistence(torch.from_numpy(x).cuda(), T, max_dim=dim)]
    for d in ([g.cpu().numpy() for g in rips_persistence_batch([x, x[:40]], T, dim)[0]], got):
        assert np.array_equal(_bits(d[0]), _bits(ref["h0"].reshape(-1, 2)))
        assert np.array_equal(_bits(d[1]), _bits(ref["h1"].reshape(-1, 2)))
        if dim == 2:
            assert np.array_equal(_bits(sorted_rows(d[2])), _bits(sorted_rows(ref["h2"])))


# four hubs joined to each other and to every leaf, the last two after the
# leaves: the triangle of the longest edge and the third hub has every leaf
# among its earlier neighbours (the list holds 768); with 1300 leaves the graph
# is too sparse for the rank table
@pytest.mark.parametrize("leaves", [767, 768, 900, 1300])
def test_many_earlier_neighbours_of_a_triangle(leaves):
    from flashph_b200 import rips_persistence
    rng = np.random.default_rng(leaves)
    x = np.zeros((leaves + 4, leaves + 2), dtype=np.float32)
    x[2 + np.arange(leaves), np.arange(leaves)] = rng.uniform(1.0, 1.02, leaves)
    x[[0, 1, leaves + 2, leaves + 3], leaves:] = [(-0.7, 0), (0.7, 0), (0, 0.3), (0, -0.31)]
    ref = oracle.run(x, T, 2, fused=True)
    got = [d.cpu().numpy() for d in rips_persistence(torch.from_numpy(x).cuda(), T, max_dim=2)]
    assert ref["Q"] > 4 * leaves
    assert np.array_equal(_bits(got[1]), _bits(ref["h1"].reshape(-1, 2)))
    assert np.array_equal(_bits(sorted_rows(got[2])), _bits(sorted_rows(ref["h2"])))


def _staged(monkeypatch, x, t, dim):
    from flashph_b200 import rips_persistence
    monkeypatch.setenv("FLASHPH_PIPELINE", "staged")
    out = rips_persistence(x, t, max_dim=dim)
    monkeypatch.delenv("FLASHPH_PIPELINE")
    return out


# H2 in the native call keeps the tetrahedra that can be pivots, the stage by
# stage form all of them: the same rows in the same order, ties (the lattice)
# and the sparse end included
@pytest.mark.parametrize("n,d,t", [(120, 4, 3.0), (300, 3, 1.1), (900, 10, 2.6), (3000, 10, 1.7), (216, 0, 2.3)])
def test_h2_rows_equal_the_staged_form(monkeypatch, n, d, t):
    from flashph_b200 import rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    if d:
        x = np.random.default_rng(n).standard_normal((n, d)).astype(np.float32)
    else:
        x = np.stack(np.meshgrid(*[np.arange(6)] * 3), -1).reshape(-1, 3).astype(np.float32)
    x = torch.from_numpy(x).cuda()
    want = _staged(monkeypatch, x, t, 2)
    batch = rips_persistence_batch([x[:50], x, x[: n // 2]], t, [1, 2, 0])[1]
    for got in (rips_persistence(x, t, max_dim=2), batch):
        for a, b in zip(got, want):
            assert np.array_equal(_bits(a.cpu().numpy()), _bits(b.cpu().numpy()))


def test_row_beyond_the_shared_memory_sort(monkeypatch):
    """More than 8192 rows in one column: the native call against the stage by
    stage form, whose cofacet rows come from the radix sort."""
    from flashph_b200 import rips_persistence
    x = torch.from_numpy(_hubs(8300, 50, 3)).cuda()
    native = rips_persistence(x, T, max_dim=1)
    monkeypatch.setenv("FLASHPH_PIPELINE", "staged")
    staged = rips_persistence(x, T, max_dim=1)
    for a, b in zip(native, staged):
        assert np.array_equal(_bits(a.cpu().numpy()), _bits(b.cpu().numpy()))


def test_reduction_beyond_shared_memory_windows(monkeypatch):
    """2.8M triangle rows in the stage by stage form (beyond the 1.79M that the
    shared-memory reduction takes: the general kernel), 0.09M in the native
    call: the same rows."""
    from flashph_b200 import rips_persistence
    x = torch.from_numpy(np.random.default_rng(0).standard_normal((1000, 3)).astype(np.float32)).cuda()
    want = _staged(monkeypatch, x, 1.269, 1)
    got = rips_persistence(x, 1.269, max_dim=1)
    for a, b in zip(got, want):
        assert np.array_equal(_bits(a.cpu().numpy()), _bits(b.cpu().numpy()))
