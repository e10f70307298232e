"""The forest kernel at the edges of its three forms (one block while
8 n + E <= 40960, a cluster while 16 n + E <= 368640, a grid beyond) and of its
passes (the first holds max(4 n, threads) edges), against Kruskal over the
positions; and a batch, a block a cloud, against its clouds one by one. Masks,
labels, counts and diagrams are the same to the bit."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _kruskal(ei, ej, n):
    parent = list(range(n))

    def find(v):
        while parent[v] != v:
            parent[v] = parent[parent[v]]
            v = parent[v]
        return v

    mask = np.zeros(len(ei), np.uint8)
    for e, (a, b) in enumerate(zip(ei.tolist(), ej.tolist())):
        ra, rb = find(a), find(b)
        if ra != rb:
            mask[e] = 1
            parent[max(ra, rb)] = min(ra, rb)
    return mask, np.array([find(v) for v in range(n)], np.int32)


@pytest.mark.parametrize("n,E,kind", [
    (1, 0, "any"), (7, 0, "any"), (1, 3, "any"), (256, 1024, "any"), (257, 1029, "late"),
    (1024, 8192, "late"), (1024, 32768, "late"), (1024, 32769, "late"), (2048, 8193, "path"),
    (5000, 960, "path"), (5000, 961, "path"), (5120, 0, "any"), (300, (1 << 18) + 1, "any"),
    (8192, 237568, "late"), (8192, 237569, "late"), (20000, 48640, "path"), (20000, 48641, "path"),
    (70000, 600000, "late"), (150000, 149999, "path"), (400000, 1300000, "late")])
def test_forest_at_form_and_pass_edges(n, E, kind):
    from flashph_b200.boruvka import boruvka_mask
    rng = np.random.default_rng(n * 31 + E)
    ei = rng.integers(0, n, E).astype(np.int32)
    ej = rng.integers(0, n, E).astype(np.int32)
    if kind == "late":  # some vertices are met only by the last edges, so every pass joins components
        k = E // 2
        ei[:k] %= max(1, n // 3)
        ej[:k] %= max(1, n // 3)
    if kind == "path":  # one path in scrambled order: the longest hook chains
        k = min(E, n - 1)
        at = rng.permutation(n).astype(np.int32)
        cut = rng.permutation(k)
        ei[:k], ej[:k] = at[cut], at[cut + 1]
    want_mask, want_comp = _kruskal(ei, ej, n)
    mask, comp, (ncomp, status) = boruvka_mask(torch.from_numpy(ei).cuda(), torch.from_numpy(ej).cuda(), n)
    assert int(status.item()) == 0
    assert np.array_equal(mask.cpu().numpy(), want_mask)
    assert np.array_equal(comp.cpu().numpy(), want_comp)
    assert int(ncomp.item()) == int((want_comp == np.arange(n)).sum())


@pytest.mark.parametrize("sizes", [[2] * 5, [300, 64, 2, 501], [900] * 12 + [3], [8192] + [1500] * 17, [8193, 700, 700]])
def test_batch_forests_match_single_calls(sizes):
    from flashph_b200 import rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    rng = np.random.default_rng(sum(sizes))
    clouds = [torch.from_numpy(rng.standard_normal((n, 3)).astype(np.float32)).cuda() for n in sizes]
    # single components, several and (t = 0) no edge at all
    ts = [(3.0 if n < 400 else 1.2 * n ** (-1 / 3)) * (k % 4 != 3) for k, n in enumerate(sizes)]
    batch = rips_persistence_batch(clouds, ts, [0] * len(sizes))
    for x, t, got in zip(clouds, ts, batch):
        want = rips_persistence(x, t, max_dim=0)
        assert np.array_equal(want[0].cpu().numpy().view(np.uint32), got[0].cpu().numpy().view(np.uint32))
