"""Reductions whose windows leave room for one to four warps an SM: the short
columns go first, the others from their records on. The rows equal those of the
staged form, whose triangle rows are more than windows hold (the general
kernel), the failure paths are the same."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cloud(kind, n, d, seed=1):
    rng = np.random.default_rng(seed)
    x = rng.random((n, d)) if kind == "uniform" else rng.standard_normal((n, d))
    if kind == "sphere":
        x /= np.linalg.norm(x, axis=1, keepdims=True)
    if kind == "lattice":
        x = np.round(x * 3)
    return torch.from_numpy(x.astype(np.float32)).cuda()


def _staged(monkeypatch, x, t, dim):
    from flashph_b200 import rips_persistence
    monkeypatch.setenv("FLASHPH_PIPELINE", "staged")
    out = rips_persistence(x, t, max_dim=dim)
    monkeypatch.delenv("FLASHPH_PIPELINE")
    return out


# rows of the native call, of 2.0M to 8.5M triangles: 0.89M, 0.68M, 0.63M, 1.16M,
# 0.40M; short columns, long chains, records of more than 31 entries, ties
@pytest.mark.parametrize("kind,n,d,t", [
    ("uniform", 250000, 2, 0.0034), ("sphere", 60000, 4, 0.12), ("normal", 30000, 16, 2.78), ("normal", 40000, 5, 0.66),
    ("lattice", 32000, 3, 0.6)])
def test_short_columns_first(monkeypatch, kind, n, d, t):
    from flashph_b200 import rips_persistence
    x = _cloud(kind, n, d)
    want = _staged(monkeypatch, x, t, 1)
    for _ in range(2):
        got = rips_persistence(x, t, max_dim=1)
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.fixture
def limits():
    from flashph_b200 import _lib
    yield _lib.lib().ph_set_reduce_limits
    _lib.lib().ph_set_reduce_limits(0, 0)


def test_failure_paths(limits):
    from flashph_b200 import _lib, rips_persistence
    x, t = _cloud("uniform", 250000, 2), 0.0031
    want = rips_persistence(x, t, max_dim=1)
    limits(1, 0)
    with pytest.raises(_lib.PHError, match="iteration limit"):
        rips_persistence(x, t, max_dim=1)
    limits(0, 1_000_000)  # below the initial records: retried with larger pools
    got = rips_persistence(x, t, max_dim=1)
    limits(0, 0)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
