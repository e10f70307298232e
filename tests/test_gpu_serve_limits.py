"""A server's limits hold for requests of every size: those that run alone and
those that share a batch are refused and accepted alike."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cloud(n, d=3):
    return torch.from_numpy(np.random.default_rng(n).standard_normal((n, d)).astype(np.float32)).cuda()


@pytest.mark.parametrize("solo", [1, 1 << 30])
@pytest.mark.parametrize("pipeline", ["native", "staged"])
def test_limits_by_the_server(monkeypatch, solo, pipeline):
    from flashph_b200.serve import PersistenceServer
    monkeypatch.setenv("FLASHPH_PIPELINE", pipeline)
    x, small = _cloud(1100), _cloud(90)
    with PersistenceServer(solo_min_points=solo, max_triangles=2000, max_tetrahedra=100) as srv:
        dense, sparse = srv.submit(x, 0.8, 1), srv.submit(x, 0.1, 1)
        tets = srv.submit(small, 0.9, 2)
        with pytest.raises(ValueError, match=r"max_triangles=2000\b"):
            dense.result(timeout=120)
        with pytest.raises(ValueError, match=r"max_tetrahedra=100\b"):
            tets.result(timeout=120)
        assert len(sparse.result(timeout=120)) == 2
    # C(450, 3) = 15,086,400 triangles, above the reference's limit
    with PersistenceServer(solo_min_points=solo, max_triangles=20_000_000) as srv:
        got = srv.submit(_cloud(450), 99.0, 1).result(timeout=120)
        assert got[0].shape[0] == 450
