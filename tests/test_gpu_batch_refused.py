"""Batches of which no cloud is left for H1: each refused with the single call's
error, or done with H0, whatever the number of rows they would have had."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,limit", [([1], 0), ([1], 10), ([2, 1, 2], 10), ([0, 1, 0, 2], 10), ([0, 1], 0)])
def test_no_cloud_left(dims, limit):
    from flashph_b200 import _lib, rips_persistence
    from flashph_b200.batch import rips_persistence_batch
    from flashph_b200.persistence import _compute_native
    rng = np.random.default_rng(len(dims))
    x = [torch.from_numpy(rng.standard_normal((60 + 9 * k, 3)).astype(np.float32)).cuda() for k in range(len(dims))]
    rips_persistence_batch(x, 1.5, dims)  # the edge kernel's trial of this batch's sizes is done
    before = _lib.launch_count()
    got = rips_persistence_batch(x, 1.5, dims, max_triangles=limit)
    refused = _lib.launch_count() - before
    for p, dim, g in zip(x, dims, got):
        if dim == 0:
            want = rips_persistence(p, 1.5, max_dim=0)[0]
            assert len(g) == 1 and torch.equal(g[0].view(torch.int32), want.view(torch.int32))
            continue
        with pytest.raises(ValueError) as e:
            _compute_native(p, 1.5, dim, p.device, max_triangles=limit)
        assert isinstance(g, ValueError) and str(g) == str(e.value) and f"max_triangles={limit}." in str(g)
    if limit:
        return  # the exact totals are more launches
    # nothing of the reduction ran
    before = _lib.launch_count()
    rips_persistence_batch(x, 1.5, dims)
    assert refused < _lib.launch_count() - before - 8
