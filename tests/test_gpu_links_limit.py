"""Calls over the triangle limit whose triangles the link pass counts: the error
has the exact total, wherever in the pass the limit is met, and a limit of just
that total is kept to. Warps bring their counts together every 16 edges, so
graphs of more edges than 16 a warp, with a warp an edge and with eight lanes."""
from __future__ import annotations

import re

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,t", [(6000, 3, 0.42), (60000, 3, 0.13), (3000, 8, 2.2)])
def test_total_in_the_error(n, d, t):
    from flashph_b200.cohomology import count_triangles
    from flashph_b200.persistence import _compute_native
    from flashph_b200.rips import rips_filtration
    x = torch.from_numpy(np.random.default_rng(n).standard_normal((n, d)).astype(np.float32)).cuda()
    filt = rips_filtration(x, t)
    E = filt.edge_i.shape[0]
    total = int(count_triangles(filt)[-1].item())
    assert 4.0 * E * E / n <= 2e8  # else the total is counted before the links
    for limit in (0, 1, total // 50, total // 2, total - 1):
        with pytest.raises(ValueError) as e:
            _compute_native(x, t, 1, x.device, max_triangles=limit)
        assert int(re.search(r"count (\d+)", str(e.value)).group(1)) == total
    assert len(_compute_native(x, t, 1, x.device, max_triangles=total)) == 2
