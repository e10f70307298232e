"""The short scan at its tile (4096) and range (65,536) edges: the place of
each forest edge's row is the exclusive prefix count of the mask."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 31, 4095, 4096, 4097, 8193, 61440, 65535, 65536, 65537])
@pytest.mark.parametrize("share", [0.0, 0.4, 1.0])
def test_h0_rows_at_short_scan_edges(E, share):
    from flashph_b200.boruvka import h0_rows
    rng = np.random.default_rng(E)
    mask = (rng.random(E) < share).astype(np.uint8)
    filt = np.sort(rng.random(E).astype(np.float32))
    rows = h0_rows(torch.from_numpy(filt).cuda(), torch.from_numpy(mask).cuda(), E + 3).cpu().numpy()
    k = int(mask.sum())
    assert np.array_equal(rows[:k, 1], filt[mask == 1])
    assert np.all(np.isinf(rows[k:, 1])) and np.all(rows[:, 0] == 0)
