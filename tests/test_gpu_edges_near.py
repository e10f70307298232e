"""Edges from blocks in grid order (large clouds of up to four dimensions)
against the direct kernel, through the whole native call: the same number of
edges and triangles and the same H0 and H1 rows, bit for bit."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(x, t, mode, dim=1):
    """Edges, triangles and rows of one native call with the given edge mode
    (0: by size, 2: the direct kernel)."""
    from flashph_b200 import _lib as L
    lib, res = L.lib(), ctypes.c_void_p()
    s = L.stream_handle(x.device)
    rc = lib.ph_rips_persistence(x.data_ptr(), x.shape[0], x.shape[1], t, dim, 1 << 28, 1 << 28, mode,
                                 ctypes.byref(res), s)
    assert rc == L.PH_OK, lib.ph_last_error()
    rows = [int(lib.ph_result_rows(res, k)) for k in range(dim + 1)]
    buf = torch.empty(sum(rows), 2, dtype=torch.float32, device=x.device)
    L.call("ph_result_copy_all", res, buf.data_ptr(), 0, s)
    torch.cuda.synchronize()
    stat = [int(lib.ph_result_stat(res, k)) for k in (0, 1)]
    lib.ph_result_free(res)
    return stat, rows, buf.view(torch.int32).cpu()


def _check(x, t, dim=1):
    x = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()
    near, direct = _run(x, t, 0, dim), _run(x, t, 2, dim)
    assert near[0] == direct[0] and near[1] == direct[1]
    assert torch.equal(near[2], direct[2])
    return near[0]


# n^2 (d + 8) past 5e8 takes the grid form: just past it, remainders of a block
@pytest.mark.parametrize("n,d,t", [
    (7500, 1, 0.001), (7169, 2, 0.05), (9001, 2, 0.02), (7041, 3, 0.1), (12801, 3, 0.15), (6500, 4, 0.3),
    (20011, 4, 0.25), (100003, 2, 0.006)])
def test_gaussian_clouds(n, d, t):
    edges, _ = _check(np.random.default_rng(n).standard_normal((n, d)), t)
    assert edges > n // 4


def test_wide_threshold_keeps_every_block():
    """A threshold near the cloud's size: all pairs of blocks are listed."""
    x = np.random.default_rng(5).standard_normal((7200, 3)) * 0.01
    edges, _ = _check(x, 0.03, dim=0)
    assert edges > 5_000_000
    _check(x, float("inf"), dim=0)


def test_uneven_and_degenerate_clouds():
    rng = np.random.default_rng(6)
    x = np.concatenate([rng.standard_normal((8000, 3)) * 1e-3, rng.standard_normal((60, 3)) * 1e6])
    _check(x[rng.permutation(len(x))], 2e-4)  # outliers: one cell holds nearly all points
    line = np.zeros((7600, 3))
    line[:, 1] = rng.uniform(0, 100, 7600)
    _check(line, 0.02)  # two coordinates constant
    _check(np.repeat(rng.standard_normal((2500, 2)), 3, axis=0), 0.01)  # duplicates
    far = rng.standard_normal((8000, 3)) + 1e4
    _check(far, 0.1)  # far from the origin


def test_lattice_ties_on_the_strict_threshold():
    x = np.stack(np.meshgrid(np.arange(90), np.arange(90), indexing="ij"), -1).reshape(-1, 2)
    assert _check(x, 1.0)[0] == 0  # strict: unit distances are not below it
    assert _check(x, 1.25)[0] == 2 * 90 * 89


def test_points_that_are_not_finite():
    rng = np.random.default_rng(8)
    x = rng.standard_normal((8000, 3))
    x[::40, 1] = np.nan
    x[7::200, 0] = np.inf
    x[9::200, 2] = -np.inf
    _check(x, 0.1)
    x[:] = np.nan
    assert _check(x, 0.1)[0] == 0
