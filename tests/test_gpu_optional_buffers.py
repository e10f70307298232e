"""Calls for which the buffers that they can do without are not to be had
(ph_set_optional_buffer_limit takes those above a size as such, as on a device
without memory to spare): the rank tables, the scratch of the faster edge
kernels and of the triangle totals, and the first guess of the triangle and
tetrahedron rows, so that these are counted, sized and counted again. The
diagrams and the errors are those of the calls that had them."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit():
    from flashph_b200 import _lib
    yield _lib.lib().ph_set_optional_buffer_limit
    _lib.lib().ph_set_optional_buffer_limit(0)


def _cloud(n, d, seed=1):
    return torch.from_numpy(np.random.default_rng(seed).standard_normal((n, d)).astype(np.float32)).cuda()


def _same(a, b):
    assert type(a) is type(b)
    if isinstance(a, Exception):
        assert str(a) == str(b)
        return
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))


# with a rank table and without one, rows up to H2, the tetrahedra counted
# before and after the H1 reduction, the grid-ordered and the screened edges
@pytest.mark.parametrize("n,d,t,dim", [
    (2, 3, 9.0, 2), (300, 3, 1.1, 2), (150, 8, 3.6, 2), (3000, 10, 1.7, 2), (900, 8, 3.0, 1), (9000, 3, 0.25, 1),
    (9000, 12, 2.2, 1), (7000, 5, 0.9, 0)])
@pytest.mark.parametrize("most", [1, 300_000])
def test_single_call(limit, n, d, t, dim, most):
    from flashph_b200 import rips_persistence
    x = _cloud(n, d, n)
    want = rips_persistence(x, t, max_dim=dim)
    limit(most)
    _same(rips_persistence(x, t, max_dim=dim), want)


def test_over_the_triangle_limit(limit):
    from flashph_b200 import rips_persistence
    x = _cloud(1500, 3)
    messages = []
    for most in (0, 1):
        limit(most)
        with pytest.raises(ValueError, match="max_triangles") as e:
            rips_persistence(x, 9.0, max_dim=1)
        messages.append(str(e.value))
    assert messages[0] == messages[1]


# dense and sparse clouds, dimensions 0 to 2, one cloud over the triangle limit
# and two over the tetrahedron limit (dropped from H2 after their count; one has all 487,635 of 60 points)
@pytest.mark.parametrize("most", [1, 20_000])
def test_batch(limit, most):
    from flashph_b200.batch import rips_persistence_batch
    x = [_cloud(300, 3, 1), _cloud(120, 4, 2), _cloud(700, 3, 3), _cloud(60, 2, 4), _cloud(200, 8, 5), _cloud(2, 1, 6),
         _cloud(400, 3, 7)]
    ts, dims = [1.0, 3.0, 0.4, 9.0, 3.2, 9.0, 9.0], [2, 2, 1, 2, 0, 2, 1]
    want = rips_persistence_batch(x, ts, dims, max_triangles=200_000, max_tetrahedra=400_000)
    assert [isinstance(w, Exception) for w in want] == [False, True, False, True, False, False, True]
    limit(most)
    got = rips_persistence_batch(x, ts, dims, max_triangles=200_000, max_tetrahedra=400_000)
    for a, b in zip(got, want):
        _same(a, b)
