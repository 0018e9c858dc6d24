"""Slot lists of the mixed second-order apply that name a first derivative more than once: the transpose of the defect
correction counts once, so that <A u, y> = <u, A^T y> (both sums run over the same products in FP64: 1e-11 of their
magnitudes, as for lists without repeats), and a repeated slot's ybar adds up."""
import numpy as np
import pytest

from perix_b200 import api
from test_gpu_apply_rows import _geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,lists", [(2, ([0, 0, 4], [1, 3, 1, 2], [0, 1, 0, 1, 0, 2])),
                                       (3, ([2, 5, 2, 2], [0, 0, 8, 1], [7, 1, 1]))])
def test_repeated_first_derivatives(dim, lists):
    n = 203 if dim == 2 else 157
    x, off, ids, src, delta = _geometry(n, dim, (9, 33) if dim == 2 else (14, 70), n, symmetric=True)
    c = api.Context(0)
    c.set_geometry(x, np.full(n, 1.0 / n), off, ids + 1, delta, delta / 3.0, dim)
    c.gbuild(2, api.MIXED, allow_degenerate=True)
    rng = np.random.default_rng(dim)
    u = rng.standard_normal(n)
    for slots in lists:
        out = c.apply(u, slots)
        y = rng.standard_normal((n, len(slots)))
        ubar = c.apply_adjoint(y, slots)
        dot = np.abs(out * y).sum() + np.abs(u * ubar).sum()
        assert abs((out * y).sum() - (u * ubar).sum()) <= 1e-11 * dot
        distinct = sorted(set(slots))
        z = np.stack([y[:, [k for k, s in enumerate(slots) if s == d]].sum(axis=1) for d in distinct], 1)
        once = c.apply_adjoint(z, distinct)
        assert np.abs(ubar - once).max() <= 1e-11 * np.abs(once).max()
