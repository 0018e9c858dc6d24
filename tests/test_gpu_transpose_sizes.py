"""The apply's transpose on both sides of the sizes from which it takes two passes (800,000 bonds in 2D; in 3D bonds times
operators asked for plus two, 2.9 million in FP64 and 8 million mixed), against sums in NumPy: a jittered lattice, every row length with kernels of its
own, both precisions.  The scratch of the two passes (8 bytes a bond) shows which way a call went.

Tolerance: a node's value is a sum of K m products of two, m own and m reverse bonds, in another order than NumPy's: at most
(2 K m + 6) eps of the sum of their magnitudes each."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _lattice(dim, m, seed):
    rng = np.random.default_rng(seed)
    q = np.indices(m).reshape(dim, -1)[::-1].T.astype(np.float64)
    h = 1.0 / max(m)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5 + rng.uniform(-0.1, 0.1, q.shape)) * h
    return x, h


@pytest.mark.parametrize("precision", [px.FP64, px.MIXED])
@pytest.mark.parametrize("dim,order,m,slots", [
    (2, 1, (170, 170), [0, 1]), (2, 1, (180, 180), [0, 1]), (2, 2, (180, 180), [4, 1, 4, 0]), (2, 2, (170, 170), [0, 1, 2, 3, 4]),
    (2, 3, (181, 183), [8, 2, 5]), (3, 1, (21, 21, 20), [0, 1, 2]), (3, 1, (14, 15, 16), [2]), (3, 2, (16, 16, 17), list(range(9))),
    (3, 2, (14, 14, 15), list(range(9))), (3, 2, (22, 21, 20), [8]), (3, 2, (25, 23, 24), [8]), (3, 2, (20, 21, 21), list(range(9))), (3, 1, (30, 31, 31), [0, 1, 2])])
def test_transpose_on_both_sides(dim, order, m, slots, precision):
    x, h = _lattice(dim, m, sum(m))
    n = len(x)
    delta = (4.015 if order == 3 else 3.015) * h
    c = px.Context(0)
    c.set_geometry_points(x, np.full(n, h ** dim), delta, delta, h, dim)
    c.gbuild(order, precision, allow_degenerate=True)
    off, ids = c.get_families()
    ids = ids.astype(np.int64) - 1
    src = np.repeat(np.arange(n), np.diff(off))
    y = np.random.default_rng(order).standard_normal((n, len(slots)))
    held = c.device_bytes()
    got = c.apply_adjoint(y, slots)
    defect = precision == px.MIXED and order == 2 and max(slots) >= dim  # first derivatives join the scatter
    used = len(set(slots) | set(range(dim) if defect else ()))
    two = c.nb >= 800000 if dim == 2 else c.nb * (used + 2) >= (8000000 if precision == px.MIXED else 2900000)
    again = c.apply_adjoint(y, slots)
    assert np.array_equal(got, again)
    more = c.device_bytes() - held
    assert (more >= 12 * c.nb) == two  # the reverse bonds take 4, the scratch 8
    if defect:  # the correction's transpose is tested by the identity of the inner products
        u = np.random.default_rng(3).standard_normal(n)
        out = c.apply(u, slots)
        dot = np.abs(out * y).sum() + np.abs(u * got).sum()
        assert abs((out * y).sum() - (u * got).sum()) <= 1e-11 * dot
        return
    g = c.get_ops()
    s = (g[:, slots] * y[src]).sum(axis=1)
    sa = (np.abs(g[:, slots]) * np.abs(y[src])).sum(axis=1)
    ref = np.bincount(ids, s, n) - np.bincount(src, s, n)
    scale = np.bincount(ids, sa, n) + np.bincount(src, sa, n)
    k = int(np.diff(off).max())
    assert np.all(np.abs(got - ref) <= (2 * len(slots) * k + 6) * 2 * EPS * scale)
