"""Family-sum apply and its transpose where the operator row has kernels of its own (2, 3, 5 or 9 operators) and
where it has not (third order in 3D, 19), against NumPy sums over the cache's own operators.

The families are ragged (short ones, ones past two strides of the lane group), irregular, and not symmetric: a third
of the bonds has no reverse.  n is no multiple of a block's nodes; the slot lists are all operators in order, a
subset out of order, and one with a repeat.

Tolerance: a sum of m products, in any order and with or without fused multiply-adds, is within
(m + 4) eps sum|terms| of the exact sum, on both sides; m is at most the family's length times the slots, plus two
for the difference u_j - u_i.  Mixed second order adds the defect correction, whose coefficients are not read back:
its families are symmetric, and <A u, y> = <u, A^T y> is asserted instead."""
import numpy as np
import pytest

from perix_b200 import api

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
SLOTS = {2: ([0, 1], [1], [1, 0, 1]), 3: ([0, 1, 2], [2], [2, 0, 2]),
         5: ([0, 1, 2, 3, 4], [3, 1], [4, 4, 0]), 9: (list(range(9)), [7, 0, 3], [8, 5, 5, 2]),
         19: (list(range(19)), [18, 4], [6, 6, 1])}


def _geometry(n, dim, fam, seed, symmetric=False):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, 3))
    x[:, :dim] = rng.uniform(0.0, 1.0, (n, dim))
    near = np.zeros((n, n), bool)
    for i in range(n):
        d = np.linalg.norm(x - x[i], axis=1)
        d[i] = np.inf
        near[i, np.argsort(d)[:min(n - 1, int(rng.integers(fam[0], fam[1] + 1)))]] = True
    if symmetric:
        near |= near.T
    src, ids = np.nonzero(near)
    off = np.concatenate([[0], np.cumsum(near.sum(axis=1))])
    delta = float(np.linalg.norm(x[ids] - x[src], axis=1).max()) * 1.01
    return x, np.asarray(off, np.int32), ids.astype(np.int32), src, delta


@pytest.mark.parametrize("dim,order,n,fam", [(2, 1, 61, (3, 19)), (3, 1, 50, (5, 40)), (2, 2, 203, (9, 33)),
                                             (3, 2, 157, (14, 70)), (2, 3, 97, (16, 40)), (3, 3, 83, (40, 75)),
                                             (2, 2, 12, (11, 11))])
@pytest.mark.parametrize("precision", [api.FP64, api.MIXED])
def test_apply_rows_against_sums(dim, order, n, fam, precision):
    defect = precision == api.MIXED and order == 2   # second derivatives corrected by their operators' defects
    x, off, ids, src, delta = _geometry(n, dim, fam, 7 * n + dim, symmetric=defect)
    rng = np.random.default_rng(n)
    c = api.Context(0)
    c.set_geometry(x, np.full(n, 1.0 / n), off, ids + 1, delta, delta / 3.0, dim)
    c.gbuild(order, precision, allow_degenerate=True)
    g = c.get_ops()
    u = rng.standard_normal(n)
    m = int(np.diff(off).max()) + 6
    for slots in SLOTS[c.nop]:
        out = c.apply(u, slots)
        y = rng.standard_normal((n, len(slots)))
        ubar = c.apply_adjoint(y, slots)
        if defect:
            dot = np.abs(out * y).sum() + np.abs(u * ubar).sum()
            assert abs((out * y).sum() - (u * ubar).sum()) <= 1e-11 * dot
            first = [k for k, s in enumerate(slots) if s < dim]
        else:
            first = list(range(len(slots)))
        du = u[ids] - u[src]
        for k in first:
            t = g[:, slots[k]] * du
            ref, scale = np.zeros(n), np.zeros(n)
            np.add.at(ref, src, t)
            np.add.at(scale, src, np.abs(g[:, slots[k]]) * (np.abs(u[ids]) + np.abs(u[src])))
            assert np.all(np.abs(out[:, k] - ref) <= 2 * m * EPS * scale)
        if defect:
            continue
        s = (g[:, slots] * y[src]).sum(axis=1)
        sa = (np.abs(g[:, slots]) * np.abs(y[src])).sum(axis=1)
        ref, scale, cnt = np.zeros(n), np.zeros(n), np.zeros(n)
        # the transpose adds the bonds whose reverse exists (m's own family lists the source) and subtracts its own
        pair = {(int(i), int(j)): t for t, (i, j) in enumerate(zip(src, ids))}
        rev = np.array([pair.get((int(j), int(i)), -1) for i, j in zip(src, ids)])
        has = rev >= 0
        np.add.at(ref, src[has], s[rev[has]])
        np.add.at(ref, src, -s)
        np.add.at(scale, src[has], sa[rev[has]])
        np.add.at(scale, src, sa)
        np.add.at(cnt, src, 1.0)
        assert np.all(np.abs(ubar - ref) <= 2 * (2 * cnt + len(slots) + 6) * EPS * scale)


def test_adjoint_without_scratch_and_on_two_streams():
    """Without room for the scratch the one-pass kernel answers; calls on two streams do not share it at one time."""
    torch = pytest.importorskip("torch")
    x, off, ids, src, delta = _geometry(3001, 3, (60, 120), 5)
    n = x.shape[0]
    c = api.Context(0)
    c.set_geometry(x, np.full(n, 1.0 / n), off, ids + 1, delta, delta / 3.0, 3)
    c.gbuild(2, api.FP64, allow_degenerate=True)
    g = c.get_ops()
    slots = list(range(9))
    ys = [torch.randn(n, 9, dtype=torch.float64, device="cuda") for _ in range(8)]
    outs = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in ys]
    ones = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in ys]
    c.apply_adjoint_d(ys[0].data_ptr(), slots, outs[0].data_ptr())  # reverse bonds and scratch are there
    c.synchronize()
    with_scratch = c.device_bytes()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k, (y, o) in enumerate(zip(ys, outs)):
        c.set_stream(streams[k & 1].cuda_stream)
        c.apply_adjoint_d(y.data_ptr(), slots, o.data_ptr())
    torch.cuda.synchronize()
    c2 = api.Context(0)
    c2.set_geometry(x, np.full(n, 1.0 / n), off, ids + 1, delta, delta / 3.0, 3)
    c2.gbuild(2, api.FP64, allow_degenerate=True)
    c2.set_memory_limit(c2.device_bytes() + 4 * c2.nb + 64)  # the reverse bonds fit, the scratch does not
    for y, o in zip(ys, ones):
        c2.apply_adjoint_d(y.data_ptr(), slots, o.data_ptr())
    c2.synchronize()
    assert c2.device_bytes() < with_scratch
    m = int(np.diff(off).max())
    scale = np.zeros(n)
    for y, o, e in zip(ys, outs, ones):
        sa = (np.abs(g) * np.abs(y.cpu().numpy()[src])).sum(axis=1)
        scale[:] = 0.0
        np.add.at(scale, src, sa)
        np.add.at(scale, ids, sa)
        assert np.all(np.abs((o - e).cpu().numpy()) <= 2 * (2 * 4 * m + 15) * EPS * scale)
