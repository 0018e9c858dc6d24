"""The tensor-core g-build's solve (Gauss-Jordan, a few lanes a row) for every system size that takes it: 2, 3, 5 and 9
monomials.  The operators must reproduce their own definition, sum_t g^k_t xi_t^p = k! [p = k] over the node's bonds, and
a node whose family cannot carry the order is reported and gets zero operators.

Tolerance: Gauss-Jordan on an n x n symmetric positive definite system leaves a residual of at most 4 n^2 eps cond(A)
relative to |A| |X|, which here is at most sum_t |g^k_t| |xi_t^p|; the weights (between exp(-4) and 1, the rim correction
a factor of 1/2 at least for the bonds kept here) raise the condition number of the plain moment matrix, formed here, by at
most 2 e^4."""
import math

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _monomials(xi, dim, order):
    cols, fact = [], []
    for k in range(1, order + 1):
        for p in range(k, -1, -1):
            for q in range(k - p, -1, -1) if dim == 3 else (k - p,):
                r = k - p - q
                cols.append(xi[:, 0] ** p * xi[:, 1] ** q * (xi[:, 2] ** r if dim == 3 else 1.0))
                fact.append(math.factorial(p) * math.factorial(q) * math.factorial(r))
    return np.stack(cols, 1), np.array(fact, float)


@pytest.mark.parametrize("dim,order,n,fam", [(2, 1, 37, 8), (3, 1, 41, 12), (2, 2, 65, 20), (3, 2, 50, 40),
                                             (2, 3, 70, 33), (3, 2, 180, 150)])
def test_operators_reproduce_their_definition(dim, order, n, fam):
    rng = np.random.default_rng(10 * dim + order)
    x = np.zeros((n, 3))
    x[:, :dim] = rng.uniform(0.0, 1.0, (n, dim))
    d = np.linalg.norm(x[:, None] - x[None], axis=2)
    np.fill_diagonal(d, np.inf)
    keep = [np.sort(np.argsort(d[i])[:1 if i == 7 else fam - i % 5]) for i in range(n)]  # node 7: one bond only
    off = np.concatenate([[0], np.cumsum([len(k) for k in keep])]).astype(np.int32)
    ids = np.concatenate(keep).astype(np.int32)
    src = np.repeat(np.arange(n), np.diff(off))
    delta = 2.0 * d[src, ids].max()  # every bond inside half the horizon: no rim bond, weights above exp(-1)
    c = px.Context(0)
    c.set_geometry(x, np.full(n, 1.0 / n), off, ids + 1, delta, delta / 50.0, dim)
    c.gbuild_set_schedule(2)
    bad, first = c.gbuild(order, px.FP64, allow_degenerate=True)
    assert bad >= 1 and first <= 8
    g = c.get_ops()
    assert not g[off[7]:off[8]].any()
    m, fact = _monomials((x[ids] - x[src]) / delta, dim, order)
    scale = _monomials(np.full((1, 3), 1.0 / delta), dim, order)[0][0]  # operators carry 1 / delta^|k|
    checked = 0
    for i in range(n):
        b = slice(off[i], off[i + 1])
        if not g[b].any():
            continue
        gi, mi = g[b] / scale, m[b]
        cond = 2.0 * math.exp(4.0) * np.linalg.cond(mi.T @ mi)
        tol = 4.0 * g.shape[1] ** 2 * EPS * cond
        if tol > 1e-3:
            continue
        res = np.abs(gi.T @ mi - np.diag(fact))
        assert np.all(res <= tol * (np.abs(gi).T @ np.abs(mi) + np.diag(fact)))
        checked += 1
    assert checked >= n // 2
