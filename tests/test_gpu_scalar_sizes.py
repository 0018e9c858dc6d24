"""Poisson and diffusion assembly on both sides of the size where a lane takes two bonds at a time (9,472 nodes: the
blocks that the chip holds at once), against NumPy sums over the cache's own operators.

Tolerance: an off-diagonal entry is one product of a sum of two or three operators, (dim + 2) eps of the sum of their
magnitudes; the diagonal and the right-hand side add a family of m of them, (m + dim + 4) eps of the sum of magnitudes,
on both sides."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize("precision", [px.FP64, px.MIXED])
@pytest.mark.parametrize("dim,shape", [(2, (98, 96)), (2, (104, 92)), (3, (21, 21, 21)), (3, (24, 20, 20))])
@pytest.mark.parametrize("kind", [0, 1])
def test_scalar_assembly_either_side_of_the_size_rule(kind, dim, shape, precision):
    rng = np.random.default_rng(sum(shape))
    h = 1.0 / shape[0]
    q = np.indices(shape).reshape(dim, -1)[::-1].T.astype(np.float64)
    n = len(q)
    x = np.zeros((n, 3))
    x[:, :dim] = (q + 0.5 + rng.uniform(-0.2, 0.2, q.shape)) * h
    off, ids = px.families(x, 3.015 * h, dim == 3)
    c = px.Context(0)
    c.set_geometry(x, np.full(n, h ** dim), off, ids, 3.015 * h, h, dim)
    c.gbuild(2, precision, allow_degenerate=True)
    g = c.get_ops()
    c.csr_build_pattern(1)
    rowptr, cols = px.csr_pattern(off, ids, None, 1)
    u, uold, f = rng.standard_normal((3, n))
    coef, dt = 0.7, 1e-2
    kv, rhs = c.assemble_scalar(kind, coef, u, f_node=f, dt=dt if kind else 0.0, uold=uold if kind else None)
    src, nbr = np.repeat(np.arange(n), np.diff(off)), ids - 1
    second = [s for s, p in enumerate([(1, 0), (0, 1), (2, 0), (1, 1), (0, 2)]) if max(p) == 2] if dim == 2 else [3, 6, 8]
    co = (coef if kind == 0 else -coef) * g[:, second].sum(1)
    mag = abs(coef) * np.abs(g[:, second]).sum(1)
    m = np.diff(off)
    dsum, dmag, rsum, rmag = (np.zeros(n) for _ in range(4))
    np.add.at(dsum, src, co)
    np.add.at(dmag, src, mag)
    np.add.at(rsum, src, co * (u[nbr] - u[src]))
    np.add.at(rmag, src, mag * (np.abs(u[nbr]) + np.abs(u[src])))
    row = np.repeat(np.arange(n), np.diff(rowptr))
    where = {(r, k): e for e, (r, k) in enumerate(zip(row, cols))}
    at = np.array([where[(i, j)] for i, j in zip(src, nbr)])
    diag = np.array([where[(i, i)] for i in range(n)])
    tol = 2 * (m + dim + 4) * EPS
    assert np.all(np.abs(kv[at] + co) <= 2 * (dim + 2) * EPS * mag)
    assert np.all(np.abs(kv[diag] - (dsum - (1.0 / dt if kind else 0.0))) <= tol * (dmag + (1.0 / dt if kind else 0.0)))
    base = f if kind == 0 else (u - uold) / dt - f
    size = np.abs(f) + ((np.abs(u) + np.abs(uold)) / dt if kind else 0.0)
    assert np.all(np.abs(rhs - (base + rsum)) <= tol * (rmag + size))
