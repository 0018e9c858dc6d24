"""The implicit Cahn-Hilliard run's Newton systems on slices (exact patterns) against its CSR path, which serves any
other pattern: the same run once on the exact pattern and once on a pattern widened by one unused block.

Node counts are below and past one slice of 32, no multiple of it, and past the lanes-a-node steps of the solver;
ghost nodes are mixed among the slices, and one run has none.

Tolerance: both paths solve every Newton system to |r| <= lin_rtol |F| and iterate to |F| <= newton_rtol |F_0| or
|dU| <= 1e-14 |U|, so the states differ by the linear tolerance times the update, far below
(steps) x 100 max(lin_rtol, newton_rtol) |U|."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
CHI, KAPPA, M0, DT = 2.5, 1e-4, 1.0, 1e-6


def _pair(nx, ny, ghosts):
    L = px.lattice(2, nx, ny, 0, [0.0, nx / 32.0, 0.0, ny / 32.0])
    mirror = L.mirror if ghosts else None
    delta = 3.015 * L.dxyz[0] * (1.0 + 1e-6)
    off, ids = px.families(L.coords, delta, False, mirror=mirror)
    rowptr, cols = px.csr_pattern(off, ids, L.mirror if ghosts else np.zeros(L.n, np.int32), 2)
    # one more block, to a node far away, in the rows of node 0: no exact pattern any more
    lo, hi = rowptr[0], rowptr[1]
    far = L.n - 1
    wide = np.sort(np.concatenate([cols[lo:hi], [2 * far, 2 * far + 1]])).astype(cols.dtype)
    cols2 = np.concatenate([wide, wide, cols[rowptr[2]:]])
    rowptr2 = rowptr.copy()
    rowptr2[1] += 2
    rowptr2[2:] += 4
    out = []
    for rp, cl in ((rowptr, cols), (rowptr2, cols2)):
        c = px.Context(0)
        c.set_geometry(L.coords, L.vols, off, ids, delta, L.dxyz[0], 2, mirror=mirror)
        c.gbuild(2, px.FP64, allow_degenerate=True)
        c.ch_build_geometry()
        c.csr_set_pattern(rp, cl, 2)
        out.append(c)
    return L, out


@pytest.mark.parametrize("nx,ny,ghosts", [(8, 9, True), (5, 5, False), (32, 17, True), (90, 75, True), (300, 260, True)])
def test_slices_against_csr_path(nx, ny, ghosts):
    L, (exact, general) = _pair(nx, ny, ghosts)
    c0 = 0.5 + np.random.default_rng(nx).uniform(-0.01, 0.01, L.n)
    steps = 3
    u, E, st = exact.ch_run(c0, CHI, KAPPA, M0, DT, steps)
    v, F, sv = general.ch_run(c0, CHI, KAPPA, M0, DT, steps)
    tol = steps * 100 * 1e-12
    for d in (0, 1):
        assert np.abs(u[d::2] - v[d::2]).max() <= tol * np.abs(v[d::2]).max()
    assert abs(E - F) <= tol * abs(F)
    assert st["max_lin_relres"] <= 1e-12 and st["steps"] == sv["steps"] == steps


def test_slices_give_way_to_memory():
    """Without room for the slices the CSR path answers; slices that are there make room for a later allocation."""
    L, (exact, general) = _pair(40, 40, True)
    c0 = 0.5 + np.random.default_rng(1).uniform(-0.01, 0.01, L.n)
    v = general.ch_run(c0, CHI, KAPPA, M0, DT, 2)[0]
    u = exact.ch_run(c0, CHI, KAPPA, M0, DT, 2)[0]
    held = exact.device_bytes()
    exact.set_memory_limit(held + 16 * (exact.nb + L.n))  # the gradient's CSR values take twice that
    E, dk, g, st = exact.ch_gradient(c0, CHI, KAPPA, M0, DT, 2)
    assert exact.device_bytes() < held
    exact.set_memory_limit(0)
    assert abs(E - general.ch_gradient(c0, CHI, KAPPA, M0, DT, 2)[0]) <= 1e-10 * abs(E)
    assert np.abs(u - v)[0::2].max() <= 2e-10 and np.isfinite(dk) and np.isfinite(g).all()
