"""The implicit run's scalars lie on one of two pages, in turn until the faster is known: repeated runs and a gradient on one
context, and the runs of new ones, give the same bits wherever they lie."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _context(m):
    L = px.lattice(2, m, m, 0, [0.0, 1.0, 0.0, 1.0])
    delta = 3.015 * L.dxyz[0] * (1.0 + 1e-6)
    off, ids = px.families(L.coords, delta, False, mirror=L.mirror)
    c = px.Context(0)
    c.set_geometry(L.coords, L.vols, off, ids, delta, L.dxyz[0], 2, mirror=L.mirror)
    c.gbuild(2, px.FP64)
    c.ch_build_geometry()
    c.csr_build_pattern(2)
    return c, 0.5 + np.random.default_rng(m).uniform(-0.01, 0.01, L.n)


@pytest.mark.parametrize("m", [9, 48, 130])
def test_same_bits_on_either_page(m):
    out, grads = [], []
    for _ in range(3):
        c, c0 = _context(m)
        for k in range(4):
            u, E, st = c.ch_run(c0, 2.5, 1e-4, 1.0, 1e-6, 3)
            out.append((u, E, st["newton_iters"], st["lin_iters"]))
            if k == 1:
                grads.append(c.ch_gradient(c0, 2.5, 1e-4, 1.0, 1e-6, 2)[:3])
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and o[1:] == out[0][1:]
    for g in grads[1:]:
        assert g[:2] == grads[0][:2] and np.array_equal(g[2], grads[0][2])
