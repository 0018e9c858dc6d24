"""Patterns of three and more unknowns built on the device: rows and columns entry for entry against the host's, and block
positions and diagonal slots through assemblies that use every block, bit for bit against the same pattern given by the
caller (whose positions a check of its rows finds)."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape,ndof", [(3, (9, 8, 7), 3), (3, (6, 5, 5), 5), (2, (19, 17), 4), (2, (13, 11), 2)])
def test_built_pattern_and_given_one(dim, shape, ndof):
    L = px.lattice(dim, *(tuple(shape) + (0,) * (3 - dim)), sum(([0.0, s / shape[0]] for s in shape), []))
    delta = 3.015 * L.dxyz[0] * (1.0 + 1e-6)
    off, ids = px.families(L.coords, delta, dim == 3, mirror=L.mirror)
    rowptr, cols = px.csr_pattern(off, ids, L.mirror, ndof)
    rng = np.random.default_rng(ndof)
    n, nb = L.n, int(off[-1])
    u = rng.uniform(0.2, 0.8, n * ndof)
    uold = u + rng.uniform(-0.05, 0.05, n * ndof)
    health = (rng.uniform(size=nb) > 0.2).astype(np.float64)
    vel, mob = rng.uniform(-1, 1, n * dim), rng.uniform(0.1, 0.3, n)
    out = []
    for built in (True, False):
        c = px.Context(0)
        c.set_geometry(L.coords, L.vols, off, ids, delta, L.dxyz[0], dim, mirror=L.mirror)
        c.gbuild(2, px.FP64)
        if built:
            assert c.csr_build_pattern(ndof) == cols.size
            r, k = c.csr_get_pattern()
            assert np.array_equal(r, rowptr) and np.array_equal(k, cols)
        else:
            c.csr_set_pattern(rowptr, cols, ndof)
        if ndof == dim:
            prm = dict(C11=3.0, C12=1.1, C66=0.95, rho=0.5, dt=0.1, b=(0.1, -0.2, 0.3))
            out.append(c.assemble_cached(prm, u, uold, vel, dim, health, 1))
        else:
            c.ch_build_geometry()
            prm = dict(C11=1.35, C12=0.58, C66=0.385, A=0.3, Kh=0.9, Ch=-0.25, Omega=0.06, cref=0.5, chi=2.5, kappa=1e-2,
                       dt=0.1, kres=1e-4, rho=1.0)
            out.append(c.assemble_stress_ch(prm, mob, u, uold, health, vel))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    own = np.repeat(np.arange(rowptr.size - 1), np.diff(rowptr)) == cols
    assert np.count_nonzero(out[0][0][own]) == n * ndof  # every diagonal entry is there
