"""CSR assembly on exact block patterns (k_csr_block.cu) against the kernels that serve any pattern (k_csr.cu): the
same systems on the device-built pattern and on that pattern with one foreign column node added to every row list, for
Poisson and diffusion, implicit dynamic fracture, Cahn-Hilliard and stress-coupled Cahn-Hilliard, in 2D and 3D, node
counts that leave a partial tile, families up to ~110 bonds in 2D (one tile of four nodes a block), a mirror node
outside its ghost's family, broken bonds, and a value array that is only 8-byte aligned.

Tolerance: both paths form the same bond terms with at most three roundings' difference (the block kernels multiply by
1/V_i where the others divide) and sum m of them in another order, so an entry differs by at most (m + 4) eps times
the sum of its terms' magnitudes; a diagonal entry is the sum of its row's off-diagonal blocks plus the nodal term, a
right-hand side the sum of K_IJ (u_j - u_i) plus the nodal term."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _mesh(ctx, dim, shape, horizon, far_mirror):
    import perix_b200 as px
    L = px.lattice(dim, *(tuple(shape) + (0,) * (3 - len(shape))), [0.0, 1.0] + [0.0, shape[1] / shape[0]] +
                   ([0.0, shape[2] / shape[0]] if dim == 3 else []))
    delta = horizon * L.dxyz[0] * (1.0 + 1e-6)
    off, ids = px.families(L.coords, delta, dim == 3, mirror=L.mirror)
    mirror = L.mirror.copy()
    if far_mirror:  # one ghost names a bulk node far outside its family
        g = int(np.nonzero(mirror > 0)[0][0])
        mirror[g] = L.nbulk
    ctx.set_geometry(L.coords, L.vols, off, ids, delta, L.dxyz[0], dim, mirror=mirror)
    ctx.gbuild(2, px.FP64)
    return L, off, ids, mirror


def _widened(off, ids, mirror, nd, n):
    """The pattern with one more column node in every list: (rowptr, cols, where the exact pattern's entries went)."""
    lists = []
    for i in range(n):
        have = set((ids[off[i]:off[i + 1]] - 1).tolist()) | {i}
        if mirror is not None and mirror[i] > 0:
            have.add(int(mirror[i]) - 1)
        foreign = next(k for k in range(n - 1, -1, -1) if k not in have)
        lists.append((sorted(have), sorted(have | {foreign})))
    rowptr, cols, keep = [0], [], []
    for exact, wide in lists:
        for _ in range(nd):
            for node in wide:
                for c in range(nd):
                    if node in set(exact):
                        keep.append(len(cols))
                    cols.append(node * nd + c)
            rowptr.append(len(cols))
    return np.asarray(rowptr, np.int32), np.asarray(cols, np.int32), np.asarray(keep)


def _check(exact, wide, keep, rowptr, cols, nd, fam, ulen, nodal):
    """exact / wide: (kvals, rhs) of the two paths on one system; ulen: per dof range of the unknowns."""
    ka, ra = exact
    kb, rb = wide
    assert not np.delete(kb, keep).any()  # the foreign columns stay zero
    kb = kb[keep]
    rows = np.repeat(np.arange(rowptr.size - 1), np.diff(rowptr))
    own = rows // nd == cols // nd
    absum = np.zeros((rowptr.size - 1, nd))  # per row and column dof: sum of the off-diagonal magnitudes
    np.add.at(absum, (rows[~own], cols[~own] % nd), np.abs(kb[~own]))
    m = fam.max() + 4
    tol = np.where(own, m * EPS * (absum[rows, cols % nd] + np.abs(kb) + nodal[cols % nd]), 4 * EPS * np.abs(kb))
    assert (np.abs(ka - kb) <= tol).all()
    rtol = m * EPS * (absum @ ulen + np.abs(rb) + np.tile(nodal, rb.size // nd))
    assert (np.abs(ra - rb) <= rtol).all()


CASES = [(2, (13, 11), 3.015, False), (2, (9, 9), 3.015, True), (2, (15, 14), 6.015, False), (3, (6, 5, 5), 3.015, False),
         (3, (5, 4, 4), 3.015, True)]


@pytest.mark.parametrize("dim,shape,horizon,far_mirror", CASES)
@pytest.mark.parametrize("kind", ["poisson", "diffusion", "dynfrac", "ch", "stress", "stress_fracture"])
def test_block_pattern_matches_general(ctx, kind, dim, shape, horizon, far_mirror):
    if kind == "ch" and dim == 3:
        pytest.skip("two-dof Cahn-Hilliard is compared in 2D")
    nd = {"poisson": 1, "diffusion": 1, "dynfrac": dim, "ch": 2}.get(kind, dim + 2)
    L, off, ids, mirror = _mesh(ctx, dim, shape, horizon, far_mirror)
    n, nb = L.n, int(off[-1])
    rng = np.random.default_rng(7)
    u = rng.uniform(0.2, 0.8, n * nd)
    uold = u + rng.uniform(-0.05, 0.05, n * nd)
    health = (rng.uniform(size=nb) > 0.2).astype(np.float64)
    vel = rng.uniform(-1, 1, n * dim)
    mob = rng.uniform(0.1, 0.3, n)
    if nd > 1:
        ctx.ch_build_geometry()

    def assemble():
        if kind in ("poisson", "diffusion"):
            t = kind == "diffusion"
            return ctx.assemble_scalar(int(t), 0.7, u, f_node=vel[:n].copy(), dt=1e-2 if t else 0.0, uold=uold if t else None)
        if kind == "dynfrac":
            prm = dict(C11=3.0, C12=1.1, C66=0.95, rho=0.5, dt=0.1, b=(0.1, -0.2, 0.3))
            return ctx.assemble_cached(prm, u, uold, vel, dim, health, 1)
        if kind == "ch":
            return ctx.assemble_ch(1e-2, 2.5, 0.1, mob, u, uold)
        prm = dict(C11=1.35, C12=0.58, C66=0.385, A=0.3, Kh=0.9, Ch=-0.25, Omega=0.06, cref=0.5, chi=2.5, kappa=1e-2, dt=0.1,
                   kres=1e-4, rho=1.0 if kind == "stress_fracture" else 0.0)
        frac = kind == "stress_fracture"
        return ctx.assemble_stress_ch(prm, mob, u, uold, health if frac else None, vel if frac else None)

    ctx.csr_build_pattern(nd)
    rowptr, cols = ctx.csr_get_pattern()
    exact = assemble()
    wr, wc, keep = _widened(off, ids, mirror, nd, n)
    ctx.csr_set_pattern(wr, wc, nd)
    wide = assemble()
    fam = np.diff(off)
    # nodal terms: at most 1/dt, 1/(c(1-c)), rho/dt^2 times O(1) values
    _check(exact, wide, keep, rowptr, cols, nd, fam, np.full(nd, 0.7), np.full(nd, 200.0))
    # the caller's own copy of the exact pattern takes the block path too
    ctx.csr_set_pattern(rowptr, cols, nd)
    again = assemble()
    assert np.array_equal(again[0], exact[0]) and np.array_equal(again[1], exact[1])


def test_ch_values_at_an_odd_address(ctx):
    import torch
    L, off, ids, mirror = _mesh(ctx, 2, (11, 10), 3.015, False)
    ctx.ch_build_geometry()
    nnz = ctx.csr_build_pattern(2)
    u = torch.rand(2 * L.n, dtype=torch.float64, device="cuda") * 0.6 + 0.2
    mob = torch.rand(L.n, dtype=torch.float64, device="cuda")
    out = []
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    for shift in (0, 1):
        kv = torch.full((nnz + 1,), 7.0, dtype=torch.float64, device="cuda")[shift:shift + nnz]
        rhs = torch.empty(2 * L.n, dtype=torch.float64, device="cuda")
        ctx.assemble_ch_d(1e-2, 2.5, 0.1, mob.data_ptr(), u.data_ptr(), u.data_ptr(), kv.data_ptr(), rhs.data_ptr())
        out.append((kv.clone(), rhs))
    ctx.set_stream(None)
    assert kv.data_ptr() % 16 == 8
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
