"""Block positions as the device pattern's sort leaves them, against those that the check of a caller's pattern finds: the
same assembled values, bit for bit.  List lengths around 32, 64 and 128 (the sort's sizes), mirrors in and outside the
family, a node without a mirror, families that list a node twice or the node itself (no exact pattern: both go through the
general path), one to three unknowns."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _families(n, dim, length, kind, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, 3))
    x[:, :dim] = rng.uniform(0.0, 1.0, (n, dim))
    d = np.linalg.norm(x[:, None] - x[None], axis=2)
    np.fill_diagonal(d, np.inf)
    fam = [rng.permutation(np.argsort(d[i])[:length - int(rng.integers(0, 3))]) for i in range(n)]
    mirror = np.zeros(n, np.int32)
    far = np.argsort(np.where(np.isinf(d), -1.0, d), axis=1)
    for i in range(0, n, 3):
        mirror[i] = 1 + (fam[i][0] if i % 2 else far[i, -1])  # in the family, outside it
    if kind == "twice":
        fam[5] = np.concatenate([fam[5], fam[5][:1]])
    if kind == "self":
        fam[7] = np.concatenate([fam[7], [7]])
    off = np.concatenate([[0], np.cumsum([len(f) for f in fam])]).astype(np.int32)
    ids = np.concatenate(fam).astype(np.int32)
    src = np.repeat(np.arange(n), np.diff(off))
    delta = 1.01 * np.linalg.norm(x[ids] - x[src], axis=1).max()
    return x, off, ids + 1, delta, mirror


@pytest.mark.parametrize("kind", ["plain", "twice", "self"])
@pytest.mark.parametrize("n,length", [(40, 9), (60, 30), (61, 31), (80, 62), (90, 63), (150, 126), (160, 128), (200, 180)])
def test_positions_of_built_and_given_pattern_agree(n, length, kind):
    x, off, ids, delta, mirror = _families(n, 2, length, kind, n + length)
    vals = []
    for built in (True, False):
        c = px.Context(0)
        c.set_geometry(x, np.full(n, 1.0 / n), off, ids, delta, delta / 3.0, 2, mirror=mirror)
        c.gbuild(2, px.FP64, allow_degenerate=True)
        if built:
            nnz = c.csr_build_pattern(1)
        else:
            rowptr, cols = px.csr_pattern(off, ids, mirror, 1)
            c.csr_set_pattern(rowptr, cols, 1)
            assert nnz == cols.size
        u = np.random.default_rng(1).standard_normal(n)
        vals.append(c.assemble_scalar(0, 0.7, u, f_node=u))
    assert np.array_equal(vals[0][0], vals[1][0]) and np.array_equal(vals[0][1], vals[1][1])


@pytest.mark.parametrize("ndof", [2, 3])
def test_positions_with_several_unknowns(ndof):
    """The diagonal slots too: the pattern built on the device and the host's, read back and compared through the dense
    rows of an assembly that touches every block (ndof 2: Cahn-Hilliard, 3: nothing assembled, the pattern alone)."""
    L = px.lattice(2, 19, 17, 0, [0.0, 1.0, 0.0, 1.0])
    delta = 3.015 * L.dxyz[0] * (1.0 + 1e-6)
    off, ids = px.families(L.coords, delta, False, mirror=L.mirror)
    rowptr, cols = px.csr_pattern(off, ids, L.mirror, ndof)
    out = []
    for built in (True, False):
        c = px.Context(0)
        c.set_geometry(L.coords, L.vols, off, ids, delta, L.dxyz[0], 2, mirror=L.mirror)
        c.gbuild(2, px.FP64)
        if built:
            assert c.csr_build_pattern(ndof) == cols.size
        else:
            c.csr_set_pattern(rowptr, cols, ndof)
        if ndof == 2:
            c.ch_build_geometry()
            c0 = 0.5 + np.random.default_rng(2).uniform(-0.01, 0.01, L.n)
            out.append(c.ch_gradient(c0, 2.5, 1e-4, 1.0, 1e-6, 2))
    if ndof == 2:
        assert out[0][0] == out[1][0] and out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])
