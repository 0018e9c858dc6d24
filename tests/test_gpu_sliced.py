"""The sliced step (k_epf_sliced.cu) where its second copy of the bond streams can go wrong: node counts around the
slice of 32, families of very different length in one slice, bonds broken by the caller, by another schedule, by a
restored snapshot and by the step itself, changed constants, a memory cap without room for the copy; against the
lane-group kernel (variant 1) from the same state, in mixed precision against a staged one (variant 6), which reads the
same FP32 packed coefficients (the lane groups form them from FP32 operators).

Tolerance: both kernels add the same bond forces P e (identical coefficients and displacements) in another order, so an
acceleration differs by at most (m + 8) eps sum |P| |e| / rho, m the family size (the sums of magnitudes are formed from the
operators here: the forces of a truncated family cancel far below them).  A difference d_n of the displacements grows
along the central difference as d_{n+1} <= (2 + k) d_n + d_{n-1} + dt^2 err + 3 eps |u|, k = dt^2 sum |P| / rho, evaluated
step by step.  Damage decisions are identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLICED = [17, 18, 19, 20]
EPS = np.finfo(np.float64).eps


def _mesh(dim, shape, seed=0):
    import perix_b200 as px
    rng = np.random.default_rng(seed)
    h = 1e-3
    q = np.indices(shape).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5 + rng.uniform(-0.2, 0.2, q.shape)) * h
    off, ids = px.families(x, 3.015 * h, dim == 3)
    return x, np.full(len(x), h ** dim), off, ids, h


def _setup(ctx, dim, shape, sc=4e-3, precision=0):
    import perix_b200 as px
    SHAPE[0] = shape
    x, vol, off, ids, h = _mesh(dim, shape)
    ctx.set_geometry(x, vol, off, ids, 3.015 * h, h, dim)
    C = px.elastic_constants(dim, False, 72e9, 0.22)
    rng = np.random.default_rng(5)
    health = (rng.uniform(size=int(off[-1])) > 0.1).astype(np.uint8)
    ctx.epf_setup(*C, 2440.0, sc=sc, tension_only=True, health0=health, precision=precision)
    ctx.epf_set_bcs([])
    u = (rng.standard_normal((len(x), dim)) * sc * h * 0.8).reshape(-1)
    return u, off, 0.5 * h / np.sqrt(C[0] / 2440.0), C


def _bound(ctx, u, off, dim, C, dt, steps):
    """(acceleration, displacement after `steps` steps) bounds for the state u, C scaled up to 1.5 and u doubled at most."""
    x, vol, off, ids, h = _mesh(dim, SHAPE[0])
    ctx.gbuild(2, 0)
    g = np.abs(ctx.get_ops())
    i = np.repeat(np.arange(len(off) - 1), np.diff(off))
    second = list(range(dim, g.shape[1]))
    P = 1.5 * (C[0] + C[1] + 2 * C[2]) * g[:, second].sum(1)  # above every row sum of |P|
    e = np.abs(u.reshape(-1, dim))
    de = 2.0 * (e[ids - 1] + e[i]).max(1)
    F, K = np.zeros(len(off) - 1), np.zeros(len(off) - 1)
    np.add.at(F, i, P * de)
    np.add.at(K, i, 2 * P)
    m = int(np.diff(off).max())
    err = (m + 8) * EPS * F.max() / 2440.0
    k = dt * dt * K.max() / 2440.0
    d, dp = 0.0, 0.5 * dt * dt * err
    for _ in range(steps):
        d, dp = (2 + k) * d + dp + dt * dt * err + 3 * EPS * 2 * e.max(), d
    return err, d


SHAPE = [None]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("variant", SLICED)
@pytest.mark.parametrize("dim,shape", [(2, (4, 8)), (2, (3, 11)), (2, (31, 1)), (2, (23, 29)), (3, (4, 4, 4)), (3, (5, 5, 5)),
                                       (3, (7, 6, 9))])
def test_sliced_steps_match_other_schedules(ctx, dim, shape, variant, precision):
    import perix_b200 as px
    try:
        u0, off, dt, C = _setup(ctx, dim, shape, precision=precision)
    except px.PxbError as e:
        assert e.status == 3  # a line of nodes cannot carry the operators
        return
    out = []
    for v in (6 if precision else 1, variant):
        _setup(ctx, dim, shape, precision=precision)
        ctx.epf_set_variant(v)
        ctx.epf_start(u0, None, dt)
        ctx.epf_advance(4)
        out.append(ctx.epf_state())
    (ua, pa, ha, ta), (ub, pb, hb, tb) = out
    assert np.array_equal(ha, hb) and ta == tb
    assert (ha == 0).any()
    assert np.abs(ua - ub).max() <= _bound(ctx, u0, off, dim, C, dt, 4)[1]


@pytest.mark.parametrize("dim,shape", [(2, (23, 29)), (3, (7, 6, 9))])
def test_words_follow_health_and_constants(ctx, dim, shape):
    """Everything that writes health or the coefficients between sliced launches: set_state, a snapshot restore, a step
    of another schedule, set_constants, and the per-step rate call."""
    u0, off, dt, C = _setup(ctx, dim, shape)
    nb = int(off[-1])
    kill = (np.random.default_rng(9).uniform(size=nb) > 0.5).astype(np.uint8)

    def script(variant, other):
        _setup(ctx, dim, shape)
        ctx.epf_set_variant(variant)
        ctx.epf_start(u0, None, dt)
        assert ctx.L.pxb_epf_snapshot(ctx.h) == 0
        seen = []

        def look():
            u, up, h, _ = ctx.epf_state()
            seen.append((u, h))
        ctx.epf_advance(2)
        look()
        u, up, h, t = ctx.epf_state()
        ctx.epf_set_state(u, up, h & kill, t)  # the caller breaks bonds
        ctx.epf_advance(2)
        look()
        ctx.epf_set_variant(other)  # another schedule breaks some
        ctx.epf_advance(2)
        ctx.epf_set_variant(variant)
        ctx.epf_advance(2)
        look()
        assert ctx.L.pxb_epf_restore(ctx.h) == 0  # bonds come back
        ctx.epf_advance(2)
        look()
        ctx.epf_set_constants(1.5 * C[0], 1.5 * C[1], 1.5 * C[2], 2440.0)
        ctx.epf_advance(2)
        look()
        a, nbk = ctx.epf_rate(2.0 * u0)
        _, _, h, _ = ctx.epf_state()
        seen.append((a, h))
        return seen, nbk

    ref, nref = script(1, 1)
    err, d = _bound(ctx, u0, off, dim, C, dt, 10)
    for v in SLICED:
        got, n = script(v, 2)
        assert n == nref
        for (ua, ha), (ub, hb) in zip(ref[:-1], got[:-1]):
            assert np.array_equal(ha, hb)
            assert np.abs(ua - ub).max() <= d
        (aa, ha), (ab, hb) = ref[-1], got[-1]
        assert np.array_equal(ha, hb)
        assert np.abs(aa - ab).max() <= err


def test_no_room_for_the_copy():
    import perix_b200 as px
    c = px.Context(0)
    try:
        u0, off, dt, _ = _setup(c, 3, (7, 6, 9))
        c.epf_start(u0, None, dt)
        c.set_memory_limit(c.device_bytes() + 4096)
        with pytest.raises(px.PxbError) as e:
            c.epf_set_variant(17)
        assert e.value.status == 4
        c.epf_advance(1)  # the schedule in effect goes on
        c.set_memory_limit(0)
        c.epf_set_variant(17)
        c.epf_advance(1)
    finally:
        c.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("keep", [0, 3])
@pytest.mark.parametrize("dim,shape", [(2, (4, 8)), (2, (23, 29)), (3, (5, 5, 5)), (3, (7, 6, 9))])
def test_sliced_adjoint_matches_reverse_only_kernel(ctx, dim, shape, keep, precision):
    """The reverse sweep on the slices (adjoint schedule 5) against the unstaged reverse-only kernel (1), with a health
    mask that differs between a bond and its reverse.  With k as in _bound but over the larger of the operators' row and
    column sums, the adjoint's magnitude and the difference of the two sweeps grow along the transposed central difference
    as M_{n+1} <= (2 + k) M_n + M_{n-1} and d_{n+1} <= (2 + k) d_n + d_{n-1} + (m + 10) eps (2 + k) M_n; dC adds one term a
    bond and step in trees of fewer than 256 levels."""
    import ctypes
    import torch
    steps = 7
    u0, off, dt, C = _setup(ctx, dim, shape, sc=0.0, precision=precision)
    x, vol, off, ids, h = _mesh(dim, shape)
    ctx.gbuild(2, 0)
    g = np.abs(ctx.get_ops())[:, dim:].sum(1)
    i = np.repeat(np.arange(len(off) - 1), np.diff(off))
    row, col = np.zeros(len(off) - 1), np.zeros(len(off) - 1)
    np.add.at(row, i, g)
    np.add.at(col, ids - 1, g)
    k = 2 * dt * dt * (C[0] + C[1] + 2 * C[2]) * max(row.max(), col.max()) / 2440.0
    dev = torch.device("cuda", 0)
    ctx.set_stream(torch.cuda.current_stream(dev).cuda_stream)
    rng = np.random.default_rng(3)
    u = torch.tensor(u0, device=dev)
    gN = torch.tensor(rng.standard_normal(u0.size), device=dev)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    out = []
    for v, schedule in ((6, 1), (17, 5)):
        ctx.epf_set_variant(6)
        assert ctx.L.pxb_epf_record_d(ctx.h, p(u), None, ctypes.c_double(dt), steps, keep, None, None) == 0
        ctx.epf_set_adjoint_schedule(schedule)
        ub, vb = torch.empty_like(u), torch.empty_like(u)
        dC = torch.zeros(3, dtype=torch.float64, device=dev)
        assert ctx.L.pxb_epf_adjoint_recorded_d(ctx.h, p(gN), None, p(ub), p(vb), p(dC)) == 0
        out.append((ub.cpu().numpy(), vb.cpu().numpy(), dC.cpu().numpy()))
    ctx.epf_set_adjoint_schedule(-1)
    ctx.set_stream(None)
    m = int(np.diff(off).max())
    M, Mp, d, dp = float(gN.abs().max()), 0.0, 0.0, 0.0
    terms, emax = 0.0, 2 * float(u.abs().max()) * (2 + k) ** steps
    for _ in range(steps + 1):
        terms += 4 * dim * dt * dt / 2440.0 * g.sum() * M * emax
        d, dp = (2 + k) * d + dp + (m + 10) * EPS * (2 + k) * M, d
        M, Mp = (2 + k) * M + Mp, M
    (ua, va, ca), (ub, vb, cb) = out
    assert np.abs(ua - ub).max() <= d and np.abs(va - vb).max() <= dt * d
    assert np.abs(ca - cb).max() <= 256 * EPS * terms + terms * d / M
    # and far closer than that in practice: the bounds above are for the worst case
    assert np.linalg.norm(ua - ub) <= 1e-10 * np.linalg.norm(ua)
    assert np.abs(ca - cb).max() <= 1e-9 * np.abs(ca).max()
