"""Set-up calls that give no stream-ordered result leave nothing queued behind them: a program may put the context on
another stream straight after them (the autograd wrappers do at every call)."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _lattice(dim, m):
    h = 1.0 / m
    q = np.indices((m,) * dim).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5) * h
    return x, np.full(len(x), h ** dim), 3.015 * h * (1 + 1e-6), h


def _on(ctx, stream):
    ctx.set_stream(stream.cuda_stream)


@pytest.mark.parametrize("dim,m,ndof", [(2, 700, 1), (2, 400, 2), (3, 44, 1), (3, 32, 3)])
def test_built_pattern_is_there(dim, m, ndof):
    """Sizes whose last kernel runs for 30 us and more."""
    torch = pytest.importorskip("torch")
    x, vol, delta, h = _lattice(dim, m)
    c = px.Context(0)
    s = torch.cuda.Stream()
    _on(c, s)
    c.set_geometry_points(x, vol, delta, delta, h, dim)
    for _ in range(3):
        nnz = c.csr_build_pattern(ndof)
        assert s.query()
    assert nnz >= ndof * ndof * (c.nb + len(x))


@pytest.mark.parametrize("dim,shape", [(2, 300), (3, 36)])
@pytest.mark.parametrize("variant", [17, 20])
def test_selected_schedule_is_there(dim, shape, variant):
    """set_variant of a schedule with streams of its own, and both autotuners answering from their cache."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    x, vol, delta, h = _lattice(dim, shape)
    s = torch.cuda.Stream()
    u = np.zeros(len(x) * dim)
    for k in range(2):  # the second context takes the first one's choice
        c = px.Context(0)
        _on(c, s)
        c.set_geometry_points(x, vol, delta, delta, h, dim)
        c.epf_setup(*px.elastic_constants(dim, False, 72e9, 0.22), 2440.0, sc=0.01, tension_only=True)
        c.epf_set_bcs([])
        c.epf_start(u, None, 1e-9)
        c.epf_set_variant(variant)
        assert s.query()
        c.epf_set_variant(1)
        c.epf_autotune(steps=4, use_cache=True)
        assert s.query()
        assert c.L.pxb_epf_autotune_rate(c.h, u.ctypes.data_as(C.c_void_p), 2, 1, None, None) == 0
        assert s.query()
