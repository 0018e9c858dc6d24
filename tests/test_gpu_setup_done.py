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
