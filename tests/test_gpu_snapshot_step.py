"""A saved explicit state includes the length of its last step, which the variable-step form of the next one needs: after a
clamped step, the autotuner (which runs steps of its own) and a restored snapshot leave the run where it was, bit for bit."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _context(dim, m):
    h = 1.0 / m
    q = np.indices((m,) * dim).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5) * h
    delta = 3.015 * h * (1 + 1e-6)
    off, ids = px.families(x, delta, dim == 3)
    c = px.Context(0)
    c.set_geometry(x, np.full(len(x), h ** dim), off, ids, delta, h, dim)
    C = px.elastic_constants(dim, False, 72e9, 0.22)
    c.epf_setup(*C, 2440.0, sc=4e-3, tension_only=True)
    c.epf_set_bcs([])
    return c, np.random.default_rng(m).standard_normal(len(x) * dim) * 1e-3 * h, 0.4 * h / np.sqrt(C[0] / 2440.0)


@pytest.mark.parametrize("dim,m", [(2, 30), (3, 9)])
@pytest.mark.parametrize("first,second", [(5.5, 12.0), (5.0, 9.25)])
def test_step_length_survives(dim, m, first, second):
    ends = []
    for what in ("run", "tuned", "restored"):
        c, u0, dt = _context(dim, m)
        c.epf_start(u0, None, dt)
        c.epf_advance_to(first * dt)
        if what == "tuned":
            c.epf_autotune(steps=3, use_cache=False)
            c.epf_set_variant(1)
        if what == "restored":
            assert c.L.pxb_epf_snapshot(c.h) == 0
            c.epf_advance_to((first + 2.75) * dt)
            assert c.L.pxb_epf_restore(c.h) == 0
        c.epf_advance_to(second * dt)
        ends.append(c.epf_state())
    for u, up, h, t in ends[1:]:
        assert t == ends[0][3] and np.array_equal(h, ends[0][2])
        assert np.array_equal(u, ends[0][0]) and np.array_equal(up, ends[0][1])
