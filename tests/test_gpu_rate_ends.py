"""The per-step rate call on page-locked buffers, whose ends are read and written by the GPU in the host's memory, against
the same call on pageable ones: the same kernel on the same state, so every value and count is equal.

16-byte aligned buffers and buffers 8 bytes off, odd and even numbers of values, node counts around a slice and a block,
sliced and other schedules; the buffers' contents change between calls, the first of which is queued, the later ones
replayed; guard values around the result stay as they are."""
import ctypes as C

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
H = 1e-3


def _context(dim, shape, variant, precision):
    rng = np.random.default_rng(sum(shape))
    q = np.indices(shape).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5 + rng.uniform(-0.2, 0.2, q.shape)) * H
    off, ids = px.families(x, 3.015 * H, dim == 3)
    c = px.Context(0)
    c.set_geometry(x, np.full(len(x), H ** dim), off, ids, 3.015 * H, H, dim)
    c.epf_setup(*px.elastic_constants(dim, False, 72e9, 0.22), 2440.0, sc=4e-3, tension_only=True, precision=precision)
    c.epf_set_bcs([])
    c.epf_set_variant(variant)
    return c, len(x) * dim


@pytest.mark.parametrize("precision", [px.FP64, px.MIXED])
@pytest.mark.parametrize("variant", [1, 6, 17, 20])
@pytest.mark.parametrize("dim,shape", [(2, (11, 9)), (2, (32, 31)), (3, (7, 7, 7)), (3, (8, 9, 7)), (2, (70, 67))])
def test_rate_on_pinned_buffers_equals_pageable(dim, shape, variant, precision):
    torch = pytest.importorskip("torch")
    for shift in (0, 1):
        plain, nd = _context(dim, shape, variant, precision)
        pinned, _ = _context(dim, shape, variant, precision)
        u = torch.empty(nd + 4, dtype=torch.float64).pin_memory()
        a = torch.full((nd + 4,), 7.25, dtype=torch.float64).pin_memory()
        rng = np.random.default_rng(nd)
        for call in range(4):
            w = rng.standard_normal(nd) * H * (1e-3 if call < 3 else 4e-3)
            u[shift:shift + nd] = torch.from_numpy(w)
            nb = C.c_longlong(-1)
            ptr = lambda t: C.cast(t.data_ptr() + 8 * shift, C.POINTER(C.c_double))  # noqa: E731
            st = pinned.L.pxb_epf_rate(pinned.h, ptr(u), ptr(a), C.byref(nb))
            assert st == 0
            ref, broken = plain.epf_rate(w)
            assert np.array_equal(a[shift:shift + nd].numpy(), ref) and nb.value == broken
            assert (a[:shift] == 7.25).all() and (a[shift + nd:] == 7.25).all()
