"""The per-step rate call on page-locked buffers of more than 4 MB with a schedule that does not write to the host itself
(the copy engines carry them), just below and above that size, against the same call on pageable buffers: the same kernel on
the same state, so every value and count is equal, first call and replays."""
import ctypes as C

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
H = 1e-3


@pytest.mark.parametrize("m,above", [((511, 512), False), ((512, 513), True)])
@pytest.mark.parametrize("variant", [1, 17])
def test_large_pinned_rate_equals_pageable(m, above, variant):
    torch = pytest.importorskip("torch")
    q = np.indices(m).reshape(2, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :2] = (q + 0.5) * H
    n = len(x)
    assert (16 * n > 4 << 20) == above
    ctxs = []
    for _ in range(2):
        c = px.Context(0)
        c.set_geometry_points(x, np.full(n, H * H), 3.015 * H, 3.015 * H, H, 2)
        c.epf_setup(*px.elastic_constants(2, False, 72e9, 0.22), 2440.0, sc=4e-3, tension_only=True)
        c.epf_set_bcs([])
        assert c.L.pxb_epf_set_rate_chunks(c.h, 1) == 0
        c.epf_set_variant(variant)
        ctxs.append(c)
    plain, pinned = ctxs
    u = torch.empty(2 * n, dtype=torch.float64).pin_memory()
    a = torch.zeros(2 * n, dtype=torch.float64).pin_memory()
    rng = np.random.default_rng(n)
    for call in range(3):
        w = rng.standard_normal(2 * n) * H * (1e-3 if call < 2 else 4e-3)
        u.copy_(torch.from_numpy(w))
        nb = C.c_longlong(-1)
        p = lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_double))  # noqa: E731
        assert pinned.L.pxb_epf_rate(pinned.h, p(u), p(a), C.byref(nb)) == 0
        ref, broken = plain.epf_rate(w)
        assert np.array_equal(a.numpy(), ref) and nb.value == broken
