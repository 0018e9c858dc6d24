"""The default reverse sweep on both sides of the 3D size below which it is the staged one (4,736 nodes), against the
unstaged reverse-only kernel (schedule 1).  Bounds as for the sliced sweep on small meshes: the two differ by the order of
their sums, far below 1e-10 of the gradients after eight steps."""
import ctypes as C

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,sliced", [((15, 17, 18), False), ((16, 16, 18), False), ((16, 16, 19), True), ((17, 18, 18), True)])
def test_default_sweep_around_the_line(shape, sliced):
    torch = pytest.importorskip("torch")
    h = 1e-3
    q = np.indices(shape).reshape(3, -1)[::-1].T.astype(np.float64)
    rng = np.random.default_rng(sum(shape))
    x = (q + 0.5 + rng.uniform(-0.1, 0.1, q.shape)) * h
    n = len(x)
    assert (n >= 4736) == sliced
    c = px.Context(0)
    c.set_geometry_points(x, np.full(n, h ** 3), 3.015 * h, 3.015 * h, h, 3)
    Cs = px.elastic_constants(3, False, 72e9, 0.22)
    c.epf_setup(*Cs, 2440.0, sc=0.0, tension_only=True, health0=(rng.uniform(size=c.nb) > 0.05).astype(np.uint8))
    c.epf_set_bcs([])
    dt = C.c_double(0.4 * h / np.sqrt(Cs[0] / 2440.0))
    u = torch.tensor(rng.standard_normal(3 * n) * 1e-6, device="cuda")
    g = torch.tensor(rng.standard_normal(3 * n), device="cuda")
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert c.L.pxb_epf_record_d(c.h, p(u), None, dt, 8, 0, None, None) == 0
    out = []
    for schedule in (1, -1):
        c.epf_set_adjoint_schedule(schedule)
        held = c.device_bytes()
        ub, dC = torch.empty_like(u), torch.zeros(3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert c.L.pxb_epf_adjoint_recorded_d(c.h, p(g), None, p(ub), None, p(dC)) == 0
        c.synchronize()
        out.append((ub.cpu().numpy(), dC.cpu().numpy()))
    assert (c.device_bytes() - held > 52 * c.nb) == sliced  # the sliced sweep's own operators
    (ua, ca), (ub, cb) = out
    assert np.linalg.norm(ua - ub) <= 1e-10 * np.linalg.norm(ua)
    assert np.abs(ca - cb).max() <= 1e-9 * np.abs(ca).max()
