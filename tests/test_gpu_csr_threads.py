"""Assemblies of two contexts in two host threads whose longest families need different amounts of shared memory, both
above the 48 KB that a kernel may use unasked: every launch of each succeeds and gives its context's values."""
import threading

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
PRM = dict(C11=1.35, C12=0.58, C66=0.385, A=0.3, Kh=0.9, Ch=-0.25, Omega=0.06, cref=0.5, chi=2.5, kappa=1e-4, dt=1e-4,
           kres=1e-6, rho=0.0)


def _context(torch, horizon, m=30):
    h = 1.0 / m
    q = np.indices((m, m)).reshape(2, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :2] = (q + 0.5) * h
    c = px.Context(0)
    c.set_geometry_points(x, np.full(len(x), h * h), horizon * h, horizon * h, h, 2)
    c.gbuild(2, px.FP64)
    c.ch_build_geometry()
    nnz = c.csr_build_pattern(4)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(horizon * 10))
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    u = 0.4 + 0.2 * rnd(len(x), 4)
    mob = u[:, 0] * (1 - u[:, 0])
    torch.cuda.synchronize()
    return c, u, u * 0.99, mob.contiguous(), torch.zeros(nnz, dtype=torch.float64, device="cuda"), torch.zeros_like(u)


def test_two_threads_with_different_families():
    torch = pytest.importorskip("torch")
    cases = [_context(torch, 5.2), _context(torch, 8.4)]  # about 84 and 220 blocks a row at most
    torch.cuda.synchronize()

    def assemble(k):
        c, u, uold, mob, kv, rhs = cases[k]
        c.assemble_stress_ch_d(PRM, mob.data_ptr(), u.data_ptr(), uold.data_ptr(), kv.data_ptr(), rhs.data_ptr())

    refs = []
    for k, (c, _, _, _, kv, rhs) in enumerate(cases):
        assemble(k)
        c.synchronize()
        refs.append((kv.clone(), rhs.clone()))
    torch.cuda.synchronize()
    errors = []

    def loop(k):
        try:
            for _ in range(2000):
                assemble(k)
            cases[k][0].synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (_, _, _, _, kv, rhs), (a, b) in zip(cases, refs):
        assert torch.equal(kv, a) and torch.equal(rhs, b)
