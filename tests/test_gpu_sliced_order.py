"""The sliced schedules' copy of health and constants where a program changes streams, or captures, between the calls that
write it and those that read it.  Each result is compared with the lane-group kernel (variant 1) on the same state, which
reads the health bytes and the operators themselves.

Tolerance: both kernels add the same bond forces in another order, at most (m + 8) eps sum |P| |e| / rho apart, m the family
size; a wrong mask or coefficient moves an acceleration by whole bond forces."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
H, RHO = 1e-3, 2440.0


class Case:
    def __init__(self, dim, shape):
        self.torch = pytest.importorskip("torch")
        rng = np.random.default_rng(sum(shape))
        q = np.indices(shape).reshape(dim, -1)[::-1].T.astype(np.float64)
        x = np.zeros((len(q), 3))
        x[:, :dim] = (q + 0.5 + rng.uniform(-0.2, 0.2, q.shape)) * H
        off, ids = px.families(x, 3.015 * H, dim == 3)
        self.C = px.elastic_constants(dim, False, 72e9, 0.22)
        self.nb, self.dim, self.n = int(off[-1]), dim, len(x)
        self.masks = [(rng.uniform(size=self.nb) > f).astype(np.uint8) for f in (0.1, 0.6)]
        self.u = self.torch.tensor((rng.standard_normal(len(x) * dim) * 4e-6), device="cuda")
        self.ctxs = []
        for variant in (1, 17):
            c = px.Context(0)
            c.set_geometry(x, np.full(len(x), H ** dim), off, ids, 3.015 * H, H, dim)
            c.epf_setup(*self.C, RHO, sc=4e-3, tension_only=True, health0=self.masks[0])
            c.epf_set_bcs([])
            c.epf_set_variant(variant)
            self.ctxs.append(c)
        c = self.ctxs[0]
        c.gbuild(2, 0)
        g = np.abs(c.get_ops())[:, dim:].sum(1)
        i = np.repeat(np.arange(len(off) - 1), np.diff(off))
        F = np.zeros(len(x))
        np.add.at(F, i, 1.5 * (self.C[0] + self.C[1] + 2 * self.C[2]) * g * 2 * float(self.u.abs().max()))
        self.tol = (int(np.diff(off).max()) + 8) * EPS * F.max() / RHO
        self.torch.cuda.synchronize()

    def state(self, c, mask):
        z = np.zeros(self.n * self.dim)
        c.epf_set_state(z, z, self.masks[mask], 0.0)

    def force(self, c, out=None):
        a = self.torch.empty_like(self.u) if out is None else out
        c.epf_force_frozen_d(self.u.data_ptr(), a.data_ptr())
        return a

    def close_to(self, a, b):
        assert float((a - b).abs().max()) <= self.tol

    def reference(self, mask, scale=1.0):
        c = self.ctxs[0]
        self.state(c, mask)
        c.epf_set_constants(*[scale * v for v in self.C], RHO)
        a = self.force(c)
        c.synchronize()
        return a


SHAPES = [(2, (23, 29)), (3, (7, 6, 9))]


@pytest.mark.parametrize("dim,shape", SHAPES)
def test_captured_force_follows_health(dim, shape):
    k = Case(dim, shape)
    torch, c = k.torch, k.ctxs[1]
    ref = [k.reference(0), k.reference(1)]
    assert float((ref[0] - ref[1]).abs().max()) > 1e6 * k.tol
    k.force(c)
    c.synchronize()
    out = torch.empty_like(k.u)
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        c.set_stream(s.cuda_stream)
        k.force(c, out)
    for mask in (1, 0, 1):
        k.state(c, mask)
        graph.replay()
        torch.cuda.synchronize()
        k.close_to(out, ref[mask])
    k.state(c, 0)
    k.force(c, out)  # and uncaptured calls go on as before
    c.synchronize()
    k.close_to(out, ref[0])
    c.set_stream(None)


@pytest.mark.parametrize("legacy", [False, True])
@pytest.mark.parametrize("dim,shape", SHAPES)
def test_force_on_another_stream_waits_for_the_refresh(dim, shape, legacy):
    """The words are refreshed by a call on one stream, late; a call on another stream needs them, and the constants that a
    third one writes.  The late stream is torch's default (the legacy) one or another."""
    k = Case(dim, shape)
    torch, c = k.torch, k.ctxs[1]
    ref = [k.reference(0), k.reference(1), k.reference(1, 1.5)]
    a, b = torch.cuda.default_stream() if legacy else torch.cuda.Stream(), torch.cuda.Stream()
    outs = [torch.empty_like(k.u) for _ in range(5)]
    torch.cuda.synchronize()
    late = lambda s: torch.cuda._sleep(20_000_000)  # noqa: E731
    k.force(c, outs[0])
    c.synchronize()
    k.close_to(outs[0], ref[0])
    k.state(c, 1)
    c.set_stream(a.cuda_stream)
    with torch.cuda.stream(a):
        late(a)
    k.force(c, outs[1])  # refreshes the words, once the stream gets there
    c.set_stream(b.cuda_stream)
    k.force(c, outs[2])
    c.set_stream(a.cuda_stream)
    with torch.cuda.stream(a):
        late(a)
    c.epf_set_constants(*[1.5 * v for v in k.C], RHO)
    c.set_stream(b.cuda_stream)
    k.force(c, outs[3])
    with torch.cuda.stream(b):
        late(b)
    k.force(c, outs[4])  # reads coefficients that the next call may write
    c.set_stream(a.cuda_stream)
    c.epf_set_constants(*k.C, RHO)
    k.force(c, outs[0])
    torch.cuda.synchronize()
    for o, r in zip(outs, (ref[1], ref[1], ref[1], ref[2], ref[2])):
        k.close_to(o, r)
    c.set_stream(None)


@pytest.mark.parametrize("dim,shape", SHAPES)
def test_recording_and_sweep_on_changing_streams(dim, shape):
    """Recordings and reverse sweeps on two streams in turn, the first of each pair late, give what one stream gives: the
    same kernels on the same values, but for dC, whose blocks are added in any order."""
    import ctypes as C
    k = Case(dim, shape)
    torch, c = k.torch, k.ctxs[1]
    g = torch.randn_like(k.u)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    dt = 0.4 * H / np.sqrt(k.C[0] / RHO)
    got = []
    for order in ((0, 0), (0, 1), (1, 0), (1, 1)):
        uN, ub, vb = (torch.empty_like(k.u) for _ in range(3))
        dC = torch.zeros(3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        c.set_stream(s[order[0]].cuda_stream)
        with torch.cuda.stream(s[order[0]]):
            torch.cuda._sleep(20_000_000)
        assert c.L.pxb_epf_record_d(c.h, p(k.u), None, C.c_double(dt), 6, 4, p(uN), None) == 0
        c.set_stream(s[order[1]].cuda_stream)
        assert c.L.pxb_epf_adjoint_recorded_d(c.h, p(g), None, p(ub), p(vb), p(dC)) == 0
        torch.cuda.synchronize()
        got.append((uN, ub, vb, dC))
    for o in got[1:]:
        for x, y in zip(o[:3], got[0]):
            assert torch.equal(x, y)
        assert float((o[3] - got[0][3]).abs().max()) <= 1e-9 * float(got[0][3].abs().max())
    c.set_stream(None)
