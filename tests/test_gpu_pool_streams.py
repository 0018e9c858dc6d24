"""The set-up buffers that a context keeps, where other streams and threads are at work: a capture that another thread has
under way, and work that still runs on a stream that the context has left."""
import threading

import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _cloud(n, dim, seed):
    rng = np.random.default_rng(seed)
    m = int(round(n ** (1.0 / dim)))
    q = np.indices((m,) * dim).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5 + rng.uniform(-0.2, 0.2, q.shape)) / m
    return x, np.full(len(x), 1.0 / len(x)), 3.015 / m, 1.0 / m


def _set_up(c, mesh, dim):
    x, vol, delta, h = mesh
    c.set_geometry_points(x, vol, delta, delta, h, dim)
    c.gbuild(2, px.FP64)
    return c.csr_build_pattern(1)


def test_set_up_leaves_another_threads_capture_alone():
    torch = pytest.importorskip("torch")
    mesh = _cloud(4000, 2, 1)
    c = px.Context(0)
    _set_up(c, mesh, 2)
    x = torch.ones(1000, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    failed = []

    def work():
        try:
            for _ in range(3):
                _set_up(c, mesh, 2)
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        y += x
        t = threading.Thread(target=work)
        t.start()
        t.join()
        y += x
    graph.replay()
    torch.cuda.synchronize()
    assert not failed and float(y.sum()) == 2000.0


def test_blocks_in_use_on_a_left_stream_are_not_taken():
    """An assembly waits on a stream that the context leaves; the next mesh is set up meanwhile, twice."""
    torch = pytest.importorskip("torch")
    mesh, other = _cloud(4000, 2, 1), _cloud(4000, 2, 2)
    c = px.Context(0)
    nnz = _set_up(c, mesh, 2)
    n = len(mesh[0])
    u = torch.sin(torch.arange(n, dtype=torch.float64, device="cuda"))
    kv = [torch.zeros(nnz, dtype=torch.float64, device="cuda") for _ in range(2)]
    rhs = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    import ctypes as C
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def assemble(k):
        assert c.L.pxb_assemble_scalar_d(c.h, 0, C.c_double(0.7), C.c_double(0.0), None, C.c_double(0.0), p(u), None,
                                         p(kv[k]), p(rhs[k])) == 0

    assemble(0)
    c.synchronize()
    c.set_stream(a.cuda_stream)
    with torch.cuda.stream(a):
        torch.cuda._sleep(40_000_000)
    assemble(1)
    c.set_stream(b.cuda_stream)
    for _ in range(2):
        _set_up(c, other, 2)
    torch.cuda.synchronize()
    assert torch.equal(kv[0], kv[1]) and torch.equal(rhs[0], rhs[1])
    c.set_stream(None)
