"""What a context keeps beyond what its calls asked for: counted where a limit is watched, and given back on request."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _mesh(m, dim=2):
    q = np.indices((m,) * dim).reshape(dim, -1)[::-1].T.astype(np.float64)
    x = np.zeros((len(q), 3))
    x[:, :dim] = (q + 0.5) / m
    return x, np.full(len(x), 1.0 / len(x)), 3.015 / m * (1 + 1e-6), 1.0 / m


def _set_up(c, m, dim=2):
    x, vol, delta, h = _mesh(m, dim)
    c.set_geometry_points(x, vol, delta, delta, h, dim)
    c.gbuild(2, px.FP64)
    c.csr_build_pattern(1)


def test_reused_blocks_count_whole():
    """A mesh set up in the blocks of a slightly larger one holds those blocks; under a limit it takes none that is larger
    than what it needs, and holds what a new context under that limit holds (which takes blocks of its own temporaries)."""
    fresh, again, capped = px.Context(0), px.Context(0), px.Context(0)
    fresh.set_memory_limit(1 << 30)
    _set_up(fresh, 190)
    _set_up(again, 200)
    _set_up(again, 190)
    assert again.device_bytes() > fresh.device_bytes()
    _set_up(capped, 200)
    capped.set_memory_limit(1 << 30)
    _set_up(capped, 190)
    assert capped.device_bytes() == fresh.device_bytes()


def test_idle_blocks_are_given_back():
    torch = pytest.importorskip("torch")
    c = px.Context(0)
    _set_up(c, 400)
    _set_up(c, 20)
    c.synchronize()
    before = torch.cuda.mem_get_info()[0]
    c.set_memory_limit(0)
    assert torch.cuda.mem_get_info()[0] - before >= 64 << 20  # 160,000 nodes' operators alone are 170 MB
    _set_up(c, 400)


def _explicit(m=24):
    x, vol, delta, h = _mesh(m, 3)
    c = px.Context(0)
    c.set_geometry_points(x, vol, delta, delta, h, 3)
    C = px.elastic_constants(3, False, 72e9, 0.22)
    c.epf_setup(*C, 2440.0, sc=0.0, tension_only=True)
    c.epf_set_bcs([])
    return c, len(x), 0.4 * h / np.sqrt(C[0] / 2440.0)


def test_slices_are_kept_only_while_they_are_used():
    c, n, dt = _explicit(12)
    c.epf_start(np.zeros(3 * n), None, dt)
    before = c.device_bytes()
    c.epf_set_variant(18)
    c.epf_advance(3)
    assert c.device_bytes() > before + 50 * c.nb
    c.epf_set_variant(6)
    assert c.device_bytes() < before + c.nb
    c.epf_advance(3)
    c.epf_autotune(steps=4)
    held = c.device_bytes() - before
    assert held > 50 * c.nb if c.epf_variant()[0] >= 17 else held < c.nb


def test_slices_give_way_to_a_recording():
    """Every state of a recording fits under the limit without the slices, not beside them: the recording is made, by the
    schedule that was current before, and the sweep goes on from it."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    steps = 40
    u = None
    got = []
    for variant in (6, 17):
        c, n, dt = _explicit()
        if u is None:
            u = torch.tensor(np.random.default_rng(2).standard_normal(3 * n) * 1e-6, device="cuda")
            g = torch.randn_like(u)
            torch.cuda.synchronize()
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        c.epf_set_variant(6)
        limit = c.device_bytes() + 8 * 3 * n * (steps + 8) + (1 << 20)  # the states, the loop's vectors and times
        c.epf_set_variant(variant)
        assert c.epf_variant()[0] == variant
        c.set_memory_limit(limit)
        uN, ub = torch.empty_like(u), torch.empty_like(u)
        assert c.L.pxb_epf_record_d(c.h, p(u), None, C.c_double(dt), steps, 0, p(uN), None) == 0
        assert c.epf_variant()[0] == 6
        c.set_memory_limit(0)
        assert c.L.pxb_epf_adjoint_recorded_d(c.h, p(g), None, p(ub), None, None) == 0
        c.synchronize()
        got.append((uN, ub))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_pattern_temporaries_make_room():
    """A limit that holds the built pattern and its value buffers, but not the build's temporaries beside them."""
    c = px.Context(0)
    _set_up(c, 120)
    rows, cols = c.csr_get_pattern()
    held = c.device_bytes()
    x, vol, delta, h = _mesh(120)
    d = px.Context(0)
    d.set_geometry_points(x, vol, delta, delta, h, 2)
    d.gbuild(2, px.FP64)
    d.set_memory_limit(held + 4096)  # the build's lists take 4 bytes a bond more
    assert d.csr_build_pattern(1) == cols.size
    r, k = d.csr_get_pattern()
    assert np.array_equal(r, rows) and np.array_equal(k, cols)
