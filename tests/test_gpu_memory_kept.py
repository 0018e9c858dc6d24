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
