"""Families built on the device against the host build, entry for entry: cells with few members (candidates laid end to
end), with more than 16 and with more than a warp's 32 (one by one), nodes with more passes than votes are kept for
(about 45 members a cell in 3D), empty cells and nodes without partners, node counts that are no multiple of a warp's
run.  Built twice on one context, the second time from the first build's released buffers, with another size between."""
import numpy as np
import pytest

import perix_b200 as px

pytestmark = pytest.mark.gpu


def _cloud(dim, n, per_cell, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, 3))
    x[:, :dim] = rng.uniform(-0.3, 0.7, (n, dim))
    if n > 40:
        x[n // 2] = x[n // 3]                # two nodes in one place
        x[n - 1, :dim] = 9.0                 # and one on its own, beyond empty cells
    return x, (per_cell / n) ** (1.0 / dim)


@pytest.mark.parametrize("dim,n,per_cell", [(3, 2003, 45), (3, 3001, 27), (3, 1501, 4), (2, 1999, 55), (2, 1203, 20),
                                            (2, 1001, 9), (2, 502, 2), (3, 1, 4), (2, 2, 1), (3, 5, 5), (2, 33, 33)])
def test_device_families_match_host(dim, n, per_cell):
    c = px.Context(0)
    for k, m in enumerate((n, max(1, n // 2), n)):
        x, radius = _cloud(dim, m, min(per_cell, m), 10 * n + k)
        off, ids = px.families(x, radius, dim == 3)
        if off[-1] == 0:
            continue
        c.set_geometry_points(x, np.full(m, 1.0 / m), radius, radius, radius / 3.0, dim)
        off_d, ids_d = c.get_families()
        assert np.array_equal(off, off_d) and np.array_equal(ids, ids_d)


def test_released_buffers_stay_within_the_limit():
    """Idle blocks do not count as held, and give way when the context's limit leaves no room for them."""
    x, radius = _cloud(3, 20011, 27, 3)
    y, ry = _cloud(3, 5003, 27, 4)
    c = px.Context(0)
    args = lambda p, r: (p, np.full(len(p), 1.0 / len(p)), r, r, r / 3.0, 3)  # noqa: E731
    c.set_geometry_points(*args(x, radius))
    c.gbuild(2, px.FP64, allow_degenerate=True)
    held = c.device_bytes()
    c.set_geometry_points(*args(y, ry))
    c.gbuild(2, px.FP64, allow_degenerate=True)
    assert c.device_bytes() < held / 2
    # each array fits beside what is held, none beside what is held and idle
    c.set_memory_limit(held)
    c.set_geometry_points(*args(y, ry))
    c.gbuild(2, px.FP64, allow_degenerate=True)
    ops = c.get_ops()
    c.set_memory_limit(c.device_bytes() // 2)
    with pytest.raises(px.api.PxbError) as e:
        c.gbuild(3, px.FP64, allow_degenerate=True)
    assert e.value.status == 2 or "limit" in str(e.value)
    c.set_memory_limit(0)
    c.gbuild(2, px.FP64, allow_degenerate=True)
    assert np.array_equal(ops, c.get_ops())
