"""The sliced step's clear-hold test (k_epf_sliced.cu): a bond of length class q = floor(|xi| / step (1 - 1e-9)) is taken as
holding without its positions being read when |e|^2 < ((s_c (1 - 1e-6) - 1e-12) step)^2 q^2.  Since q step <= |xi|, its stretch
is at most |e| / |xi| < s_c.  This checks, in the kernels' arithmetic, that no class exceeds its bond's length and that no
bond the test clears breaks under the reference's FP64 stretch (ExplicitPDDOFracElement.cpp:239-266), for every class width
the ids leave, lattice and random bonds, and displacements at the bound along and against the bond.  Host arithmetic."""
import numpy as np
import pytest

from test_epf_clear_bound import _bonds, _kernel_e2, _ref_stretch


@pytest.mark.parametrize("qbits", [0, 1, 3, 7])
def test_length_classes_never_clear_a_breaking_bond(qbits):
    rng = np.random.default_rng(31)
    for sc in (1e-6, 1e-4, 4e-3, 0.1, 0.5):
        xi = _bonds(rng, 1e-3, 20000)
        r2 = xi[:, 0] * xi[:, 0] + xi[:, 1] * xi[:, 1] + xi[:, 2] * xi[:, 2]
        r = np.sqrt(r2)
        step = np.sqrt(r2.max()) / (1 << qbits)
        q = np.minimum((1 << qbits) - 1, (r * (1.0 / step) * (1.0 - 1.0e-9)).astype(np.int64))
        assert (q * step <= r).all()
        m = sc * (1.0 - 1.0e-6) - 1.0e-12
        clear = (m * m * step * step if m > 0 else 0.0) * (q * q).astype(np.float64)
        unit = xi / r[:, None]
        for direction in (unit, -unit, rng.standard_normal(xi.shape)):
            d = direction / np.linalg.norm(direction, axis=1)[:, None]
            for f in (0.5, 1.0 - 1e-9, 1.0, 1.0 + 1e-9):
                e = d * (np.sqrt(clear) * f)[:, None]
                cleared = _kernel_e2(e) < clear
                s = _ref_stretch(xi, e)
                assert not (cleared & (np.abs(s) > sc)).any()
        assert qbits < 7 or (q[r > 0.99e-3] > 0).all()  # with seven bits a lattice's shortest bond has a class
