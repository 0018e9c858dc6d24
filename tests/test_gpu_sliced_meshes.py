"""Of the meshes that the sliced schedules are compared on, the line of nodes alone cannot carry the operators: the others
must not be refused as degenerate (the comparison passes over a refused mesh)."""
import pytest

import perix_b200 as px
from test_gpu_sliced import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [px.FP64, px.MIXED])
@pytest.mark.parametrize("dim,shape", [(2, (4, 8)), (2, (3, 11)), (2, (31, 1)), (2, (23, 29)), (3, (4, 4, 4)), (3, (5, 5, 5)),
                                       (3, (7, 6, 9))])
def test_only_the_line_is_degenerate(ctx, dim, shape, precision):
    if shape == (31, 1):
        with pytest.raises(px.PxbError) as e:
            _setup(ctx, dim, shape, precision=precision)
        assert e.value.status == 3
    else:
        _setup(ctx, dim, shape, precision=precision)
