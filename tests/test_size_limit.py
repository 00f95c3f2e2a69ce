"""Grids whose arrays the kernels' 32-bit byte offsets cannot address are refused before anything is allocated, with
or without a GPU."""
import pytest

from qasmhd_b200 import lib as L

FLAGS = (0,) * 8


@pytest.mark.parametrize("dim,n", [(1, ((1 << 29) - 8, 1, 1)), (2, (1 << 15, 1 << 14, 1)), (3, (1 << 10, 1 << 10, 1 << 9)),
                                   (1, ((1 << 31) - 1, 1, 1)), (3, ((1 << 31) - 1,) * 3)], ids=str)
def test_refused_before_allocation(dim, n):
    with pytest.raises(L.QasError) as e:
        L.Context(dim, *n, 1.0, 1.0, 1.0, 5.0 / 3.0, 1, 4, 3, 1, FLAGS, FLAGS, FLAGS)
    assert e.value.status == L.QAS_ERR_NOMEM
