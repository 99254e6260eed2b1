"""Row kernels at the products per row where a row takes a larger CTA."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_row_kernels import check_product

pytestmark = pytest.mark.gpu


def _constant(rng, rows, cols, per, hi):
    """`per` entries in every row, at distinct columns."""
    start, step = rng.integers(0, cols, (rows, 1)), 1 + 2 * rng.integers(0, 3, (rows, 1))
    col = np.sort((start + step * np.arange(per)) % cols, axis=1)
    return sp.csr_matrix((rng.integers(1, hi, col.size, dtype=np.uint64), col.reshape(-1),
                          np.arange(rows + 1) * per), shape=(rows, cols))


# 64 x 768 and 256 x 1,024 products a row, and one position of B less; rows
# enough for the smaller CTAs they would take otherwise.  (Widths prime to the
# steps of 1, 3 and 5.)
@pytest.mark.parametrize("rows,a,b", [(1300, 64, 768), (1300, 64, 767), (700, 256, 1024), (700, 256, 1023),
                                      (320, 256, 1024)])
@pytest.mark.parametrize("n", [1501, 5003])
@pytest.mark.parametrize("vt,bhi", [("VAL_U32", 9), ("VAL_U32", 2 ** 23), ("VAL_U64", 9)])
def test_rows_of_many_products(native, engine, vt, bhi, n, rows, a, b):
    rng = np.random.default_rng(n + b)
    A = _constant(rng, rows, 311, a, 2 if bhi > 9 else 9)
    B = _constant(rng, 311, n, b, 9)
    B.data[::4096] = bhi - 1      # 2^23: too wide to pack, and 256 of them in a count stay below 2^32
    check_product(native, engine, A, B, getattr(native, vt))
