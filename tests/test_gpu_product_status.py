"""What a product leaves behind when counts overflow, and when its call is done."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _upload(eng, M, vt):
    M = M.tocsr()
    M.sort_indices()
    return eng.upload(M.indptr, M.indices, cols=M.shape[1], val=M.data.astype(np.uint64), valtype=vt)


def _rows(lists, cols):
    """CSR of (columns, values) per row."""
    rp = np.concatenate([[0], np.cumsum([len(c) for c, _ in lists])])
    return sp.csr_matrix((np.concatenate([np.asarray(v, np.uint64) for _, v in lists]),
                          np.concatenate([np.asarray(c, np.int64) for c, _ in lists]), rp), shape=(len(lists), cols))


# widths of the last product's output: the warp bin's, the dense bin's (one
# window), and rows enough to leave the small products' kernels
@pytest.mark.parametrize("n,rows", [(1500, 40), (1500, 3000), (5000, 40), (5000, 3000)])
@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
def test_a_count_that_wraps_to_zero_keeps_its_column(native, vt, n, rows):
    """A B wraps its first column to exactly 0 in every row; its columns reach
    D's rows all the same: the chain reports the overflow and C's structure is
    the Boolean product, its counts modulo the type."""
    bits = 32 if vt == "VAL_U32" else 64
    eng = native.Engine(device=0, valtype=getattr(native, vt))
    rng = np.random.default_rng(n)
    k = 60
    A = _rows([([0, 1], [2 ** (bits // 2), 3])] * rows, 2)
    B = _rows([([0], [2 ** (bits // 2)]), (np.arange(1, k), rng.integers(1, 9, k - 1))], k)
    # D's first row alone holds the odd columns
    D = _rows([(np.arange(1, n, 2), np.full(n // 2, 5))] +
              [(2 * np.sort(rng.choice(n // 2, 90, replace=False)), rng.integers(1, 9, 90)) for _ in range(k - 1)], n)
    C, _, rc = eng.chain([_upload(eng, M, getattr(native, vt)) for M in (A, B, D)], pairs=[(0, 1), (-1, 2)])
    assert rc == native.EOVERFLOW
    rp, col, val = C.download()
    ab = np.zeros(k, object)
    ab[1:] = [3 * int(x) for x in B.toarray()[1, 1:]]
    d = D.toarray().astype(object)
    want = [int(x) % 2 ** bits for x in ab @ d]
    cols = np.nonzero((d != 0).any(axis=0))[0]
    assert np.array_equal(rp, np.arange(rows + 1) * cols.size)
    assert np.array_equal(col.reshape(rows, -1), np.tile(cols, (rows, 1)))
    assert np.array_equal(val.reshape(rows, -1)[[0, -1]].astype(np.uint64), np.array([[want[c] for c in cols]] * 2, np.uint64))
    eng.close()


def test_spgemm_returns_with_its_result_written(native):
    """Rows of a single-pass product are copied into the result last: the call
    waits for that, nothing of it is left on the stream."""
    import torch

    eng = native.Engine(device=0)
    st = torch.cuda.Stream()
    eng.set_stream(st.cuda_stream)
    rng = np.random.default_rng(2)
    m, k, n = 20000, 60, 3000
    A = _rows([([r % k, (r * 7 + 1) % k] if (r * 7 + 1) % k != r % k else [r % k], [1] * (2 if (r * 7 + 1) % k != r % k else 1))
               for r in range(m)], k)
    B = _rows([(np.sort(rng.choice(n, 2000, replace=False)), rng.integers(1, 9, 2000)) for _ in range(k)], n)
    a, b = _upload(eng, A, native.VAL_U32), _upload(eng, B, native.VAL_U32)
    for _ in range(5):
        C = eng.spgemm(a, b)      # some 50M entries to copy
        assert st.query()
        C.free()
    a.free(), b.free()
    eng.close()
