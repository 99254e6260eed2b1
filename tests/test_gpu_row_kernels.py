"""Row kernels at the edges of their ranges, against exact integer products."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def upload(native, engine, M, vt):
    M = M.tocsr()
    M.sort_indices()
    return engine.upload(M.indptr, M.indices, cols=M.shape[1], val=M.data.astype(np.uint64), valtype=vt)


def check_product(native, engine, A, B, vt):
    """Structure and uint64 values against scipy (whose arithmetic is modulo
    2^64, exact for the sums drawn here)."""
    ref = (A.astype(np.uint64) @ B.astype(np.uint64)).tocsr()
    ref.sum_duplicates()
    ref.sort_indices()
    C = engine.spgemm(upload(native, engine, A, vt), upload(native, engine, B, vt))
    rp, col, val = C.download()
    assert np.array_equal(rp, ref.indptr)
    assert np.array_equal(col, ref.indices)
    assert np.array_equal(val.astype(np.uint64), ref.data)


def random_csr(rng, rows, cols, lens, lo=1, hi=4):
    lens = np.minimum(np.asarray(lens), cols)
    c = np.concatenate([rng.choice(cols, int(k), replace=False) for k in lens]) if lens.sum() else np.zeros(0, int)
    r = np.repeat(np.arange(rows), lens)
    v = rng.integers(lo, hi, c.size, dtype=np.uint64)
    return sp.csr_matrix((v, (r, c)), shape=(rows, cols))


@pytest.mark.parametrize("n,terms", [(40, 60), (1500, 60), (5000, 300), (60000, 40)])
def test_uint64_counts_carry_between_their_halves(native, engine, n, terms):
    """Many terms near 2^32 and 2^50 land on the same columns, so the counters'
    low halves wrap many times (warp, dense and hash bins)."""
    rng = np.random.default_rng(n)
    A = random_csr(rng, 50, terms, np.full(50, terms), lo=2 ** 16 - 2, hi=2 ** 16 + 2)
    lens = rng.integers(1, min(n, 40), terms)
    B = random_csr(rng, terms, n, lens, lo=2 ** 16 - 2, hi=2 ** 16 + 2)
    big = rng.random(B.nnz) < 0.3
    B.data[big] = rng.integers(2 ** 33, 2 ** 34, int(big.sum()), dtype=np.uint64)
    check_product(native, engine, A, B, native.VAL_U64)


@pytest.mark.parametrize("n", [40, 5000, 60000])
@pytest.mark.parametrize("over", [0, 1])
def test_uint64_overflow_is_seen_at_its_exact_limit(native, engine, n, over):
    """A count of exactly 2^64 - 1 is no overflow, 2^64 is one; the last term
    only carries out of the low half."""
    k = 80
    top = [2 ** 63, 2 ** 62, 2 ** 62 - 2 ** 32, 2 ** 32 - (k - 4)]
    vals = np.array(top + [1] * (k - 4), np.uint64)      # sums to 2^64
    assert sum(int(v) for v in vals) == 2 ** 64
    if not over:
        vals[-1] = 0
    A = sp.csr_matrix(np.ones((1, k), np.uint64))
    cols = np.stack([np.full(k, n - 1), np.arange(k) % (n - 1)], 1)
    B = sp.csr_matrix((np.stack([vals, np.ones(k, np.uint64)], 1).reshape(-1),
                       (np.repeat(np.arange(k), 2), cols.reshape(-1))), shape=(k, n))
    Am, Bm = upload(native, engine, A, native.VAL_U64), upload(native, engine, B, native.VAL_U64)
    h = ctypes.c_void_p()
    rc = native.lib().rmcm_spgemm(engine._h, Am._h, Bm._h, ctypes.byref(h))
    C = native.Matrix(engine, h.value)
    assert rc == (native.EOVERFLOW if over else native.OK)
    if not over:
        rp, col, val = C.download()
        assert col[-1] == n - 1 and int(val[-1]) == 2 ** 64 - 1
