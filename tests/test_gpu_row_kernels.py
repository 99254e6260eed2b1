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


# B row lengths around the points where a row kernel changes how an entry's
# products are spread (4 | 5, 64 | 65), around whole blocks of 128, and empty
SPREAD = np.array([0, 1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129, 255, 257, 300])


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("n", [127, 128, 129, 2047, 2048, 2049, 4100, 10300, 22528, 22529, 40960])
def test_row_kernels_at_their_widths(native, engine, n, vt):
    """Every width at which another kernel, CTA size or window takes the rows;
    rows from one entry to more than a CTA lists at a time; some rows of a
    uint64 product stay below 2^32, some do not."""
    rng = np.random.default_rng(n)
    k = 1500
    B = random_csr(rng, k, n, rng.choice(SPREAD, k), hi=6)
    m = 260
    a_len = np.concatenate([rng.integers(1, 60, m - 4), [k, 1030, 513, 511]])
    A = random_csr(rng, m, k, a_len, hi=6)
    if vt == "VAL_U64":
        A.data[A.indptr[5]:A.indptr[40]] *= np.uint64(2 ** 34)
    check_product(native, engine, A, B, getattr(native, vt))


@pytest.mark.parametrize("n", [900, 5000])
def test_safe_and_risky_rows_in_one_product(native, engine, n):
    """uint32 rows whose bound passes 2^32 (none overflows: their large values
    meet different columns) beside rows that cannot."""
    rng = np.random.default_rng(n)
    k = 300
    B = random_csr(rng, k, n, rng.integers(20, 200, k), hi=3)
    A = random_csr(rng, 200, k, rng.integers(2, 60, 200), hi=4)
    A = A.tolil()
    for r in range(0, 200, 7):           # two entries of 2^30 and B rows of ones that do not meet
        A[r, k - 1] = 2 ** 31
        A[r, k - 2] = 2 ** 31
    A = A.tocsr().astype(np.uint64)
    B = B.tolil()
    B[k - 1, :] = 0
    B[k - 2, :] = 0
    B[k - 1, 0:n // 3:2] = 1
    B[k - 2, 1:n // 3:2] = 1
    B = B.tocsr().astype(np.uint64)
    B.eliminate_zeros()
    check_product(native, engine, A, B, native.VAL_U32)


@pytest.mark.parametrize("n", [600, 3000])
def test_ones_and_repeated_columns(native, engine, n):
    """Leaves are matrices of ones, and may hold a column twice in a row."""
    rng = np.random.default_rng(n)
    k, m = 400, 300
    lens = rng.choice(SPREAD, k)
    col = [np.sort(rng.integers(0, n, x)) for x in lens]          # with repeats
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    bc = np.concatenate(col).astype(np.int32)
    A = random_csr(rng, m, k, rng.integers(1, 80, m), hi=2)
    B = sp.csr_matrix((np.ones(bc.size, np.uint64), bc, rp), shape=(k, n))
    ref = (A.astype(np.uint64) @ B).tocsr()
    ref.sum_duplicates()
    ref.sort_indices()
    for vt in (native.VAL_U32, native.VAL_U64):
        Am = engine.upload(A.indptr, A.indices, cols=k, valtype=vt)
        Bm = engine.upload(rp, bc, cols=n, valtype=vt)
        rp2, col2, val2 = engine.spgemm(Am, Bm).download()
        assert np.array_equal(rp2, ref.indptr) and np.array_equal(col2, ref.indices)
        assert np.array_equal(val2.astype(np.uint64), ref.data)


def test_heavy_rows_are_split_below_the_general_threshold(native, engine):
    """Rows of 2^17 products and more in a small product go to several CTAs."""
    rng = np.random.default_rng(3)
    k, n = 4000, 6000
    B = random_csr(rng, k, n, rng.choice(SPREAD, k), hi=4)
    lens = np.concatenate([rng.integers(1, 40, 120), [k, k, 3000]])
    A = random_csr(rng, lens.size, k, lens, hi=4)
    for vt in (native.VAL_U32, native.VAL_U64):
        check_product(native, engine, A, B, vt)


@pytest.mark.parametrize("avg", [1, 3, 9, 40, 200])
@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
def test_analysis_at_every_row_length(native, engine, avg, vt):
    """The average row sets the lanes per row; rows past 64 times that many
    entries, past a piece of the grid's and past two pieces go other ways."""
    rng = np.random.default_rng(avg)
    k, n = 6000, 700
    lens = np.concatenate([rng.integers(0, 2 * avg + 1, 900), [130, 257, 600, 2047, 2048, 2049, 4096, 4097, 6000]])
    A = random_csr(rng, lens.size, k, rng.permutation(lens), hi=5)
    B = random_csr(rng, k, n, rng.integers(0, 6, k), hi=5)
    check_product(native, engine, A, B, getattr(native, vt))
    ones = sp.csr_matrix((np.ones(A.nnz, np.uint64), A.indices, A.indptr), shape=A.shape)
    check_product(native, engine, ones, B, getattr(native, vt))


@pytest.mark.parametrize("n", [40, 5000, 60000])
@pytest.mark.parametrize("over", [0, 1])
def test_uint32_overflow_is_seen_at_its_exact_limit(native, engine, n, over):
    """A count of 2^32 - 1 is no overflow, 2^32 is one, beside columns whose
    totals alone pass 2^32."""
    k = 70
    vals = np.array([2 ** 31, 2 ** 30, 2 ** 30 - (k - 3)] + [1] * (k - 3), np.uint64)     # sums to 2^32
    if not over:
        vals[-1] = 0
    cols = np.stack([np.full(k, n - 1), np.arange(k) % (n - 1)], 1)
    other = np.where(np.arange(k) < n - 1, 2 ** 31, 1).astype(np.uint64)[: k]
    other[n - 1:] = 1
    B = sp.csr_matrix((np.stack([vals, other], 1).reshape(-1), (np.repeat(np.arange(k), 2), cols.reshape(-1))),
                      shape=(k, n))
    A = sp.csr_matrix(np.ones((1, k), np.uint64))
    h = ctypes.c_void_p()
    Am, Bm = upload(native, engine, A, native.VAL_U32), upload(native, engine, B, native.VAL_U32)
    rc = native.lib().rmcm_spgemm(engine._h, Am._h, Bm._h, ctypes.byref(h))
    C = native.Matrix(engine, h.value)
    assert rc == (native.EOVERFLOW if over else native.OK)
    if not over:
        rp, col, val = C.download()
        assert col[-1] == n - 1 and int(val[-1]) == 2 ** 32 - 1


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("n", [41000, 100003, 2 ** 22, 2 ** 22 + 1, 2 ** 24, 2 ** 24 + 1])
def test_sorted_rows_at_their_limits(native, engine, n, vt):
    """Rows of exactly 33, 127..129, 255..257, 511..513 and 1023..1025 products
    on outputs around the widest whose columns fit a key; few distinct columns,
    the last one among them; B rows of every length up to one of 1,025."""
    rng = np.random.default_rng(n % 1000)
    want = [33, 64, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025]
    parts = [1, 2, 7, 8, 9, 31, 64, 65, 200]
    brow, acol, alen = [], [], []
    for w in want:
        for style in range(3):
            left, used = w, 0
            while left:
                x = left if style == 0 else min(left, int(rng.choice(parts[: 4 + 5 * (style == 1)])))
                acol.append(len(brow))
                brow.append(x)
                left -= x
                used += 1
            alen.append(used)
    k = len(brow)
    pool = np.unique(np.concatenate([rng.integers(0, n, 1500), [0, n - 1]]))
    cols = [np.sort(rng.choice(pool, x, replace=False)) for x in brow]
    cols[0][-1] = n - 1
    rp = np.concatenate([[0], np.cumsum(brow)])
    B = sp.csr_matrix((rng.integers(1, 50, rp[-1], dtype=np.uint64), np.concatenate(cols), rp), shape=(k, n))
    ap = np.concatenate([[0], np.cumsum(alen)])
    A = sp.csr_matrix((rng.integers(1, 50, k, dtype=np.uint64), np.array(acol), ap), shape=(len(alen), k))
    check_product(native, engine, A, B, getattr(native, vt))


@pytest.mark.parametrize("terms", [40, 200, 700])
def test_sorted_rows_report_overflow(native, engine, terms):
    """Equal columns that only together pass the value type, in one lane's
    share of the sorted row and across many lanes'."""
    n = 60000
    for vt, top in ((native.VAL_U32, 32), (native.VAL_U64, 64)):
        each = -(-2 ** top // terms)
        for over in (0, 1):
            v = np.full(terms, each if over else each - 1, np.uint64)
            rp = np.arange(terms + 1, dtype=np.int64)
            col = np.full(terms, 12345, np.int32)
            Am = engine.upload(np.array([0, terms]), np.arange(terms, dtype=np.int32), cols=terms, valtype=vt)
            Bm = engine.upload(rp, col, cols=n, val=v, valtype=vt)
            h = ctypes.c_void_p()
            rc = native.lib().rmcm_spgemm(engine._h, Am._h, Bm._h, ctypes.byref(h))
            C = native.Matrix(engine, h.value)
            assert rc == (native.EOVERFLOW if over else native.OK)
            if not over:
                assert int(C.download()[2][0]) == terms * (each - 1)


def _estimates(mats, dims):
    """The estimates in float64 from sums of logarithms."""
    L = len(mats)
    c = np.zeros((L, L))
    after = {}
    for i in range(L - 1, -1, -1):
        rp, col = mats[i]
        lens = np.diff(rp)
        now = {i: np.minimum(1.0, lens / dims[i + 1])}
        for j, r in after.items():
            with np.errstate(divide="ignore"):
                t = np.concatenate([np.log1p(-r)[col], [0.0]])
            sums = np.where(lens > 0, np.add.reduceat(t, rp[:-1]), 0.0)
            now[j] = -np.expm1(sums)
            c[i, j] = now[j].sum() * dims[j + 1]
        after = now
    return c


@pytest.mark.parametrize("length", [2, 3, 5, 9, 16])
@pytest.mark.parametrize("n", [7, 900, 30000])
def test_estimates_at_every_row_length(native, engine, length, n):
    """Rows of every class of lanes (1 .. 4, 5 .. 8, ... entries), around the
    length a CTA shares and the length a cluster takes, empty rows; chains from
    one target to fifteen (1, 2, 4, 8 and 16 lanes a group).  A row's product of
    up to 9,000 factors is off by at most 9,000 roundings of a value below 1,
    1e-12; the densities here are above 1e-4, and their errors average out over
    the rows: 1e-9 relative, the parity tolerance of the estimates."""
    rng = np.random.default_rng(n + length)
    mats, dims = [], [n]
    special = [0, 1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128, 129, 130, 255, 257, 2047, 2049, 4095, 4096, 4097,
               8192, 9000]
    for i in range(length):
        cols = int(rng.integers(9001, 12000)) if i < length - 1 else 5000
        rows = dims[-1]
        lens = rng.integers(0, 12, rows)
        at = rng.choice(rows, min(rows, len(special)), replace=False)
        lens[at] = rng.permutation(special)[: at.size]
        lens = np.minimum(lens, cols)
        rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
        col = np.concatenate([np.sort(rng.choice(cols, int(k), replace=False)) for k in lens]).astype(np.int32)
        mats.append((rp, col))
        dims.append(cols)
    chain = [engine.upload(rp, col, cols=dims[i + 1]) for i, (rp, col) in enumerate(mats)]
    got = engine.estimate(chain)
    again = engine.estimate(chain)
    assert np.array_equal(got, again)
    want = _estimates(mats, dims)
    np.testing.assert_allclose(got, want, rtol=1e-9, atol=0)


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
def test_bucketed_rows(native, vt):
    """Rows of an output wider than a window, from the fewest products the rank
    bin takes to several times what a CTA holds: uniform columns, columns in one
    narrow range (a bucket too full: the bitmap kernel's rows), one column many
    times, the first and the last column; B rows of every length."""
    eng = native.Engine(device=0)
    rng = np.random.default_rng(11)
    n = 700_001
    k = 3000
    lens = rng.choice([1, 2, 5, 9, 31, 33, 63, 64, 65, 128, 129, 200], k)
    cols = []
    for i, x in enumerate(lens):
        if i < 1500:
            c = rng.choice(n, x, replace=False)                       # anywhere
        elif i < 2300:
            c = 5000 + rng.choice(600, x, replace=False)              # one narrow range
        else:
            c = np.concatenate([[0, n - 1, 77][: min(3, x)], 100 + rng.choice(n - 200, max(0, x - 3), replace=False)])
            c = np.unique(c)
            while c.size < x:
                c = np.unique(np.concatenate([c, rng.integers(100, n - 2, x - c.size)]))
        cols.append(np.sort(c))
    rp = np.concatenate([[0], np.cumsum(lens)])
    B = sp.csr_matrix((rng.integers(1, 30, rp[-1], dtype=np.uint64), np.concatenate(cols), rp), shape=(k, n))
    picks = []
    for lo, hi in ((0, 1500), (1500, 2300), (2300, 3000), (0, 3000)):
        for take in (20, 60, 90, 150, 240, 400, 690):
            picks.append(np.sort(lo + rng.choice(hi - lo, take, replace=False)))
    ap = np.concatenate([[0], np.cumsum([p.size for p in picks])])
    A = sp.csr_matrix((rng.integers(1, 30, ap[-1], dtype=np.uint64), np.concatenate(picks), ap), shape=(len(picks), k))
    f = np.array([lens[p].sum() for p in picks])
    assert f.min() < 1100 and (f > 8448).sum() > 3 and (f > 33792).sum() > 1
    check_product(native, eng, A, B, getattr(native, vt))
    eng.close()


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("k", [248, 256, 257])
def test_every_index_of_full_matrices_is_heavy(native, vt, k):
    """Widths that are multiples of the sampling step: a full matrix shows
    every column to the heavy-index selection, not one in eight."""
    eng = native.Engine(device=0)
    eng.set_tuning(gemm_min_mflops=1)
    rng = np.random.default_rng(k)
    A = sp.csr_matrix(rng.integers(1, 40, (520, k), dtype=np.uint64))
    B = sp.csr_matrix(rng.integers(1, 40, (k, 264), dtype=np.uint64))
    eng.set_profiling(1)
    check_product(native, eng, A, B, getattr(native, vt))
    assert eng.product_stats()[-1]["gemm_inner"] == k
    eng.close()


@pytest.mark.parametrize("m", [1, 3, 1023, 1024, 1025, 2047, 2048, 2049, 8191, 8192, 8193])
@pytest.mark.parametrize("n", [1500, 50000])
def test_small_products_at_the_limits_of_their_plan(native, engine, m, n):
    """Row counts around the one-kernel plan's tiles and its end and the
    one-tile scan's; rows of every bin, many of one kind or a few of each, and
    rows without products."""
    rng = np.random.default_rng(m + n)
    k = 600
    B = random_csr(rng, k, n, rng.choice(np.array([0, 1, 2, 3, 7, 12, 40, 90]), k), hi=6)
    for lens in (rng.integers(0, 3, m), rng.choice([0, 1, 2, 5, 9, 30, 110], m)):
        if lens.sum() > 40000:
            lens[rng.random(m) < 0.8] = 1
        A = random_csr(rng, m, k, lens, hi=6)
        for vt in (native.VAL_U32, native.VAL_U64):
            check_product(native, engine, A, B, vt)
    empty = sp.csr_matrix((m, k), dtype=np.uint64)
    check_product(native, engine, empty, B, native.VAL_U32)


@pytest.mark.parametrize("m", [8194, 20480, 20481, 4096 * 2048, 4096 * 2048 + 1])
def test_row_pointers_over_many_tiles(native, engine, m):
    """The scan of the row lengths at whole tiles and their remainders, and at
    the count of tiles where their sums get a launch of their own; long gaps of
    empty rows, the last row empty or not."""
    rng = np.random.default_rng(m)
    k = 50
    B = random_csr(rng, k, 300, rng.integers(0, 5, k), hi=6)
    for last in (0, 1):
        lens = (rng.random(m) < 0.3).astype(np.int64)
        lens[m // 3: m // 2] = 0
        lens[-1] = last
        rp = np.concatenate([[0], np.cumsum(lens)])
        A = sp.csr_matrix((rng.integers(1, 6, rp[-1], dtype=np.uint64), rng.integers(0, k, rp[-1]), rp), shape=(m, k))
        check_product(native, engine, A, B, native.VAL_U32)


@pytest.mark.parametrize("vt,hi", [("VAL_U32", 4), ("VAL_U32", 5000), ("VAL_U64", 4), ("VAL_U64", 2 ** 20)])
def test_long_rows_of_the_tensor_part(native, vt, hi):
    """Panels of rows about the length where they are filled in by pieces, at a
    piece's edges and beyond, with heavy inner indices and light ones of every
    length, one limb of values and several."""
    eng = native.Engine(device=0)
    eng.set_tuning(gemm_min_mflops=1)
    rng = np.random.default_rng(hi)
    k, n = 60000, 1000
    rows = [0, 5000, 16384, 16385, 24576, 24577, 32768, 60000] + [16385] * 40 + [900] * 40
    A = random_csr(rng, len(rows), k, rows, lo=1, hi=hi)
    lens = rng.integers(0, 4, k)
    lens[rng.permutation(k)[:400]] = n
    B = random_csr(rng, k, n, lens, lo=1, hi=min(hi, 6))
    eng.set_profiling(1)
    check_product(native, eng, A, B, getattr(native, vt))
    # an index in the sample of A's columns is heavy: 7 of 8 with 16 entries each
    st = eng.product_stats()[-1]
    assert st["gemm_inner"] >= 300, st
    eng.close()


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("rows", [3, 304, 305, 700])
def test_bucketed_rows_few_and_many(native, engine, rows, vt):
    """Rank-bin rows about the count (two an SM) up to which every row takes the
    larger CTAs; products from the fewest to beyond a smaller CTA's."""
    rng = np.random.default_rng(rows)
    n, k = 500_003, 400
    B = random_csr(rng, k, n, rng.choice([3, 20, 40, 130], k), hi=30)
    A = random_csr(rng, rows, k, rng.choice([30, 60, 190, 280], rows), hi=30)
    check_product(native, engine, A, B, getattr(native, vt))


@pytest.mark.parametrize("vt,hi,bhi", [("VAL_U32", 4, 4), ("VAL_U32", 4, 2 ** 20), ("VAL_U64", 4, 4),
                                       ("VAL_U64", 2 ** 20, 2 ** 24)])
@pytest.mark.parametrize("n", [97, 128, 2049, 22528])
def test_split_rows(native, engine, n, vt, hi, bhi):
    """Rows split over CTAs: windows of one block and at their limits, B packed
    and not, counts within 32 bits and beyond, B rows of every length class."""
    rng = np.random.default_rng(n)
    k = 30000
    lens = np.minimum(rng.choice([0, 1, 4, 5, 9, 40, 64, 65, 200], k), n)
    hub = rng.integers(0, n, 40)
    rows = np.repeat(np.arange(k), lens)
    cols = np.concatenate([rng.permutation(n)[:x] for x in lens])
    cols[rng.random(cols.size) < 0.02] = hub[0]
    B = sp.csr_matrix((rng.integers(1, bhi, cols.size, dtype=np.uint64), (rows, cols)), shape=(k, n))
    B.sum_duplicates()
    A = random_csr(rng, 40, k, [29000, 12000, 30000] + [30] * 37, hi=hi)
    if vt == "VAL_U32" and bhi > 4:
        A.data[:] = 1
        B.data[:] = 1 + B.data % 2
        B.data[::50000] = bhi      # too wide to pack beside the widest columns, sums within 32 bits
    check_product(native, engine, A, B, getattr(native, vt))
