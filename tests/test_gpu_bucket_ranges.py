"""Rank-bin rows at the limits of what the bucket kernel's CTAs take."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_row_kernels import check_product

pytestmark = pytest.mark.gpu

RANK = 5                                        # the rank bin's place in bin_rows
EDGES = [2816, 5632, 11264, 33792]              # one and two fills of 128 threads, one and three of 512


def _operands(rng, lens, per, n):
    """A with lens[r] entries in row r, B with `per` entries in every row (so a
    row has lens[r] x per products)."""
    k = max(lens)
    A = sp.csr_matrix((rng.integers(1, 30, sum(lens), dtype=np.uint64),
                       np.concatenate([np.sort(rng.permutation(k)[:x]) for x in lens]),
                       np.concatenate([[0], np.cumsum(lens)])), shape=(len(lens), k))
    step = n // per                              # one column of every `step`
    col = np.arange(per) * step + rng.integers(0, step, (k, per))
    B = sp.csr_matrix((rng.integers(1, 30, k * per, dtype=np.uint64), col.reshape(-1), np.arange(k + 1) * per),
                      shape=(k, n))
    return A, B


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("n", [70_001, 2 ** 19, 2 ** 19 + 1, 2 ** 20])
@pytest.mark.parametrize("per", [8, 31, 32, 64])
def test_rows_about_whole_fills(native, engine, per, n, vt):
    """Products up to an edge and past it, through B rows shorter and longer than
    those of which a CTA makes another pass; many rows of each, so that both CTA
    sizes run."""
    rng = np.random.default_rng(per)
    lens = [x for e in EDGES for x in (e // per, e // per + 1)] * 40
    engine.set_profiling(1)
    try:
        engine.product_stats()
        check_product(native, engine, *_operands(rng, lens, per, n), getattr(native, vt))
        assert engine.product_stats()[-1]["bin_rows"][RANK] == len(lens)
    finally:
        engine.set_profiling(0)


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("more", [0, 1])
def test_rows_up_to_two_an_sm(native, engine, more, vt):
    """The count of rows up to which all of them take the larger CTAs."""
    import torch

    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(rows)
    lens = [int(x) for x in rng.choice([60, 141, 282, 600], rows)]
    engine.set_profiling(1)
    try:
        engine.product_stats()
        check_product(native, engine, *_operands(rng, lens, 40, 300_007), getattr(native, vt))
        assert engine.product_stats()[-1]["bin_rows"][RANK] == rows
    finally:
        engine.set_profiling(0)


@pytest.mark.parametrize("vt", ["VAL_U32", "VAL_U64"])
@pytest.mark.parametrize("n", [70_001, 2 ** 17, 2 ** 17 + 1, 2 ** 19, 2 ** 19 + 1])
@pytest.mark.parametrize("rows", [90, 400])
def test_rows_through_short_rows_of_b(native, engine, rows, n, vt):
    """B rows of 1, 1.5, 2 and 3 positions on average, some rows taken and some
    left in one product."""
    rng = np.random.default_rng(n)
    per = np.repeat([1, 2, 3], 1300)
    rp = np.concatenate([[0], np.cumsum(per)])
    third = n // 3                               # one column of each third
    col = np.concatenate([np.arange(x) for x in per]) * third + rng.integers(0, third, rp[-1])
    B = sp.csr_matrix((rng.integers(1, 30, col.size, dtype=np.uint64), col, rp), shape=(per.size, n))
    first = [0, 650, 1300, 2600]                 # 1,300 rows of B from here: 1, 1.5, 2 and 3 positions
    picks = [first[r % 4] + np.sort(rng.permutation(1300)[: 1100 + r // 2]) for r in range(rows)]
    ap = np.concatenate([[0], np.cumsum([p.size for p in picks])])
    A = sp.csr_matrix((rng.integers(1, 30, ap[-1], dtype=np.uint64), np.concatenate(picks), ap), shape=(rows, per.size))
    check_product(native, engine, A, B, getattr(native, vt))
