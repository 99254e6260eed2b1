"""Orders of chains whose costs are not numbers below the largest double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check_pairs(pairs, n):
    """A post-order of n matrices: every one used once, in order, and at each
    step the top of the stack is what stands beside it."""
    stack = []

    def take(k):
        return stack.pop() if k < 0 else (int(k), int(k))

    assert len(pairs) == n - 1
    for k, l in pairs:
        right = take(l)
        left = take(k)
        assert left[1] + 1 == right[0]
        stack.append((left[0], right[1]))
    assert stack == [(0, n - 1)]


@pytest.mark.parametrize("n", [3, 4, 16])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e308])
def test_costs_without_a_smallest_one(engine, n, bad):
    """Every interval, the last ones only, and one interval in the middle."""
    for where in ("all", "last", "one"):
        c = np.triu(np.arange(1.0, n * n + 1).reshape(n, n))
        if where == "all":
            c[np.triu_indices(n)] = bad
        elif where == "last":
            c[:, n - 1] = bad
        else:
            c[1, 2] = bad
        split, cost, pairs = engine.order(c)
        _check_pairs(pairs, n)
        for i in range(n):
            for j in range(i + 1, n):
                assert i <= split[i, j] < j


def test_chain_into_a_type_without_vertices(native, engine):
    """Densities over zero columns are 0 / 0."""
    ones = [(np.arange(7) * 2, np.tile([0, 3], 6)), (np.arange(6), np.array([0, 1, 2, 0, 1])), (np.zeros(4), np.zeros(0))]
    mats = [engine.upload(rp.astype(np.int64), col.astype(np.int32), cols=n)
            for (rp, col), n in zip(ones, (5, 3, 0))]
    C, _, rc = engine.chain(mats)
    assert rc == native.OK and C.shape == (6, 0) and C.nnz == 0
    C.free()
