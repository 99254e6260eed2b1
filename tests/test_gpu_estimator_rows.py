"""Estimates of matrices whose long rows lie together, evenly or not, and of
more long rows than the device takes a cluster each."""
import numpy as np
import pytest

from test_gpu_row_kernels import _estimates

pytestmark = pytest.mark.gpu


def _lengths(kind, rows, sms):
    if kind == "sorted":             # by degree: the longest rows are neighbours
        return np.maximum(1, 9000 // (np.arange(rows) + 1))
    if kind == "even":               # every warp has as long a row as the others
        return np.full(rows, 700)
    if kind == "huge":               # evenly long, and long enough to be shared all the same
        return np.full(rows, 4096)
    lens = np.full(rows, 2)          # one cluster each for 2 SMs' worth of rows, or eight rows a cluster
    long = 2 * sms + (1 if kind == "more" else 0)
    lens[5:5 + long] = np.resize([4097, 8192, 8193, 9000], long)
    return lens


@pytest.mark.parametrize("length", [2, 4, 16])
@pytest.mark.parametrize("kind", ["sorted", "even", "huge", "clusters", "more"])
def test_estimates_of_neighbouring_long_rows(native, engine, kind, length):
    """Against sums of logarithms in float64: a row's product of up to 9,000
    factors is off by at most 9,000 roundings of a value below 1, 1e-12, its
    densities are above 1e-4; 1e-9 relative is the parity tolerance."""
    import torch

    rows = 300 if kind in ("even", "huge") else 1000
    lens = _lengths(kind, rows, torch.cuda.get_device_properties(0).multi_processor_count)
    rng = np.random.default_rng(length)
    cols = 9500
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(cols, int(k), replace=False)) for k in lens]).astype(np.int32)
    # every second matrix leads back to the rows' type, two entries a row
    back = np.sort(rng.integers(0, rows, (cols, 2)), axis=1).astype(np.int32).reshape(-1)
    brp = np.arange(cols + 1, dtype=np.int64) * 2
    mats = [(rp, col) if i % 2 == 0 else (brp, back) for i in range(length)]
    dims = [rows if i % 2 == 0 else cols for i in range(length + 1)]
    up = [engine.upload(rp, col, cols=cols), engine.upload(brp, back, cols=rows)]
    got = engine.estimate([up[i % 2] for i in range(length)])
    assert np.array_equal(got, engine.estimate([up[i % 2] for i in range(length)]))
    np.testing.assert_allclose(got, _estimates(mats, dims), rtol=1e-9, atol=0)
    for m in up:
        m.free()
