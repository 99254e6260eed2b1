"""Panels of the tensor-core part at the limits of their shared memory."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a process of its own: the first panel it gathers has this size, nothing
# before has raised the kernel's limit
SCRIPT = """
import numpy as np, scipy.sparse as sp, resmcm_ari_gb300 as rg
k, vt, ahi = {k}, rg.{vt}, {ahi}
eng = rg.Engine(device=0)
eng.set_tuning(gemm_min_mflops=1)
eng.set_profiling(1)
rng = np.random.default_rng(k)
A = rng.integers(1, ahi, (160, k), dtype=np.uint64)
A[:, 0] = ahi - 1
B = rng.integers(1, 3, (k, 200), dtype=np.uint64)
up = lambda M: eng.upload(np.arange(M.shape[0] + 1) * M.shape[1], np.tile(np.arange(M.shape[1]), M.shape[0]),
                          cols=M.shape[1], val=M.reshape(-1), valtype=vt)
rp, col, val = eng.spgemm(up(A), up(B)).download()
st = eng.product_stats()[-1]
# (the panel's rows are padded to 64 indices)
assert -(-st["gemm_inner"] // 64) == -(-k // 64) and st["gemm_limbs"] == {limbs}, st
assert np.array_equal(val.reshape(160, 200).astype(np.uint64), A @ B)
"""


# one limb of 24,576 indices fills 48 KB with A's row, as two of 12,288 and
# three of 8,192 do; one panel step less and more.  (Odd widths: the sample
# then shows every column.)
@pytest.mark.parametrize("vt,ahi,limbs,k", [("VAL_U32", 3, 1, 24575), ("VAL_U64", 3, 1, 24575), ("VAL_U64", 3, 1, 24511),
                                            ("VAL_U64", 3, 1, 24639), ("VAL_U64", 2 ** 16, 2, 12287),
                                            ("VAL_U64", 2 ** 24, 3, 8191)])
def test_panels_of_48_kb(native, vt, ahi, limbs, k):
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(vt=vt, ahi=ahi, k=k, limbs=limbs)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
