"""Right-canonical jobs on both sides of the lines of their dispatch: tall (V
tracked), square and up to twice as wide (theta^T, no V, the left site by a product),
wider (V tracked); sizes around the 64 x 64 tiles of that product, kept counts below
and at the rank, and null directions.  Checked like test_gpu_svd_kernel.py's jobs
(same tolerances) against complex128 LAPACK.
"""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chil,chim,chir,k", [
    (33, 40, 32, 50),       # tall 66 x 64
    (32, 40, 32, 64),       # square
    (32, 40, 33, 63),       # 64 x 66: one tile, its last columns in a second
    (33, 20, 64, 33),       # 66 x 128: rank 40 of 66
    (32, 8, 63, 40),        # 64 x 126: rank 16, 24 null directions kept
    (32, 40, 64, 64),       # 64 x 128: twice as wide
    (5, 4, 9, 10),          # 10 x 18: rank 8
    (96, 96, 130, 129),     # 192 x 260: the factorised form
    (1, 1, 1, 2),
])
def test_widths(built_lib, cuda, chil, chim, chir, k):
    rng = np.random.default_rng(100 * chil + chir)
    a, b, g = make_job_inputs(rng, chil, chim, chir, 2, scale=1.0 / chim)
    rc, res, _ = run_batch(built_lib, cuda, [(a, b, g, k, False)])
    assert rc == 0, _native.last_error()
    check_job((a, b, g, k, False), res[0], 2)
