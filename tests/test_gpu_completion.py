"""The orthonormal completion of null directions: none, some and all kept columns missing,
more elements than threads, shares of rows that do not divide, in both forms.
Checked like test_gpu_svd_kernel.py's jobs (same tolerances) against complex128 LAPACK.
"""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chil,chir,rank,k", [
    (1, 1, 1, 2), (3, 5, 1, 6), (5, 3, 2, 6), (16, 17, 3, 32), (33, 33, 0, 40), (33, 30, 7, 60),
    (100, 40, 9, 80), (40, 90, 9, 80), (128, 128, 100, 256), (700, 6, 2, 12), (6, 700, 2, 12),
    (300, 290, 1, 130)])
@pytest.mark.parametrize("lc", [True, False])
def test_missing_directions(built_lib, cuda, chil, chir, rank, k, lc):
    """theta of rank 2 rank at most, exact zeros behind it; k kept."""
    rng = np.random.default_rng(chil + 10 * chir)
    chim = max(rank, 1)
    a, b, g = make_job_inputs(rng, chil, chim, chir, 2, rank=rank, scale=0.5)
    g = np.eye(4, dtype=np.complex64)                  # (keeps the rank: half of the site's columns)
    b[:, 1] = 0                                        # exact zero columns of theta
    spec = (a, b, g, k, lc)
    rc, res, _ = run_batch(built_lib, cuda, [spec, spec])
    assert rc == 0, _native.last_error()
    for out in res:
        check_job(spec, out, 2)
    assert np.array_equal(res[0]["a"], res[1]["a"]) and np.array_equal(res[0]["b"], res[1]["b"])
