"""The factorised start at the widths where its panel kernels change (64, 128, 256,
384, 512 and 640 columns) and at ragged last panels, square and tall, in both forms.
Checked like test_gpu_svd_kernel.py's jobs (same tolerances) against complex128 LAPACK.
"""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,extra", [(64, 0), (66, 2), (96, 34), (128, 64), (130, 0), (256, 2),
                                        (258, 0), (384, 30), (386, 0), (512, 2), (514, 0),
                                        (640, 0), (642, 0)])
@pytest.mark.parametrize("lc", [True, False])
def test_widths(built_lib, cuda, cols, extra, lc):
    """theta of cols + extra rows and cols columns, or its transpose's shape."""
    rng = np.random.default_rng(cols + extra)
    long, short = (cols + extra) // 2, cols // 2
    chil, chir = (long, short) if lc else (short, long)
    a, b, g = make_job_inputs(rng, chil, short, chir, 2, scale=1.0 / short)
    k = short + 1
    rc, res, _ = run_batch(built_lib, cuda, [(a, b, g, k, lc)])
    assert rc == 0, _native.last_error()
    check_job((a, b, g, k, lc), res[0], 2)
