"""Gram sweeps at the sizes where their tiles end: 8-column blocks (padding
blocks, odd block counts), 64-row tasks of the apply warps, the slot lengths, and
jobs that accumulate V.  Checked like test_gpu_svd_kernel.py's jobs (same
tolerances) against complex128 LAPACK.
"""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chil,chir", [
    (1, 2), (4, 4), (4, 5), (8, 9), (12, 12), (16, 17), (31, 32), (32, 33), (36, 37), (63, 65),
    (64, 64), (65, 60), (128, 100), (129, 128), (250, 140), (257, 255), (300, 40)])
@pytest.mark.parametrize("lc", [True, False])
def test_sizes(built_lib, cuda, chil, chir, lc):
    """theta of 2 chil x 2 chir, from 2 x 4 to 600 x 80, in both forms."""
    rng = np.random.default_rng(1000 * chil + chir)
    chim = max(chil, chir)
    a, b, g = make_job_inputs(rng, chil, chim, chir, 2, scale=1.0 / chim)
    k = max(1, min(chil, chir))
    rc, res, _ = run_batch(built_lib, cuda, [(a, b, g, k, lc)])
    assert rc == 0, _native.last_error()
    check_job((a, b, g, k, lc), res[0], 2)


def test_mixed_shapes_in_one_call(built_lib, cuda):
    """Jobs of different lengths, widths and forms in one slot class, more visits
    than the SMs have slots."""
    rng = np.random.default_rng(5)
    specs = []
    for q in range(70):
        chil, chir = int(rng.integers(20, 65)), int(rng.integers(3, 65))
        a, b, g = make_job_inputs(rng, chil, 64, chir, 2, scale=0.1)
        specs.append((a, b, g, min(chil, chir), bool(q % 3)))
    rc, res, _ = run_batch(built_lib, cuda, specs)
    assert rc == 0, _native.last_error()
    for spec, out in zip(specs, res):
        check_job(spec, out, 2)


@pytest.mark.parametrize("chil,chir", [(255, 256), (288, 280), (289, 150), (512, 200)])
@pytest.mark.parametrize("lc", [True, False])
def test_buffers_fewer_than_slots(built_lib, cuda, chil, chir, lc):
    """The longest slots (512, 576 and 1024 rows), where several visits pass through
    one column buffer; right-canonical: V rows beside it."""
    rng = np.random.default_rng(7000 * chil + chir)
    specs = []
    for _ in range(3):
        a, b, g = make_job_inputs(rng, chil, chir, chir, 2, scale=1.0 / chir)
        specs.append((a, b, g, chir, lc))
    rc, res, _ = run_batch(built_lib, cuda, specs)
    assert rc == 0, _native.last_error()
    for spec, out in zip(specs, res):
        check_job(spec, out, 2)


@pytest.mark.parametrize("n", [20, 70, 130])
def test_infinite_entry_is_reported(built_lib, cuda, n):
    """The column sort keeps a valid order when norms overflow; the call ends with
    its error and the next one is right."""
    rng = np.random.default_rng(n)
    a, b, g = make_job_inputs(rng, n, n, n, 2, scale=1.0 / n)
    bad = a.copy()
    bad[n // 2, 1, n // 3] = np.inf
    rc, _, _ = run_batch(built_lib, cuda, [(bad, b, g, n, True)])
    assert rc == _native.MPS_ERR_NONFINITE
    rc, res, _ = run_batch(built_lib, cuda, [(a, b, g, n, True)])
    assert rc == 0, _native.last_error()
    check_job((a, b, g, n, True), res[0], 2)
