"""A caller's own tolerance is the one that decides, also where its square is no float."""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol,rc", [(0.0, 0), (1e-6, 0), (1e-18, _native.MPS_ERR_NOT_CONVERGED),
                                    (1e-30, _native.MPS_ERR_NOT_CONVERGED)])
def test_tolerance(built_lib, cuda, tol, rc):
    """Cosines of rounding noise, 1e-8 and more, never pass one of 1e-18 or 1e-30."""
    rng = np.random.default_rng(4)
    spec = make_job_inputs(rng, 32, 32, 32, 2) + (64, True)
    got, res, p = run_batch(built_lib, cuda, [spec], params=_native.SvdParams(20, tol))
    assert got == rc, _native.last_error()
    if rc == 0:
        check_job(spec, res[0], 2)
    else:
        assert p.sweeps_out == 20 and res[0]["status"] & _native.STATUS_NOT_CONVERGED
