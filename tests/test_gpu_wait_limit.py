"""A caller's wait_limit bounds the sweeps' waits, and nothing else cuts them short: the
warps of a CTA that wait for its loader hold on for as long as the loader may poll.
"""
import time

import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


def test_a_raised_limit_is_waited_for(built_lib, cuda):
    """One wait targets a round that never completes (the stall hook), so a call takes
    its limit's polls: 32 times the limit, 32 times as long (about 0.07 s and 2.3 s)."""
    rng = np.random.default_rng(3)
    a, b, g = make_job_inputs(rng, 64, 64, 64, 2)          # 128 columns: 15 rounds per sweep
    assert run_batch(built_lib, cuda, [(a, b, g, 64, True)])[0] == 0       # (loads the kernels)
    seconds = []
    for limit in (1 << 18, 32 << 18):
        t0 = time.perf_counter()
        rc, _, _ = run_batch(built_lib, cuda, [(a, b, g, 64, True)],
                             params=_native.SvdParams(0, 0.0, 0, 0, limit, 1))
        seconds.append(time.perf_counter() - t0)
        assert rc == _native.MPS_ERR_TIMEOUT
    assert seconds[1] > 24 * seconds[0], seconds
