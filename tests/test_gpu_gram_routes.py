"""Gram sweeps where the loader claims ahead (more than four visits an SM and round) and
where the list of jobs is longer than a CTA's copy of it (256), and the sweeps queued
ahead of the host from several threads and streams at once.  Checked like
test_gpu_svd_kernel.py's jobs (same tolerances) against complex128 LAPACK.
"""
import threading

import numpy as np
import pytest
import torch

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, make_job_inputs, run_batch

pytestmark = pytest.mark.gpu


def _specs(rng, count, top):
    specs = []
    for q in range(count):
        chil, chir = int(rng.integers(1, top + 1)), int(rng.integers(1, top + 1))
        if q == 0:
            chil = chir = top                          # 2 top columns: the call's rounds and pairs
        a, b, g = make_job_inputs(rng, chil, max(chil, chir), chir, 2, scale=1.0 / top)
        specs.append((a, b, g, min(chil, chir), bool(q % 3)))
    return specs


@pytest.mark.parametrize("count,top", [(300, 64), (120, 64)])
def test_many_visits(built_lib, cuda, count, top):
    """128 columns: 8 visits a job and round, 2400 and 960 for at most 608 slots."""
    specs = _specs(np.random.default_rng(count), count, top)
    rc, res, _ = run_batch(built_lib, cuda, specs)
    assert rc == 0, _native.last_error()
    for spec, out in zip(specs, res):
        check_job(spec, out, 2)


def test_threads_and_streams(built_lib, cuda):
    """Calls of two threads, each on a stream of its own, at the same time."""
    work = [[_specs(np.random.default_rng(10 * t + i), 3 + i, 12 + 9 * i) for i in range(5)]
            for t in range(2)]
    results, errors = [[], []], []

    def calls(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for specs in work[t]:
                    results[t].append(run_batch(built_lib, cuda, specs))
        except Exception as e:                         # noqa: BLE001 (raised in the main thread)
            errors.append(e)
    threads = [threading.Thread(target=calls, args=(t,)) for t in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
    for t in range(2):
        for specs, (rc, res, _) in zip(work[t], results[t]):
            assert rc == 0
            for spec, out in zip(specs, res):
                check_job(spec, out, 2)
