"""Scratch of the read-outs: bounded for states near a GPU's capacity, and the routes
that take less give the same results (against complex128 NumPy) and stay inside it.
"""
import ctypes

import numpy as np
import pytest
import torch

from mpsim_gb300 import _native
from test_gpu_readout_tiles import CHAINS, EPS, _chain

GUARD = 4096


def _ints(values):
    return (ctypes.c_int * len(values))(*values)


def _lean_marginals(chis, d):
    n, mx = len(chis) - 1, max(chis)
    cells = sum(c * c for c in chis[:n]) + 2 * (1 + d) * mx * mx
    return (cells * 8 + n * d * 4 + 1024 + 255) // 256 * 256


@pytest.mark.parametrize("n,chi,d", [(48, 128, 2), (1000, 800, 2), (1500, 590, 3), (40000, 256, 2)])
def test_marginal_scratch_is_bounded(built_lib, n, chi, d):
    """At most 16 GiB, or the left environments of a state too large for that: 1 / d of the
    state, not twice it."""
    chis = [1] + [chi] * (n - 1) + [1]
    need = built_lib.mps_marginals_workspace_bytes(_ints(chis), n, d)
    assert 0 < need <= max(16 << 30, _lean_marginals(chis, d))


@pytest.mark.gpu
@pytest.mark.parametrize("d,bonds", CHAINS + [(2, [1, 2, 4, 70, 70, 70, 4, 2, 1])])
def test_marginals_in_the_least_scratch(built_lib, cuda, d, bonds):
    rng = np.random.default_rng(sum(bonds) + 1)
    sites = _chain(rng, d, bonds)
    n = len(sites)
    # (of a few sites the products are fewer than the environments' scratch)
    nbytes = min(_lean_marginals(bonds, d),
                 built_lib.mps_marginals_workspace_bytes(_ints(bonds), n, d))
    dev = [torch.from_numpy(s).to(cuda) for s in sites]
    ptrs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in dev])
    ws = torch.full((nbytes + GUARD,), 0x5a, dtype=torch.uint8, device=cuda)
    out = np.full((n, d), np.nan, np.float32)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(size):
        return built_lib.mps_site_marginals(stream, ptrs, _ints(bonds), n, d,
                                            ctypes.c_void_p(ws.data_ptr()), size,
                                            out.ctypes.data_as(ctypes.c_void_p))
    assert call(nbytes - 256) == _native.MPS_ERR_WORKSPACE
    assert call(nbytes) == 0, _native.last_error()
    assert bool((ws[nbytes:] == 0x5a).all())

    def norm(chain):
        e = np.ones((1, 1), np.complex128)
        for s in chain:
            s = s.astype(np.complex128)
            e = np.einsum("ab,axc,bxd->cd", e, s, s.conj(), optimize=True)
        return e[0, 0].real

    # n products of terms d max(bonds) long (see test_gpu_readout_tiles.py), one rounding
    tol = (n * 2 * (d * max(bonds) + 8) + 1) * EPS * norm(sites)
    for i in range(n):
        for x in range(d):
            cut = [s.copy() for s in sites]
            cut[i][:, [y for y in range(d) if y != x]] = 0
            assert abs(out[i, x] - norm(cut)) <= tol
