"""Scratch of the read-outs: bounded for states near a GPU's capacity, and the routes
that take less give the same results (against complex128 NumPy) and stay inside it.
"""
import ctypes

import numpy as np
import pytest
import torch

from mpsim_gb300 import MPS, _native
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


@pytest.mark.parametrize("nbits,chi,n,d", [(4096, 256, 64, 2), (1, 1, 1, 2), (4 * 10 ** 6, 1, 1000, 2),
                                           (10 ** 6, 16, 5000, 3), (10 ** 6, 256, 64, 2)])
def test_amplitude_scratch_is_bounded(built_lib, nbits, chi, n, d):
    """Two environments and 256 MiB, or a product of every digit, if that is more; it
    does not grow with the chain."""
    need = built_lib.mps_amplitudes_workspace_bytes(nbits, chi, n, d)
    env = nbits * chi * 8
    assert (d + 2) * env <= need <= max((d + 2) * env, 2 * env + (256 << 20))


@pytest.mark.gpu
def test_amplitudes_of_a_chain_listed_in_parts(cuda):
    """More sites than lists fit in 256 MiB (470 of them here), the last part shorter.  Sites
    of bond 1 with entries of modulus 1; a complex product is off by 2 sqrt(2) 2^-24."""
    rng = np.random.default_rng(2)
    n, count = 500, 140000
    phase = np.exp(2j * np.pi * rng.random((n, 1, 2, 1))).astype(np.complex64)
    bits = rng.integers(0, 2, (count, n), dtype=np.int8)
    ref = np.ones(count, np.complex128)
    for i in range(n):
        ref *= phase[i, 0, bits[:, i], 0].astype(np.complex128)
    mps = MPS.from_sites([torch.from_numpy(t).to(cuda) for t in phase], 2)
    assert np.max(np.abs(mps.amplitudes(bits) - ref)) <= n * 2 * np.sqrt(2) * EPS * np.max(np.abs(ref))


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
