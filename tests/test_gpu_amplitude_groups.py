"""Sampled amplitudes through their grouping by digit: one and several chunks of 4096
bitstrings, both row tiles (64 x 64 ones from 152 tiles on), digits that a site does not
have, and the smallest workspace, against complex128 NumPy.

Bound: an entry of a site's product sums k complex terms, whose rounding errors add like
a random walk: 2 sqrt(k + 4) 2^-24 of the product's 2-norm for random sites, and at
most n times that over a chain of n, relative to the 2-norm over all amplitudes.  (Operands
of 11 bits would be off by some 5e-4 a site, 40 times as much at k = 256.)
"""
import ctypes

import numpy as np
import pytest
import torch

from mpsim_gb300 import MPS, _native
from test_gpu_readout_tiles import EPS, _chain

pytestmark = pytest.mark.gpu
GUARD = 4096


def _bits(rng, d, count, n):
    bits = rng.integers(0, d, (count, n)).astype(np.int8)
    bits[: count // 2, ::2] = 0                       # groups of uneven length
    return bits


def _exact(sites, bits):
    env = np.ones((len(bits), 1), np.complex128)
    for i, s in enumerate(sites):
        out = np.zeros((len(bits), s.shape[2]), np.complex128)
        for x in range(s.shape[1]):
            out[bits[:, i] == x] = env[bits[:, i] == x] @ s[:, x].astype(np.complex128)
        env = out
    return env[:, 0]


def _check(got, ref, bonds):
    tol = (len(bonds) - 1) * 2 * np.sqrt(max(bonds) + 4) * EPS
    assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("d,bonds,count", [
    (2, [1, 2, 256, 64, 1], 3000),                    # 64 x 64 tiles, one chunk
    (2, [1, 2, 130, 256, 200, 16, 1], 4100),          # the same, a second chunk of 4
    (3, [1, 3, 40, 130, 7, 1], 9000),
    (2, [1, 5, 33, 7, 1], 4096),                      # 32 x 32 tiles
    (2, [1, 5, 33, 7, 1], 4097),
    (5, [1, 5, 20, 1], 12289),
    (2, [1, 1, 1, 1], 140000)])                       # 35 chunks: more than a warp counts
def test_chunks_and_tiles(cuda, d, bonds, count):
    rng = np.random.default_rng(count + sum(bonds))
    sites = _chain(rng, d, bonds)
    bits = _bits(rng, d, count, len(sites))
    mps = MPS.from_sites([torch.from_numpy(s).to(cuda) for s in sites], d)
    _check(mps.amplitudes(bits), _exact(sites, bits), bonds)


def _call(lib, cuda, sites, bits, d, bonds, nbytes):
    """mps_amplitudes in a workspace of nbytes, nothing written beyond."""
    n, count = len(sites), len(bits)
    dev = [torch.from_numpy(s).to(cuda) for s in sites]
    ptrs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in dev])
    chis = (ctypes.c_int * (n + 1))(*bonds)
    b = torch.from_numpy(bits).to(cuda)
    out = torch.full((count,), float("nan"), dtype=torch.complex64, device=cuda)
    ws = torch.full((nbytes + GUARD,), 0x5a, dtype=torch.uint8, device=cuda)
    rc = lib.mps_amplitudes(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ptrs, chis, n, d,
                            ctypes.c_void_p(b.data_ptr()), count, ctypes.c_void_p(out.data_ptr()),
                            ctypes.c_void_p(ws.data_ptr()), nbytes)
    torch.cuda.synchronize()
    assert bool((ws[nbytes:] == 0x5a).all())
    return rc, out.cpu().numpy()


@pytest.mark.parametrize("d,bonds,count", [(2, [1, 33, 20, 2, 1], 300), (3, [1, 40, 9, 1], 5000),
                                           (2, [1, 2, 256, 64, 1], 3000)])
def test_digits_a_site_does_not_have(built_lib, cuda, d, bonds, count):
    rng = np.random.default_rng(count)
    sites = _chain(rng, d, bonds)
    n = len(sites)
    bits = _bits(rng, d, count, n)
    rows = rng.choice(count, count // 5, replace=False)
    bits[rows, rng.integers(0, n, len(rows))] = rng.choice([-128, -1, d, 127], len(rows))
    nbytes = built_lib.mps_amplitudes_workspace_bytes(count, max(bonds), n, d)
    rc, got = _call(built_lib, cuda, sites, bits, d, bonds, nbytes)
    assert rc == 0, _native.last_error()
    assert np.all(got[rows] == 0)
    _check(got, _exact(sites, bits), bonds)


@pytest.mark.parametrize("d,bonds,count", [
    (2, [1, 2] + [4] * 27 + [2, 1], 5),               # no room for the groups
    (2, [1, 2, 1, 1, 2, 1], 9000),
    (3, [1, 40, 9, 40, 1], 700)])                     # room for them
def test_smallest_workspace(built_lib, cuda, d, bonds, count):
    rng = np.random.default_rng(count)
    sites = _chain(rng, d, bonds)
    bits = _bits(rng, d, count, len(sites))
    bits[1, 2] = d
    nbytes = (count * d * max(bonds) + 2 * count * max(bonds)) * 8
    rc, _ = _call(built_lib, cuda, sites, bits, d, bonds, nbytes - 8)
    assert rc == _native.MPS_ERR_WORKSPACE
    rc, got = _call(built_lib, cuda, sites, bits, d, bonds, nbytes)
    assert rc == 0 and got[1] == 0
    _check(got, _exact(sites, bits), bonds)
