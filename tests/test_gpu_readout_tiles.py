"""The contraction kernels at the edges of their tiles (32 / 64 rows and columns,
8 / 16 of K), every conjugation and operand order, grouped amplitudes and the
two-directional sweeps on odd chains, against complex128 NumPy.

Bounds: an FP32 dot product of k complex terms is off by at most about
2 (k + 4) 2^-24 |row| |column|; the sweeps chain n such products of well
conditioned random sites, n times that of one site.
"""
import ctypes

import numpy as np
import pytest
import torch

from mpsim_gb300 import MPS, _native

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _rand(rng, *shape):
    return (rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 17), (32, 32, 16), (33, 65, 15), (64, 64, 8),
                                   (65, 130, 9), (7, 200, 300), (1300, 1281, 20), (5, 4, 0)])
@pytest.mark.parametrize("conj_a,conj_b", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("order", ["nn", "tt", "strided"])
def test_cgemm(built_lib, cuda, m, n, k, conj_a, conj_b, order):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    batch = 3 if m * n < 20000 else 1
    a, b = _rand(rng, batch, m, k), _rand(rng, batch, k, n)
    if order == "nn":
        ta, tb, sa, sb = a, b, (k, 1), (n, 1)
    elif order == "tt":
        ta, tb, sa, sb = a.transpose(0, 2, 1).copy(), b.transpose(0, 2, 1).copy(), (1, m), (1, k)
    else:                                          # neither stride is 1
        ta, tb = np.zeros((batch, m, 2 * k), np.complex64), np.zeros((batch, k, 3 * n), np.complex64)
        ta[..., ::2], tb[..., ::3] = a, b
        sa, sb = (2 * k, 2), (3 * n, 3)
    da, db = torch.from_numpy(ta).to(cuda), torch.from_numpy(tb).to(cuda)
    c = torch.full((batch, m, n), float("nan"), dtype=torch.complex64, device=cuda)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = built_lib.mps_cgemm(stream, m, n, k, p(da), sa[0], sa[1], conj_a, p(db), sb[0], sb[1],
                             conj_b, p(c), n, 1, batch, ta[0].size, tb[0].size, m * n)
    assert rc == 0, _native.last_error()
    x, y = a.astype(np.complex128), b.astype(np.complex128)
    x, y = (x.conj() if conj_a else x), (y.conj() if conj_b else y)
    ref = x @ y
    bound = 2 * (k + 4) * EPS * np.linalg.norm(x, axis=2)[:, :, None] * \
        np.linalg.norm(y, axis=1)[:, None, :]
    assert np.all(np.abs(c.cpu().numpy() - ref) <= bound + 1e-30)


def _chain(rng, d, bonds):
    return [(_rand(rng, bonds[i], d, bonds[i + 1]) / np.sqrt(2 * bonds[i] * d)).astype(np.complex64)
            for i in range(len(bonds) - 1)]


def _mps(sites, d, cuda):
    return MPS.from_sites([torch.from_numpy(s).to(cuda) for s in sites], d)


CHAINS = [(2, [1, 2, 1]), (2, [1, 2, 5, 1]), (2, [1, 33, 65, 31, 64, 1]), (3, [1, 3, 40, 130, 7, 2, 1]),
          (2, [1, 17, 1, 40, 9, 1])]


@pytest.mark.parametrize("d,bonds", CHAINS)
def test_sweeps(cuda, d, bonds):
    rng = np.random.default_rng(sum(bonds))
    sites = _chain(rng, d, bonds)
    other = _chain(rng, d, [1] + [b + 3 for b in bonds[1:-1]] + [1])
    n = len(sites)
    a, b = _mps(sites, d, cuda), _mps(other, d, cuda)

    def env(x, y):
        e = np.ones((1, 1), np.complex128)
        for s, t in zip(x, y):
            e = np.einsum("ab,axc,bxd->cd", e, s.astype(np.complex128), t.astype(np.complex128).conj())
        return e[0, 0]

    scale = np.sqrt(abs(env(sites, sites)) * abs(env(other, other)))
    tol = n * 2 * (d * max(bonds) + 8) * EPS
    assert abs(a.inner_product(b) - env(sites, other)) <= tol * scale
    assert abs(a.inner_product(a) - env(sites, sites)) <= tol * abs(env(sites, sites))
    marg = a.site_marginals()
    norm = abs(env(sites, sites))
    for i in range(n):
        for x in range(d):
            cut = [s.copy() for s in sites]
            for y in range(d):
                if y != x:
                    cut[i][:, y] = 0
            assert abs(marg[i, x] - env(cut, cut).real) <= tol * norm + EPS * norm


@pytest.mark.parametrize("d,bonds", CHAINS)
@pytest.mark.parametrize("count", [1, 31, 65, 700])
def test_amplitudes(cuda, d, bonds, count):
    rng = np.random.default_rng(count + sum(bonds))
    sites = _chain(rng, d, bonds)
    bits = rng.integers(0, d, (count, len(sites))).astype(np.int8)
    bits[: count // 2] = 0                            # one digit only in half of the rows
    got = _mps(sites, d, cuda).amplitudes(bits)
    for row, v in zip(bits, got):
        e, size = np.ones((1, 1), np.complex128), 1.0
        for s, x in zip(sites, row):
            m = s[:, x].astype(np.complex128)
            e, size = e @ m, size * np.linalg.norm(m)
        tol = len(sites) * 2 * (max(bonds) + 4) * EPS
        assert abs(v - e[0, 0]) <= tol * size + 1e-30
