"""Truncated SVDs of degenerate thetas: equal, zero and repeated columns, exact ties,
spectra of thirty decades.  Columns cancel to rounding noise and to norms whose squares
are no normal floats; the factors stay finite and the isometric one an isometry.
Checked like test_gpu_svd_kernel.py's jobs (same tolerances) against complex128 LAPACK.
"""
import numpy as np
import pytest

from mpsim_gb300 import _native
from test_gpu_svd_kernel import check_job, run_batch

pytestmark = pytest.mark.gpu


def _theta(kind, m, n, rng):
    x = rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))
    r = min(m, n)
    if kind == "constant":
        return np.ones((m, n), complex)
    if kind == "zero columns":
        x[:, ::3] = 0
        x[1::4] = 0
    elif kind == "repeated columns":
        x[:, 1::2] = x[:, 0:2 * (n // 2):2]
    elif kind == "repeated rows":
        x[1::2] = x[0:2 * (m // 2):2]
    elif kind == "permutation":
        x = np.zeros((m, n), complex)
        x[np.arange(r), rng.permutation(n)[:r]] = 1
    elif kind == "thirty decades":
        u, _, vh = np.linalg.svd(x, full_matrices=False)
        x = (u * 10.0 ** -np.linspace(0, 30, r)) @ vh
    return x


KINDS = ["constant", "zero columns", "repeated columns", "repeated rows", "permutation",
         "thirty decades"]


def _spec(kind, chil, chir, k, lc):
    """The job whose merged theta (identity gate) is this matrix."""
    m, n = 2 * chil, 2 * chir
    th = _theta(kind, m, n, np.random.default_rng(m + 1000 * n))
    if m >= n:
        a, b = th.reshape(chil, 2, n), np.eye(n).reshape(n, 2, chir)
    else:
        a, b = np.eye(m).reshape(chil, 2, m), th.reshape(m, 2, chir)
    return a.astype(np.complex64), b.astype(np.complex64), np.eye(4, dtype=np.complex64), k, lc


def _check(lib, cuda, specs, precision=_native.PRECISION_PLAIN):
    p = _native.SvdParams()
    p.precision = precision
    rc, res, _ = run_batch(lib, cuda, specs, params=p)
    assert rc == 0, _native.last_error()
    for spec, out in zip(specs, res):
        check_job(spec, out, 2)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("chil,chir,lc", [(8, 20, True), (33, 40, True), (40, 70, True), (64, 100, True),
                                          (70, 40, False), (100, 64, False), (60, 130, False)])
def test_rotations_accumulated(built_lib, cuda, kind, chil, chir, lc):
    """Jobs that accumulate V: every rotation of noise has to be one."""
    _check(built_lib, cuda, [_spec(kind, chil, chir, 2 * min(chil, chir), lc)])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("chil,chir,lc", [(8, 8, True), (33, 40, False), (40, 70, False), (64, 64, True),
                                          (64, 64, False), (100, 64, True), (64, 100, False),
                                          (128, 128, False), (300, 40, True)])
def test_left_factor_read_off_the_columns(built_lib, cuda, kind, chil, chir, lc):
    """Jobs without V: columns too short to be made orthogonal are completed, not divided
    by their norms; all singular vectors kept, and half of them."""
    k = 2 * min(chil, chir)
    _check(built_lib, cuda, [_spec(kind, chil, chir, k, lc), _spec(kind, chil, chir, k // 2, lc)])


@pytest.mark.parametrize("kind,chil,chir,lc", [
    ("constant", 384, 384, True), ("constant", 384, 384, False), ("repeated rows", 384, 384, True),
    ("repeated columns", 400, 400, False), ("repeated rows", 400, 400, True),
    ("constant", 450, 450, False), ("constant", 600, 60, True), ("repeated rows", 600, 60, True)])
def test_exactly_dependent_columns_end(built_lib, cuda, kind, chil, chir, lc):
    """Columns of an exactly dependent set shrink with every sweep; they are followed no
    further than they can be made orthogonal, within the sweep cap (768 columns: the
    factorised start's most; 800 and 900: without it; 1200 rows: column by column)."""
    _check(built_lib, cuda, [_spec(kind, chil, chir, min(chil, chir), lc)])


@pytest.mark.parametrize("kind", ["constant", "zero columns", "permutation", "thirty decades"])
@pytest.mark.parametrize("chil,chir", [(64, 64), (100, 64), (128, 128)])
def test_mixed(built_lib, cuda, kind, chil, chir):
    _check(built_lib, cuda, [_spec(kind, chil, chir, 2 * chir, True)], _native.PRECISION_MIXED)


@pytest.mark.parametrize("chil,chir,lc", [(64, 64, False), (288, 288, True), (288, 288, False),
                                          (150, 290, False), (512, 200, True), (600, 100, True)])
def test_constant_theta_keeps_its_accuracy(built_lib, cuda, chil, chir, lc):
    """Every product of a constant theta's factors sums equal terms, whose roundings all go
    one way.  In parts of 32 terms (two FMAs each) and their sums a product of K terms is
    off by (64 + K / 32) 2^-25 at most, 3e-6 here; twice that for the isometry and for the
    two factors' product beside what random thetas show (a single sum of K: 2 K 2^-25)."""
    spec = _spec("constant", chil, chir, 8, lc)
    rc, res, _ = run_batch(built_lib, cuda, [spec])
    assert rc == 0, _native.last_error()
    left = res[0]["a"].reshape(2 * chil, 8).astype(np.complex128)
    right = res[0]["b"].reshape(8, 2 * chir).astype(np.complex128)
    gram = left.conj().T @ left if lc else right @ right.conj().T
    assert np.max(np.abs(gram - np.eye(8))) <= 6e-6
    assert np.linalg.norm(left @ right - 1) <= 6e-6 * np.sqrt(left.shape[0] * right.shape[1])
