"""The largest eigenvalue of a symmetric 5x5 (adfvm_gb300/csrc/eig5.cuh, the viscosity's) against
LAPACK: within 4e-15 of the Frobenius norm (the reduction and LAPACK each err by a small multiple
of 2^-53 times it), on matrices with separated, coinciding and nearly coinciding largest
eigenvalues, graded and nearly diagonal ones, one-sided spectra and extreme scales; NaN for a
non-finite entry, 0 for the zero matrix."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope='module')
def eig5():
    out = os.path.join(tempfile.mkdtemp(prefix='eig5_'), 'eig5.so')
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-shared', '-fPIC', '-I' + os.path.join(ROOT, 'include'),
                           '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc'),
                           os.path.join(ROOT, 'tests', 'native', 'eig5_host.cpp'), '-o', out])
    lib = C.CDLL(out)
    dp = C.POINTER(C.c_double)
    lib.eig5_host.argtypes = [dp, C.c_int, dp]

    def run(a):
        a = np.ascontiguousarray(a, np.float64)
        r = np.empty(len(a))
        lib.eig5_host(a.ctypes.data_as(dp), len(a), r.ctypes.data_as(dp))
        return r
    return run


def _matrices(kind, n=4000):
    rng = np.random.default_rng(23)
    a = rng.standard_normal((n, 5, 5))
    a = a + a.transpose(0, 2, 1)
    q = np.linalg.qr(rng.standard_normal((n, 5, 5)))[0]
    spread = lambda w: np.einsum('nij,nj,nkj->nik', q, w, q)
    if kind == 'graded':
        s = 10.0 ** np.array([0, -3, -6, -9, -12])
        return a * s[:, None] * s
    if kind == 'nearly diagonal':
        return np.where(np.eye(5) > 0, a, 1e-9 * a)
    if kind == 'double':
        w = rng.standard_normal((n, 5)) - 3
        w[:, 0] = w[:, 1] = 2.0
        return spread(w)
    if kind == 'nearly double':
        w = rng.standard_normal((n, 5)) - 3
        w[:, 0], w[:, 1] = 2.0, 2.0 - 10.0 ** rng.uniform(-14, -1, n)
        return spread(w)
    if kind == 'identity':
        return np.eye(5) * rng.standard_normal((n, 1, 1))
    if kind == 'negative':
        return spread(-1 - rng.random((n, 5)))
    if kind == 'rank one':
        v = rng.standard_normal((n, 5, 1))
        return v @ v.transpose(0, 2, 1)
    if kind == 'tiny':
        return a * 1e-200
    if kind == 'huge':
        return a * 1e150
    return a


@pytest.mark.parametrize('kind', ['random', 'graded', 'nearly diagonal', 'double', 'nearly double', 'identity',
                                  'negative', 'rank one', 'tiny', 'huge'])
def test_largest_eigenvalue_matches_lapack(eig5, kind):
    a = _matrices(kind)
    a = (a + a.transpose(0, 2, 1)) / 2
    norm = np.sqrt((a / np.abs(a).max(axis=(1, 2), keepdims=True)) ** 2).sum(axis=(1, 2)) ** 0.5 * \
        np.abs(a).max(axis=(1, 2))
    err = np.abs(eig5(a) - np.linalg.eigvalsh(a)[:, -1]) / norm
    print(kind, err.max())
    assert err.max() <= 4e-15


def test_zero_and_non_finite(eig5):
    a = np.zeros((3, 5, 5))
    a[1, 2, 3] = a[1, 3, 2] = np.nan
    a[2, 0, 0], a[2, 1, 1] = 1.0, np.inf
    r = eig5(a)
    assert r[0] == 0 and np.isnan(r[1]) and np.isnan(r[2])
