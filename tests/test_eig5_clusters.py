"""The largest eigenvalue of a symmetric 5x5 (adfvm_gb300/csrc/eig5.cuh) where two to five eigenvalues
nearly coincide, against LAPACK: within 4e-15 of the Frobenius norm, as for other matrices (the
reduction and LAPACK each err by a small multiple of 2^-53 times it). Its conversions: low is x
truncated to a float, zero below 2^-120, high is exact. On the host and, marked gpu, on the device."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INCLUDES = ['-I' + os.path.join(ROOT, 'include'), '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc')]
SPREADS = [10.0 ** -k for k in range(4, 17)]
SIZES = [2, 3, 4, 5]


def _build(where):
    out = os.path.join(tempfile.mkdtemp(prefix='eig5_'), 'eig5.so')
    source = os.path.join(ROOT, 'tests', 'native', 'eig5_parts_host.cpp' if where == 'host' else 'eig5_probe.cu')
    if where == 'host':
        subprocess.check_call(['g++', '-O2', '-std=c++17', '-shared', '-fPIC'] + INCLUDES + [source, '-o', out])
    else:
        subprocess.check_call([os.environ.get('NVCC', 'nvcc'), '-gencode', 'arch=compute_103a,code=sm_103a', '-O3',
                               '-std=c++17', '--expt-relaxed-constexpr', '-shared', '-Xcompiler', '-fPIC'] + INCLUDES +
                              [source, '-o', out])
    lib = C.CDLL(out)

    def call(name, x, per, out_type):
        x = np.ascontiguousarray(x)
        r = np.empty(x.size // per, out_type)
        f = getattr(lib, name + '_' + where)
        st = f(x.ctypes.data_as(C.c_void_p), C.c_int(len(r)), r.ctypes.data_as(C.c_void_p))
        assert where == 'host' or st == 0
        return r
    return call


@pytest.fixture(scope='module', params=['host', pytest.param('device', marks=pytest.mark.gpu)])
def eig5(request):
    return _build(request.param)


def _error(eig5, a):
    a = (a + a.transpose(0, 2, 1)) / 2
    norm = np.sqrt((a * a).sum(axis=(1, 2)))
    return np.abs(eig5('eig5', a, 25, np.float64) - np.linalg.eigvalsh(a)[:, -1]) / norm


@pytest.mark.parametrize('spread', SPREADS)
def test_all_five_nearly_equal(eig5, spread):
    rng = np.random.default_rng(31)
    n = 50000
    a = np.eye(5) * rng.standard_normal((n, 1, 1)) + spread * rng.standard_normal((n, 5, 5))
    assert _error(eig5, a).max() <= 4e-15


@pytest.mark.parametrize('size', SIZES)
def test_clusters_of_any_size_and_spread(eig5, size):
    rng = np.random.default_rng(size)
    n = 50000
    q = np.linalg.qr(rng.standard_normal((n, 5, 5)))[0]
    w = rng.standard_normal((n, 5)) - 4
    w[:, :size] = rng.standard_normal((n, 1)) + 10.0 ** rng.uniform(-16, -1, (n, 1)) * rng.standard_normal((n, size))
    assert _error(eig5, np.einsum('nij,nj,nkj->nik', q, w, q)).max() <= 4e-15


def test_the_conversions(eig5):
    rng = np.random.default_rng(5)
    x = np.ldexp(rng.uniform(1, 2, 200000), rng.integers(-140, 100, 200000)) * rng.choice([-1.0, 1.0], 200000)
    x[:3] = 0.0, -0.0, 2.0 ** -120
    with np.errstate(over='ignore', under='ignore'):
        f = x.astype(np.float32)
    f = np.where(np.abs(f.astype(np.float64)) > np.abs(x), np.nextafter(f, np.float32(0)), f)
    want = np.where(np.abs(x) < 2.0 ** -120, np.float32(0), f)
    assert np.array_equal(eig5('low', x, 1, np.float32), want)
    normal = want[np.abs(want) >= 2.0 ** -120]
    assert np.array_equal(eig5('high', normal, 1, np.float64), normal.astype(np.float64))
    assert np.array_equal(eig5('high', np.zeros(2, np.float32), 1, np.float64), np.zeros(2))
