"""The FP32 contexts' pairs of floats (adfvm_gb300/csrc/ff32.cuh) against extended precision: what they
take comes out correctly rounded (they give up, with nothing written, where their error could decide
a rounding), which is nearly all of a flow's values; values out of their range, infinities and NaN
are refused with nothing written."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
AIR = (0.4, 717.5)


@pytest.fixture(scope='module')
def lib():
    out = os.path.join(tempfile.mkdtemp(prefix='ff32_'), 'ff.so')
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-ffp-contract=off', '-shared', '-fPIC',
                           '-I' + os.path.join(ROOT, 'include'), '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc'),
                           os.path.join(ROOT, 'tests', 'native', 'ff_host.cpp'), '-o', out])
    return C.CDLL(out)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _states(mach, n=20000):
    rng = np.random.default_rng(4)
    T, p = 300 * (1 + 0.1 * rng.standard_normal(n)), 1e5 * (1 + 0.1 * rng.standard_normal(n))
    rho = p / (AIR[0] * AIR[1] * T)
    U = mach * 347 * rng.standard_normal((n, 3))
    s = np.empty((n, 6), np.float32)
    s[:, 0] = rho
    s[:, 1:4] = rho[:, None] * U
    s[:, 4] = rho * (AIR[1] * T + 0.5 * (U ** 2).sum(1))
    s[:, 5] = 1 / s[:, 0]
    return s


@pytest.mark.parametrize('mach', [0.0, 1e-3, 0.1, 1.0, 5.0])
@pytest.mark.parametrize('gauge', [(0.0, 0.0), (1e5, 300.0)])
def test_primitives(lib, mach, gauge):
    s = _states(mach)
    out, ok = np.empty((len(s), 2), np.float32), np.empty(len(s), np.int32)
    lib.ff_prims(_p(np.array(AIR + gauge)), _p(s), len(s), _p(out), _p(ok))
    ok = ok.astype(bool)
    assert ok.mean() > 0.9
    d = s.astype(np.longdouble)
    e = d[:, 4] - (d[:, 1:4] ** 2).sum(1) * d[:, 5] / 2
    for got, want in ((out[:, 0], AIR[0] * e - gauge[0]), (out[:, 1], e * d[:, 5] / np.longdouble(AIR[1]) - gauge[1])):
        assert np.array_equal(got[ok], want.astype(np.float32)[ok])


def test_kinetic_gradient(lib):
    s, rng = _states(0.3), np.random.default_rng(8)
    n, obja, gauge = len(s), 0.7, (1e5, 300.0)
    v = np.empty((n, 6), np.float32)
    v[:, :3] = 100 * rng.standard_normal((n, 3))
    v[:, 3], v[:, 4] = 30 * rng.standard_normal(n), 1e4 * rng.standard_normal(n)
    v[:, 5] = 10.0 ** rng.uniform(-9, 0, n)
    g, ok = np.zeros((n, 5), np.float32), np.empty(n, np.int32)
    lib.ff_kinetic(_p(np.array(AIR + gauge)), C.c_double(obja), _p(v), n, _p(g), _p(ok))
    ok = ok.astype(bool)
    assert ok.mean() > 0.99
    d = v.astype(np.longdouble)
    T, p, V = d[:, 3] + gauge[1], d[:, 4] + gauge[0], d[:, 5]
    Rg = np.longdouble(AIR[1] * AIR[0])
    q = (d[:, :3] ** 2).sum(1) / 2 * obja * V
    want = np.stack([obja * p / (Rg * T) * d[:, k] * V for k in range(3)] + [-q * p / (Rg * T * T), q / (Rg * T)], 1)
    assert np.array_equal(g[ok], want.astype(np.float32)[ok]) and not g[~ok].any()


@pytest.mark.parametrize('column,value', [(0, 0.0), (0, -1.0), (0, np.inf), (0, np.nan), (0, 1e13), (1, np.inf),
                                          (2, np.nan), (3, 1e20), (4, 1e-20), (4, np.inf), (4, np.nan), (1, 1e3)])
def test_out_of_range(lib, column, value):
    s = _states(0.1)[:3].copy()
    s[1, column] = value          # (rhoU 1e3: no internal energy is left)
    out, ok = np.full((3, 2), 9, np.float32), np.empty(3, np.int32)
    lib.ff_prims(_p(np.array(AIR + (1e5, 300.0))), _p(s), 3, _p(out), _p(ok))
    assert list(ok) == [1, 0, 1] and np.all(out[1] == 9)
