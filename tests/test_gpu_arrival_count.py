"""The reductions that a last-arriving block completes (the sensitivity, the adjoint viscosity's sums):
with their arrival count left where calls that overlapped may leave it, the next call gives the
same bits as ever."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest
import torch

from adfvm_gb300 import _lib as L
from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope='module')
def probe():
    L.lib()
    out = os.path.join(tempfile.mkdtemp(prefix='arrival_'), 'arrival_probe.so')
    where = os.path.dirname(L.LIB_PATH)
    subprocess.check_call([os.environ.get('NVCC', 'nvcc'), '-gencode', 'arch=compute_103a,code=sm_103a', '-O2',
                           '-std=c++17', '--expt-relaxed-constexpr', '-shared', '-cudart', 'shared', '-Xcompiler', '-fPIC',
                           '-I' + os.path.join(ROOT, 'include'), '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc'),
                           os.path.join(ROOT, 'tests', 'native', 'arrival_probe.cu'), '-o', out, '-L' + where,
                           '-l:' + os.path.basename(L.LIB_PATH), '-Xlinker', '-rpath=' + where])
    return C.CDLL(out)


@pytest.mark.parametrize('value', [0, 1, 2, 1000, 70000])
@pytest.mark.parametrize('sizes', [(1,), (700, 3), (300000, 0, 257), (5000,) * 17])
def test_sensitivity(probe, value, sizes):
    g = [torch.arange(n, dtype=torch.float64, device='cuda') % 7 - 3 for n in sizes]
    p = [torch.arange(n, dtype=torch.float64, device='cuda') % 5 - 2 for n in sizes]
    want = sum(float((a * b).sum()) for a, b in zip(g, p))          # (whole numbers: exact)
    k = len(sizes)
    partials = torch.empty(1024 * k, dtype=torch.float64, device='cuda')
    tail = torch.empty(2, dtype=torch.float64, device='cuda')
    torch.cuda.synchronize()
    out = C.c_double()
    st = probe.sensitivity_after(C.c_uint(value), k, (C.c_void_p * k)(*[t.data_ptr() for t in g]),
                                 (C.c_void_p * k)(*[t.data_ptr() for t in p]), (C.c_int64 * k)(*sizes),
                                 C.c_void_p(partials.data_ptr()), C.c_void_p(tail.data_ptr()), C.byref(out))
    assert st == 0
    assert out.value == want


def test_a_context(probe):
    case = cases.box(12)
    rcf = RCF(case.build_mesh(), case.bc, objective=case.objective, **case.config)
    rng = np.random.default_rng(9)
    x = [torch.as_tensor(a).cuda() for a in cases.conservative(case)]
    seeds = [torch.as_tensor(rng.standard_normal(t.shape)).cuda() for t in x]

    def both():
        a = [t.clone() for t in seeds]
        its = rcf.adjoint_viscosity(*x, a, 1e-4, 'turkel', 1.0)
        return [rcf.sensitivity([t.reshape(-1) for t in x], [t.reshape(-1) for t in seeds]), its] + a
    want = both()
    for value in (1, 3, 1000):
        assert probe.set_counters(rcf._ctx, C.c_uint(value)) == 0
        got = both()
        assert got[:2] == want[:2]
        assert all(torch.equal(p, q) for p, q in zip(got[2:], want[2:]))
