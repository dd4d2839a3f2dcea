"""The FP64 arithmetic of the large meshes' face kernels on the integer pipes
(adfvm_gb300/csrc/soft64.cuh) and the face kernels that use it.

* soft_mul: the bits of the IEEE product for significands of every length (ties and exact products
  among them) while the result is normal; a zero of either sign for zeros; zero for results below
  2^-1022 (2^-1021 at most).
* soft_rcp, soft_rsqrt: within 0.502 units in the last place of the exact value (numpy long
  double) inside their window 2^[-64, 64], flagged outside it and for 0, inf, NaN.
* Meshes above the small-grid limit (their flux and VJP take this path): step and adjoint against
  the oracle within 1e-12, taped and untaped; a uniform flow (1/eps = 1e30 of the entropy fix);
  a state with non-finite cells, whose faces are evaluated again with the hardware operations:
  the same non-finite entries as the oracle and 1e-12 elsewhere; seeds scaled by 2^100 (again
  evaluated by the hardware) and by 2^-1040 and 2^-900: the VJP is linear, so its results scale
  with them - 2^100 and 2^-900 within 1e-13 (the two paths round alike but for the reciprocals
  held in the tape, which both read), 2^-1040 within the absolute 2^-1020 that results below
  2^-1021 may lose at each of the step's few hundred products."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF
from oracle import torch_ref
from tests import golden_cases as G

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMALL_ITEMS = 32 * 4 * 152 * 8          # SMALL_WARPS warps (csrc/ctx.cuh)


@pytest.fixture(scope='module')
def probe():
    out = os.path.join(tempfile.mkdtemp(prefix='soft64_'), 'soft64_probe.so')
    subprocess.check_call([os.environ.get('NVCC', 'nvcc'), '-gencode', 'arch=compute_103a,code=sm_103a', '-O3',
                           '-std=c++17', '--expt-relaxed-constexpr', '-shared', '-Xcompiler', '-fPIC',
                           '-I' + os.path.join(ROOT, 'include'), '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc'),
                           os.path.join(ROOT, 'tests', 'native', 'soft64_probe.cu'), '-o', out])
    lib = C.CDLL(out)
    dp = C.POINTER(C.c_double)
    lib.soft64_probe.argtypes = [dp, dp, dp, C.c_int]

    def run(x, y):
        x, y = np.ascontiguousarray(x, np.float64), np.ascontiguousarray(y, np.float64)
        r = np.empty((5, len(x)))
        assert lib.soft64_probe(x.ctypes.data_as(dp), y.ctypes.data_as(dp), r.ctypes.data_as(dp), len(x)) == 0
        return r
    return run


def _numbers(rng, n, lo, hi):
    """Random significands, a third of them cut to a random length or ending in ones, both signs."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    cut = rng.integers(0, 52, n, dtype=np.uint64)
    kind = rng.integers(0, 6, n)
    m = np.where(kind == 0, (m >> cut) << cut, m)
    m = np.where(kind == 1, m | ((np.uint64(1) << cut) - np.uint64(1)), m)
    e = rng.integers(1023 + lo, 1023 + hi, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.parametrize('lo,hi', [(-60, 60), (-500, 500), (-1022, 300)])
def test_product_has_the_bits_of_the_hardware(probe, lo, hi):
    rng = np.random.default_rng(17)
    n = 400000
    x, y = _numbers(rng, n, lo, hi), _numbers(rng, n, lo, hi)
    x[:64] = np.where(np.arange(64) % 2, 0.0, -0.0)
    y[32:96] = 0.0
    with np.errstate(under='ignore'):
        want = x * y
    got = probe(x, y)[0]
    normal = np.abs(want) >= 2.0 ** -1021
    assert normal.sum() > n // 3
    assert np.array_equal(got[normal].view(np.uint64), want[normal].view(np.uint64))
    assert not got[np.abs(want) < 2.0 ** -1022].any()
    edge = ~normal & (np.abs(want) >= 2.0 ** -1022)
    assert np.all((got[edge] == 0) | (got[edge] == want[edge]))


def test_reciprocal_and_square_root_round_within_0502_ulp(probe):
    rng = np.random.default_rng(18)
    x = _numbers(rng, 400000, -64, 64)
    r = probe(x, x)
    ulps = lambda got, exact: (np.abs(got.astype(np.longdouble) - exact) /
                               np.spacing(np.abs(exact.astype(np.float64))).astype(np.longdouble)).astype(float)
    xl = x.astype(np.longdouble)
    assert not r[2].any()
    e = ulps(r[1], 1 / xl).max()
    print('soft_rcp', e)
    assert e <= 0.502
    pos = x > 0
    assert not r[4][pos].any() and r[4][~pos].all()
    e = ulps(r[3][pos], 1 / np.sqrt(xl[pos])).max()
    print('soft_rsqrt', e)
    assert e <= 0.502
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -65, 2.0 ** 66, 1e300])
    r = probe(odd, odd)
    assert r[2].all() and r[4].all()


@pytest.fixture(scope='module')
def large():
    """A box whose faces are just past the small-grid limit, and its oracle."""
    case = cases.box(38)
    mesh = case.build_mesh()
    assert SMALL_ITEMS < mesh.nFaces < 1.1 * SMALL_ITEMS and mesh.nFaces % 128
    prob = torch_ref.Problem(mesh, case.bc, case.config, case.objective)
    return case, mesh, prob, RCF(mesh, case.bc, objective=case.objective, **case.config)


def _state(case, kind, seed=5):
    rng = np.random.default_rng(seed)
    x = [torch.as_tensor(a) for a in cases.conservative(case)]
    if kind == 'uniform':
        x[1] = torch.zeros_like(x[1])
        x[1][:, 0] = 40.0 * x[0][:, 0]
        x[2] = torch.full_like(x[2], 2.6e5)
    else:
        x[0] = x[0] * (1 + 1e-3 * torch.as_tensor(rng.standard_normal(x[0].shape)))
    seeds = [torch.as_tensor(rng.standard_normal(t.shape)) / max(1.0, float(t.abs().max())) for t in x]
    return x, seeds


@pytest.mark.parametrize('kind', ['noise', 'uniform'])
@pytest.mark.parametrize('taped', [True, False])
def test_large_mesh_matches_oracle(large, kind, taped):
    case, mesh, prob, rcf = large
    x, seeds = _state(case, kind)
    ref = prob.step(*x, case.dt)
    d, s = [t.cuda() for t in x], [t.cuda() for t in seeds]
    kw = dict(stages=rcf.stage_buffer(), tape=rcf.tape_buffer()) if taped else {}
    out = rcf.step(*d, case.dt, **kw)
    for i in range(3):
        assert G.rel_err(out[i].cpu().numpy(), ref[i].numpy()) < 1e-12, (kind, i)
    assert abs(out[3] - float(ref[3])) <= 1e-12 * abs(float(ref[3]))
    a = rcf.adjoint_step(*d, case.dt, s, obja=1.0, **kw)
    if kind == 'uniform':
        # (|U_L.n - U_R.n| is at its kink in a uniform flow: the VJP is one of its one-sided values)
        assert all(bool(torch.isfinite(t).all()) for t in a[:3])
        return
    refa = torch_ref.vjp_step(prob, *x, case.dt, None, seeds, obja=1.0)
    for i in range(3):
        assert G.rel_err(a[i].cpu().numpy(), refa[i].numpy()) < 1e-12, (kind, i)


def test_non_finite_cells_match_oracle(large):
    case, mesh, prob, rcf = large
    x, _ = _state(case, 'noise')
    x[0][1234, 0] = float('nan')
    x[2][30000, 0] = float('inf')
    x[1][20000, 1] = 1e200
    ref = prob.step(*x, case.dt)
    d = [t.cuda() for t in x]
    out = rcf.step(*d, case.dt, want_scalars=False)
    for i in range(3):
        got, want = out[i].cpu().numpy(), ref[i].numpy()
        fine = np.isfinite(want)
        assert 0 < (~fine).sum() < fine.size // 2
        assert np.array_equal(np.isfinite(got), fine)
        small = fine & (np.abs(np.where(fine, want, 0)) < 1e8)      # (cells 1e200 has not reached)
        assert np.abs(got[small] - want[small]).max() <= 1e-12 * np.abs(want[small]).max()


@pytest.mark.parametrize('power', [100, -900, -1040])
def test_vjp_scales_with_its_seeds(large, power):
    case, mesh, prob, rcf = large
    x, seeds = _state(case, 'noise')
    d = [t.cuda() for t in x]
    kw = dict(stages=rcf.stage_buffer(), tape=rcf.tape_buffer())
    rcf.step(*d, case.dt, **kw)
    base = rcf.adjoint_step(*d, case.dt, [t.cuda() for t in seeds], obja=0.0, **kw)
    scaled = rcf.adjoint_step(*d, case.dt, [torch.ldexp(t, torch.tensor(power)).cuda() for t in seeds], obja=0.0, **kw)
    for i in range(3):
        got, want = scaled[i], torch.ldexp(base[i], torch.tensor(power, device='cuda'))
        if power < -1000:
            assert float((got - want).abs().max()) <= 2.0 ** -1010
        else:
            assert float((got - want).abs().max()) <= 1e-13 * float(want.abs().max())


def test_a_captured_step_and_adjoint_repeat(large):
    case, mesh, prob, rcf = large
    x, seeds = _state(case, 'noise')
    d, s = [t.cuda() for t in x], [t.cuda() for t in seeds]
    kw = dict(stages=rcf.stage_buffer(), tape=rcf.tape_buffer())
    out, adj = [torch.empty_like(t) for t in d], [torch.empty_like(t) for t in d]
    run = lambda: (rcf.step(*d, case.dt, out=out, want_scalars=False, **kw),
                   rcf.adjoint_step(*d, case.dt, s, out=adj, source_grad=False, **kw))
    run()
    want = [t.clone() for t in out + adj]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run()
    for t in out + adj:
        t.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out + adj, want))
