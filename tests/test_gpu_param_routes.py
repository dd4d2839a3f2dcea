"""Mesh gradients of a mesh past the small-grid limit on every route: with memory for a whole step's
tape, for one stage's and for none (the forward values then come from the face kernel itself, by the
same arithmetic), and captured before the context has a tape; each with nothing kept of the step, with
its stages, and with its stages and tape. Against the oracle within 1e-12, and the same bits whatever
the memory."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import pytest
import torch

from adfvm_gb300.solver import RCF
from tests import golden_cases as G
from tests.test_gpu_param_tape import large          # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TAPE = 61


@pytest.fixture(scope='module')
def probe():
    out = os.path.join(tempfile.mkdtemp(prefix='param_tape_'), 'param_tape_probe.so')
    subprocess.check_call([os.environ.get('NVCC', 'nvcc'), '-gencode', 'arch=compute_103a,code=sm_103a', '-O2',
                           '-std=c++17', '--expt-relaxed-constexpr', '-shared', '-Xcompiler', '-fPIC',
                           '-I' + os.path.join(ROOT, 'include'), '-I' + os.path.join(ROOT, 'adfvm_gb300', 'csrc'),
                           os.path.join(ROOT, 'tests', 'native', 'param_tape_probe.cu'), '-o', out])
    return C.CDLL(out)


@pytest.mark.parametrize('kept', ['nothing', 'stages', 'tape'])
def test_the_same_bits_on_every_route(large, probe, kept):          # noqa: F811
    case, mesh, x, seeds, ref = large
    d, s = [t.cuda() for t in x], [t.cuda() for t in seeds]
    one = 8 * TAPE * mesh.nFaces
    # (the limit, what the context then holds - a whole step's takes 3.6 of a stage's -; a step with its
    # own tape needs none)
    routes = {'none': (0, 0), 'one stage': (one, 1), 'four stages': (4 * one, 2), 'whole': (1 << 40, 2),
              'just too little': (one - 1, 0)}
    results = {}
    for name, (limit, held) in routes.items():
        rcf = RCF(mesh, case.bc, objective=case.objective, **case.config)
        probe.limit_tape(rcf._ctx, C.c_size_t(limit))
        kw = {}
        if kept != 'nothing':
            kw['stages'] = rcf.stage_buffer()
            if kept == 'tape':
                kw['tape'] = rcf.tape_buffer()
            rcf.step(*d, case.dt, **kw)
        for again in range(2):                                      # (the first call and a later one)
            a = rcf.adjoint_step(*d, case.dt, s, params='mesh', **kw)
            results[name, again] = list(a[:3]) + list(a[4])
        assert probe.tape_held(rcf._ctx) == (0 if kept == 'tape' else held)
        if held == 0:
            # captured before there is a tape: the route without one
            probe.limit_tape(rcf._ctx, C.c_size_t(1 << 40))
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                a = rcf.adjoint_step(*d, case.dt, s, params='mesh', **kw)
            assert probe.tape_held(rcf._ctx) == 0
            g.replay()
            results[name, 'captured'] = list(a[:3]) + list(a[4])
        torch.cuda.synchronize()
    want = results['none', 0]
    for i in range(3):
        assert G.rel_err(want[i].cpu().numpy(), ref[i].numpy()) < 1e-12
    for k, field in enumerate(RCF.MESH_GRAD_FIELDS):
        assert G.rel_err(want[3 + k].cpu().numpy(), ref[4][k].numpy()) < 1e-12, field
    names = ['rhoa', 'rhoUa', 'rhoEa'] + list(RCF.MESH_GRAD_FIELDS)
    differ = [(route, n, float((p - q).abs().max() / q.abs().max())) for route, r in results.items()
              for n, p, q in zip(names, r, want) if not torch.equal(p, q)]
    assert not differ
