"""Mesh gradients of meshes past the small-grid limit, which are formed from face tapes: against the
oracle within 1e-12, with the step's own tape and without; the state adjoint's bits are the same with
and without the gradients; a captured call (which makes no tape of its own) gives the same gradients
within 1e-12."""
import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF
from oracle import torch_ref
from tests import golden_cases as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def large():
    case = cases.box(38)
    mesh = case.build_mesh()
    rng = np.random.default_rng(12)
    x = [torch.as_tensor(a) for a in cases.conservative(case)]
    x[0] = x[0] * (1 + 1e-3 * torch.as_tensor(rng.standard_normal(x[0].shape)))
    seeds = [torch.as_tensor(rng.standard_normal(t.shape)) / max(1.0, float(t.abs().max())) for t in x]
    prob = torch_ref.Problem(mesh, case.bc, case.config, case.objective)
    ref = torch_ref.vjp_step_params(prob, *x, case.dt, None, seeds, 1.0, 'mesh')
    return case, mesh, x, seeds, ref


@pytest.mark.parametrize('taped', [False, True])
def test_mesh_gradient_matches_oracle(large, taped):
    case, mesh, x, seeds, ref = large
    rcf = RCF(mesh, case.bc, objective=case.objective, **case.config)
    d, s = [t.cuda() for t in x], [t.cuda() for t in seeds]
    kw = dict(stages=rcf.stage_buffer(), tape=rcf.tape_buffer()) if taped else {}
    if taped:
        rcf.step(*d, case.dt, **kw)
    plain = rcf.adjoint_step(*d, case.dt, s, **kw)
    a = rcf.adjoint_step(*d, case.dt, s, params='mesh', **kw)
    for i in range(3):
        assert torch.equal(a[i], plain[i]), i
        assert G.rel_err(a[i].cpu().numpy(), ref[i].numpy()) < 1e-12
    for k, field in enumerate(RCF.MESH_GRAD_FIELDS):
        assert G.rel_err(a[4][k].cpu().numpy(), ref[4][k].numpy()) < 1e-12, field


def test_captured_gradients(large):
    case, mesh, x, seeds, ref = large
    rcf = RCF(mesh, case.bc, objective=case.objective, **case.config)
    d, s = [t.cuda() for t in x], [t.cuda() for t in seeds]
    rcf.adjoint_step(*d, case.dt, s, params='mesh')          # (makes the context's buffers)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a = rcf.adjoint_step(*d, case.dt, s, params='mesh')
    g.replay()
    for k, field in enumerate(RCF.MESH_GRAD_FIELDS):
        assert G.rel_err(a[4][k].cpu().numpy(), ref[4][k].numpy()) < 1e-12, field
