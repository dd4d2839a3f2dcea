"""The FP64 stage update of meshes whose cells are past the small-grid limit (its gather's products are
on the integer pipes): a step with sources against the oracle within 1e-12, and a state with NaN,
infinite and 1e200 entries, whose cells gather again with the hardware's products: the same
non-finite entries as the oracle and 1e-12 elsewhere."""
import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF
from oracle import torch_ref
from tests import golden_cases as G

pytestmark = pytest.mark.gpu

SMALL_ITEMS = 32 * 4 * 152 * 8          # SMALL_WARPS warps (csrc/ctx.cuh)


@pytest.fixture(scope='module')
def large():
    case = cases.box(54)
    mesh = case.build_mesh()
    assert SMALL_ITEMS < mesh.nInternalCells < 1.02 * SMALL_ITEMS and mesh.nInternalCells % 256
    rng = np.random.default_rng(6)
    x = [torch.as_tensor(a) for a in cases.conservative(case)]
    x[0] = x[0] * (1 + 1e-3 * torch.as_tensor(rng.standard_normal(x[0].shape)))
    S = [1e-3 * t / case.dt for t in x]
    prob = torch_ref.Problem(mesh, case.bc, case.config, case.objective)
    return case, x, S, prob, RCF(mesh, case.bc, objective=case.objective, **case.config)


@pytest.mark.parametrize('sources', [False, True])
def test_step_matches_oracle(large, sources):
    case, x, S, prob, rcf = large
    ref = prob.step(*x, case.dt, S) if sources else prob.step(*x, case.dt)
    out = rcf.step(*[t.cuda() for t in x], case.dt, S=[t.cuda() for t in S] if sources else None)
    for i in range(3):
        assert G.rel_err(out[i].cpu().numpy(), ref[i].numpy()) < 1e-12, i
    assert abs(out[3] - float(ref[3])) <= 1e-12 * abs(float(ref[3]))
    assert abs(out[4] - float(ref[4])) <= 1e-12 * abs(float(ref[4]))


def test_non_finite_cells_match_oracle(large):
    case, x, S, prob, rcf = large
    x = [t.clone() for t in x]
    x[0][1234, 0] = float('nan')
    x[2][30000, 0] = float('inf')
    x[1][120000, 1] = 1e200
    ref = prob.step(*x, case.dt)
    out = rcf.step(*[t.cuda() for t in x], case.dt, want_scalars=False)
    for i in range(3):
        got, want = out[i].cpu().numpy(), ref[i].numpy()
        fine = np.isfinite(want)
        assert 0 < (~fine).sum() < fine.size // 2
        assert np.array_equal(np.isfinite(got), fine)
        small = fine & (np.abs(np.where(fine, want, 0)) < 1e8)      # (cells 1e200 has not reached)
        assert np.abs(got[small] - want[small]).max() <= 1e-12 * np.abs(want[small]).max()
