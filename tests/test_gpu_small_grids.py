"""The launch shapes of small meshes: one-warp blocks up to a limit, full blocks above it. One step
and its adjoint against the oracle where a block is partly filled, and on a mesh whose cells
take the one shape and whose faces the other. Within 1e-12 (max|x-ref|/max|ref| per field), the
bound of every FP64 step here; dtc and the objective within 1e-12 of their own size. The adjoint is
compared on the boxes only: the quiet ends of the tube keep velocities at roundoff level, which
puts |U_L.n - U_R.n| of the Roe entropy fix at its kink, where no two evaluation orders agree."""
import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF
from oracle import torch_ref
from tests import golden_cases as G

pytestmark = pytest.mark.gpu

SMALL_ITEMS = 32 * 4 * 152 * 8          # SMALL_WARPS warps (csrc/ctx.cuh)


def _case(name, n):
    if name == 'tube':
        return cases.sod(n)
    return cases.box(n)


@pytest.mark.parametrize('name,n', [('tube', 7), ('tube', 31), ('tube', 32), ('tube', 33), ('tube', 257),
                                    ('box', 8), ('box', 26), ('box', 27), ('box', 38)])
def test_step_and_adjoint_at_the_edges_of_a_block(name, n):
    case = _case(name, n)
    mesh = case.build_mesh()
    if name == 'box' and n in (26, 27):
        assert (mesh.nInternalCells <= 32 * 4 * 152) == (n == 26)
    if n == 38:
        assert mesh.nInternalCells < SMALL_ITEMS < mesh.nFaces
    prob = torch_ref.Problem(mesh, case.bc, case.config, case.objective)
    rng = np.random.default_rng(3)
    x = [torch.as_tensor(a) for a in cases.conservative(case)]
    x[0] = x[0] * (1 + 1e-3 * torch.as_tensor(rng.standard_normal(x[0].shape)))
    seeds = [torch.as_tensor(rng.standard_normal(t.shape)) / max(1.0, float(t.abs().max())) for t in x]
    ref = prob.step(*x, case.dt)
    obja = 0.0 if case.objective == 'none' else 1.0
    refa = torch_ref.vjp_step(prob, *x, case.dt, None, seeds, obja=obja)
    rcf = RCF(mesh, case.bc, objective=case.objective, **case.config)
    d = [t.cuda() for t in x]
    st, tp = rcf.stage_buffer(), rcf.tape_buffer()
    out = rcf.step(*d, case.dt, stages=st, tape=tp)
    a = rcf.adjoint_step(*d, case.dt, [t.cuda() for t in seeds], obja=obja, stages=st, tape=tp)
    for i in range(3):
        assert G.rel_err(out[i].cpu().numpy(), ref[i].numpy()) < 1e-12, (name, n, i)
        assert torch.isfinite(a[i]).all()
        if name == 'box':
            assert G.rel_err(a[i].cpu().numpy(), refa[i].numpy()) < 1e-12, (name, n, i)
    assert abs(out[3] - float(ref[3])) <= 1e-12 * abs(float(ref[3]))
    assert abs(out[4] - float(ref[4])) <= 1e-12 * max(abs(float(ref[4])), 1e-300)


@pytest.mark.parametrize('name', ['tube', 'box', 'cylinder', 'channel'])
@pytest.mark.parametrize('steps', [1, 2, 5])
def test_a_device_run_is_its_steps(name, steps):
    """RCF.run_device (whose steps write the next one's primitives and its dt on the device) against
    the same steps one call at a time with the dt rule on the host: the same bits. The histories
    cover each kind of objective: none, a cell sum, a face sum, the vane's."""
    case = {'tube': lambda: cases.sod(100), 'box': lambda: cases.box(8), 'cylinder': lambda: cases.cylinder(32, 16),
            'channel': lambda: cases.vane_channel(32, 12)}[name]()
    config = dict(case.config, fixedTimeStep=False)
    rcf = RCF(case.build_mesh(), case.bc, objective=case.objective, **config)
    x = [torch.as_tensor(a).cuda() for a in cases.conservative(case)]
    y = [t.clone() for t in x]
    dt, want = case.dt, []
    for _ in range(steps):
        r = rcf.step(*x, dt)
        x = list(r[:3])
        want.append((dt, r[3], r[4]))
        dt = min(2 * rcf.CFL / r[3], dt * rcf.stepFactor)
    hist = rcf.run_device(*y, steps, case.dt).cpu().numpy()
    assert all(torch.equal(a, b) for a, b in zip(x, y))
    assert np.array_equal(hist[:, :steps].T, np.array(want))
