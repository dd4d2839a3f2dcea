"""RCF.run_fixed (the adjoint sweep's primal pass): steps of one size in one device run, and of
several sizes one by one, against the same steps one call at a time: the same bits and objectives.
The objectives are a cell sum, a face sum, the vane's and a caller's function."""
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF

pytestmark = pytest.mark.gpu


def _mean_T(fields, solver):
    return fields[1].mean()


@pytest.mark.parametrize('name,precision', [('box', 'fp64'), ('box', 'fp32'), ('cylinder', 'fp64'),
                                            ('cylinder', 'mixed'), ('channel', 'fp64'), ('function', 'fp64')])
@pytest.mark.parametrize('sizes', [(1.0,), (1.0, 1.0, 1.0), (1.0, 0.5, 1.0)])
@pytest.mark.parametrize('sources', [False, True])
def test_run_fixed_is_its_steps(name, precision, sizes, sources):
    case = {'box': lambda: cases.box(7), 'cylinder': lambda: cases.cylinder(32, 16), 'function': lambda: cases.box(6),
            'channel': lambda: cases.vane_channel(32, 12)}[name]()
    objective = _mean_T if name == 'function' else case.objective
    rcf = RCF(case.build_mesh(), case.bc, objective=objective, precision=precision, **case.config)
    td = torch.float32 if precision == 'fp32' else torch.float64
    x = [torch.as_tensor(a).to(td).cuda() for a in cases.conservative(case)]
    S = [1e-3 * t / case.dt for t in x] if sources else None
    y, dts, want = [t.clone() for t in x], [case.dt * s for s in sizes], []
    for dt in dts:
        r = rcf.step(*x, dt, S=S)
        x = list(r[:3])
        want.append(r[4])
    assert rcf.run_fixed(y, dts, S) == want
    assert all(torch.equal(a, b) for a, b in zip(x, y))
