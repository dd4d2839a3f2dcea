"""A flow that has gone non-finite stops the adjoint sweep's primal pass, whatever form its steps take
(one device run for steps of one size, one call each for several sizes): AFVM_ERR_NONFINITE, with
built-in objectives and with none, and AFVM_ERR_BAD_ARG for a step size that is not finite, as
RCF.step gives them."""
import numpy as np
import pytest
import torch

from adfvm_gb300 import _lib as L
from adfvm_gb300 import cases
from adfvm_gb300.adjoint import Adjoint
from adfvm_gb300.solver import RCF

pytestmark = pytest.mark.gpu


def _setup(name, precision, objective=None):
    case = {'box': lambda: cases.box(6), 'cylinder': lambda: cases.cylinder(32, 16),
            'channel': lambda: cases.vane_channel(32, 12)}[name]()
    rcf = RCF(case.build_mesh(), case.bc, objective=objective or case.objective, precision=precision, **case.config)
    return case, rcf, [np.array(a) for a in cases.conservative(case)]


def _device(rcf, x):
    td = torch.float32 if rcf.dtype == np.float32 else torch.float64
    return [torch.as_tensor(a).to(td).cuda() for a in x]


@pytest.mark.parametrize('name,precision,objective', [('box', 'fp64', None), ('box', 'fp32', None), ('box', 'fp64', 'none'),
                                                      ('cylinder', 'mixed', None), ('channel', 'fp64', None)])
@pytest.mark.parametrize('sizes', [(1.0,), (1.0, 1.0, 1.0), (1.0, 0.5, 1.0)])
def test_run_fixed_reports_a_non_finite_flow(name, precision, objective, sizes):
    case, rcf, x = _setup(name, precision, objective)
    x[2][5] = np.nan
    with pytest.raises(L.AfvmError) as e:
        rcf.run_fixed(_device(rcf, x), [case.dt * s for s in sizes])
    assert e.value.status == L.AFVM_ERR_NONFINITE


@pytest.mark.parametrize('sizes', [(float('inf'),), (float('inf'), float('inf')), (1.0, float('nan'))])
def test_run_fixed_refuses_a_non_finite_step_size(sizes):
    case, rcf, x = _setup('box', 'fp64')
    with pytest.raises(L.AfvmError) as e:
        rcf.run_fixed(_device(rcf, x), [case.dt * s for s in sizes])
    assert e.value.status == L.AFVM_ERR_BAD_ARG


@pytest.mark.parametrize('objective', [None, 'none'])
@pytest.mark.parametrize('sizes', [(1.0, 1.0, 1.0, 1.0), (1.0, 1.0, 0.5, 1.0)])
def test_a_sweep_of_a_non_finite_flow_stops(objective, sizes):
    case, rcf, x = _setup('box', 'fp64', objective)
    adjoint = Adjoint(rcf)
    pert = [tuple(np.ones_like(a) for a in x)]
    adjoint.run(x, 4, [case.dt * s for s in sizes], 2, pert)           # (a finite flow goes through)
    x[0][7] = np.nan
    with pytest.raises(L.AfvmError) as e:
        adjoint.run(x, 4, [case.dt * s for s in sizes], 2, pert)
    assert e.value.status == L.AFVM_ERR_NONFINITE
