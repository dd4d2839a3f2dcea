"""The FP32 and mixed adjoint's kernels at the edges of their launch shapes: meshes whose faces and
record pieces leave a warp or a block partly filled, on either side of the small-mesh limits. One
adjoint step against the FP64 one (itself held to autograd elsewhere) within the bounds that the
reduced precisions have against FP64 autograd: 1e-4 (fp32) and 1e-6 (mixed) of a field's largest
value. (box 41 is left out: its middle faces have U_L.n = U_R.n to roundoff, the kink of the Roe
entropy fix, where FP32 and FP64 take different sides.)"""
import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF
from tests import golden_cases as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision,tol', [('fp32', 1e-4), ('mixed', 1e-6)])
@pytest.mark.parametrize('name,n', [('box', 7), ('box', 27), ('box', 38), ('cylinder', 40)])
def test_adjoint_step_at_the_edges_of_a_block(name, n, precision, tol):
    case = cases.cylinder(n, n // 2 + 1) if name == 'cylinder' else cases.box(n)
    mesh = case.build_mesh()
    x = [torch.as_tensor(a) for a in cases.conservative(case)]
    rng = np.random.default_rng(5)
    seeds = [torch.as_tensor(rng.standard_normal(t.shape)) / max(1.0, float(t.abs().max())) for t in x]
    out = {}
    for p in ('fp64', precision):
        rcf = RCF(mesh, case.bc, objective=case.objective, precision=p, **case.config)
        td = torch.float32 if p == 'fp32' else torch.float64
        out[p] = rcf.adjoint_step(*[t.to(td).cuda() for t in x], case.dt, [t.to(td).cuda() for t in seeds], obja=1.0)
    for i in range(3):
        e = G.rel_err(out[precision][i].double().cpu().numpy(), out['fp64'][i].cpu().numpy())
        assert e < tol, (name, n, i, e)
