"""The rounding error of the adjoint viscosity's field M, cell by cell: against the formulas of
adFVM/postpro.py:491-697 in extended precision on periodic boxes (all faces central).

Bound: the root mean square over the cells of M's relative error, without the common factor of its
norm, may be 5 % above what it is when every quotient and root is an IEEE division and square root
(measured with such a build: ERROR); the mean over 1,728 cells of independent roundings scatters by
1.7 %, over 8,000 by 0.8 %."""
import numpy as np
import pytest
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF

pytestmark = pytest.mark.gpu

ERROR = {(12, 'turkel'): 2.682e-16, (12, 'abarbanel'): 2.525e-16, (20, 'turkel'): 2.769e-16, (20, 'abarbanel'): 2.535e-16}
NOISE = {12: 1e-2, 20: 1e-3}
UREF, PREF = 33.0, 1e5


def _state(case, n):
    rng = np.random.default_rng(n)
    rho, rhoU, rhoE = [np.array(a) for a in cases.conservative(case)]
    rho *= 1 + NOISE[n] * rng.standard_normal(rho.shape)
    rhoE *= 1 + NOISE[n] * rng.standard_normal(rhoE.shape)
    return rho, rhoU, rhoE


def _extended(case, m, state, kind):
    """The largest eigenvalue of every cell's symmetrised matrix, up to a common factor."""
    L = lambda a: np.asarray(a).astype(np.longdouble)
    n, nIF = m.nInternalCells, m.nInternalFaces
    g, Cp = L(1.4), L(1004.5)
    Cv = Cp / g
    rho, rhoU, rhoE = [L(a) for a in state]
    U = rhoU / rho
    E = rhoE / rho - (U * U).sum(axis=1, keepdims=True) / 2
    p, T = ((g - 1) * rho * E)[:, 0], (E / Cv)[:, 0]
    own, nbr = np.array(m.owner), np.array(m.neighbour)
    for patch in m.boundary.values():       # a cyclic ghost is its partner's owner
        f = np.arange(patch['nFaces'])
        nbr[patch['startFace'] + f] = own[m.boundary[patch['neighbourPatch']]['startFace'] + f]
    w, N = L(m.weights).reshape(-1), L(m.normals)
    central = lambda a: (a[own].T * w + a[nbr].T * (1 - w)).T
    c = np.sqrt(g * T * (Cp - Cv))
    gU, gp, gc = np.zeros((n, 3, 3), np.longdouble), np.zeros((n, 3), np.longdouble), np.zeros((n, 3), np.longdouble)
    UF, pF, cF = central(U), central(p), central(c)
    faces, V = np.asarray(m.cellFaces).reshape(n, 6), L(m.volumes).reshape(-1)
    for k in range(6):
        f = faces[:, k]
        N_V = N[f] * (np.where(own[f] == np.arange(n), 1, -1) * L(m.areas).reshape(-1)[f] / V)[:, None]
        gU += UF[f][:, :, None] * N_V[:, None, :]
        gp += pF[f][:, None] * N_V
        gc += cF[f][:, None] * N_V
    dU = gU[:, 0, 0] + gU[:, 1, 1] + gU[:, 2, 2]
    cc = np.sqrt(g * p / rho[:, 0])
    r, rc, p, d = [t[:, None] for t in (rho[:, 0], rho[:, 0] * cc, p, dU)]
    grho = g * (gp - cc[:, None] * p) / cc[:, None] ** 2
    A = np.zeros((n, 5, 5), np.longdouble)
    A[:, range(5), range(5)] = d / 2
    A[:, 1:4, 1:4] -= gU
    A[:, 4, 4] -= (g - 1) * dU / 2
    if kind == 'turkel':
        A[:, 0, 0] -= (g - 1) * dU / 2
        A[:, 0, 1:4] += gc / 2 - gp / rc
        A[:, 1:4, 0] += gc / 2 - (g - 1) * gp / (2 * rc)
        A[:, 1:4, 4] -= gp * PREF / (2 * g * p * r * UREF)
        A[:, 4, 1:4] -= (gp - cc[:, None] ** 2 * grho) * UREF / PREF
        A[:, 0, 4] -= (d * PREF / (2 * rc * UREF))[:, 0]
    else:
        b, s = cc[:, None] / np.sqrt(g), np.sqrt(g - 1)
        gb = gc / np.sqrt(g)
        A[:, 0, 1:4] += gb / 2 - b * grho / r
        A[:, 1:4, 0] += gb / 2
        A[:, 1:4, 4] += s * gb / 2 - s * b * gp / (2 * p)
        A[:, 4, 1:4] += s * gb / 2 - 2 * s * gb / (g - 1)
        A[:, 0, 4] -= s * dU / 2
    S = (A + A.transpose(0, 2, 1)) / 2
    # a Rayleigh quotient in extended precision errs by the square of its vector's error
    v = np.linalg.eigh(S.astype(np.float64))[1][:, :, -1].astype(np.longdouble)
    return np.einsum('ni,nij,nj->n', v, S, v) / (v * v).sum(axis=1)


@pytest.mark.parametrize('n,kind', list(ERROR))
def test_the_viscosity_rounds_as_with_divisions(n, kind):
    case = cases.box(n)
    m = case.build_mesh()
    state = _state(case, n)
    rcf = RCF(m, case.bc, objective=case.objective, **case.config)
    d = [torch.as_tensor(t).cuda() for t in state]
    a = [torch.zeros_like(t) for t in d]
    _, M, _ = rcf.adjoint_viscosity(*d, a, 1e-4, kind, 1.0, want_fields=True)
    ratio = M.cpu().numpy()[:m.nInternalCells] / _extended(case, m, state, kind)
    error = ratio / ratio.mean() - 1
    assert float(np.sqrt((error * error).mean())) <= 1.05 * ERROR[n, kind]
