"""The adjoint viscosity's heat equation where diffusion is strong against the volume (coefficients up
to 1e4 and 1e6 times it) and the fields are smooth: against the solution in extended precision. There
the matrix product has to be one of differences, V p + sum w (p - p_nb).

Tolerance: four times the error that the same conjugate gradients have in numpy in 64 bits (the
iterations differ in the order of their sums only). With diagonal p - sum w p_nb in the place of the
differences the numpy iteration errs 17 to 240 times as much on these inputs, which a CPU test checks."""
import numpy as np
import pytest
import scipy.linalg
import torch

from adfvm_gb300 import cases
from adfvm_gb300.solver import RCF

CELLS = 200
STRENGTHS = [1e4, 1e6]


def _slots(m):
    """Per cell and face slot: the face, the neighbour (the cell itself across a boundary), and
    whether there is one."""
    n = m.nInternalCells
    f = np.asarray(m.cellFaces).reshape(n, 6)
    inside = f < m.nInternalFaces
    here = np.arange(n)[:, None]
    other = np.where(m.owner[f] == here, m.neighbour[f], m.owner[f])
    return f, np.where(inside, other, here), inside


def _fields(m, seed):
    """V times smooth fields, n x 5."""
    rng = np.random.default_rng(seed)
    x = m.cellCentres[:m.nInternalCells] @ rng.standard_normal((3, 5)) + rng.random(5)
    return m.volumes.reshape(-1, 1) * (1 + 0.5 * np.sin(2 * np.pi * x))


def _product(V, w, o, p):
    return V[:, None] * p + sum(w[:, k:k + 1] * (p - p[o[:, k]]) for k in range(6))


def _short_product(V, w, o, p):
    return (V + w.sum(axis=1))[:, None] * p - sum(w[:, k:k + 1] * p[o[:, k]] for k in range(6))


def _exact(V, w, o, a):
    """The solution in extended precision: LU in 64 bits, refined."""
    n = len(V)
    A = np.diag(V + w.sum(axis=1))
    for k in range(6):
        np.add.at(A, (np.arange(n), o[:, k]), -w[:, k])
    lu = scipy.linalg.lu_factor(A)
    V, w, a = [t.astype(np.longdouble) for t in (V, w, a)]
    x = np.zeros(a.shape, np.longdouble)
    for _ in range(12):
        x = x + scipy.linalg.lu_solve(lu, (a - _product(V, w, o, x)).astype(np.float64))
    return x


def _conjugate_gradients(V, w, o, a, product=_product):
    """The kernel's iteration (csrc/viscosity.cu) in numpy."""
    rdiag = 1 / (V + w.sum(axis=1))[:, None]
    ratio = lambda s, t: np.divide(s, t, out=np.zeros_like(s), where=t != 0)
    x = a / V[:, None]
    r = a - _product(V, w, o, x)
    p = r * rdiag
    rz, rr, limit = (r * p).sum(axis=0), (r * r).sum(axis=0), 1e-26 * (a * a).sum(axis=0)
    it = 0
    while it % 4 or not (rr <= limit).all():
        assert it < 500
        q = product(V, w, o, p)
        alpha = ratio(rz, (p * q).sum(axis=0))
        x, r = x + alpha * p, r - alpha * q
        before, rz, rr = rz, (r * (r * rdiag)).sum(axis=0), (r * r).sum(axis=0)
        p = r * rdiag + ratio(rz, before) * p
        it += 1
    return x


def _setup(strength, seed):
    case = cases.duct(CELLS)
    m = case.build_mesh()
    f, o, inside = _slots(m)
    V = m.volumes.reshape(-1)
    g = (m.areas.reshape(-1) / m.deltas.reshape(-1))[f] * inside
    return case, m, f, o, inside, V, strength / np.max(g / V[:, None]), _fields(m, seed)


def _error(x, exact):
    return float(np.abs(x - exact).max() / np.abs(exact).max())


@pytest.mark.parametrize('strength', STRENGTHS)
@pytest.mark.parametrize('seed', [0, 1])
def test_the_tolerance_tells_the_products_apart(strength, seed):
    case, m, f, o, inside, V, dt, a = _setup(strength, seed)
    w = dt * (m.areas.reshape(-1) / m.deltas.reshape(-1))[f] * inside
    exact = _exact(V, w, o, a)
    assert _error(_conjugate_gradients(V, w, o, a, _short_product), exact) > \
        8 * _error(_conjugate_gradients(V, w, o, a), exact)


@pytest.mark.gpu
@pytest.mark.parametrize('strength', STRENGTHS)
@pytest.mark.parametrize('seed', [0, 1])
def test_strong_diffusion_of_smooth_fields(strength, seed):
    case, m, f, o, inside, V, dt, a = _setup(strength, seed)
    rcf = RCF(m, case.bc, objective=case.objective, **case.config)
    x = [torch.as_tensor(t).cuda() for t in cases.conservative(case)]
    got = [torch.as_tensor(np.ascontiguousarray(t)).cuda() for t in (a[:, :1], a[:, 1:4], a[:, 4:])]
    it, _, DT = rcf.adjoint_viscosity(*x, got, dt, 'uniform', 1.0, want_fields=True)
    w = (dt * (m.areas.reshape(-1) * DT.cpu().numpy() / m.deltas.reshape(-1)))[f] * inside
    exact = _exact(V, w, o, a)
    out = np.concatenate([t.cpu().numpy() for t in got], axis=1) / V[:, None]
    assert _error(out, exact) <= 4 * _error(_conjugate_gradients(V, w, o, a), exact), it
