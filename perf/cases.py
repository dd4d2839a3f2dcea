"""The calls whose speed is measured: what a user of the solver runs, from one small tube to the
128^3 box, through the public entry points of ``adfvm_gb300``.

``call`` is the entry point, ``mesh`` and its sizes the workload, ``precision`` the context's:

* ``run``      RCF.run_device: time steps resident on the GPU (the solver's time loop)
* ``step``     RCF.step with source terms: one primal step
* ``pair``     RCF.step keeping its stages and tape, then RCF.adjoint_step reading them: one step
               of an adjoint sweep, forward and backward
* ``mesh``     RCF.adjoint_step with the gradients of the ten mesh tensors, nothing kept
* ``solve``    autograd.solve and its backward pass: the solver inside a torch program
* ``sweep``    Adjoint.run: the checkpointed sweep with a source sensitivity
* ``map``      RCF.map and Adjoint.map on host arrays: the reference's two compiled functions
* ``viscosity``  RCF.adjoint_viscosity: the stabilisation of an adjoint field
* ``serve``    SensitivityServer.serve: requests on small meshes, slots made before

A solver (mesh tables, work buffers) is made once per mesh and reused for every state, as a
program that steps, sweeps or serves does.
"""
import functools
import math

import numpy as np
import torch

from adfvm_gb300 import adjoint, autograd, cases, serving
from adfvm_gb300.solver import RCF

GRADS = ('areas', 'volumesL', 'volumesR', 'weights', 'deltas', 'normals', 'deltasUnit', 'linearWeights',
         'quadraticWeights', 'volumes')


def listed():
    return [
        # the 1-D validation case: 1,000 cells, adaptive dt; a step is a few microseconds of work
        dict(name='tube1000_run_fp64', call='run', mesh='tube', a=1000, b=0, precision='fp64', steps=40),
        # the smallest box of the serving mix, one sweep step of it
        dict(name='box16_pair_fp32', call='pair', mesh='box', a=16, b=0, precision='fp32', steps=1),
        # six requests of the small meshes of the serving mix in flight together
        dict(name='serve_small_mixed', call='serve', mesh='small', a=16, b=0, precision='mixed', steps=20),
        # the precision study's cylinder: walls, far field, drag objective
        dict(name='cyl256x128_pair_mixed', call='pair', mesh='cylinder', a=256, b=128, precision='mixed', steps=1),
        # the vane objective's channel through the reference's own call surface, arrays on the host
        dict(name='channel64x24_map_fp64', call='map', mesh='channel', a=64, b=24, precision='fp64', steps=1),
        # a whole checkpointed sweep as the adjoint driver runs it
        dict(name='cyl128x64_sweep_fp64', call='sweep', mesh='cylinder', a=128, b=64, precision='fp64', steps=10),
        # shape gradients: an odd box, nothing kept from the primal step
        dict(name='box47_mesh_fp64', call='mesh', mesh='box', a=47, b=0, precision='fp64', steps=1),
        # the adjoint workload's box inside a torch program, checkpoints every second step
        dict(name='box64_solve_fp64', call='solve', mesh='box', a=64, b=0, precision='fp64', steps=4),
        # an adjoint field smoothed between sweep steps
        dict(name='box64_viscosity_fp64', call='viscosity', mesh='box', a=64, b=0, precision='fp64', steps=1),
        # a large primal step with sources, nothing kept
        dict(name='box96_step_fp64', call='step', mesh='box', a=96, b=0, precision='fp64', steps=1),
        # the headline workload in both precisions: primal + adjoint of 2,097,152 cells
        dict(name='box128_pair_fp64', call='pair', mesh='box', a=128, b=0, precision='fp64', steps=1),
        dict(name='box128_pair_fp32', call='pair', mesh='box', a=128, b=0, precision='fp32', steps=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(['run', 'run', 'step', 'step', 'pair', 'pair', 'pair', 'mesh', 'solve', 'sweep', 'map',
                       'viscosity', 'serve'])
    precision = rng.choice(['fp64', 'fp32', 'mixed'])
    mesh = rng.choice(['box', 'box', 'cylinder', 'channel', 'tube'])
    steps = 1
    if call == 'serve':
        return dict(call=call, mesh='small', a=rng.randint(12, 24), b=0, precision=rng.choice(['fp64', 'mixed']),
                    steps=10 * rng.randint(1, 3))
    if call == 'mesh':
        precision = 'fp64'
    if call == 'sweep' and mesh == 'tube':
        mesh = 'channel'                 # the tube has no objective to sweep back from
    top = {'run': 64, 'step': 110, 'pair': 112, 'mesh': 56, 'solve': 56, 'sweep': 40, 'map': 56, 'viscosity': 64}[call]
    if call == 'run':
        steps = rng.randint(4, 40)
    if call == 'solve':
        steps = rng.randint(2, 4)
    if call == 'sweep':
        steps = 2 * rng.randint(2, 6)
    if mesh == 'box':
        a, b = _log(rng, 12, top), 0
    elif mesh == 'cylinder':
        a, b = _log(rng, 32, 256), _log(rng, 16, 128)
    elif mesh == 'channel':
        a, b = _log(rng, 32, 160), _log(rng, 12, 64)
    else:
        a, b = _log(rng, 100, 4000), 0
    return dict(call=call, mesh=mesh, a=a, b=b, precision=precision, steps=steps)


# ------------------------------------------------------------------ set-up

@functools.lru_cache(maxsize=32)
def _workload(mesh, a, b):
    if mesh == 'tube':
        return cases.sod(a)
    if mesh == 'box':
        return cases.box(a)
    if mesh == 'cylinder':
        return cases.cylinder(a, b)
    return cases.vane_channel(a, b)


@functools.lru_cache(maxsize=4)
def _solver(mesh, a, b, precision):
    w = _workload(mesh, a, b)
    gauge = cases.gauge(w) if precision != 'fp64' and mesh == 'box' else None
    return RCF(w.mesh, w.bc, objective=w.objective, precision=precision, gauge=gauge, **w.config)


@functools.lru_cache(maxsize=4)
def _base(mesh, a, b):
    """The workload's initial state and the cell volumes on the GPU, FP64."""
    w = _workload(mesh, a, b)
    return [torch.as_tensor(np.ascontiguousarray(v), device='cuda') for v in cases.conservative(w) + (w.mesh.volumes,)]


def _fields(case, seed, dtype):
    """A state (the workload's initial field with 0.1 % of density noise), a smooth source
    perturbation and the adjoint of a kinetic-energy-like functional with noise, from the seed."""
    rho, rhoU, rhoE, V = _base(case['mesh'], case['a'], case['b'])
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed))
    noise = lambda t: torch.randn(t.shape, generator=g, device='cuda', dtype=torch.float64)
    x = [rho * (1 + 1e-3 * noise(rho)), rhoU, rhoE]
    U = rhoU / rho + noise(rhoU)
    s = [V * (-0.5 * (U * U).sum(1, keepdim=True)), V * U, V * (1e-2 + 1e-3 * noise(rho))]
    return [t.to(dtype).contiguous().clone() for t in x], [t.to(dtype).contiguous() for t in s]


def _source(case, seed):
    return cases.source_field(_workload(case['mesh'], case['a'], case['b']).mesh, scale=1e-3, seed=int(seed) % 100003)


def _keys(a):
    """The meshes of a serve case: boxes of side a and a + 8, and a cylinder."""
    return ['box%d' % a, 'cyl64x32', 'box%d' % (a + 8)]


@functools.lru_cache(maxsize=1)
def _server(a, precision, steps):
    s = serving.SensitivityServer(precision=precision, k=10, nPrimal=steps)
    s.warm(_keys(a) * 2)
    return s


def _requests(case, seed):
    return [serving.Request(rid=i, key=k, seed=(int(seed) * 7 + i) % 1000003, nPrimal=case['steps'])
            for i, k in enumerate(_keys(case['a']) * 2)]


def prepare(case, seed):
    call = case['call']
    if call == 'serve':
        server = _server(case['a'], case['precision'], case['steps'])
        return dict(case=case, server=server, requests=serving.prepare(_requests(case, seed), server.lib))
    key = (case['mesh'], case['a'], case['b'])
    w = _workload(*key)
    solver = _solver(*key, case['precision'])
    x, seeds = _fields(case, seed, torch.float32 if case['precision'] == 'fp32' else torch.float64)
    s = dict(case=case, solver=solver, x=x, seeds=seeds, dt=w.dt)
    if call == 'step':
        s['S'] = [torch.as_tensor(v, device='cuda').to(x[0].dtype) for v in _source(case, seed)]
    if call == 'pair':
        s['stages'], s['tape'] = solver.stage_buffer(), solver.tape_buffer()
    if call == 'sweep':
        s['driver'] = adjoint.Adjoint(solver)
        s['host'] = [t.double().cpu().numpy() for t in x]
        s['dS'] = [_source(case, seed)]
    if call == 'map':
        s['driver'] = adjoint.Adjoint(solver)
        s['host'] = [t.double().cpu().numpy() for t in x]
        s['hostSeeds'] = [t.double().cpu().numpy() for t in seeds]
        s['hostSource'] = _source(case, seed)
    return s


# ------------------------------------------------------------------ one pass

def run(state):
    case = state['case']
    call = case['call']
    if call == 'serve':
        state['server'].serve(state['requests'], realtime=False)
        return [r.sensitivity for r in state['requests']]
    solver, x, dt = state['solver'], state['x'], state['dt']
    if call == 'run':
        y = [t.clone() for t in x]
        hist = solver.run_device(*y, case['steps'], dt)
        return y + [hist]
    if call == 'step':
        return list(solver.step(*x, dt, S=state['S']))
    if call == 'pair':
        p = solver.step(*x, dt, stages=state['stages'], tape=state['tape'])
        r = solver.adjoint_step(*x, dt, state['seeds'], stages=state['stages'], tape=state['tape'])
        return list(p) + list(r[:3]) + list(r[3])
    if call == 'mesh':
        r = solver.adjoint_step(*x, dt, state['seeds'], params='mesh')
        return list(r[:3]) + list(r[3]) + list(r[4])
    if call == 'solve':
        leaves = [t.detach().requires_grad_(True) for t in x]
        S = [torch.zeros_like(t).requires_grad_(True) for t in x]
        out = autograd.solve(solver, *leaves, S=S, nSteps=case['steps'], dt=dt, checkpoint_every=2)
        loss = out[3].sum() + sum((o * s).sum() for o, s in zip(out, state['seeds']))
        loss.backward()
        return [t.detach() for t in out] + [t.grad for t in leaves + S]
    if call == 'sweep':
        sens, adj, record = state['driver'].run(state['host'], case['steps'], dt, case['steps'] // 2,
                                                perturbations=state['dS'])
        return [sens, adj, record['objective']]
    if call == 'map':
        inputs = solver.mapInputs(*state['host'], dt, sources=state['hostSource'])
        primal = solver.map(*inputs)
        adj = state['driver'].map(*inputs, *state['hostSeeds'], np.zeros((1, 1)), np.ones((1, 1)), 0.0)
        return primal + adj
    a = [t.clone() for t in state['seeds']]
    solver.adjoint_viscosity(*x, a, dt, kind='turkel', scaling=1e-3)
    return a


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(case):
    a, b = case['a'], case['b']
    if case['mesh'] == 'box':
        return a ** 3, 3 * a ** 3 + 3 * a ** 2, 6 * a ** 2
    if case['mesh'] == 'tube':
        return a, 5 * a + 1, 4 * a + 2
    if case['mesh'] == 'cylinder':
        return a * b, 4 * a * b + a, 2 * a * b + 2 * a
    return a * b, 4 * a * b + a + b, 2 * a * b + 2 * a + 2 * b


def work(case):
    """Bytes: the mesh (per face its two cells, area, delta, weight, normal, unit delta, linear and
    quadratic weights; per cell its volume and six faces), the call's inputs and its outputs, each
    once, whatever the steps in between. Flops: one evaluation of the face flux (450) and of its
    transpose (500) per face and stage, 250 and 350 per cell for the gradient, the update and their
    transposes."""
    if case['call'] == 'serve':
        a = case['a']
        cells = 2 * (a ** 3 + (a + 8) ** 3 + 64 * 32)
        faces = 2 * (3 * a ** 3 + 3 * (a + 8) ** 3 + 4 * 64 * 32)
        es, ss, fwd, rev = (8 if case['precision'] == 'fp64' else 4), 8, 2 * case['steps'], case['steps']
        state = cells * 10 * 8
    else:
        cells, faces, ghosts = _sizes(case)
        es = 8 if case['precision'] == 'fp64' else 4
        ss = 4 if case['precision'] == 'fp32' else 8
        n = case['steps']
        fwd, rev, state = {'run': (n, 0, 10), 'step': (1, 0, 15), 'pair': (1, 1, 23), 'mesh': (1, 1, 18),
                           'solve': (2 * n, n, 35), 'sweep': (2 * n, n, 15), 'map': (1, 1, 30),
                           'viscosity': (0, 0, 15)}[case['call']]
        state = cells * state * ss
        if case['call'] == 'mesh':
            state += 8 * (22 * faces + 2 * cells)
    mesh = faces * (8 + 17 * es) + cells * (24 + es)
    flops = 3 * (fwd * (450 * faces + 250 * cells) + rev * (500 * faces + 350 * cells))
    if case['call'] == 'viscosity':
        flops = 2500 * cells
    return dict(bytes=float(mesh + state), flops=float(flops))


# ------------------------------------------------------------------ the same results in 64 bits
#
# The finite-volume residual (Green-Gauss gradients, second-order reconstruction, Roe or
# Lax-Friedrichs flux, viscous flux), the SSP-RK3 step and its derivative by torch's own
# differentiation, on the mesh tensors and boundary dicts that the case hands the solver.

class _Exact(object):
    def __init__(self, w):
        m = w.mesh
        f = lambda v, *s: torch.as_tensor(np.ascontiguousarray(v, np.float64), device='cuda').reshape(*s)
        i = lambda v, *s: torch.as_tensor(np.ascontiguousarray(v, np.int64), device='cuda').reshape(*s)
        self.cfg = dict(Cp=1004.5, gamma=1.4, Pr=0.7, mu=None, riemannSolver='eulerRoe',
                        boundaryRiemannSolver='eulerRoe')
        self.cfg.update(w.config)
        self.g, self.Cp = self.cfg['gamma'], self.cfg['Cp']
        self.Cv = self.Cp / self.g
        self.objective = w.objective
        self.n, self.nIF, self.nF = m.nInternalCells, m.nInternalFaces, m.nFaces
        self.own, self.nbr = i(m.owner, -1), i(m.neighbour, -1)
        self.cf, self.cn, self.co = i(m.cellFaces, -1, 6), i(m.cellNeighbours, -1, 6), f(m.cellOwner, -1, 6)
        shapes = dict(normals=(-1, 3), deltasUnit=(-1, 3), linearWeights=(-1, 2), quadraticWeights=(-1, 2, 3))
        self.t = {k: f(getattr(m, k), *shapes.get(k, (-1, 1))) for k in GRADS}
        # faces by kind, ghosts by source cell and boundary condition
        src = torch.empty(self.nF - self.nIF, dtype=torch.int64, device='cuda')
        central, char, wall = [torch.arange(self.nIF, device='cuda')], [], []
        self.bcs, self.patch = [], {}
        for name in m.sortedPatches:
            p = m.boundary[name]
            s, k = int(p['startFace']), int(p['nFaces'])
            r = torch.arange(s, s + k, device='cuda')
            b = {q: w.bc[q][name] for q in 'UTp'}
            self.patch[name] = r
            src[r - self.nIF] = self.own[r]
            if p['type'] == 'cyclic':
                q = int(m.boundary[p['neighbourPatch']]['startFace'])
                src[r - self.nIF] = self.own[q:q + k]
                central.append(r)
            elif b['p']['type'] in ('CBC_UPT', 'CBC_TOTAL_PT'):
                char.append(r)
            else:
                wall.append(r)
            values = {q: {c: f(v, k, -1) for c, v in b[q].items() if isinstance(v, np.ndarray)} for q in 'UTp'}
            self.bcs.append((r - self.nIF, {q: b[q]['type'] for q in 'UTp'}, values))
        self.src = src
        cat = lambda v: torch.cat(v) if v else torch.empty(0, dtype=torch.int64, device='cuda')
        self.central, self.char, self.wall = cat(central), cat(char), cat(wall)

    def mu(self, T):
        if self.cfg['mu'] is None:
            return 1.4792e-06 * T ** 1.5 / (T + 116.)
        return T * 0 + float(self.cfg['mu'])

    def ghosts(self, U, T, p):
        gU, gT, gp = U[self.src], T[self.src], p[self.src]
        U0, T0 = gU, gT
        for r, kind, v in self.bcs:
            if kind['p'] == 'CBC_UPT':
                gU = gU.index_copy(0, r, v['p']['U0'])
                gT = gT.index_copy(0, r, v['p']['T0'])
                gp = gp.index_copy(0, r, v['p']['p0'])
            elif kind['p'] == 'CBC_TOTAL_PT':
                d, Tt, pt = v['p']['direction'], v['p']['Tt'], v['p']['pt']
                un = (U0[r] * d).sum(1, keepdim=True)
                gU = gU.index_copy(0, r, un * d)
                gT = gT.index_copy(0, r, Tt - 0.5 * un * un / self.Cp)
                gp = gp.index_copy(0, r, pt * (T0[r] / Tt) ** (self.g / (self.g - 1)))
            else:
                if kind['U'] == 'fixedValue':
                    gU = gU.index_copy(0, r, v['U']['value'])
                if kind['T'] == 'fixedValue':
                    gT = gT.index_copy(0, r, v['T']['value'])
                if kind['p'] == 'fixedValue':
                    gp = gp.index_copy(0, r, v['p']['value'])
        return torch.cat([U, gU]), torch.cat([T, gT]), torch.cat([p, gp])

    def primitives(self, u):
        rho = u[:, 0:1]
        U = u[:, 1:4] / rho
        e = u[:, 4:5] / rho - 0.5 * (U * U).sum(1, keepdim=True)
        return self.ghosts(U, e / self.Cv, (self.g - 1) * rho * e)

    def gradient(self, q):
        """(cells and ghosts, k) -> (cells and ghosts, k, 3)."""
        t, out = self.t, 0
        for s in range(6):
            face, o = self.cf[:, s], self.co[:, s:s + 1]
            w = t['weights'][face]
            w = w + o - 2 * w * o
            N = t['areas'][face] * t['normals'][face] * (2 * o - 1)
            q_f = q[:self.n] * (1 - w) + q[self.cn[:, s]] * w
            out = out + q_f.unsqueeze(2) * N.unsqueeze(1)
        out = out / t['volumes'].unsqueeze(2)
        return torch.cat([out, out[self.src]])

    def riemann(self, name, N, UL, TL, pL, UR, TR, pR):
        g = self.g
        dot = lambda x, y: (x * y).sum(1, keepdim=True)
        R = self.Cv * (g - 1)
        rL, rR = pL / (R * TL), pR / (R * TR)
        unL, unR = dot(UL, N), dot(UR, N)
        HL, HR = self.Cp * TL + 0.5 * dot(UL, UL), self.Cp * TR + 0.5 * dot(UR, UR)
        cL, cR = (g * R * TL).sqrt(), (g * R * TR).sqrt()
        flux = lambda r, U, H, p, un: torch.cat([r * un, r * un * U + p * N, r * un * H], 1)
        mean = 0.5 * (flux(rL, UL, HL, pL, unL) + flux(rR, UR, HR, pR, unR))
        qL, qR = torch.cat([rL, rL * UL, rL * HL - pL], 1), torch.cat([rR, rR * UR, rR * HR - pR], 1)
        if name == 'eulerLaxFriedrichs':
            return mean - 0.5 * torch.maximum(unL.abs() + cL, unR.abs() + cR) * (qR - qL)
        sL, sR = rL.sqrt(), rR.sqrt()
        U, H = (UL * sL + UR * sR) / (sL + sR), (HL * sL + HR * sR) / (sL + sR)
        k = 0.5 * dot(U, U)
        a2 = (g - 1) * (H - k)
        a = a2.sqrt()
        un = dot(U, N)
        eps = 0.5 * (unL - unR).abs() + 0.5 * (cL - cR).abs() + 1e-30
        l1, l2, l3 = (torch.where(v < 2 * eps, 0.25 * v * v / eps + eps, v)
                      for v in (un.abs(), (un + a).abs(), (un - a).abs()))
        d = qR - qL
        dr, dm, dE = d[:, 0:1], d[:, 1:4], d[:, 4:5]
        v2, v3 = 0.5 * (l2 - l3), 0.5 * (l2 + l3) - l1
        v4 = (g - 1) * (k * dr - dot(U, dm) + dE)
        v5 = un * dr - dot(dm, N)
        v6, v7 = v3 * v4 / a2 - v2 * v5 / a, v3 * v5 - v2 * v4 / a
        return mean - 0.5 * torch.cat([l1 * dr + v6, l1 * dm + U * v6 - v7 * N, l1 * dE + H * v6 - un * v7], 1)

    def residual(self, u, want=False):
        t = self.t
        U, T, p = self.primitives(u)
        J = self.value(U, T, p) if want else None
        gU, gT, gp = self.gradient(U), self.gradient(T), self.gradient(p)
        R = torch.zeros_like(u)
        lam = torch.zeros_like(u[:, 0:1])
        for kind, r in (('central', self.central), ('char', self.char), ('wall', self.wall)):
            if not len(r):
                continue
            o, n = self.own[r], self.nbr[r]
            N, D, delta = t['normals'][r], t['deltasUnit'][r], t['deltas'][r]
            lw, qw = t['linearWeights'][r], t['quadraticWeights'][r]
            side = lambda q, gq, c, d, k: (q[c] + (q[d] - q[c]) * lw[:, k:k + 1] +
                                           (gq[c] * qw[:, k].unsqueeze(1)).sum(2))
            if kind == 'wall':
                TF, UF, gTF, gUF = T[n], U[n], gT[n], gU[n]
                rho = p[n] / (self.Cv * (self.g - 1) * TF)
                un = (UF * N).sum(1, keepdim=True)
                F = torch.cat([rho * un, rho * un * UF + p[n] * N,
                               rho * un * (self.Cp * TF + 0.5 * (UF * UF).sum(1, keepdim=True))], 1)
            else:
                L = [side(q, gq, o, n, 0) for q, gq in ((U, gU), (T, gT), (p, gp))]
                if kind == 'char':
                    F = self.riemann(self.cfg['boundaryRiemannSolver'], N, *L, U[n], T[n], p[n])
                    TF, UF, gTF, gUF = T[n], U[n], gT[n], gU[n]
                else:
                    Q = [side(q, gq, n, o, 1) for q, gq in ((U, gU), (T, gT), (p, gp))]
                    F = self.riemann(self.cfg['riemannSolver'], N, *L, *Q)
                    UF, TF = 0.5 * (L[0] + Q[0]), 0.5 * (L[1] + Q[1])
                    gTF, gUF = 0.5 * (gT[o] + gT[n]), 0.5 * (gU[o] + gU[n])
            mu = self.mu(TF)
            fix = lambda q, gq: gq + (((q[n] - q[o]) / delta - (gq * D.unsqueeze(1)).sum(2)).unsqueeze(2) *
                                      D.unsqueeze(1))
            gTn = (fix(T, gTF) * N.unsqueeze(1)).sum(2)
            G = fix(U, gUF)
            tr = (G[:, 0, 0] + G[:, 1, 1] + G[:, 2, 2]).unsqueeze(1)
            sigma = mu * (((G + G.transpose(1, 2)) * N.unsqueeze(1)).sum(2) - 2. / 3 * tr * N)
            q = mu * (self.Cp / self.cfg['Pr']) * gTn + (sigma * UF).sum(1, keepdim=True)
            F = F - torch.cat([torch.zeros_like(q), sigma, q], 1)
            speed = (UF * N).sum(1, keepdim=True).abs() + (self.Cp * TF * (self.g - 1)).sqrt()
            wL = t['areas'][r] / t['volumesL'][r]
            R = R.index_add(0, o, F * wL)
            lam = lam.index_add(0, o, speed * wL)
            inner = r < self.nIF
            if bool(inner.any()):
                q = r[inner]
                wR = t['areas'][q] / t['volumesR'][q]
                R = R.index_add(0, self.nbr[q], -(F[inner] * wR))
                lam = lam.index_add(0, self.nbr[q], speed[inner] * wR)
        return R, lam, J

    def value(self, U, T, p):
        o, t, n = self.objective, self.t, self.n
        gas = self.Cv * (self.g - 1)
        if o == 'none':
            return torch.zeros((), dtype=torch.float64, device='cuda')
        if o == 'kinetic_energy':
            return (0.5 * p[:n] / (gas * T[:n]) * (U[:n] ** 2).sum(1, keepdim=True) * t['volumes']).sum()
        if isinstance(o, str):
            r = self.patch[o.split(':', 1)[1]]
            b, i = self.nbr[r], self.own[r]
            shear = self.mu(T[b]) * (U[b] - U[i])[:, 0:1] / t['deltas'][r]
            return ((p[b] * t['normals'][r][:, 0:1] - shear) * t['areas'][r]).sum()
        c = torch.as_tensor(o['planeCells'], device='cuda', dtype=torch.int64)
        A = torch.as_tensor(o['planeAreas'], device='cuda')
        d = torch.as_tensor(o['normal'], device='cuda')
        m = p[c] / (gas * T[c]) * (U[c] * d).sum(1, keepdim=True) * A
        M2 = (U[c] ** 2).sum(1, keepdim=True) / (self.g * gas * T[c])
        pt = p[c] * (1 + 0.5 * (self.g - 1) * M2) ** (self.g / (self.g - 1))
        J = o['a'] * ((o['ptin'] - pt) / o['ptin'] * m).sum() / m.sum()
        k = float(self.mu(torch.tensor(o['Tw'], dtype=torch.float64))) * self.Cp / self.cfg['Pr']
        num = den = 0
        for name, wt in o['heat'].items():
            r, wt = self.patch[name], torch.as_tensor(wt, device='cuda')
            num = num + (k * (o['Tw'] - T[self.own[r]]) / t['deltas'][r] * t['areas'][r] * wt).sum()
            den = den + (t['areas'][r] * wt).sum()
        return J + o['b'] * (num / den if float(den) else 0.0)

    def step(self, u, dt, S):
        R, _, _ = self.residual(u)
        u1 = u - dt * (R - S)
        R, lam, J = self.residual(u1, want=True)
        u2 = 0.75 * u + 0.25 * u1 - 0.25 * dt * (R - S)
        R, _, _ = self.residual(u2)
        return u / 3 + 2. / 3 * u2 - 2. / 3 * dt * (R - S), lam.max().detach(), J

    def smoothed(self, u, a, dt, scaling):
        """The 'turkel' artificial viscosity of the state and the implicit diffusion of a by it."""
        t, n, g = self.t, self.n, self.g
        U, T, p = self.primitives(u)
        c = (g * (self.Cp - self.Cv) * T).sqrt()
        w, o, b = t['weights'], self.own, self.nbr
        mid = lambda q: torch.index_copy(q[b].clone(), 0, self.central,
                                         (q[o] * w + q[b] * (1 - w))[self.central])
        wL = t['areas'] / t['volumesL']
        wR = t['areas'][:self.nIF] / t['volumesR']

        def grad(q):
            qn = q.unsqueeze(2) * t['normals'].unsqueeze(1)
            z = torch.zeros((n,) + tuple(qn.shape[1:]), dtype=torch.float64, device='cuda')
            z = z.index_add(0, o, qn * wL.unsqueeze(2))
            return z.index_add(0, b[:self.nIF], -qn[:self.nIF] * wR.unsqueeze(2))
        gU, gp, gc = grad(mid(U)), grad(mid(p))[:, 0], grad(mid(c))[:, 0]
        c, p, T = c[:n], p[:n], T[:n]
        div = (gU[:, 0, 0] + gU[:, 1, 1] + gU[:, 2, 2])
        rho = p / (self.Cv * (g - 1) * T)
        gr = g * (gp - c * p) / (c * c)
        M = torch.diag_embed(div.unsqueeze(1).expand(n, 5) / 2).clone()
        M[:, 0, 1:4] += gc / 2 - gp / (rho * c)
        M[:, 1:4, 0] += gc / 2 - (g - 1) * gp / (2 * rho * c)
        M[:, 1:4, 4] -= gp * 1e5 / (2 * g * p * rho * 33.)
        M[:, 4, 1:4] -= (gp - c * c * gr) * 33. / 1e5
        M[:, 1:4, 1:4] -= gU
        M[:, 0, 4] -= div * 1e5 / (2 * rho * c * 33.)[:, 0]
        M[:, 0, 0] -= (g - 1) * div / 2
        M[:, 4, 4] -= (g - 1) * div / 2
        e = np.linalg.eigvalsh(((M + M.transpose(1, 2)) / 2).cpu().numpy())[:, -1:]
        e = torch.as_tensor(e, device='cuda')
        V = t['volumes']
        e = e * scaling / ((e * e * V).sum() / V.sum()).sqrt()
        e = torch.cat([e, e[self.src]])
        k = (dt * t['areas'] * (e[o] * w + e[b] * (1 - w)) / t['deltas'])[:self.nIF]
        o, b = o[:self.nIF], b[:self.nIF]

        def apply(q):
            f = k * (q[o] - q[b])
            return (V * q).index_add(0, o, f).index_add(0, b, -f)
        diag = V.index_add(0, o, k).index_add(0, b, k)
        q = a / V
        r = a - apply(q)
        z = r / diag
        s, rz = z, (r * z).sum(0)
        for _ in range(400):
            if bool((r.norm(dim=0) <= 1e-15 * a.norm(dim=0)).all()):
                break
            y = apply(s)
            alpha = torch.where(rz > 0, rz / (s * y).sum(0), rz * 0)
            q, r = q + alpha * s, r - alpha * y
            z = r / diag
            new = (r * z).sum(0)
            s = z + torch.where(rz > 0, new / rz, rz * 0) * s
            rz = new
        return q * V


def exact(case, seed):
    call, steps = case['call'], case['steps']
    split = lambda u: [u[:, 0:1], u[:, 1:4], u[:, 4:5]]
    cat = lambda v: torch.cat([torch.as_tensor(x, device='cuda').double() for x in v], 1)
    if call == 'serve':
        out = []
        for r in serving.prepare(_requests(case, seed), serving.MeshLibrary()):
            w = serving.make_case(r.key)
            w.build_mesh()
            e = _Exact(w)
            u, S, J = cat(r.inputs[0]), torch.zeros(e.n, 5, dtype=torch.float64, device='cuda', requires_grad=True), 0
            for _ in range(steps):
                u, _, j = e.step(u, w.dt, S)
                J = J + j
            out.append(float((torch.autograd.grad(J, S)[0] * cat(r.inputs[1])).sum()) / steps)
        return out
    w = _workload(case['mesh'], case['a'], case['b'])
    e = _Exact(w)
    x, seeds = _fields(case, seed, torch.float32 if case['precision'] == 'fp32' else torch.float64)
    u, a, dt = cat(x), cat(seeds), w.dt
    zero = torch.zeros_like(u)
    if call == 'viscosity':
        return split(e.smoothed(u, a, dt, 1e-3))
    if call in ('run', 'step'):
        S = cat(_source(case, seed)) if call == 'step' else zero
        hist = []
        with torch.no_grad():
            for _ in range(steps):
                u, dtc, J = e.step(u, dt, S)
                hist.append((dt, float(dtc), float(J)))
                if not w.config.get('fixedTimeStep'):
                    dt = min(2 * w.config.get('CFL', 1.2) / float(dtc), dt * w.config.get('stepFactor', 1.2))
        if call == 'run':
            return split(u) + [torch.tensor(hist, dtype=torch.float64).T]
        return split(u) + [hist[0][1], hist[0][2]]
    u.requires_grad_(True)
    S = (cat(_source(case, seed)) if call == 'map' else zero).requires_grad_(True)
    if call in ('solve', 'sweep'):
        v, J, dts = u, [], []
        for _ in range(steps):
            v, dtc, j = e.step(v, dt, S)
            J.append(j)
            dts.append(dt)
            if call == 'solve' and not w.config.get('fixedTimeStep'):
                dt = min(2 * w.config.get('CFL', 1.2) / float(dtc), dt * w.config.get('stepFactor', 1.2))
        total = sum(J) + ((v * a).sum() if call == 'solve' else 0)
        gu, gS = torch.autograd.grad(total, [u, S]) if total.requires_grad else (zero, zero)
        J = torch.stack([j.detach() for j in J])
        if call == 'solve':
            return split(v.detach()) + [J] + split(gu) + split(gS)
        return [[float((gS * cat(_source(case, seed))).sum()) / steps], split(gu), J.tolist()]
    leaves = []
    if call == 'mesh':
        for k in GRADS:
            e.t[k] = e.t[k].requires_grad_(True)
            leaves.append(e.t[k])
    v, dtc, J = e.step(u, dt, S)
    g = torch.autograd.grad((v * a).sum() + J, [u, S] + leaves, allow_unused=True)
    adj = split(g[0]) + split(g[1])
    if call == 'mesh':
        return adj + [torch.zeros_like(t) if x is None else x for x, t in zip(g[2:], leaves)]
    v, J = v.detach(), J.detach()
    if call == 'map':
        return split(v) + [dtc.reshape(1, 1), J.reshape(1, 1)] + adj
    return split(v) + [float(dtc), float(J)] + adj
