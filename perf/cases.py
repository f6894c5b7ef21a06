"""Performance cases: the work a user of this framework has it do, through its public entry points.

Every case is one pass of a program that keeps one model (a module with its mesh loaded and
``sw_mpas_init_block`` done) on the GPU and gives it new states, perturbations or adjoints:

* the drop-in module routines on host arrays, one step per call, as the reference's driver and
  its demo scripts call them (``step``, ``tlm_adj``);
* many nonlinear steps in one call (``forward``);
* a window's tangent-linear sweep followed by the adjoint of its result, the product a
  variational analysis or a singular-vector iteration asks for (``gradient``), or the adjoint
  sweep alone, for a batch of cost functions of the final state (``adjoint``);
* one RK4 step as an autograd function, forward and backward (``autograd``).

The meshes are the bisected icosahedra of levels 3 to 7 (642 to 163842 cells) with the time step
each of them is run with (75 s on level 7, twice that per coarser level).  States are random smooth
stream functions with winds up to 40 m/s, in geostrophic balance, over eight Gaussian mountains;
perturbations are independent, 0.1 m/s in u and 1 m in h.

Sweeps and forwards in precision 1 compute their stencils in 32 bits, so their results are good
to 32 bits: the program takes them on as float32 (which is what it would store or hand to its
minimiser), and ``run`` returns them so.  Precision 0 and the module routines return float64.
"""
from __future__ import annotations

import functools
import gc
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'mpas-sw-tl-ad_b200'))

from module_sw_mpas import MpasSwModule  # noqa: E402
from mpsw import ic  # noqa: E402
from mpsw.mesh import icosahedral_mesh  # noqa: E402
from mpsw.torch_api import Engine, rk4_step  # noqa: E402

# namelist settings: the default physics; del2 viscosity with bottom drag; everything on
PHYSICS = {
    'default': dict(visc2=0.0, visc4=0.0, drag=False, wind=False),
    'visc2': dict(visc2=1.0e5, visc4=0.0, drag=True, wind=False),
    'full': dict(visc2=1.0e5, visc4=5.0e14, drag=True, wind=True),
}
APVM = 0.5


def _dt(level):
    return 75.0 * 2 ** (7 - level)


def _case(name, kind, level, steps=1, members=1, precision=0, physics='default', snapshots=0):
    c = dict(kind=kind, level=level, steps=steps, members=members, precision=precision, physics=physics,
             snapshots=snapshots)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one model step per call on host arrays: the reference driver's time loop
        _case('step_l5', 'step', 5),
        # one tangent-linear and one adjoint step per call: the reference's demo scripts
        _case('tlm_adj_l5', 'tlm_adj', 5),
        # a day of the plain FP64 forward on the coarse mesh, in quarters
        _case('forward_f64_l5', 'forward', 5, steps=72),
        # the high-resolution forward with 32-bit stencils, one hour
        _case('forward_f32_l7', 'forward', 7, steps=48, precision=1),
        # one differentiable step inside a PyTorch program
        _case('autograd_l5', 'autograd', 5),
        # a single FP64 gradient: the plain form of a tangent-linear / adjoint window
        _case('gradient_f64_l5_b1', 'gradient', 5, steps=32),
        # one block of a block-Lanczos singular-vector iteration
        _case('gradient_f64_l6_b8', 'gradient', 6, steps=8, members=8),
        # batched gradients on the coarse mesh
        _case('gradient_f32_l5_b64', 'gradient', 5, steps=16, members=64, precision=1),
        # an odd number of members, with viscosity and bottom drag
        _case('gradient_f32_l6_b13_visc', 'gradient', 6, steps=8, members=13, precision=1, physics='visc2'),
        # gradients of 64 cost functions of the final state
        _case('adjoint_f32_l6_b64', 'adjoint', 6, steps=12, members=64, precision=1),
        # a long window reversed from a few snapshots
        _case('adjoint_f32_l6_b16_binomial', 'adjoint', 6, steps=20, members=16, precision=1, snapshots=3),
        # batched gradients at high resolution: the headline workload
        _case('gradient_f32_l7_b64', 'gradient', 7, steps=6, members=64, precision=1),
    ]


def _cells(level):
    return 10 * 4 ** level + 2


def _cost(c):
    """Rough size of a pass, in cell updates of one member and RK stage."""
    k = {'step': 1, 'tlm_adj': 6, 'autograd': 6, 'forward': 1, 'gradient': 6, 'adjoint': 4}[c['kind']]
    return k * 4 * _cells(c['level']) * c['steps'] * (c['members'] if c['kind'] in ('gradient', 'adjoint') else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(['step', 'tlm_adj', 'forward', 'forward', 'autograd', 'gradient', 'gradient', 'gradient',
                           'adjoint', 'adjoint'])
        level = rng.randint(3, 7)
        steps, members, precision, snapshots = rng.randint(1, 12), 1, 0, 0
        physics = rng.choice(['default', 'default', 'default', 'visc2', 'full'])
        if kind == 'forward':
            steps = round(math.exp(rng.uniform(math.log(4), math.log(96))))
            precision = rng.randint(0, 1)
        elif kind in ('gradient', 'adjoint'):
            steps = round(math.exp(rng.uniform(math.log(4), math.log(32))))
            members = round(math.exp(rng.uniform(0.0, math.log(64))))
            precision = rng.randint(0, 1)
            if kind == 'adjoint' and rng.random() < 0.3:
                snapshots = rng.randint(2, 4)
        c = _case(None, kind, level, steps, members, precision, physics, snapshots)
        # FP64 members cost twice the bytes of FP32 ones
        if _cost(c) * (2 if precision == 0 and members > 1 else 1) <= most:
            return c


# ---- the model a program keeps --------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _mesh(level):
    """(unit-sphere mesh, Earth-sized mesh, topography) of a level."""
    unit = icosahedral_mesh(level)
    mesh = ic.scale_mesh(unit)
    return unit, mesh, ic.mountains(mesh, 1000)


def _wind_source(level):
    return np.random.default_rng(7).standard_normal((1, 30 * 4 ** level)) * 0.1


def _configure(level, physics):
    mesh, b = _mesh(level)[1:]
    m = MpasSwModule()
    m.nvertlevels = 1
    m.ncells, m.nedges, m.nvertices = mesh['nCells'], mesh['nEdges'], mesh['nVertices']
    m.maxedges, m.maxedges2, m.vertexdegree = mesh['maxEdges'], mesh['maxEdges2'], mesh['vertexDegree']
    m.r3, m.ntracers = 3, 1
    m.var_allocation()
    m.on_a_sphere = True
    for k, v in mesh.items():
        if isinstance(v, np.ndarray):
            setattr(m, k.lower(), v.T)
    m.fvertex = 2.0 * ic.OMEGA * np.sin(mesh['latVertex'])
    m.fedge = 2.0 * ic.OMEGA * np.sin(mesh['latEdge'])
    m.h_s = b
    p = PHYSICS[physics]
    m.config_dt = _dt(level)
    m.config_test_case = 7
    m.config_apvm_upwinding = APVM
    m.config_h_mom_eddy_visc2, m.config_h_mom_eddy_visc4 = p['visc2'], p['visc4']
    m.config_bottom_drag, m.config_wind_stress = p['drag'], p['wind']
    if p['wind']:
        m.u_src = _wind_source(level)
    return m


_kept = {}


def _model(level, physics, twins):
    """The program's model on this mesh (one is kept at a time); twins: with the module's
    tangent-linear and adjoint variables."""
    key = (level, physics, twins)
    if key not in _kept:
        _kept.clear()
        gc.collect()
        m = _configure(level, physics)
        if twins:
            m.var_allocation_tlm()
            m.var_allocation_adj()
        u, h = _flow(level, 0, 'cpu')
        m.u[0, 0], m.h[0, 0] = u.numpy(), h.numpy()
        m.sw_mpas_init_block()
        _kept[key] = m, Engine(m)
    return _kept[key]


# ---- inputs ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _geometry(level, device):
    mesh, b = _mesh(level)[1:]
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=device)  # noqa: E731
    xyz = lambda s: t(np.stack([mesh[a + s] for a in 'xyz'], 1) / ic.A_EARTH)  # noqa: E731
    return (xyz('Cell'), xyz('Vertex'), t(mesh['verticesOnEdge'].astype(np.int64) - 1), t(mesh['dvEdge']),
            t(2.0 * ic.OMEGA * np.sin(mesh['latCell'])), t(b))


def _flow(level, seed, device):
    """A balanced state: psi a random sum of smooth waves (amplitudes falling as the cube of the
    wavenumber), u its discrete rotated gradient scaled to 40 m/s, h = 5500 m + f psi / g - b."""
    xc, xv, voe, dv, f, b = _geometry(level, device)
    rng = np.random.default_rng(seed)
    psi_c, psi_v = torch.zeros_like(f), torch.zeros_like(xv[:, 0])
    for _ in range(24):
        n = rng.uniform(1.0, 12.0)
        d = rng.standard_normal(3)
        k = torch.as_tensor(n * d / np.linalg.norm(d), device=device)
        a, ph = rng.standard_normal() * n ** -3.0, rng.uniform(0.0, 2.0 * math.pi)
        psi_c += a * torch.sin(xc @ k + ph)
        psi_v += a * torch.sin(xv @ k + ph)
    u = -(psi_v[voe[:, 1]] - psi_v[voe[:, 0]]) / dv
    s = 40.0 / u.abs().max()
    # the additive constant of psi is free: the mean depth stays 5500 m
    return u * s, 5500.0 + f * (psi_c - psi_c.mean()) * s / ic.GRAVITY - b


def _members(level, B, seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    du = 0.1 * torch.randn(30 * 4 ** level, B, generator=g, dtype=torch.float64, device=device)
    dh = torch.randn(_cells(level), B, generator=g, dtype=torch.float64, device=device)
    return du, dh


def _inputs(case, seed):
    """State (u, h) and members (du, dh) of a case, on the GPU."""
    u, h = _flow(case['level'], seed, 'cuda')
    du, dh = _members(case['level'], case['members'], seed, 'cuda')
    return u, h, du, dh


def prepare(case, seed):
    kind = case['kind']
    m, engine = _model(case['level'], case['physics'], kind == 'tlm_adj')
    u, h, du, dh = _inputs(case, seed)
    if kind in ('step', 'tlm_adj', 'forward'):  # the module's routines work on host arrays
        u, h, du, dh = (x.cpu().numpy() for x in (u, h, du[:, 0], dh[:, 0]))
    return dict(case=case, module=m, engine=engine, u=u, h=h, du=du, dh=dh)


def run(state):
    c, m, e = state['case'], state['module'], state['engine']
    u, h, du, dh = state['u'], state['h'], state['du'], state['dh']
    if c['kind'] == 'step':
        m.u[0, 0], m.h[0, 0] = u, h
        for _ in range(c['steps']):
            m.sw_rk4()
        return m.u[0, 0].copy(), m.h[0, 0].copy()
    if c['kind'] == 'tlm_adj':  # the tangent-linear steps carry the state along; the adjoint's are given it
        states = [(u, h)]
        m.u[0, 0], m.h[0, 0] = u, h
        m.u_tl[0, 0], m.h_tl[0, 0] = du, dh
        for _ in range(c['steps']):
            m.sw_rk4_tlm()
            states.append((m.u[0, 0].copy(), m.h[0, 0].copy()))
        tu, th = m.u_tl[0, 0].copy(), m.h_tl[0, 0].copy()
        m.u_ad[0, 0], m.h_ad[0, 0] = tu, th
        for n in reversed(range(c['steps'])):
            m.u[0, 0], m.h[0, 0] = states[n]
            m.sw_rk4_adj()
        return states[-1] + (tu, th, m.u_ad[0, 0].copy(), m.h_ad[0, 0].copy())
    if c['kind'] == 'forward':
        m.u[0, 0], m.h[0, 0] = u, h
        m.sw_rk4_steps(c['steps'], c['precision'])
        t = np.float32 if c['precision'] else np.float64
        return m.u[0, 0].astype(t), m.h[0, 0].astype(t)
    if c['kind'] == 'autograd':
        u, h = u.detach().requires_grad_(), h.detach().requires_grad_()
        u1, h1 = u, h
        for _ in range(c['steps']):
            u1, h1 = rk4_step(u1, h1, e)
        gu, gh = torch.autograd.grad((u1, h1), (u, h), (du[:, 0], dh[:, 0]))
        return u1.detach(), h1.detach(), gu, gh
    t = torch.float32 if c['precision'] else torch.float64
    e.set_state(u, h)
    w = e.window(c['steps'], ckpt_every=16, storage=0 if c['snapshots'] else -1, snapshots=c['snapshots'])
    if c['kind'] == 'adjoint':
        return tuple(x.to(t) for x in w.ad(du, dh, c['precision']))
    tu, th = w.tl(du, dh, c['precision'])
    au, ah = w.ad(tu, th, c['precision'])
    return tuple(x.to(t) for x in (tu, th, au, ah))


def work(case):
    """Per RK stage: the mesh (indices in 32 bits, metrics and weights in the stencils' precision)
    and each prognostic row read and written once; per step the FP64 accumulations read and
    written once.  A tangent-linear or adjoint stage also reads the state it is linearised about."""
    C = _cells(case['level'])
    E, V = 3 * C, 2 * C
    s = 4 if case['precision'] else 8
    mesh = 4 * (14 * E + 12 * C + 6 * V) + s * (12 * E + 2 * C + 5 * V)
    rows = E + C
    forward = 4 * (mesh + 2 * s * rows) + 16 * rows
    B = case['members']
    member = 4 * (mesh + s * rows + 2 * s * rows * B) + 16 * rows * B
    f_fwd, f_mem = 4 * (110 * E + 70 * C + 20 * V), 4 * (180 * E + 120 * C + 35 * V) * B
    sweeps = {'step': 0, 'forward': 0, 'tlm_adj': 2, 'autograd': 1, 'gradient': 2, 'adjoint': 1}[case['kind']]
    n = case['steps']
    return {'bytes': float(n * (forward + sweeps * member)), 'flops': float(n * (f_fwd + sweeps * f_mem))}


# ---- the same results in 64 bits, in plain torch --------------------------------------------------
class _Model64:
    """The shallow-water equations on the mesh as sums over index tables, with the tangent linear
    by the product rule; fields are [n] (states) or [n, B] (members)."""

    def __init__(self, level, physics, device):
        mesh, b = _mesh(level)[1:]
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=device)  # noqa: E731
        index = lambda k: mesh[k].astype(np.int64) - 1  # noqa: E731
        p = PHYSICS[physics]
        self.dt, self.visc2, self.visc4 = _dt(level), p['visc2'], p['visc4']
        self.drag, self.wind = p['drag'], p['wind']
        coe, voe = index('cellsOnEdge'), index('verticesOnEdge')
        self.c1, self.c2, self.v1, self.v2 = t(coe[:, 0]), t(coe[:, 1]), t(voe[:, 0]), t(voe[:, 1])
        self.dc, self.dv = t(mesh['dcEdge']), t(mesh['dvEdge'])
        self.f, self.b = t(2.0 * ic.OMEGA * np.sin(mesh['latVertex'])), t(b)
        self.src = t(_wind_source(level)[0]) if p['wind'] else None
        dc, dv = mesh['dcEdge'], mesh['dvEdge']

        def table(idx, coef):  # slots as columns; empty ones (index -1) weigh nothing
            ok = idx >= 0
            idx = np.where(ok, idx, 0)
            return [(t(idx[:, k]), t(np.where(ok, coef, 0.0)[:, k])) for k in range(idx.shape[1])]
        eoc, eov, voc = index('edgesOnCell'), index('edgesOnVertex'), index('verticesOnCell')
        cell, vert = np.arange(mesh['nCells'])[:, None], np.arange(mesh['nVertices'])[:, None]
        aC, aV = mesh['areaCell'][:, None], mesh['areaTriangle'][:, None]
        out = np.where(coe[eoc][:, :, 0] == cell, 1.0, -1.0)
        self.div = table(eoc, out * dv[eoc] / aC)
        self.ke = table(eoc, 0.25 * dc[eoc] * dv[eoc] / aC)
        self.curl = table(eov, np.where(voe[eov][:, :, 1] == vert, 1.0, -1.0) * dc[eov] / aV)
        cov, kite = index('cellsOnVertex'), mesh['kiteAreasOnVertex']
        self.to_vertex = table(cov, kite / aV)
        part = sum(np.where(cov[voc][:, :, k] == cell, kite[voc][:, :, k], 0.0) for k in range(3))
        self.to_cell = table(voc, part / aC)
        self.perp = table(index('edgesOnEdge'), mesh['weightsOnEdge'])

    @staticmethod
    def _w(c, x):  # a coefficient per entity against a field [n] or [n, B]
        return c if x.dim() == 1 else c[:, None]

    def sum(self, tab, x):
        out = 0.0
        for i, c in tab:
            out = out + self._w(c, x) * x.index_select(0, i)
        return out

    def normal(self, x):
        return (x.index_select(0, self.c2) - x.index_select(0, self.c1)) / self._w(self.dc, x)

    def along(self, x):
        return (x.index_select(0, self.v2) - x.index_select(0, self.v1)) / self._w(self.dv, x)

    def edge_c(self, x):
        return 0.5 * (x.index_select(0, self.c1) + x.index_select(0, self.c2))

    def edge_v(self, x):
        return 0.5 * (x.index_select(0, self.v1) + x.index_select(0, self.v2))

    def dissipation(self, div, vort):
        out = 0.0
        if self.visc2 or self.visc4:
            d2 = self.normal(div) - self.along(vort)
            out = self.visc2 * d2
            if self.visc4:
                out = out - self.visc4 * (self.normal(self.sum(self.div, d2)) - self.along(self.sum(self.curl, d2)))
        return out

    def tend(self, u, h):
        """Tendencies of a state and what its tangent linear needs."""
        he, vort, hv = self.edge_c(h), self.sum(self.curl, u), self.sum(self.to_vertex, h)
        pvv = (self.f + vort) / hv
        v, gpt = self.sum(self.perp, u), self.along(pvv)
        gpn = self.normal(self.sum(self.to_cell, pvv))
        a = APVM * self.dt
        pe = self.edge_v(pvv) - a * (v * gpt + u * gpn)
        ke = self.sum(self.ke, u * u)
        F = u * he
        tu = 0.5 * (pe * self.sum(self.perp, F) + self.sum(self.perp, F * pe))
        tu = tu - self.normal(ke + ic.GRAVITY * (h + self.b)) + self.dissipation(self.sum(self.div, u), vort)
        if self.wind:
            tu = tu + self.src / 1000.0 / he
        if self.drag:
            tu = tu - 1.0e-3 * u * torch.sqrt(2.0 * self.edge_c(ke)) / he
        return tu, -self.sum(self.div, F), (u, he, vort, hv, pvv, v, gpt, gpn, pe, ke, F)

    def tend_tl(self, base, du, dh):
        u, he, vort, hv, pvv, v, gpt, gpn, pe, ke, F = (x[:, None] for x in base)
        a = APVM * self.dt
        dhe, dvort = self.edge_c(dh), self.sum(self.curl, du)
        dpvv = (dvort - pvv * self.sum(self.to_vertex, dh)) / hv
        dgpn = self.normal(self.sum(self.to_cell, dpvv))
        dpe = self.edge_v(dpvv) - a * (self.sum(self.perp, du) * gpt + v * self.along(dpvv) + du * gpn + u * dgpn)
        dke = self.sum(self.ke, 2.0 * u * du)
        dF = du * he + u * dhe
        dtu = 0.5 * (dpe * self.sum(self.perp, F) + pe * self.sum(self.perp, dF) + self.sum(self.perp, dF * pe + F * dpe))
        dtu = dtu - self.normal(dke + ic.GRAVITY * dh) + self.dissipation(self.sum(self.div, du), dvort)
        if self.wind:
            dtu = dtu - self.src[:, None] / 1000.0 * dhe / he ** 2
        if self.drag:
            k = torch.sqrt(2.0 * self.edge_c(ke))
            dtu = dtu - 1.0e-3 * (du * k / he + u * self.edge_c(dke) / (k * he) - u * k * dhe / he ** 2)
        return dtu, -self.sum(self.div, dF)

    def rk4(self, f, u, h):
        """One RK4 step with the tendencies f(stage, u, h)."""
        dt = self.dt
        tu, th = f(0, u, h)
        nu, nh = u + dt / 6.0 * tu, h + dt / 6.0 * th
        for k, c, w in ((1, dt / 2.0, dt / 3.0), (2, dt / 2.0, dt / 3.0), (3, dt, dt / 6.0)):
            tu, th = f(k, u + c * tu, h + c * th)
            nu, nh = nu + w * tu, nh + w * th
        return nu, nh

    def step(self, u, h, keep=None):
        def f(k, pu, ph):
            tu, th, base = self.tend(pu, ph)
            if keep is not None:
                keep.append(base)
            return tu, th
        return self.rk4(f, u, h)

    def step_tl(self, bases, du, dh):
        return self.rk4(lambda k, pu, ph: self.tend_tl(bases[k], pu, ph), du, dh)

    def step_ad(self, bases, au, ah):
        """The transpose of step_tl, by differentiating it (it is linear)."""
        with torch.enable_grad():
            x = torch.zeros_like(au).requires_grad_(), torch.zeros_like(ah).requires_grad_()
            return torch.autograd.grad(self.step_tl(bases, *x), x, (au, ah))


@torch.no_grad()
def exact(case, seed):
    u, h, du, dh = _inputs(case, seed)
    M = _Model64(case['level'], case['physics'], 'cuda')
    states = [(u, h)]
    for _ in range(case['steps']):
        states.append(M.step(*states[-1]))
    kind = case['kind']
    if kind in ('step', 'forward'):
        return states[-1]
    out = []

    def bases(n):
        keep = []
        M.step(*states[n], keep)
        return keep
    if kind in ('tlm_adj', 'gradient'):
        for n in range(case['steps']):
            du, dh = M.step_tl(bases(n), du, dh)
        out += [du, dh]
    for n in reversed(range(case['steps'])):
        du, dh = M.step_ad(bases(n), du, dh)
    out += [du, dh]
    if kind in ('tlm_adj', 'autograd'):
        out = list(states[-1]) + [x[:, 0] for x in out]
    return tuple(out)
