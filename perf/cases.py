"""Performance cases of the framework's main paths, each through the entry points a program calls.

A case is a dict of plain values with a "kind":
  jac        reactor right-hand sides and analytical Jacobians of a batch of states (PyCombustionKernels)
  rhs        reactor right-hand sides alone
  newton     factor gamma h J - I for a batch of Jacobians and solve one right-hand side each (NewtonSystems)
  integrate  adaptive ESDIRK64 integration of a batch of reactors to a time (BatchIntegrator)
  flamelet   one implicit stage of a batch of flamelets: residual, iteration matrix gamma h J - I, block-tridiagonal
             factorization and solve (FlameletBatch)
  steady     a steady flamelet library: the pseudo-transient solver, with its eigenvalue bounds, from
             Burke-Schumann profiles (FlameletBatch)
  adjoint    rate-parameter gradients of a batch of reactors: recorded integration and backward sweep (ReactorAdjoint)
Mechanisms and sizes are those of the repository's benchmark workloads and tests (h2-burke, GRI-3.0 methane).
"""
import functools
import json
import math
import os

import numpy as np
import torch

from spitfire_gb300.adjoint import ReactorAdjoint
from spitfire_gb300.flamelet import FlameletBatch, FlameletSetup, FlameletSpec
from spitfire_gb300.linalg import NewtonSystems
from spitfire_gb300.mechanism import ChemicalMechanismSpec
from spitfire_gb300.reactors import BatchIntegrator

MECHS = {'h2': 'h2-burke', 'gri': 'methane-gri30'}
NS = {'h2': 11, 'gri': 53}
NR = {'h2': 27, 'gri': 325}
DATA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'spitfire_gb300', 'data')
F64 = torch.float64
ATM = 101325.


# ------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one state of a small mechanism: a reactor inside a user's own time loop, where the call's latency is all
        dict(name='jac_h2_1', kind='jac', mech='h2', n=1, conf='isobaric', heat='adiabatic', open=False),
        # the small-mechanism benchmark batch
        dict(name='jac_h2_4096', kind='jac', mech='h2', n=4096, conf='isochoric', heat='adiabatic', open=False),
        # a flow solver's cut cell list or one flamelet's grid: fewer states than the GPU has resident warps, ragged
        dict(name='jac_gri_333', kind='jac', mech='gri', n=333, conf='isobaric', heat='adiabatic', open=False),
        # the benchmark's headline batch
        dict(name='jac_gri_65536', kind='jac', mech='gri', n=65536, conf='isochoric', heat='adiabatic', open=False),
        # source terms of a mid-sized mesh of stirred reactors with wall heat loss
        dict(name='rhs_gri_20011', kind='rhs', mech='gri', n=20011, conf='isobaric', heat='diathermal', open=True),
        # Newton algebra of an implicit step over a batch, both linear precisions
        dict(name='newton_54_8192', kind='newton', m=54, n=8192, precision=0),
        dict(name='newton_53_2500_fp32', kind='newton', m=53, n=2500, precision=1),
        # reactor ensembles integrated through ignition: a study of a few hundred, and of a small mechanism
        dict(name='integrate_gri_300', kind='integrate', mech='gri', n=300, conf='isobaric', t_end=1.e-4),
        dict(name='integrate_h2_1000', kind='integrate', mech='h2', n=1000, conf='isochoric', t_end=8.e-5),
        # implicit stage of a flamelet library with grids of different sizes
        dict(name='flamelet_gri_8x97', kind='flamelet', mech='gri', nf=8, points=97),
        # a whole steady library build of a few dissipation rates
        dict(name='steady_gri_3x48', kind='steady', mech='gri', nf=3, points=48),
        # parameter gradients of a small ensemble (forward with recording, and backward)
        dict(name='adjoint_gri_64', kind='adjoint', mech='gri', n=64, t_end=5.e-5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['jac', 'jac', 'rhs', 'newton', 'integrate', 'flamelet', 'steady', 'adjoint'])
    mech = rng.choice(['h2', 'gri', 'gri'])
    if kind in ('jac', 'rhs'):
        return dict(kind=kind, mech=mech, n=_log_int(rng, 1, 65536), conf=rng.choice(['isobaric', 'isochoric']),
                    heat=rng.choice(['adiabatic', 'adiabatic', 'isothermal', 'diathermal']),
                    open=rng.random() < 0.25)
    if kind == 'newton':
        return dict(kind=kind, m=rng.choice([11, 12, 53, 54]), n=_log_int(rng, 1, 16384),
                    precision=rng.choice([0, 0, 1]))
    if kind == 'integrate':
        return dict(kind=kind, mech=mech, n=_log_int(rng, 1, 300 if mech == 'gri' else 1000),
                    conf=rng.choice(['isobaric', 'isochoric']), t_end=10. ** rng.uniform(-5., -4.))
    if kind == 'flamelet':
        return dict(kind=kind, mech=mech, nf=rng.randint(1, 8), points=_log_int(rng, 24, 128))
    if kind == 'steady':
        return dict(kind=kind, mech=mech, nf=rng.randint(1, 3), points=rng.randint(24, 48))
    return dict(kind='adjoint', mech='gri', n=_log_int(rng, 1, 64), t_end=10. ** rng.uniform(-5., -4.3))


# ------------------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _mechanism(mech):
    return ChemicalMechanismSpec.bundled(MECHS[mech])


@functools.lru_cache(maxsize=None)
def _table(mech):
    with open(os.path.join(DATA, MECHS[mech] + '.json')) as f:
        return json.load(f)


@functools.lru_cache(maxsize=None)
def _weights(mech):
    d = _table(mech)
    return np.array([sum(n * d['element_mw_map'][e] for e, n in d['species'][s]['atom_map'].items())
                     for s in d['species_order']])


def _air_products(mech, phi):
    """Complete-combustion mass fractions of fuel (H2 or CH4) and air at equivalence ratios phi [n]."""
    names = _table(mech)['species_order']
    X = np.zeros((phi.size, len(names)))
    lean = np.minimum(phi, 1.)
    o2 = (0.5 if mech == 'h2' else 2.)
    X[:, names.index('N2')] = 3.76 * o2 / phi
    X[:, names.index('O2')] = o2 / phi - o2 * lean / phi
    if mech == 'h2':
        X[:, names.index('H2O')] = lean / phi
        X[:, names.index('H2')] = 1. - lean / phi
    else:
        X[:, names.index('CO2')] = lean / phi
        X[:, names.index('H2O')] = 2. * lean / phi
        X[:, names.index('CO')] = 0.5 * (1. - lean / phi)
        X[:, names.index('H2')] = 1. - lean / phi
    Y = X * _weights(mech)
    return Y / Y.sum(1, keepdims=True)


def _states(case, seed):
    """Hot reacting states: T 800-2800 K, 1-40 atm, random mixtures around complete-combustion products."""
    mech, n = case['mech'], case['n']
    rng = np.random.default_rng(seed)
    T = rng.uniform(800., 2500. if mech == 'h2' else 2800., n)
    p = ATM * np.exp(rng.uniform(0., math.log(40.), n))
    Y = rng.standard_exponential((n, NS[mech]))
    Y = 0.7 * Y / Y.sum(1, keepdims=True) + 0.3 * _air_products(mech, rng.uniform(0.5, 2., n))
    rho = p / (8314.46261815324 * T * (Y / _weights(mech)).sum(1))
    if case['conf'] == 'isochoric':
        q = np.hstack([rho[:, None], T[:, None], Y[:, :-1]])
    else:
        q = np.hstack([T[:, None], Y[:, :-1]])
    feed = _fresh(mech, np.array([0.8]))[0]
    return q, p, feed


def _fresh(mech, phi):
    """Mass fractions of unburnt fuel and air at equivalence ratios phi [n]."""
    names = _table(mech)['species_order']
    X = np.zeros((phi.size, len(names)))
    o2 = (0.5 if mech == 'h2' else 2.)
    X[:, names.index('H2' if mech == 'h2' else 'CH4')] = phi
    X[:, names.index('O2')] = o2
    X[:, names.index('N2')] = 3.76 * o2
    Y = X * _weights(mech)
    return Y / Y.sum(1, keepdims=True)


HEAT = dict(fluid_temperature=400., surface_temperature=350., h_convection=20., eps_radiation=0.5,
            surface_area_to_volume=60.)
FEED = dict(inflow_temperature=600., inflow_density=0.6, tau=2.e-3)


def _ensemble(case, seed):
    """Unburnt reactors for an integration: hot enough that part of the ensemble ignites before t_end, and slow
    enough for the default first time step of a microsecond."""
    mech, n = case['mech'], case['n']
    rng = np.random.default_rng(seed)
    if case['kind'] == 'adjoint':
        T, p = rng.uniform(1000., 1400., n), np.full(n, 10. * ATM)
    elif mech == 'h2':
        T, p = rng.uniform(1000., 1250., n), ATM * np.exp(rng.uniform(0., math.log(4.), n))
    else:
        T, p = rng.uniform(1200., 1600., n), ATM * np.exp(rng.uniform(0., math.log(20.), n))
    Y = _fresh(mech, rng.uniform(0.5, 2., n))
    rho = p / (8314.46261815324 * T * (Y / _weights(mech)).sum(1))
    cols = [rho[:, None]] if case.get('conf') == 'isochoric' else []
    return np.hstack(cols + [T[:, None], Y[:, :-1]]), p


def _setups(case, seed):
    rng = np.random.default_rng(seed)
    m = _mechanism(case['mech'])
    air = m.stream('TPX', (rng.uniform(300., 500.), ATM, 'O2:1 N2:3.76'))
    fuel = m.stream('TPX', (rng.uniform(300., 400.), ATM, 'H2:1 N2:1' if case['mech'] == 'h2' else 'CH4:1'))
    out = []
    for k in range(case['nf']):
        # grids from two thirds of `points` up to `points`, dissipation rates over two decades
        nz = case['points'] - (case['points'] // 3) * k // max(case['nf'], 2)
        chi = 10. ** (rng.uniform(-1., 0.) + 2. * k / max(case['nf'], 2))
        out.append(FlameletSetup(FlameletSpec(mech_spec=m, oxy_stream=air, fuel_stream=fuel, grid_points=int(nz),
                                              stoich_dissipation_rate=float(chi),
                                              initial_condition='Burke-Schumann')))
    return out


def _newton_inputs(case, seed):
    """Jacobians shaped as chemistry makes them: every column is one species' destruction rate, shared out among a
    third of the others; rates over nine decades. gamma h as an implicit step of such a system has it."""
    n, m = case['n'], case['m']
    gen = torch.Generator(device='cuda').manual_seed(int(seed))
    r = lambda *s: torch.rand(*s, generator=gen, dtype=F64, device='cuda')
    rate = 10. ** (9. * r(n, m))
    share = torch.where(r(n, m, m) < 1. / 3., r(n, m, m) / m, 0.)         # [column, row]
    J = rate[:, :, None] * (share - torch.diag_embed(0.5 + r(n, m)))
    return J.reshape(n, m * m), 10. ** (-9. + 4. * r(n)), r(n, m) - 0.5


def prepare(case, seed):
    kind = case['kind']
    dev = lambda a: torch.tensor(a, dtype=F64, device='cuda')
    if kind in ('jac', 'rhs'):
        g = _mechanism(case['mech']).griffon
        q, p, feed = _states(case, seed)
        feed = dev(feed)
        kw = dict(HEAT) if case['heat'] == 'diathermal' else {}
        if case['open']:
            kw.update(FEED, inflow_Y_ptr=feed.data_ptr())
        params = g.reactor_params(case['conf'], heat_transfer=case['heat'], open_=case['open'], **kw)
        return dict(case=case, g=g, q=dev(q), p=dev(p), params=params, feed=feed)
    if kind == 'newton':
        J, gh, b = _newton_inputs(case, seed)
        return dict(case=case, J=J, gh=gh, b=b, system=NewtonSystems(case['n'], case['m'], case['precision']))
    if kind == 'integrate':
        q, p = _ensemble(case, seed)
        return dict(case=case, q=dev(q), p=dev(p), bi=BatchIntegrator(_mechanism(case['mech']), case['conf']))
    if kind == 'adjoint':
        q, p = _ensemble(case, seed)
        return dict(case=case, q=dev(q), p=dev(p), adj=ReactorAdjoint(_mechanism(case['mech'])))
    fb = FlameletBatch(_setups(case, seed))
    state = fb.initial_state()
    if kind == 'steady':
        return dict(case=case, fb=fb, state=state)
    return dict(case=case, fb=fb, state=state, prefactor=torch.tensor(_prefactors(case['nf']), device='cuda'))


def _prefactors(nf):
    """gamma h of every flamelet's time step, two decades around a microsecond."""
    return 0.25e-6 * 10. ** np.linspace(-1., 1., nf)


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'jac':
        return state['g'].reactor_jac_batch(state['params'], state['q'], pressures=_pressures(state))
    if kind == 'rhs':
        return state['g'].reactor_rhs_batch(state['params'], state['q'], pressures=_pressures(state))
    if kind == 'newton':
        system = state['system'].factor(state['J'], state['gh'])
        return [system.solve(state['b']), system.A]
    if kind == 'integrate':
        out = state['bi'].run(state['q'], pressures=_pressures(state), stop_at_time=case['t_end'], max_attempts=20000)
        return [out['q'], out['t'], out['status']]
    if kind == 'adjoint':
        traj = state['adj'].forward(state['q'], state['p'], t_end=case['t_end'])
        return [traj.q_end, traj.tau_s, state['adj'].backward(traj)['theta']]
    fb = state['fb']
    if kind == 'steady':
        s, converged, iterations = fb.steady_solve_psitc(state['state'])
        return [s, converged.int()]
    rhs = fb.rhs(state['state'])
    matrix = fb.jacobian(state['state'], scale_and_offset=True, prefactor=state['prefactor']).clone()
    fb.factor()
    return [rhs, matrix, fb.solve(rhs)]


def _pressures(state):
    return state['p'] if state['case']['conf'] == 'isobaric' else None


# -------------------------------------------------------------------------------------------------------- work
def _rhs_flops(mech):
    # per species: NASA7 polynomials and a Gibbs factor (80); per reaction: forward and reverse constants, two
    # mass-action products and the net rates (70)
    return 80. * NS[mech] + 70. * NR[mech]


def _jac_flops(mech):
    # the right-hand side, each reaction's derivatives (50) and its column entries (4 species on 4 rows), and the
    # dense third-body and closure part of each entry
    return _rhs_flops(mech) + 82. * NR[mech] + 4. * NS[mech] ** 2


def work(case):
    kind = case['kind']
    if kind in ('jac', 'rhs'):
        mech, n = case['mech'], case['n']
        iso = case['conf'] == 'isobaric'
        neq = NS[mech] + (0 if iso else 1)
        doubles = 2 * neq + (1 if iso else 0) + (neq * neq if kind == 'jac' else 0)
        return dict(bytes=8. * n * doubles, flops=n * (_jac_flops(mech) if kind == 'jac' else _rhs_flops(mech)))
    if kind == 'newton':
        n, m = case['n'], case['m']
        return dict(bytes=8. * n * (2 * m * m + 2 * m + 1), flops=n * (2. / 3. * m ** 3 + 2. * m * m))
    if kind in ('integrate', 'adjoint'):
        mech, n = case['mech'], case['n']
        neq = NS[mech] + 1
        # steps grow by a tenth from 1 us to the end time, about half as many again through an ignition, at least 40;
        # a step is one Jacobian, one factorization and about fifteen right-hand sides and solves
        steps = max(40., 1.5 * math.log(1. + 0.1 * case['t_end'] / 1.e-6) / math.log(1.1))
        step = _jac_flops(mech) + 2. / 3. * neq ** 3 + 15. * (_rhs_flops(mech) + 2. * neq * neq)
        if kind == 'adjoint':  # six stage Jacobians, five factorizations, two outputs' solves and products, parameters
            step += 6. * _jac_flops(mech) + 5. * 2. / 3. * neq ** 3 + 2. * 6. * 4. * neq * neq + 12. * 10. * NR[mech]
        outputs = 2 * neq + 2 + (2 * (2 * NR[mech] + neq) if kind == 'adjoint' else 0)
        return dict(bytes=8. * n * outputs, flops=n * steps * step)
    ns = NS[case['mech']]
    points = sum(case['points'] - (case['points'] // 3) * k // max(case['nf'], 2) - 2 for k in range(case['nf']))
    solve = points * (2. * ns ** 3 + 6. * ns * ns)     # block inverses and the block sweeps
    if kind == 'steady':
        # about 40 iterations, every other with a new Jacobian and its eigenvalues (10 n^3)
        return dict(bytes=8. * points * ns * 2,
                    flops=40. * points * _rhs_flops(case['mech'])
                    + 20. * (solve + points * (_jac_flops(case['mech']) + 10. * ns ** 3)))
    return dict(bytes=8. * points * (ns * ns + 6. * ns),
                flops=points * (_rhs_flops(case['mech']) + _jac_flops(case['mech'])) + solve)


# ------------------------------------------------------------------------------------------------------- exact
class _Chemistry:
    """Mass-action kinetics with NASA7 thermodynamics in plain 64-bit torch, from the mechanism's data file."""

    def __init__(self, mech, device):
        d = _table(mech)
        names = d['species_order']
        t = lambda a: torch.tensor(np.array(a), dtype=F64, device=device)
        self.Ru, self.pref = d['gas_constant'], d['ref_pressure']
        self.M = t(_weights(mech))
        cps = [d['species'][s]['cp'] for s in names]
        self.tmin, self.tmid, self.tmax = (t([c[j] for c in cps]) for j in (1, 2, 3))
        self.lo, self.hi = t([c[4] for c in cps]).T, t([c[5] for c in cps]).T
        rx, ns = d['reactions'], len(names)
        one = ns  # index of a column of ones beside the concentrations
        sides = []
        for side in (1, 2):
            lists = [[names.index(s) for s, v in r[side].items() for _ in range(int(v))] for r in rx]
            most = max(map(len, lists))
            sides.append(torch.tensor([x + [one] * (most - len(x)) for x in lists], device=device).T)
        self.reac, self.prod = sides
        nu = np.zeros((len(rx), ns))
        for r, x in enumerate(rx):
            for s, v in x[1].items():
                nu[r, names.index(s)] += v
            for s, v in x[2].items():
                nu[r, names.index(s)] -= v
        self.nu = t(nu)                                    # reactants minus products
        self.rev = t([1. if r[3] else 0. for r in rx])
        self.A, self.b, self.E = (t([r[j] for r in rx]) for j in (4, 5, 6))
        body = [i for i, r in enumerate(rx) if r[0] != 'simple']
        eff = np.array([[rx[i][7].get(s, rx[i][8]) for s in names] for i in body])
        self.eff = t(eff)
        self.body = torch.tensor(body, device=device)
        self.simple_body = torch.tensor([rx[i][0] == 'three-body' for i in body], device=device)
        fall = [rx[i] if rx[i][0] in ('Lindemann', 'Troe') else None for i in body]
        self.A0, self.b0, self.E0 = (t([f[j] if f else 1. for f in fall]) for j in (9, 10, 11))
        self.troe = torch.tensor([f is not None and f[0] == 'Troe' for f in fall], device=device)
        tr = [list(f[12]) if f is not None and f[0] == 'Troe' else [0.5, 1., 1., 0.] for f in fall]
        self.tr = t(tr).T

    def thermo(self, T):
        """cp, h per unit mass [n, ns] and g/RT."""
        def pick(x):
            return torch.where((x <= self.tmid)[None], self.lo[:, None], self.hi[:, None])
        Tc = T[:, None].expand(-1, self.M.numel())
        x = torch.minimum(torch.maximum(Tc, self.tmin), self.tmax)
        R = self.Ru / self.M
        a = pick(x)
        cp = a[0] + x * (a[1] + x * (a[2] + x * (a[3] + x * a[4])))
        h = a[5] + x * (a[0] + x * (a[1] / 2 + x * (a[2] / 3 + x * (a[3] / 4 + x * a[4] / 5)))) + cp * (Tc - x)
        a = pick(Tc)
        hg = a[5] / Tc + a[0] + Tc * (a[1] / 2 + Tc * (a[2] / 3 + Tc * (a[3] / 4 + Tc * a[4] / 5)))
        s = a[0] * torch.log(Tc) + a[6] + Tc * (a[1] + Tc * (a[2] / 2 + Tc * (a[3] / 3 + Tc * a[4] / 4)))
        return R * cp, R * h, hg - s

    def rates(self, T, rho, Y):
        """Net mass production rates [n, ns]."""
        C = rho[:, None] * Y / self.M
        Ce = torch.cat([C, torch.ones_like(C[:, :1])], 1)
        iT, lT = 1. / T[:, None], torch.log(T)[:, None]
        k = lambda A, b, E: A * torch.exp(b * lT - E / self.Ru * iT)
        kf = k(self.A, self.b, self.E)
        g = self.thermo(T)[2]
        kr = kf * self.rev * torch.exp(torch.log(self.pref / self.Ru * iT) * self.nu.sum(1) - g @ self.nu.T)
        product = lambda idx: functools.reduce(torch.mul, [Ce[:, i] for i in idx])
        q = kf * product(self.reac) - kr * product(self.prod)
        conc = C @ self.eff.T
        pr = k(self.A0, self.b0, self.E0) / kf[:, self.body] * conc
        a, T3, T1, T2 = self.tr
        Tc = T[:, None]
        fc = (1 - a) * torch.where(T3 > 1e-8, torch.exp(-Tc / T3), 0.) \
            + a * torch.where(T1 > 1e-8, torch.exp(-Tc / T1), 0.) + torch.where(T2 > 1e-8, torch.exp(-T2 * iT), 0.)
        lpr, lfc = torch.log10(torch.clamp(pr, min=1e-300)), torch.log10(fc)
        c = lpr - 0.4 - 0.67 * lfc
        F = torch.pow(10., lfc / (1. + (c / (0.75 - 1.27 * lfc - 0.14 * c)) ** 2))
        factor = torch.where(self.simple_body, conc, torch.where(self.troe, F, 1.) * pr / (1. + pr))
        q = q * torch.ones_like(q).index_copy(1, self.body, factor)
        return -(q @ self.nu) * self.M

    def reactor(self, q, p, case, feed):
        """Right-hand sides of q [n, neq]."""
        iso = case['conf'] == 'isobaric'
        o = 0 if iso else 1
        T, Y = q[:, o], q[:, o + 1:]
        Y = torch.cat([Y, 1. - Y.sum(1, keepdim=True)], 1)
        im = (Y / self.M).sum(1)
        rho = p / (self.Ru * T * im) if iso else q[:, 0]
        cp, h, _ = self.thermo(T)
        e = h if iso else h - self.Ru * T[:, None] / self.M
        c = (cp * Y).sum(1) - (0. if iso else self.Ru * im)
        w = self.rates(T, rho, Y)
        dT = -(w * e).sum(1) / (rho * c)
        dY = w / rho[:, None]
        drho = torch.zeros_like(T)
        if case['heat'] == 'diathermal':
            H = HEAT
            dT = dT + H['surface_area_to_volume'] / (rho * c) * (
                H['h_convection'] * (H['fluid_temperature'] - T)
                + H['eps_radiation'] * 5.67e-8 * (H['surface_temperature'] ** 4 - T ** 4))
        if case['open']:
            Tin = torch.full_like(T, FEED['inflow_temperature'])
            _, hin, _ = self.thermo(Tin)
            ein = hin if iso else hin - self.Ru * Tin[:, None] / self.M
            f = (1. if iso else FEED['inflow_density'] / rho) / FEED['tau']
            dT = dT + f / c * ((ein - e) * feed).sum(1)
            dY = dY + (f if iso else f[:, None]) * (feed - Y)
            drho = (FEED['inflow_density'] - rho) / FEED['tau']
        if case['heat'] == 'isothermal':
            dT = torch.zeros_like(T)
        return torch.cat(([] if iso else [drho[:, None]]) + [dT[:, None], dY[:, :-1]], 1)

    def jacobian(self, f, q):
        """Column-major Jacobians [n, neq * neq] of f at q by forward differentiation."""
        cols = [torch.func.jvp(f, (q,), (torch.zeros_like(q).index_fill_(1, torch.tensor([k], device=q.device), 1.),))[1]
                for k in range(q.shape[1])]
        return torch.stack(cols, 1).reshape(q.shape[0], -1)


def _exact_flamelet(case, seed, device):
    ns = NS[case['mech']]
    chem = _Chemistry(case['mech'], device)
    closed = dict(conf='isobaric', heat='adiabatic', open=False)
    t = lambda a: torch.tensor(np.asarray(a), dtype=F64, device=device)
    every = [[], [], []]
    for s, gh in zip(_setups(case, seed), _prefactors(case['nf'])):
        n = s.nzi
        q, oxy, fuel = t(s.initial_state).reshape(n, ns), t(s.state_oxy), t(s.state_fuel)
        dz, x = t(s.dz), t(s.x)
        full = torch.cat([oxy[None], q, fuel[None]])
        below, above = full[:-2], full[2:]
        a, b = dz[:-1], dz[1:]
        major, sub, sup = -x[1:-1] / (a * b), x[1:-1] / ((a + b) * a), x[1:-1] / ((a + b) * b)
        p = torch.full((n,), s.pressure, dtype=F64, device=device)
        f = lambda u: chem.reactor(u, p, closed, None)
        Yfull = torch.cat([full[:, 1:], 1. - full[:, 1:].sum(1, keepdim=True)], 1)
        cps = chem.thermo(full[:, 0])[0]
        cpm = (cps * Yfull).sum(1)
        ddz = lambda v: (v[2:] - v[:-2]) / (a + b).reshape([-1] + [1] * (v.dim() - 1))
        slope = 0.5 * x[:n] / cpm[1:-1] * ddz(full[:, 0])  # the dissipation rate is read one point below
        flux = ((cps[1:-1, :-1] - cps[1:-1, -1:]) * ddz(full[:, 1:])).sum(1) + ddz(cpm)
        rhs = f(q) + major[:, None] * q + sub[:, None] * below + sup[:, None] * above
        rhs[:, 0] += slope * flux
        J = chem.jacobian(f, q).reshape(n, ns, ns)         # [point, column, row]
        block = J + major[:, None, None] * torch.eye(ns, dtype=F64, device=device)
        T = q[:, 0].clone()
        dcp = torch.func.jvp(lambda u: chem.thermo(u)[0], (T,), (torch.ones_like(T),))[1]
        block[:, 0, 0] -= slope * ddz(cpm) / cpm[1:-1] * (dcp * Yfull[1:-1]).sum(1)
        eye = torch.eye(ns, dtype=F64, device=device)
        block = gh * block - eye
        lower, upper = gh * sub[1:, None].expand(-1, ns), gh * sup[:-1, None].expand(-1, ns)
        # block Thomas
        G, y = [], []
        for i in range(n):
            Di, ri = block[i].T, rhs[i]
            if i:
                Di = Di - lower[i - 1][:, None] * G[-1] * upper[i - 1][None, :]
                ri = ri - lower[i - 1] * y[-1]
            G.append(torch.linalg.inv(Di))
            y.append(G[-1] @ ri)
        sol = [y[-1]]
        for i in range(n - 2, -1, -1):
            sol.append(y[i] - G[i] @ (upper[i] * sol[-1]))
        every[0].append(rhs.reshape(-1))
        every[1] += [block.reshape(-1), lower.reshape(-1), upper.reshape(-1)]
        every[2].append(torch.stack(sol[::-1]).reshape(-1))
    return [torch.cat(e) for e in every]


def exact(case, seed):
    kind = case['kind']
    device = 'cuda' if torch.cuda.is_available() else 'cpu'
    if kind in ('jac', 'rhs'):
        q, p, feed = (torch.tensor(a, dtype=F64, device=device) for a in _states(case, seed))
        chem = _Chemistry(case['mech'], device)
        rhs, jac = [], []
        for k in range(0, case['n'], 8192):
            f = lambda u: chem.reactor(u, p[k:k + 8192], case, feed)
            rhs.append(f(q[k:k + 8192]))
            if kind == 'jac':
                jac.append(chem.jacobian(f, q[k:k + 8192]))
        return (torch.cat(rhs), torch.cat(jac)) if kind == 'jac' else torch.cat(rhs)
    if kind == 'newton':
        J, gh, b = _newton_inputs(case, seed)
        A = gh[:, None, None] * J.reshape(case['n'], case['m'], case['m']).transpose(1, 2)
        A = A - torch.eye(case['m'], dtype=F64, device=device)
        return [torch.linalg.solve(A, b), A.transpose(1, 2).reshape(case['n'], -1)]
    if kind == 'flamelet':
        return _exact_flamelet(case, seed, device)
    return None  # adaptive integrations and steady solves: minutes in plain torch
