"""Rate constants at both sides of the ranges of their fixed-point form (A, b and E of both signs, the falloff ratio
k0/kinf, the temperature), in every kernel shape, against the formulas in numpy's long double."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = 'unit-rev_troe4_noN_withNTB'
SPECIES = ['A', 'B', 'C', 'D', 'E', 'N']
LD = np.longdouble
TEMPERATURES = [15.9, 16.1, 300., 1500., 6.4e4, 6.6e4]


def _mechanism(reactions):
    """The base mechanism's six species with these reactions: (reactants, products, reversible, A, b, E/R[, A0, b0, E0/R of
    a Lindemann reaction])."""
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    md = copy.deepcopy(ChemicalMechanismSpec.bundled(BASE).mech_data)
    Ru = md['gas_constant']
    rx = []
    for r in reactions:
        head = (dict(r[0]), dict(r[1]), r[2], r[3], r[4], r[5] * Ru)
        rx.append(('simple',) + head if len(r) == 6 else ('Lindemann',) + head + ({}, 1., r[6], r[7], r[8] * Ru))
    md['reactions'] = rx
    return ChemicalMechanismSpec(mech_data=md)


def _log_k(A, b, theta, T):
    """(sign, ln |A T^b exp(-theta / T)|), long double; A = 0: -inf"""
    with np.errstate(divide='ignore'):
        return np.sign(A), np.log(np.abs(LD(A))) + LD(b) * np.log(LD(T)) - LD(theta) / LD(T)


def _g_over_RT(md, s, T):
    _, _, tmid, _, lo, hi = md['species'][s]['cp']
    a = [LD(v) for v in (lo if T <= tmid else hi)]
    T = LD(T)
    h = a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5))) + a[5] / T
    return h - (a[0] * np.log(T) + T * (a[1] + T * (a[2] / 2 + T * (a[3] / 3 + T * a[4] / 4))) + a[6])


def _log_Kc(md, reac, prod, T):
    """ln of kr / kf"""
    nu = {s: reac.get(s, 0) - prod.get(s, 0) for s in SPECIES}
    port = LD(md['ref_pressure']) / (LD(md['gas_constant']) * LD(T))
    return sum(nu.values()) * np.log(port) - sum(v * _g_over_RT(md, s, T) for s, v in nu.items() if v)


def _state(present):
    Y = np.array([1. if s in present else 0. for s in SPECIES])
    return Y / Y.sum()


def _conc(spec, rho, Y):
    return {s: LD(rho) * LD(y) / LD(m) for s, y, m in zip(SPECIES, Y, spec.griffon._rec.species_mw)}


def _evaluate(spec, T, rho, Y):
    """Production rates [shape][state][species] of every kernel shape: the library's choice for one state and for many,
    8, 16 and 32 lanes, a thread per state; and the rates of the sensitivity kernels."""
    import torch
    from spitfire_gb300 import autotune as AT
    g = spec.griffon
    n = len(T)
    out = [np.array([g.production_rates_batch(T[i:i + 1], rho[i:i + 1], Y[i:i + 1]).cpu().numpy()[0] for i in range(n)])]
    reps = 800
    for knob in (0, 8, 16, 32, 1):
        AT.set_tuning(spec, 'group_rates', knob)
        AT.set_tuning(spec, 'group_sens', knob)
        k = reps if knob == 0 else 1
        out.append(g.production_rates_batch(np.tile(T, k), np.tile(rho, k), np.tile(Y, (k, 1))).cpu().numpy()[-n:])
        w, S = g.rates_sens_batch(rho, T, Y)
        out.append(w.cpu().numpy())
    torch.cuda.synchronize()
    assert g.device_status() == 0
    return out


CONSTANTS = [(A, 0.5, 2e3) for A in (1e10, -1e10, 1e-299, 1e-301, -1e-301, 1e299, 1e301)] + \
    [(A, b, 2e3) for A in (1e10, -1e10) for b in (30.9, 31.1, -30.9, -31.1)] + \
    [(A, b, s * theta) for A, b in ((1e10, 0.), (1e-100, -2.3), (-1e10, 0.)) for s in (1., -1.)
     for theta in (3.5e5, 3.599e5, 3.601e5, 3.65e5, 4e5, 6.9e5, 7.1e5)]


@pytest.mark.parametrize('A,b,theta', CONSTANTS)
def test_forward_constant(cuda, A, b, theta):
    """Irreversible A + D -> B + E. The exponent's terms are each rounded to 53 bits at most four times (the constant, the
    logarithm or reciprocal, the product, the sum), so ln k is within 4 eps of the terms' magnitudes."""
    reac, prod = {'A': 1, 'D': 1}, {'B': 1, 'E': 1}
    spec = _mechanism([(reac, prod, False, A, b, theta)])
    Y = _state('AD')
    expect, tol, use = [], [], []
    for T in TEMPERATURES:
        sign, lk = _log_k(A, b, theta, T)
        size = abs(np.log(abs(A))) + abs(b) * np.log(T) + abs(theta) / T
        use.append(abs(lk) < 680. and abs(lk - np.log(LD(abs(A)))) < 690.)  # T^b exp(-theta/T) and the rate are normal
        expect.append(sign * np.exp(lk) if use[-1] else LD(0))
        tol.append(4. * 2.3e-16 * size + 1e-14)
    use = np.array(use)
    if not use.any():
        pytest.skip('no temperature gives a normal constant')
    T = np.array(TEMPERATURES)[use]
    c = _conc(spec, 1., Y)
    q = np.array([e for e, u in zip(expect, use) if u]) * c['A'] * c['D']
    mw = spec.griffon._rec.species_mw[0]
    for w in _evaluate(spec, T, np.ones(T.size), np.tile(Y, (T.size, 1))):
        err = np.abs(w[:, 0] / (-q * LD(mw)) - 1.).astype(float)
        assert (err <= np.array(tol)[use]).all(), (err, T)


@pytest.mark.parametrize('A0', [1e16, -1e16, 1e-291, 1e301])
@pytest.mark.parametrize('b0', [-0.5, 30.9, 31.2])
@pytest.mark.parametrize('theta', [-6.9e5, -4e5, -3.5e5, 500., 3.5e5, 4e5, 6.9e5])
def test_falloff_ratio(cuda, A0, b0, theta):
    """Lindemann falloff with kinf = 1e10 and k0 = A0 T^b0 exp(-theta/T): pr / (1 + pr) of the ratio; the tolerance as
    above, the ratio's logarithm with two more rounded terms."""
    reac, prod = {'A': 1, 'D': 1}, {'B': 1, 'E': 1}
    spec = _mechanism([(reac, prod, False, 1e10, 0., 0., A0, b0, theta)])
    Y = _state('AD')
    c = _conc(spec, 1., Y)
    M = c['A'] + c['D']
    T, expect, tol = [], [], []
    for t in TEMPERATURES:
        sign, lk = _log_k(A0, b0, theta, t)
        lr = lk - np.log(LD(1e10))
        if not (abs(lr) < 600. and abs(lk - np.log(LD(abs(A0)))) < 690.):
            continue
        pr = sign * np.exp(lr) * M
        if abs(1. + pr) < 1e-3:
            continue
        T.append(t)
        expect.append(1e10 * pr / (1. + pr))
        size = abs(np.log(abs(A0) / 1e10)) + abs(b0) * np.log(t) + abs(theta) / t
        tol.append((6. * 2.3e-16 * size + 1e-14) * max(1., float(1. / abs(1. + pr))))
    if not T:
        pytest.skip('no temperature gives a normal ratio')
    q = np.array(expect) * c['A'] * c['D']
    mw = spec.griffon._rec.species_mw[0]
    for w in _evaluate(spec, np.array(T), np.ones(len(T)), np.tile(Y, (len(T), 1))):
        err = np.abs(w[:, 0] / (-q * LD(mw)) - 1.).astype(float)
        assert (err <= np.array(tol)).all(), (err, T)


def _g_terms(md, s, T):
    """Sum of the magnitudes of the terms of g/RT."""
    _, _, tmid, _, lo, hi = md['species'][s]['cp']
    a = np.abs(lo if T <= tmid else hi)
    return sum(a[k] * T ** k for k in range(5)) * 2. + a[0] * np.log(T) + a[5] / T + a[6]


def _reaction(sides, A, T):
    """reactants -> products at temperature T with kr / kf far out of range where the sides' energies differ enough: E/R halves
    what ln(kr) would be with none."""
    reac, prod = ({s: side.count(s) for s in side} for side in sides)
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    md = ChemicalMechanismSpec.bundled(BASE).mech_data
    mid = float(_log_Kc(md, reac, prod, T)) / 2. + np.log(abs(A) if A else 1.)
    return reac, prod, True, A, 0., max(0., mid * T)


REVERSIBLE = [(sides, T, A) for A in (1e10, -1e10) for sides, temps in
              ((('ABDD', 'NNNC'), (15.9, 17., 300., 1500.)), (('BD', 'NC'), (15.9, 17., 300., 1500.)),
               (('CC', 'D'), (300., 1500.))) for T in temps] + \
    [(('ABDD', 'NNNC'), T, 1e-302) for T in (15.9, 17., 300., 1500.)] + \
    [(sides, T, 0.) for sides in (('ABDD', 'NNNC'), ('NNNC', 'ABDD'), ('BD', 'NC'), ('CC', 'D'))
     for T in (15.9, 17., 300., 1500., 66000.)]


@pytest.mark.parametrize('sides,T,A', REVERSIBLE)
def test_reverse_constant(cuda, sides, T, A):
    """A state of products alone, so that the rate is the reverse one. E/R is chosen so that kf and kr are normal numbers
    although kr / kf may lie far above the range; A = 0 gives no rate whatever kr / kf is. Below 16 K and above 65,536 K both
    constants are formed in FP64, between them kf alone where A is not positive or out of range. The Gibbs energies'
    terms are rounded to 53 bits at most six times each."""
    spec = _mechanism([_reaction(sides, A, T)])
    md = spec.mech_data
    reac, prod = md['reactions'][0][1], md['reactions'][0][2]
    theta = md['reactions'][0][6] / md['gas_constant']
    Y = _state(''.join(prod))
    c = _conc(spec, 1., Y)
    product = np.prod([c[s] ** v for s, v in prod.items()])
    net = {s: reac.get(s, 0) - prod.get(s, 0) for s in SPECIES}
    i = SPECIES.index(next(iter(prod)))
    mw = LD(spec.griffon._rec.species_mw[i])
    runs = _evaluate(spec, np.array([T]), np.ones(1), Y[None])
    w, S = spec.griffon.rates_sens_batch(np.ones(1), np.array([T]), Y[None])
    assert bool(S.isfinite().all())
    if A == 0.:
        for w in runs:
            assert (w == 0.).all()
        return
    sign, lk = _log_k(A, 0., theta, T)
    lkr = lk + _log_Kc(md, reac, prod, T)
    assert abs(lk) < 700. and abs(lkr) < 700.
    expect = -net[SPECIES[i]] * mw * -sign * np.exp(lkr) * product
    size = abs(np.log(abs(A))) + abs(theta) / T + abs(sum(net.values())) * 10. + \
        sum(abs(v) * _g_terms(md, s, T) for s, v in net.items())
    for w in runs:
        assert abs(float(w[0, i] / expect - 1.)) <= 6. * 2.3e-16 * float(size) + 1e-14, (w[0, i], expect)


@pytest.mark.parametrize('b,theta', [(5e-7, 0.), (1. + 5e-7, 0.), (2. - 5e-7, 5e-7), (-1. + 9e-7, -9e-7), (0., 9e-7)])
def test_temperature_forms(cuda, b, theta):
    """b within 1e-6 of 0, 1, 2 or -1 and E/R below 1e-6 mean exactly A, A T, A T^2 or A / T, in the forward constant, in
    the reverse one and under a falloff ratio."""
    form = round(b)
    T = np.array([300., 1500., 3000.])
    for falloff in (False, True):
        reac, prod = {'B': 1, 'D': 1}, {'N': 1, 'C': 1}
        spec = _mechanism([(reac, prod, True, 1e8, b, theta) + ((1e12, -0.3, 100.) if falloff else ())])
        md = spec.mech_data
        for present in ('BD', 'CN'):
            Y = _state(present)
            c = _conc(spec, 1., Y)
            k = LD(1e8) * LD(1.) * np.array([LD(t) for t in T]) ** form
            if falloff:
                pr = np.array([np.exp(_log_k(1e12, -0.3, 100., t)[1]) for t in T]) / k * sum(c.values())
                k = k * pr / (1. + pr)
            if present == 'CN':
                k = -k * np.array([np.exp(_log_Kc(md, reac, prod, t)) for t in T])
            expect = -k * c[present[0]] * c[present[1]] * LD(spec.griffon._rec.species_mw[1])
            for w in _evaluate(spec, T, np.ones(3), np.tile(Y, (3, 1))):
                assert np.abs((w[:, 1] / expect - 1.).astype(float)).max() <= 6. * 2.3e-16 * 200. + 1e-14


def test_thermodynamics_without_numbers(cuda):
    """A species whose polynomials hold no number makes the reverse rates of its reactions none, in every kernel shape, and leaves
    the irreversible ones alone; a reference pressure of zero makes reverse constants zero where moles are lost."""
    for case in ('nan', 'zero pressure'):
        spec = _mechanism([({'A': 1, 'D': 1}, {'B': 1, 'E': 1}, True, 1e8, 0., 0.), ({'A': 1}, {'C': 1}, False, 1e3, 0., 0.),
                           ({'A': 2}, {'D': 1}, True, 1e3, 0., 0.)])
        md = copy.deepcopy(spec.mech_data)
        if case == 'nan':
            md['species']['E']['cp'] = tuple(md['species']['E']['cp'][:4]) + ([float('nan')] * 7, [float('nan')] * 7)
        else:
            md['ref_pressure'] = 0.
        spec = type(spec)(mech_data=md)
        Y = np.full(6, 1. / 6.)
        for w in _evaluate(spec, np.array([300., 1500.]), np.ones(2), np.tile(Y, (2, 1))):
            if case == 'nan':
                assert np.isnan(w[:, SPECIES.index('B')]).all() and np.isnan(w[:, SPECIES.index('E')]).all()
                assert np.isfinite(w[:, SPECIES.index('C')]).all()
            else:  # 2 A <=> D: one mole lost, so kr has a factor p_ref; A + D <=> B + E has none
                c = _conc(spec, 1., Y)
                q = 1e3 * c['A'] ** 2
                kr = np.array([np.exp(_log_Kc(md | {'ref_pressure': 1.}, {'A': 1, 'D': 1}, {'B': 1, 'E': 1}, T)) for T in (300., 1500.)])
                r = 1e8 * (c['A'] * c['D'] - kr * c['B'] * c['E'])
                mw = LD(spec.griffon._rec.species_mw[SPECIES.index('D')])
                assert np.abs((w[:, SPECIES.index('D')] / (mw * (q - r)) - 1.).astype(float)).max() < 1e-11


@pytest.mark.parametrize('knob', [0, 8, 16, 32, 1])
def test_jacobians_with_constants_of_both_forms(cuda, knob):
    """h2-burke with reversible duplicates whose A is negative, whose b or E/R is beyond the fixed-point range, and a falloff
    reaction whose k0/kinf is: rates, right-hand sides and Jacobians against the CPU oracle, 1e-10 row-normwise as for the
    mechanism itself, for one state (a wide group) and several."""
    import oracle as orc
    from helpers import colmajor, rownorm_err
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300._desc import reactor_params
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    md = copy.deepcopy(ChemicalMechanismSpec.bundled('h2-burke').mech_data)
    Ru = md['gas_constant']
    rx = [list(r) for r in md['reactions']]
    simple = [r for r in rx if r[0] == 'simple' and r[3]]
    troe = [list(r) for r in rx if r[0] == 'Troe']
    for k, change in enumerate(('negative', 'b', 'E')):
        r = list(simple[k])
        if change == 'negative':
            r[4] = -0.3 * r[4]
        elif change == 'b':
            r[4], r[5] = r[4] * 1e-99, r[5] + 32.
        else:
            r[6] = -3.7e5 * Ru
            r[4] = r[4] * 1e-150
        rx.insert(k, r)
    troe[0][10] = troe[0][5] + 32.  # the ratio's exponent
    troe[0][9] = troe[0][9] * 1e-99
    rx = [r for r in rx if r[0] != 'Troe'] + troe
    md['reactions'] = [tuple(r) for r in rx]
    spec = ChemicalMechanismSpec(mech_data=md)
    og = orc.OracleGriffon()
    spec._populate_griffon(og)
    g = spec.griffon
    d = W.h2_states(spec, 40, seed=4)
    q = W.isochoric_state(d)
    P = reactor_params('isochoric')
    neq = q.shape[1]
    ref, refJ = og.reactor_jac_batch(P, q)
    for name in ('group_rates', 'group_rhs', 'group_jac'):
        AT.set_tuning(spec, name, knob)
    w = g.production_rates_batch(d['T'], d['rho'], d['Y']).cpu().numpy()
    assert rownorm_err(w, og.production_rates_batch(d['T'], d['rho'], d['Y'])) < 1e-10
    for n in (1, 40):
        rhs, J = g.reactor_jac_batch(P, q[:n])
        assert rownorm_err(g.reactor_rhs_batch(P, q[:n]).cpu().numpy()[:, None, :], ref[:n, None, :]) < 1e-10
        assert rownorm_err(rhs.cpu().numpy()[:, None, :], ref[:n, None, :]) < 1e-10
        assert rownorm_err(colmajor(J.cpu().numpy(), neq), colmajor(refJ[:n], neq)) < 1e-10
    assert g.device_status() == 0
