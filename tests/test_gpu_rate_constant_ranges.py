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
