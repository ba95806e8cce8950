"""The group widths the library picks by batch size (one state on 8 to 256 threads, or a thread per state) against an
explicit 32-lane group, at the sizes where the rule changes width and where blocks or groups stay partly empty; and
the integrator's eight-warp groups against one warp per reactor."""
import numpy as np
import pytest

from helpers import colmajor, pair, rownorm_err

pytestmark = pytest.mark.gpu


def _sm_count():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize('mech', ['h2-burke', 'methane-gri30'])
@pytest.mark.parametrize('conf', ['isobaric', 'isochoric'])
@pytest.mark.parametrize('states', [(0, 1), (1, 1), (2, 1), (4, 1), (6, 1), (10, 1), (16, 1), (20, 1), (24, 1), (27, 1), (80, 1), (101, 3)])
def test_group_widths_agree(cuda, mech, conf, states):
    """States per SM up to and one past a line of the rule (the second number: states above that multiple of the SM
    count). Every width sums the same terms in another order: 1e-13 row-normwise, as between any two widths."""
    import torch
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300._desc import reactor_params
    spec, og = pair(mech)
    g = spec.griffon
    base = states[0] * _sm_count()
    d0 = (W.h2_states if mech == 'h2-burke' else W.gri_states)(spec, 257, seed=7)
    for n in {max(base, 1), base + states[1]}:
        d = {k: np.resize(v, (n,) + v.shape[1:]) for k, v in d0.items()}
        q = torch.tensor((W.isobaric_state if conf == 'isobaric' else W.isochoric_state)(d), device='cuda')
        p = torch.tensor(d['p'], device='cuda')
        T, rho, Y = (torch.tensor(d[k], device='cuda') for k in ('T', 'rho', 'Y'))
        P = reactor_params(conf, 'diathermal', fluid_temperature=400., surface_temperature=500., h_convection=10.,
                           eps_radiation=0.5)
        out = {}
        for width in (32, 0):
            for k in ('rates', 'sens', 'rhs', 'jac'):
                AT.set_tuning(spec, 'group_' + k, width)
            rhs, J = g.reactor_jac_batch(P, q, 0, pressures=p)
            m = min(n, 300)  # the sensitivity block of every state would be large; its widths are the Jacobian's
            w, S = g.rates_sens_batch(rho[:m], T[:m], Y[:m])
            out[width] = [g.reactor_rhs_batch(P, q, pressures=p), rhs, J, g.production_rates_batch(T, rho, Y), w, S]
        nq = q.shape[1]
        ns1 = spec.n_species + 1
        for a, b, m in zip(out[0], out[32], (0, 0, nq, 0, 0, ns1)):
            a, b = a.cpu().numpy(), b.cpu().numpy()
            if m:
                a, b = colmajor(a, m), colmajor(b, m)
            assert rownorm_err(a, b) < 1e-13
    assert g.device_status() == 0


@pytest.mark.parametrize('n', [1, 153, 305])
@pytest.mark.parametrize('conf,kw', [
    ('isobaric', {}),
    ('isochoric', dict(heat_transfer='diathermal', convection_temperature=lambda t: 400. + 1.e6 * t,
                       radiation_temperature=400., convection_coefficient=50., radiative_emissivity=0.5,
                       surface_area_to_volume=100.)),
    ('isobaric', dict(mass_transfer='open', mixing_tau=1.e-4, feed_temperature=1300., feed_mass_fractions='table'))])
def test_wide_integration_matches_one_warp_per_reactor(cuda, n, conf, kw):
    """GRI-3.0 reactors below, at and above one and two per SM, an odd and an even number of equations, with and without
    parameter tables: the same steps and status, and states within 1e-9 of the one-warp shape in the weights of the
    Newton iteration, which both converge to 1e-12 in them (the shapes differ in rounding and in the linear solves)."""
    import torch
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300.reactors import BatchIntegrator
    spec, og = pair('methane-gri30')
    d = W.ignition_batch(spec, n, seed=5, T_range=(1200., 1500.), p_log_range=(1., 10.))
    kw = dict(kw)
    if kw.get('feed_mass_fractions') == 'table':
        lean, rich = W.ch4_air_mixture(spec, 0.7), W.ch4_air_mixture(spec, 1.4)
        kw['feed_mass_fractions'] = lambda t: lean + (rich - lean) * min(max(t / 2.e-5, 0.), 1.)
    if conf == 'isochoric':
        rho = d['p'] / (8314.46261815324 * d['T0'] * (d['Y'] / spec.molecular_weights).sum(1))
        q0 = np.hstack([rho[:, None], d['q0']])
    else:
        q0 = d['q0']
    bi = BatchIntegrator(spec, conf, **kw)
    res = {}
    for knob in (2, 0):
        AT.set_tuning(spec, 'integrate_scratch', knob)
        res[knob] = bi.run(q0, pressures=d['p'] if conf == 'isobaric' else None, stop_at_time=2.e-5)
    a, b = res[0], res[2]
    assert torch.equal(a['status'], b['status']) and torch.equal(a['counts'][:, 0], b['counts'][:, 0])
    weight = torch.ones(b['q'].shape[1], dtype=torch.float64, device='cuda')  # the integrator's own error weights
    weight[1 if conf == 'isochoric' else 0] = 1.e-3
    assert float(((a['q'] - b['q']).abs() * weight).max()) < 1e-9
    assert float((a['t'] - b['t']).abs().max()) <= 1e-9 * 2.e-5
    assert spec.griffon.device_status() == 0
