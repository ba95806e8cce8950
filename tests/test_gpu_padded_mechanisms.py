"""GRI-3.0 with inert species added, for the paths that only larger systems take: more than 64 equations in the eight-warp
integrator (two parts per row), more than 64 rows in the eigenvalue bounds at every group width, more than 64 equations in
the adjoint's stage solves."""
import copy

import numpy as np
import pytest

import flamelet_cases as FC

pytestmark = pytest.mark.gpu


def padded(ns):
    """(spec, oracle): GRI-3.0's reactions on ns species, copies of N2 before the last species."""
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    import oracle as orc
    md = copy.deepcopy(ChemicalMechanismSpec.bundled('methane-gri30').mech_data)
    names = list(md['species'])
    order = names[:-1] + [f'PAD{k}' for k in range(ns - len(names))] + names[-1:]
    md['species'] = {s: copy.deepcopy(md['species'][s if s in md['species'] else 'N2']) for s in order}
    spec = ChemicalMechanismSpec(mech_data=md)
    og = orc.OracleGriffon()
    spec._populate_griffon(og)
    return spec, og


@pytest.mark.parametrize('ns', [65, 77])
@pytest.mark.parametrize('conf', ['isobaric', 'isochoric'])
def test_wide_integration_of_more_than_64_equations(cuda, ns, conf):
    """Against one warp per reactor: the same steps and status, states within 1e-9 in the weights of the Newton iteration, which
    both converge to 1e-12 in them."""
    import torch
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300.reactors import BatchIntegrator
    spec, og = padded(ns)
    d = W.ignition_batch(spec, 5, seed=5, T_range=(1200., 1500.), p_log_range=(1., 10.))
    Y = 0.9 * d['Y'] + 0.1 / ns
    q0 = np.hstack([d['T0'][:, None], Y[:, :-1]])
    if conf == 'isochoric':
        q0 = np.hstack([(d['p'] / (8314.46261815324 * d['T0'] * (Y / spec.molecular_weights).sum(1)))[:, None], q0])
    bi = BatchIntegrator(spec, conf)
    res = {}
    for knob in (2, 0):
        AT.set_tuning(spec, 'integrate_scratch', knob)
        res[knob] = bi.run(q0, pressures=d['p'] if conf == 'isobaric' else None, stop_at_time=2.e-5, max_attempts=2000)
    a, b = res[0], res[2]
    assert torch.equal(a['status'], b['status']) and torch.equal(a['counts'][:, 0], b['counts'][:, 0])
    weight = torch.ones(q0.shape[1], dtype=torch.float64, device='cuda')
    weight[1 if conf == 'isochoric' else 0] = 1.e-3
    assert float(((a['q'] - b['q']).abs() * weight).max()) < 1e-9
    assert spec.griffon.device_status() == 0


@pytest.mark.parametrize('ns,points', [(65, 9), (80, 9), (105, 9), (65, 200), (105, 200), (65, 400), (105, 400)])
def test_eigenvalue_bounds_of_more_than_64_rows(cuda, ns, points):
    """Up to one point per SM eight warps per point, up to two two, above one, against LAPACK on every point."""
    import flamelet_steady as FS
    from spitfire_gb300.flamelet import FlameletBatch, FlameletSetup, FlameletSpec
    spec, og = padded(ns)
    oxy, fuel, kw = FC.flamelet_case_setup(spec, FC.case('gri'))
    s = FlameletSetup(FlameletSpec(mech_spec=spec, initial_condition='Burke-Schumann', **dict(kw, grid_points=points)))
    rng = np.random.default_rng(5)
    q = s.initial_state.reshape(-1, ns) * (1. + 0.02 * rng.standard_normal((s.nzi, ns)))
    q[:, 1:] += 1.e-3 * rng.random((s.nzi, ns - 1)) / ns
    s.initial_state = np.abs(q).ravel()
    b = FlameletBatch([s])
    op = FS.FlameletOperator(og, s.z, s.x, s.state_oxy, s.state_fuel)
    for dt in (4. * s.max_dissipation_rate, -1.e3):  # most points are proven below the first without their eigenvalues
        vals, e = b.jacobian(b.initial_state(), eig=True, diffterm=dt)
        ref = op.expeig(s.initial_state, dt)
        assert dt > 0. or (ref > 0.).all()
        assert FC.eig_err(e.cpu().numpy(), ref, op, s.initial_state) < 1.
    assert spec.griffon.device_status() == 0


@pytest.mark.parametrize('ns', [65, 77])
def test_adjoint_of_more_than_64_equations(cuda, ns):
    """The native backward sweep against its step loop on the host (1e-9 of the largest gradient, as for GRI-3.0)."""
    import torch
    from spitfire_gb300 import workloads as W
    from spitfire_gb300.adjoint import ReactorAdjoint
    spec, og = padded(ns)
    d = W.ignition_batch(spec, 3, seed=7, T_range=(1300., 1500.), p_log_range=(5., 10.))
    Y = 0.9 * d['Y'] + 0.1 / ns
    q0 = np.hstack([d['T0'][:, None], Y[:, :-1]])
    spec._reaction_yaml_index = list(range(len(spec.mech_data['reactions'])))
    adj = ReactorAdjoint(spec, 'isobaric')
    tr = adj.forward(q0, pressures=d['p'], t_end=1.e-5, max_attempts=2000)
    a, b = adj.backward(tr), adj.backward_host(tr)
    for key in ('theta', 'q0'):
        x, y = a[key].cpu().numpy(), b[key].cpu().numpy()
        for o in range(x.shape[1]):
            assert np.abs(x[:, o] - y[:, o]).max() <= 1e-9 * np.abs(y[:, o]).max(), (key, o)
    assert spec.griffon.device_status() == 0
