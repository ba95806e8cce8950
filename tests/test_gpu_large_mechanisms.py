"""Mechanisms at the limit of the shared memory: what fits one narrow group of threads per state runs at every batch size."""
import ctypes as C

import numpy as np
import pytest

import large_mechanism as LM

pytestmark = pytest.mark.gpu

NS = 53
# doubles of one group's scratch beside the blob
DOUBLES = {'rhs': lambda lay: lay['rhs'], 'jac': lambda lay: lay['total'], 'param': lambda lay: lay['rhs'] + NS + 2,
           'flamelet_rhs': lambda lay: lay['rhs'] + NS + 2, 'flamelet_jac': lambda lay: lay['total'] + NS + 2}


def _filled(kind, wide_rest):
    """A mechanism that leaves less shared memory beside one narrow group than a wide group's reductions take."""
    def need(k, small=0):
        lay = LM.mechanism(k, small).griffon.scratch_layout()
        return lay['blob_bytes'] + 8 * DOUBLES[kind](lay) + 64
    k = LM.search(need, LM.SMEM, 500, 1400)
    small = 0
    while LM.SMEM - need(k, small) >= wide_rest:
        small += 1
    assert 0 <= LM.SMEM - need(k, small) < wide_rest
    return LM.mechanism(k, small)


@pytest.mark.parametrize('kind', ['rhs', 'jac'])
def test_reactor_calls(cuda, kind):
    """One state asks for 256 threads, whose reductions do not fit; the call takes fewer and equals the 32-lane kernel to
    rounding (1e-13 row-normwise, as between any two widths), also in the host-buffer form."""
    import torch
    from helpers import colmajor, rownorm_err
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300._desc import reactor_params
    spec = _filled(kind, 256)
    g = spec.griffon
    d = W.gri_states(spec, 3, seed=5)
    q = W.isobaric_state(d)
    P = reactor_params('isobaric')
    if kind == 'rhs':
        run = lambda n: g.reactor_rhs_batch(P, q[:n], pressures=d['p'][:n]).cpu().numpy()[:, None, :]
    else:
        run = lambda n: colmajor(g.reactor_jac_batch(P, q[:n], pressures=d['p'][:n])[1].cpu().numpy(), NS)
    AT.set_tuning(spec, 'group_' + kind, 32)
    ref = run(3)
    AT.set_tuning(spec, 'group_' + kind, 0)
    for n in (1, 3):
        assert rownorm_err(run(n), ref[:n]) < 1e-13
    if kind == 'jac':
        r, J = np.empty((3, NS)), np.empty((3, NS * NS))
        g.reactor_jac_host_batch(P, np.ascontiguousarray(q), r, J, pressures=np.ascontiguousarray(d['p']))
        torch.cuda.synchronize()
        assert rownorm_err(colmajor(J, NS), ref) < 1e-13
    assert g.device_status() == 0


def test_rate_parameter_adjoint(cuda):
    """Few items (256 threads each asked for) against the same items in a batch of 32-lane groups, to rounding."""
    import torch
    from spitfire_gb300 import _native as N
    from spitfire_gb300 import workloads as W
    from spitfire_gb300._desc import reactor_params
    spec = _filled('param', 256)
    g = spec.griffon
    nr = len(spec.mech_data['reactions'])
    d = W.gri_states(spec, 2, seed=6)
    P = reactor_params('isobaric')
    out = []
    for reps in (1, 1 + 4 * torch.cuda.get_device_properties(0).multi_processor_count):
        q = torch.tensor(np.tile(W.isobaric_state(d), (reps, 1)), device='cuda')
        p = torch.tensor(np.tile(d['p'], reps), device='cuda')
        w = torch.tensor(np.tile(np.random.default_rng(3).standard_normal((2, NS)), (reps, 1)), device='cuda')
        o = torch.zeros((2 * reps, 2 * nr), dtype=torch.float64, device='cuda')
        N.check(N.load().sf_rate_param_adjoint_batch(g.handle, C.byref(P), 2 * reps, 1, N.ptr(q), N.ptr(p), N.ptr(w),
                                                     N.ptr(o), N.stream_handle()))
        out.append(o[:2].cpu().numpy().reshape(2, nr, 2))
    assert (np.abs(out[0] - out[1]).max(1) <= 1e-12 * np.abs(out[1]).max(1)).all()
    assert g.device_status() == 0


@pytest.mark.parametrize('kind', ['flamelet_rhs', 'flamelet_jac'])
def test_flamelet_points(cuda, kind):
    """A flamelet of few points, against one call per width the other way: the same points in a batch large enough for
    narrower groups, to rounding."""
    import torch
    from spitfire_gb300.flamelet import FlameletBatch, FlameletSetup, FlameletSpec
    spec = _filled(kind, 256)
    air = spec.stream('TPX', (400., 101325., 'O2:1 N2:3.76'))
    fuel = spec.stream('TPX', (350., 101325., 'CH4:1'))
    setup = lambda: FlameletSetup(FlameletSpec(mech_spec=spec, oxy_stream=air, fuel_stream=fuel, grid_points=9,
                                               stoich_dissipation_rate=1., initial_condition='Burke-Schumann'))
    out = []
    for nf in (1, 400):
        b = FlameletBatch([setup()] * nf)
        s = b.initial_state()
        v = b.rhs(s) if kind == 'flamelet_rhs' else b.jacobian(s)
        out.append(v.reshape(-1)[:v.numel() // nf].clone())
    assert bool(torch.isfinite(out[0]).all())
    assert float((out[0] - out[1]).abs().max()) <= 1e-12 * float(out[1].abs().max())
    assert spec.griffon.device_status() == 0


@pytest.mark.parametrize('which', [0, 1])
def test_tables_up_to_the_plain_layout(cuda, which):
    """The largest mechanism whose FP64 tables and plain scratch fit a block (0: right-hand sides, 1: Jacobians) runs, the
    fixed-point constants' tables or not, in every kernel shape, and an integration of it. 1e-10 row-normwise against the
    CPU oracle: rates near equilibrium cancel to about 1e-4 of their terms."""
    import oracle as orc
    import torch
    from helpers import colmajor, rownorm_err
    from spitfire_gb300 import autotune as AT
    from spitfire_gb300 import workloads as W
    from spitfire_gb300._desc import reactor_params
    from spitfire_gb300.reactors import BatchIntegrator
    k = LM.search(lambda k: LM.plain_need(LM.mechanism(k))[which], LM.SMEM - 64, 400, 1600)
    spec = LM.mechanism(k)
    og = orc.OracleGriffon()
    spec._populate_griffon(og)
    g = spec.griffon
    d = W.gri_states(spec, 3, seed=9)
    q = W.isobaric_state(d)
    P = reactor_params('isobaric')
    ref, refJ = og.reactor_jac_batch(P, q, pressures=d['p'])
    for knob in (0, 8, 16, 32):
        AT.set_tuning(spec, 'group_rhs', knob)
        AT.set_tuning(spec, 'group_jac', knob)
        for n in (1, 3):
            r = g.reactor_rhs_batch(P, q[:n], pressures=d['p'][:n]).cpu().numpy()
            assert rownorm_err(r[:, None, :], ref[:n, None, :]) < 1e-10
            if which == 1:
                J = g.reactor_jac_batch(P, q[:n], pressures=d['p'][:n])[1].cpu().numpy()
                assert rownorm_err(colmajor(J, NS), colmajor(refJ[:n], NS)) < 1e-10
    out = BatchIntegrator(spec, 'isobaric').run(q, pressures=d['p'], stop_at_time=1.e-9, first_time_step=1.e-9,
                                                 max_attempts=3)
    assert bool(torch.isfinite(out['q']).all())
    assert g.device_status() == 0
