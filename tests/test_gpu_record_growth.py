"""Recorded integrations whose record grows: the reactors integrated again by themselves, and the rest of a batch so large
that an integration without a record takes another kernel, equal one run whose record fits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('per_sm', [1, 12, 13])
def test_regrown_record_equals_one_fitting_run(cuda, per_sm):
    import torch
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    from spitfire_gb300.reactors import BatchIntegrator
    spec = ChemicalMechanismSpec.bundled('methane-gri30')
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    n = n - 7 if per_sm <= 12 else n
    X = np.zeros((n, spec.n_species))
    X[:, spec.species_index('CH4')] = 1.
    X[:, spec.species_index('O2')] = 2.
    X[:, spec.species_index('N2')] = 7.52
    Y = X * spec.molecular_weights
    Y /= Y.sum(1, keepdims=True)
    T = np.linspace(1100., 1900., n)
    q0 = torch.tensor(np.hstack([T[:, None], Y[:, :-1]]), device='cuda')
    bi = BatchIntegrator(spec, 'isobaric', pressure=10. * 101325.)
    ip = bi.controls(stop_at_time=3.e-5, max_attempts=1024)
    one, rec = bi.record(q0, None, ip, 1024)
    steps = one['counts'][:, 0].cpu().numpy()
    assert (one['status'].cpu().numpy() != 7).all()
    capacity = int(np.quantile(steps, 0.95))  # about one reactor in twenty is integrated again
    assert steps.max() > capacity
    out, grown = bi.record(q0, None, ip, capacity)
    for k in ('q', 't', 'counts', 'status'):
        assert torch.equal(out[k], one[k]), k
    for i in range(0, n, max(1, n // 50)):
        assert torch.equal(grown[i, :steps[i]], rec[i, :steps[i]])
    full = np.nonzero(steps > capacity)[0]
    for i in full[:: max(1, full.size // 20)]:
        assert torch.equal(grown[i, :steps[i]], rec[i, :steps[i]])
    assert spec.griffon.device_status() == 0
