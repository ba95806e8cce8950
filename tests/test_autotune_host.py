"""Host logic of tune_integrator with CPU stand-ins for the launches and the knobs: which shape it keeps when the library's own
shape agrees, when it does not, and when a launch fails."""
import types

import pytest
import torch

from spitfire_gb300 import autotune as AT
from spitfire_gb300 import build


class FakeIntegrator:
    """run() in milliseconds by knobs; the library's own shape (0, 0) ends one reactor a step later if `jump`."""

    def __init__(self, jump=False, fail_at=None):
        self.mech = types.SimpleNamespace(knobs={'integrate_scratch': 2, 'integrate_warps': 5})
        self.jump, self.fail_at = jump, fail_at

    def shape(self):
        return self.mech.knobs['integrate_scratch'], self.mech.knobs['integrate_warps']

    def run(self, q0, pressures=None):
        if self.shape() == self.fail_at:
            raise ValueError('launch failed')
        t = torch.tensor([1., 2., 0.], dtype=torch.float64)
        if self.jump and self.shape() == (0, 0):
            t[1] *= 1.01
        return dict(t=t, q=torch.ones(3, 2), status=torch.ones(3, dtype=torch.int32))


@pytest.fixture
def tuner(monkeypatch):
    def use(integrator, ms):
        monkeypatch.setattr(AT, 'set_tuning', lambda mech, k, v: mech.knobs.__setitem__(k, v))
        monkeypatch.setattr(AT, 'get_tuning', lambda mech, k: mech.knobs[k])
        monkeypatch.setattr(AT, '_fitting_warps', lambda i: 8)
        monkeypatch.setattr(AT, '_time', lambda fn, reps: ms.get(integrator.shape(), 9.))
        monkeypatch.setattr(AT, '_torch', lambda: types.SimpleNamespace(
            equal=torch.equal, cuda=types.SimpleNamespace(synchronize=lambda: None)))
        return AT.tune_integrator(integrator, None)
    return use


@pytest.mark.parametrize('own,jump,expected', [(1., False, (0, 0)), (5., False, (2, 6)), (1., True, (2, 6))])
def test_shape_kept(tuner, own, jump, expected):
    f = FakeIntegrator(jump=jump)
    best, times = tuner(f, {(2, 6): 3., (0, 0): own})
    assert best == expected and f.shape() == expected
    assert ((0, 0) in times) == (not jump)


@pytest.mark.parametrize('fail_at', [(3, 8), (2, 6), (0, 0)])
def test_knobs_restored_when_a_launch_fails(tuner, fail_at):
    f = FakeIntegrator(fail_at=fail_at)
    with pytest.raises(ValueError):
        tuner(f, {})
    assert f.shape() == (2, 5)


def test_saved_choices_belong_to_the_kernels_that_were_timed(monkeypatch, tmp_path):
    """load() finds what save() wrote, and no longer once a kernel source has changed."""
    src = tmp_path / 'csrc'
    src.mkdir()
    (src / 'a.cu').write_text('one')
    (src / 'note.txt').write_text('no kernel')
    monkeypatch.setattr(build, 'CSRC', str(src))
    monkeypatch.setattr(AT, 'CACHE_DIR', str(tmp_path / 'tuning'))
    monkeypatch.setattr(AT, '_torch', lambda: types.SimpleNamespace(
        cuda=types.SimpleNamespace(get_device_name=lambda: 'a GPU')))
    knobs = {name: 0 for name in AT.KNOBS}
    knobs['group_jac'] = 16
    monkeypatch.setattr(AT, 'get_tuning', lambda mech, k: knobs[k])
    applied = {}
    monkeypatch.setattr(AT, 'set_tuning', lambda mech, k, v: applied.__setitem__(k, v))
    mech = types.SimpleNamespace(mech_data_json=lambda: {'species': 2})
    AT.save(mech, {})
    assert AT.load(mech) == knobs and applied == knobs
    (src / 'note.txt').write_text('still none')
    assert AT.load(mech) == knobs
    (src / 'a.cu').write_text('two')
    assert AT.load(mech) is None
