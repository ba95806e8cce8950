"""The integrator's workspace: its size does not depend on the number of reactors, so that one asked for at a small batch
serves a large one."""
import pytest

import large_mechanism as LM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('large', [False, True])
def test_workspace_of_a_small_batch_serves_a_large_one(cuda, large):
    """large: a mechanism that leaves shared memory for four warps per block with FP64 factors and for three with FP32 ones,
    so that the two precisions' scratch orders the other way round."""
    import torch
    from spitfire_gb300 import workloads as W
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    from spitfire_gb300.reactors import BatchIntegrator
    spec = ChemicalMechanismSpec.bundled('methane-gri30')
    if large:
        k = LM.search(lambda k: LM.mechanism(k).griffon.scratch_layout()['blob_bytes'], LM.SMEM - 64 - 23400, 600, 1400)
        spec = LM.mechanism(k)
        room = LM.SMEM - 64 - spec.griffon.scratch_layout()['blob_bytes']
        assert room // (718 * 8) == 4 and room // (771 * 8) == 3  # doubles per warp of 53 equations, FP64 and FP32
    bi = BatchIntegrator(spec, 'isobaric')
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    n = 12 * nsm + 1
    sizes = [bi.workspace_bytes(k) for k in (1, nsm, 12 * nsm, n, 100000)]
    assert len(set(sizes)) == 1, sizes
    d = W.gri_states(spec, n, seed=5)
    q = torch.tensor(W.isobaric_state(d), device='cuda')
    p = torch.tensor(d['p'], device='cuda')
    out = bi.allocate(n)
    out['ws'] = bi.allocate(1)['ws']
    bi.launch(q, p, out, bi.controls(stop_at_time=1.e-9, first_time_step=1.e-9, maximum_time_step_count=2, max_attempts=2))
    torch.cuda.synchronize()
    assert bool(torch.isfinite(out['q']).all()) and spec.griffon.device_status() == 0
