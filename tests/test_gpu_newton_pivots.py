"""Newton solves with pivots whose reciprocals are not normal numbers: subnormal, zero and near the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('m', [1, 2, 32, 33, 64, 65, 80])
def test_solve_divides_where_reciprocals_end(cuda, m, precision):
    """Diagonal factors U = diag(d) and right-hand sides 2 d or d / 2, whose quotients are exact."""
    import torch
    from spitfire_gb300 import _native as N
    f, tiny, large = (np.float64, 3e-310, 2. ** 1023) if precision == 0 else (np.float32, 3e-40, 2. ** 127)
    n = 4
    d = np.ones((n, m), dtype=f)
    want = np.full((n, m), 2.)
    for k, at in enumerate((0, m // 2, m - 1)):
        d[k, at] = tiny
    d[3, 0], want[3, 0] = large, 0.5
    b = d.astype(np.float64) * want
    lu = np.zeros((n, m * m), dtype=f)
    lu[:, ::m + 1] = d
    dev = lambda a: torch.tensor(a, device='cuda')
    lu, piv, b = dev(lu), dev(np.tile(np.arange(m, dtype=np.int32), (n, 1))), dev(b)
    A = torch.zeros((n, m * m), dtype=torch.float64, device='cuda')
    x = torch.empty_like(b)
    N.check(N.load().sf_newton_solve_batch(n, m, N.ptr(A), N.ptr(lu), N.ptr(piv), precision, 0, N.ptr(b), N.ptr(x),
                                           N.stream_handle()))
    assert np.array_equal(x.cpu().numpy(), want)
    # a zero pivot: a quotient by zero, and 0 / 0, as in IEEE arithmetic
    lu[0] = 0.
    lu[0, ::m + 1] = 1.
    lu[0, m * m - 1] = 0.
    b[0] = 1.
    N.check(N.load().sf_newton_solve_batch(1, m, N.ptr(A), N.ptr(lu), N.ptr(piv), precision, 0, N.ptr(b), N.ptr(x),
                                           N.stream_handle()))
    assert np.isposinf(x[0, m - 1].item())
