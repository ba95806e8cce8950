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


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('m', [1, 31, 33, 64, 80])
def test_quotients_are_as_accurate_as_a_division(cuda, m, precision):
    """Diagonal factors, so that a solution is a quotient per row: within 0.51 ulp of the exact one (the reciprocal's second part
    and the corrected FP32 product leave 2^-100 and 2^-46 before the rounding) where it is a normal number, over mantissas,
    signs and exponents up to quotients that leave the range on both sides, and zeros of both signs."""
    import torch
    from spitfire_gb300 import _native as N
    rng = np.random.default_rng(m)
    n = 400
    f, e = (np.float64, 500) if precision == 0 else (np.float32, 60)
    rand = lambda lo, hi: np.ldexp(rng.uniform(1., 2., (n, m)) * rng.choice([-1., 1.], (n, m)), rng.integers(lo, hi, (n, m)))
    d, b = rand(-e, e).astype(f), rand(-e, e).astype(f)
    d[0] = np.ldexp(1., rng.integers(-e, e, m))
    b[1] = np.ldexp(1., rng.integers(-e, e, m))
    d[2], b[2] = np.ldexp(d[2], e), np.ldexp(b[2], -e)  # quotients below the range
    if m == 1:  # (an infinite element times a zero of its column would spoil the others)
        d[3], b[3] = np.ldexp(d[3], -e), np.ldexp(b[3], e)  # and above
    b[4] = 0.
    b[5] = -0.
    if precision == 0:
        b[6] = np.ldexp(b[6], -1040)  # subnormal right-hand sides
    lu = np.zeros((n, m * m), dtype=f)
    lu[:, ::m + 1] = d
    dev = lambda a: torch.tensor(a, device='cuda')
    A = torch.zeros((n, m * m), dtype=torch.float64, device='cuda')
    x = torch.empty((n, m), dtype=torch.float64, device='cuda')
    lu, piv, bd = dev(lu), dev(np.tile(np.arange(m, dtype=np.int32), (n, 1))), dev(b.astype(np.float64))
    N.check(N.load().sf_newton_solve_batch(n, m, N.ptr(A), N.ptr(lu), N.ptr(piv), precision, 0, N.ptr(bd), N.ptr(x),
                                           N.stream_handle()))
    x = x.cpu().numpy()
    with np.errstate(all='ignore'):
        q = (b / d).astype(np.float64)
        exact = b.astype(np.longdouble) / d.astype(np.longdouble)
        tiny, big = np.finfo(f).tiny, np.finfo(f).max
        normal = (np.abs(exact) >= 2. * tiny) & (np.abs(exact) <= big / 2.)
        ulp = np.spacing(np.abs(q[normal]).astype(f)).astype(np.longdouble)
        assert float((np.abs(x[normal] - exact[normal]) / ulp).max()) <= 0.51
        zero = np.abs(exact) < np.finfo(f).smallest_subnormal / 4.
        assert (x[zero] == 0.).all()
        if m == 1:  # the sweeps add zeros, which leaves -0 only where there are none
            assert (np.signbit(x[4:6]) == np.signbit(q[4:6])).all()
        over = np.abs(exact) > 4. * np.longdouble(big)
        assert np.array_equal(x[over], q[over])
        rest = ~(normal | zero | over) & np.isfinite(q) & np.isfinite(x)  # within a last place of the ends of the range
        assert np.abs(x[rest] - q[rest]).max(initial=0.) <= np.maximum(np.spacing(np.abs(q[rest]).astype(f)), 0.).max(initial=0.)
