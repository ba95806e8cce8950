"""The fixed-point exponential, logarithm, reciprocal and reciprocal square root of the kernels (spitfire_gb300/csrc/fixed_point.cuh) against
numpy's long double (113 bits on the Arm host of the GPU; on narrower hosts the test is skipped), over the ranges the
rate code meets and at their ends."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(x):
    import torch
    import bench
    L = C.CDLL(bench.build_probes())
    L.bench_fixed_values.argtypes = [C.c_void_p] * 5 + [C.c_longlong, C.c_void_p]
    xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = [torch.empty_like(xd) for _ in range(4)]
    assert L.bench_fixed_values(xd.data_ptr(), *[o.data_ptr() for o in out], xd.numel(),
                                torch.cuda.current_stream().cuda_stream) == 0
    return [o.cpu().numpy() for o in out]


def _ulp(ref):
    return np.spacing(np.abs(ref).astype(np.float64)).astype(np.longdouble)


@pytest.mark.parametrize('kind', ['wide', 'kinetic', 'near_one', 'binade_ends'])
def test_accuracy(cuda, kind):
    """Bounds by the method's error analysis: 20 units of 2^-63 of the exponential's mantissa (0.51 ulp rounded), 6 units
    of 2^-64 of the reciprocal's and the reciprocal square root's (0.51 ulp), 2^-58.9 absolute of log2 (rounded to half an ulp of the result)."""
    if np.finfo(np.longdouble).nmant < 100:
        pytest.skip('needs a long double wider than the bounds')
    rng = np.random.default_rng(3)
    n = 200000
    x = {'wide': rng.uniform(-707.9, 707.9, n), 'kinetic': rng.uniform(-80., 40., n),
         'near_one': 1. + rng.uniform(-1., 1., n) * 10. ** rng.uniform(-16., -1., n),
         'binade_ends': np.ldexp(1. + rng.integers(-3, 4, n) * 2. ** -52, rng.integers(-9, 10, n))}[kind]
    e, l, r, s = _values(x)
    X = x.astype(np.longdouble)
    ref = np.exp(X)
    assert float((np.abs(e.astype(np.longdouble) - ref) / _ulp(ref)).max()) <= 0.51
    ref = 1. / X
    assert float((np.abs(r.astype(np.longdouble) - ref) / _ulp(ref)).max()) <= 0.51
    pos = X > 0
    ref = 1. / np.sqrt(X[pos])
    assert float((np.abs(s[pos].astype(np.longdouble) - ref) / _ulp(ref)).max()) <= 0.51
    ref = np.log(X[pos])
    assert float((np.abs(l[pos].astype(np.longdouble) - ref) - 0.51 * _ulp(ref)).max()) <= 2. ** -58.9 * math.log(2.)


def test_special_arguments(cuda):
    """Arguments outside the fixed-point ranges give what IEEE arithmetic gives."""
    x = np.array([0., -0., np.inf, -np.inf, np.nan, 709.78, -745.2, -708.5, 1e-310, 1.7e308, -2.])
    e, l, r, s = _values(x)
    with np.errstate(all='ignore'):
        np.testing.assert_allclose(e, np.exp(x), rtol=1e-15)
        np.testing.assert_allclose(l, np.log(x), rtol=1e-15)
        np.testing.assert_allclose(r, 1. / x, rtol=1e-15)
        np.testing.assert_allclose(s, 1. / np.sqrt(x), rtol=1e-15)
