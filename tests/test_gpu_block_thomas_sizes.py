"""Block-Thomas factorization and solves at the block sizes where the elimination's and the sweeps' thread layouts change
(one, two, three and four rows per lane, odd and even leading dimensions, one staged block or two) and the chain lengths
where a half or the middle has no neighbour, against a dense solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('bs', [1, 2, 32, 33, 53, 64, 65, 97, 119])
@pytest.mark.parametrize('nb', [1, 2, 3, 6])
def test_factor_and_solves_match_dense(cuda, bs, nb):
    """Well-conditioned matrices (condition below 1e3): forward error within 1e3 n eps < 2e-10 of a dense solve."""
    from spitfire_gb300 import griffon as G
    rng = np.random.default_rng(100 * nb + bs)
    D = rng.standard_normal((nb, bs, bs)) / np.sqrt(bs)
    for i in range(nb):  # diagonally shifted, rows permuted so that the elimination has to pivot
        D[i] = (D[i] + 3. * np.eye(bs))[rng.permutation(bs)] if nb == 1 else D[i] + 3. * np.eye(bs)
    sub, sup = 0.3 * rng.standard_normal((nb - 1, bs)), 0.3 * rng.standard_normal((nb - 1, bs))
    A = np.zeros((nb * bs, nb * bs))
    s = lambda i: slice(i * bs, (i + 1) * bs)
    low, up = np.zeros_like(A), np.zeros_like(A)
    for i in range(nb):
        A[s(i), s(i)] = low[s(i), s(i)] = up[s(i), s(i)] = D[i]
        if i:
            A[s(i), s(i - 1)] = low[s(i), s(i - 1)] = np.diag(sub[i - 1])
            A[s(i - 1), s(i)] = up[s(i - 1), s(i)] = np.diag(sup[i - 1])
    vals = np.concatenate([np.swapaxes(D, 1, 2).ravel(), sub.ravel(), sup.ravel()])
    b = rng.standard_normal(nb * bs)
    n = nb * bs
    def rel(x, M):
        ref = np.linalg.solve(M, b)
        return np.abs(x - ref).max() / np.abs(ref).max()

    fac, lv, piv, x = vals.copy(), np.zeros(n * bs), np.zeros(n, dtype=np.int32), np.zeros(n)
    G.py_btddod_full_factorize(fac, nb, bs, lv, piv)
    G.py_btddod_full_solve(fac, lv, piv, b, nb, bs, x)
    assert rel(x, A) < 2e-10
    dfac, dpiv = np.zeros(n * bs), np.zeros(n, dtype=np.int32)
    G.py_btddod_blockdiag_factorize(vals, nb, bs, dpiv, dfac)
    G.py_btddod_lowerfulltriangle_solve(dpiv, dfac, vals, b, nb, bs, x)
    assert rel(x, low) < 2e-10
    G.py_btddod_upperfulltriangle_solve(dpiv, dfac, vals, b, nb, bs, x)
    assert rel(x, up) < 2e-10
