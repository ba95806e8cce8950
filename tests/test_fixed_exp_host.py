"""The fixed-point exponential's 2^f (fix_exp2, spitfire_gb300/csrc/fixed_point.cuh), its integer operations restated on the host
with the committed constants, against 300-bit powers of two."""
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'spitfire_gb300', 'csrc')


def _constants():
    text = open(os.path.join(CSRC, 'exp_table.h')).read()
    c = [int(re.search(rf'kFixC{k} = (0x[0-9a-f]+)ull', text).group(1), 16) for k in range(1, 6)]
    body = text[text.index('kFixExpTable[256] = {'):]
    tab = [int(v, 16) for v in re.findall(r'(0x[0-9a-f]+)ull', body)]
    assert len(tab) == 256
    return c, tab


def _mulhi(a, b):
    """fix_mulhi: the high 64 bits of a product without the product of the low words"""
    ah, al, bh, bl = a >> 32, a & 0xffffffff, b >> 32, b & 0xffffffff
    return (ah * bh + (ah * bl >> 32) + (al * bh >> 32)) & (2 ** 64 - 1)


def _exp2(f, c, tab):
    v = (f << 8) & (2 ** 64 - 1)
    vh = v >> 32
    a4 = (c[3] + (vh * c[4] >> 32)) & 0xffffffff
    a3 = (c[2] + ((vh * a4 >> 32) >> 8)) & 0xffffffff
    a2 = c[1] + (vh * a3 >> 20)
    T = tab[f >> 56]
    return T + (_mulhi(T, _mulhi(v, c[0] + _mulhi(v, a2))) >> 8)


@pytest.mark.parametrize('kind', ['uniform', 'end of a table step', 'close to 1', 'close to 0'])
def test_within_20_units(kind):
    """20 units of 2^-63 (0.51 ulp of the rounded result). The two one-sided errors of c3's term, the shift (1 unit of 2^-52) and
    the 24 bits of v that vh drops (0.87), reach 8 to 16 units of the result each way at most once centred; the high
    products lose 3 units each in terms that are shifted by 8."""
    mp = pytest.importorskip('mpmath')
    mp.mp.prec = 300
    c, tab = _constants()
    rng = np.random.default_rng(8)
    f = rng.integers(0, 2 ** 64, 6000, dtype=np.uint64)
    if kind == 'end of a table step':
        f |= np.uint64(0x00fff00000000000)
    elif kind == 'close to 1':
        f = np.concatenate([f | np.uint64(0xfffff00000000000), np.arange(2 ** 64 - 200, 2 ** 64, dtype=np.uint64)])
    elif kind == 'close to 0':
        f = np.concatenate([f >> np.uint64(24), np.arange(0, 200, dtype=np.uint64)])
    worst = 0.
    for x in f.tolist():
        worst = max(worst, abs(float(_exp2(x, c, tab) - mp.power(2, mp.mpf(x) / 2 ** 64 + 63))))
    assert worst <= 20., worst
