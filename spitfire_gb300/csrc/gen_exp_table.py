"""Writes exp_table.h: the constants of the table-driven exponential in chem_device.cuh (Tang's method, ACM TOMS
15(2), 1989), computed at 300 bits with mpmath and rounded to the nearest double.

  python spitfire_gb300/csrc/gen_exp_table.py

* kExpInvL = 64/ln 2;
* kExpL1 + kExpL2 = ln 2/64: kExpL1 is ln 2/64 rounded, kExpL2 the rounded remainder;
* kExpTable[2j], kExpTable[2j+1] = head and tail of 2^(j/64), j = 0..63 (head: 2^(j/64) rounded; tail: the
  rounded remainder), interleaved so that one 16-byte load fetches both.

The fixed-point exponential's constants (fixed_point.cuh: fix_exp2):
* kFixLog2e2, 1, 0: the three 32-bit words of log2(e) 2^95, truncated;
* kFixExpTable[j] = 2^(j/256) 2^63, rounded, j = 0..255;
* kFixC1 .. kFixC5: the polynomial of W(v) = 256 (2^(v/256) - 1) = v (c1 + v (c2 + ...)) on [0, 1], the Chebyshev fit of
  degree 4 of W(v)/v, as integers scaled by 2^64 (c1, c2), 2^52 (c3) and 2^60 (c4, c5). The device's shifts and high
  products truncate; 2700 added to kFixC2 centers the error that leaves (within 16 units of 2^-63 of the result's mantissa,
  0.0079 ulp, before the final rounding).
"""
import os

import mpmath as mp


def header_text():
    """The text of exp_table.h."""
    mp.mp.prec = 300
    ln2 = mp.log(2)
    inv_l = float(64 / ln2)
    l1 = float(ln2 / 64)
    l2 = float(ln2 / 64 - mp.mpf(l1))
    tab = []
    for j in range(64):
        s = mp.power(2, mp.mpf(j) / 64)
        hi = float(s)
        tab += [hi, float(s - mp.mpf(hi))]
    lines = ['// Generated by gen_exp_table.py: constants of the table-driven exponential (Tang, ACM TOMS 15(2), 1989),',
             '// computed at 300 bits and rounded to the nearest double.',
             '#pragma once', '',
             'namespace sfgb {', '',
             f'constexpr double kExpInvL = {inv_l.hex()};  // 64 / ln 2',
             f'constexpr double kExpL1 = {l1.hex()};    // ln 2 / 64, rounded',
             f'constexpr double kExpL2 = {l2.hex()};    // ln 2 / 64 - kExpL1, rounded', '',
             '// 2^(j/64) = kExpTable[2j] + kExpTable[2j + 1], j = 0..63',
             'constexpr double kExpTable[128] = {']
    for j in range(64):
        lines.append(f'    {tab[2 * j].hex()}, {tab[2 * j + 1].hex()},')
    lines += ['};', '']
    l96 = int(mp.floor(mp.mpf(2) ** 95 / ln2))
    lines += ['// The fixed-point exponential: words of log2(e) 2^95, polynomial coefficients, 2^(j/256) 2^63.']
    lines += [f'constexpr unsigned kFixLog2e{k} = {hex((l96 >> (32 * k)) & 0xffffffff)}u;' for k in (2, 1, 0)]
    w = lambda v: ln2 if v == 0 else 256 * (mp.power(2, v / 256) - 1) / v
    c = mp.chebyfit(w, [mp.mpf(10) ** -30, 1], 5)[::-1]
    fix = [int(mp.nint(c[k] * mp.mpf(2) ** (64, 64, 52, 60, 60)[k])) + (0, 2700, 0, 0, 0)[k] for k in range(5)]
    lines += [f'constexpr unsigned long long kFixC{k + 1} = {hex(fix[k])}ull;' for k in range(5)]
    lines += ['constexpr unsigned long long kFixExpTable[256] = {']
    for j in range(0, 256, 4):
        t = [int(mp.nint(mp.power(2, mp.mpf(i) / 256) * mp.mpf(2) ** 63)) for i in range(j, j + 4)]
        lines.append('    ' + ' '.join(f'{hex(v)}ull,' for v in t))
    lines += ['};', '', '}  // namespace sfgb', '']
    return '\n'.join(lines)


def main():
    out = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'exp_table.h')
    with open(out, 'w') as f:
        f.write(header_text())
    print(out)


if __name__ == '__main__':
    main()
