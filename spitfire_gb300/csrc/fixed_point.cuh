// Fixed-point arithmetic on the integer pipes: exponential, logarithm, reciprocal and reciprocal square root of doubles.
//
// A warp FP64 instruction takes its scheduler's FP64 unit 64 to 76 cycles on GB300, an integer multiply-add 2 to 5, and
// the two pipes run side by side, so that the functions below cost no time in a kernel that the FP64 unit bounds.
#pragma once
#include <cuda_runtime.h>

#include "exp_table.h"

namespace sfgb {

// x 2^K, exact unless the result leaves the normal range; |K| beyond 2044 already takes any factor of a rate
// expression to 0 or infinity. A normal x whose result is normal has K added to its exponent field.
__device__ __forceinline__ double scale_pow2(double x, long long K)
{
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  const int k = (int)(K < -4096 ? -4096 : (K > 4096 ? 4096 : K));
  if ((unsigned)(e - 1) < 2046u && (unsigned)(e + k - 1) < 2046u)
    return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
  const int kc = k < -2044 ? -2044 : (k > 2046 ? 2046 : k);
  const int k1 = kc / 2, k2 = kc - k1;  // both within [-1022, 1023]
  const double f1 = __longlong_as_double((long long)(k1 + 1023) << 52);
  const double f2 = __longlong_as_double((long long)(k2 + 1023) << 52);
  return x * f1 * f2;
}

// ----------------------------------------------------------------------------------------- exponential
// e^x by Tang's table method (ACM TOMS 15(2), 1989) in fixed point, about 200 issue slots where the FP64 form (tab_exp,
// 11.7 FP64 instructions) takes 890 cycles of the FP64 unit:
//   y = x log2(e) = N + f with f in [0, 1) as a 64-bit fraction, from the 53-bit mantissa of x times log2(e) to 96 bits;
//   2^f = T_j (1 + p): T_j = 2^(j/256) to 64 bits, j the leading 8 bits of f, and 256 p = W(v) = v (c1 + v (c2 + ...)),
//   v the other 56 bits as a fraction. The terms shrink by 2^-8 each, so c3 .. c5 need only 32-bit products.
// The 64-bit result is within 16 units of 2^-63 before it is rounded (c4 and c5 eight bits finer than c3: with all three in
// units of 2^-52 it was 23.6, 0.5115 ulp, for fractions close to 1): at most 0.51 ulp like tab_exp, NaN and |x| >= 708 go
// to tab_exp. tab: the 128 doubles of tab_exp's table, then the 256 words of 2^(j/256).

// High 64 bits of a b without the product of the low words (within 3 units).
__device__ __forceinline__ unsigned long long fix_mulhi(unsigned long long a, unsigned long long b)
{
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
  return (unsigned long long)ah * bh + ((unsigned long long)__umulhi(ah, bl) + __umulhi(al, bh));
}

// x log2(e) = N + f 2^-64 for |x| < 2^20
__device__ __forceinline__ void fix_reduce(double x, int &N, unsigned long long &f)
{
  typedef unsigned long long u64;
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const unsigned m1 = ((((unsigned)hi & 0xfffffu) | 0x100000u) << 11) | (lo >> 21), m0 = lo << 11;
  // the leading 96 bits of the 64 x 96 bit product
  const u64 t1 = (u64)m0 * kFixLog2e1;
  const u64 t2 = (u64)m1 * kFixLog2e0 + (unsigned)t1;
  const u64 t3 = (u64)m1 * kFixLog2e1 + (unsigned)(t1 >> 32);
  const u64 t4 = (u64)m0 * kFixLog2e2 + (unsigned)t3;
  const u64 s2 = (u64)(unsigned)t4 + (unsigned)(t2 >> 32);
  const u64 t5 = (u64)m1 * kFixLog2e2 + ((u64)(unsigned)(t3 >> 32) + (unsigned)(t4 >> 32) + (unsigned)(s2 >> 32));
  const unsigned p2 = (unsigned)(t5 >> 32), p1 = (unsigned)t5, p0 = (unsigned)s2;
  // shifted right by 30 - exponent (at most 95) bits: 32 integer bits above 64 fraction bits
  int sh = 30 + 1023 - ((hi >> 20) & 0x7ff);
  sh = sh > 95 ? 95 : sh;
  const bool q1 = sh >= 32, q2 = sh >= 64;
  const unsigned w2 = q1 ? 0u : p2, w1 = q2 ? 0u : (q1 ? p2 : p1), w0 = q2 ? p2 : (q1 ? p1 : p0);
  const unsigned f0 = __funnelshift_r(w0, w1, sh), f1 = __funnelshift_r(w1, w2, sh), n = w2 >> (sh & 31);
  f = ((u64)f1 << 32) | f0;
  N = (int)n;
  if (hi < 0) {  // -(N + f) = (-N - 1) + (1 - f), or -N when f = 0
    N = f ? ~N : -N;
    f = 0ull - f;
  }
}

// 2^(f 2^-64) 2^63
__device__ __forceinline__ unsigned long long fix_exp2(unsigned long long f, const unsigned long long *tab)
{
  typedef unsigned long long u64;
  const u64 T = tab[(unsigned)(f >> 56)];
  const u64 v = f << 8;
  const unsigned vh = (unsigned)(v >> 32);
  const unsigned a4 = (unsigned)kFixC4 + __umulhi(vh, (unsigned)kFixC5);     // units of 2^-60
  const unsigned a3 = (unsigned)kFixC3 + (__umulhi(vh, a4) >> 8);            // units of 2^-52
  const u64 a2 = kFixC2 + (((u64)vh * a3) >> 20);
  const u64 W = fix_mulhi(v, kFixC1 + fix_mulhi(v, a2));
  return T + (fix_mulhi(T, W) >> 8);
}

// R 2^-63 2^N, R in [2^63, 2^64), rounded to nearest, as a normal double
__device__ __forceinline__ double fix_to_double(unsigned long long R, int N)
{
  const unsigned long long m = (R >> 11) + ((unsigned)(R >> 10) & 1u);  // 53 bits; the leading one adds to the exponent
  return __longlong_as_double((long long)(m + ((unsigned long long)(unsigned)(N + 1022) << 52)));
}

// Logarithms to base 2 in fixed point: 32 integer bits (signed) over 64 fraction bits. A rate constant is kept as its
// logarithm until the one fix_exp2 that forms it: log2 k = log2 A + b log2 T - (E/R) log2(e) / T, and the reverse
// constant's logarithm adds the species' -g/RT log2(e), so that the two constants of a reaction take no FP64 instruction
// (8 before, with the exponential already in fixed point). Sums wrap only beyond 2^31, far outside the range of doubles.
struct Fix96 {
  unsigned f0, f1;
  int n;
};
__device__ __forceinline__ Fix96 fix96(int n, unsigned long long f) { return Fix96{(unsigned)f, (unsigned)(f >> 32), n}; }
// The carry chains keep their partial words in registers of their own until every input is read: the compiler may hold
// equal input words in one register, also with an output.
__device__ __forceinline__ Fix96 operator+(Fix96 a, Fix96 b)
{
  Fix96 r;
  asm("{\n\t.reg .u32 t0, t1, t2;\n\tadd.cc.u32 t0, %3, %6;\n\taddc.cc.u32 t1, %4, %7;\n\taddc.u32 t2, %5, %8;\n\t"
      "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\tmov.u32 %2, t2;\n\t}"
      : "=r"(r.f0), "=r"(r.f1), "=r"(r.n)
      : "r"(a.f0), "r"(a.f1), "r"(a.n), "r"(b.f0), "r"(b.f1), "r"(b.n));
  return r;
}
__device__ __forceinline__ Fix96 operator-(Fix96 a, Fix96 b)
{
  Fix96 r;
  asm("{\n\t.reg .u32 t0, t1, t2;\n\tsub.cc.u32 t0, %3, %6;\n\tsubc.cc.u32 t1, %4, %7;\n\tsubc.u32 t2, %5, %8;\n\t"
      "mov.u32 %0, t0;\n\tmov.u32 %1, t1;\n\tmov.u32 %2, t2;\n\t}"
      : "=r"(r.f0), "=r"(r.f1), "=r"(r.n)
      : "r"(a.f0), "r"(a.f1), "r"(a.n), "r"(b.f0), "r"(b.f1), "r"(b.n));
  return r;
}

// a b 2^-32 2^-SHIFT as a Fix96 (SHIFT 1 to 31) for 64-bit a, b; the dropped bits are below the result's last one.
template <int SHIFT>
__device__ __forceinline__ Fix96 fix_product(unsigned long long a, unsigned long long b)
{
  typedef unsigned long long u64;
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
  const u64 t2 = (u64)ah * bl + __umulhi(al, bl);
  const u64 t3 = (u64)al * bh + (unsigned)t2;
  const u64 t4 = (u64)ah * bh + ((u64)(unsigned)(t2 >> 32) + (unsigned)(t3 >> 32));
  const unsigned p1 = (unsigned)t3, p2 = (unsigned)t4, p3 = (unsigned)(t4 >> 32);
  return Fix96{__funnelshift_r(p1, p2, SHIFT), __funnelshift_r(p2, p3, SHIFT), (int)(p3 >> SHIFT)};
}

// 2^y as a double, 0 or infinity beyond its range
__device__ __forceinline__ double fix96_exp2(Fix96 y, const unsigned long long *tab)
{
  const unsigned long long R = fix_exp2(((unsigned long long)y.f1 << 32) | y.f0, tab);
  if ((unsigned)(y.n + 1022) < 2045u) return fix_to_double(R, y.n);
  return scale_pow2(fix_to_double(R, 0), y.n);
}


// 1 / m for m = M 2^-63 in [1, 2), as a 64-bit fraction of (1/2, 1], within 6 units: the FP32 reciprocal of the leading
// bits and two Newton steps y + y (1 - m y), the first with 32-bit products.
__device__ __forceinline__ unsigned long long fix_rcp(unsigned long long M)
{
  typedef unsigned long long u64;
  const unsigned mh = (unsigned)(M >> 32), ml = (unsigned)M;
  const float f = __frcp_rn(__int_as_float(0x3f800000 | (int)((mh >> 8) & 0x7fffffu)));
  const unsigned y0 = __float2uint_rz(f * 4294967296.f);  // saturates at 2^32 - 1
  const long long e0 = (long long)(0x8000000000000000ull - ((u64)mh * y0 + __umulhi(ml, y0)));
  const long long c0 = (long long)(int)(e0 >> 10) * (int)(y0 >> 1);
  const u64 s1 = ((u64)y0 << 32) + (u64)(c0 >> 20);
  const u64 y1 = y0 > 0xff000000u && (s1 >> 63) == 0 ? ~0ull : s1;  // past 1
  const long long e1 = (long long)(0x8000000000000000ull - fix_mulhi(M, y1));
  const long long c1 = (long long)(int)e1 * (int)(unsigned)(y1 >> 33);
  const u64 s2 = y1 + (u64)(c1 >> 30);
  return y1 > 0xff00000000000000ull && (s2 >> 63) == 0 ? ~0ull : s2;
}

// 1 / x to within 0.51 ulp; zeros, subnormals, values that are not finite and results that are not normal divide.
__device__ __forceinline__ double fix_reciprocal(double x)
{
  const int hi = __double2hiint(x);
  const int e = (hi >> 20) & 0x7ff;
  if ((unsigned)(e - 1) >= 2044u) return 1. / x;
  const unsigned long long M = ((unsigned long long)__double_as_longlong(x) << 11) | 0x8000000000000000ull;
  const double y = fix_to_double(fix_rcp(M), 1022 - e);
  return __hiloint2double(__double2hiint(y) | (hi & 0x80000000), __double2loint(y));
}

// 1 / sqrt(x) to within 0.51 ulp, the same way: a 2^(2q) = x with a in [1/4, 1), the FP32 reciprocal square root and two
// Newton steps y + y (1 - a y^2) / 2. Arguments that are not normal and positive go to rsqrt.
__device__ __forceinline__ double fix_rsqrt(double x)
{
  typedef unsigned long long u64;
  const int hi = __double2hiint(x);
  if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u) return rsqrt(x);
  const u64 M = ((u64)__double_as_longlong(x) << 11) | 0x8000000000000000ull;
  const int e1 = (hi >> 20) - 1022;  // x = M 2^-64 2^e1
  const int odd = e1 & 1, q = (e1 + odd) >> 1;
  const u64 a = M >> odd;
  const float f = rsqrtf(__int_as_float(((126 - odd) << 23) | (int)((unsigned)(M >> 40) & 0x7fffffu)));
  const unsigned y0 = __float2uint_rz(f * 2147483648.f);  // saturates at 2^32 - 1
  const long long d0 = (long long)(0x4000000000000000ull - fix_mulhi(a, (u64)y0 * y0));
  const long long c0 = (long long)(int)(d0 >> 11) * (int)(y0 >> 1);
  const u64 s1 = ((u64)y0 << 32) + (u64)(c0 >> 19);
  const u64 y1 = y0 > 0xff000000u && (s1 >> 63) == 0 ? ~0ull : s1;  // past 2
  const long long d1 = (long long)(0x4000000000000000ull - fix_mulhi(a, fix_mulhi(y1, y1)));
  const long long c1 = (long long)(int)d1 * (int)(unsigned)(y1 >> 33);
  const u64 s2 = y1 + (u64)(c1 >> 30);
  return fix_to_double(y1 > 0xff00000000000000ull && (s2 >> 63) == 0 ? ~0ull : s2, -q);
}

// log2 of a normal positive x as a Fix96, within 2^-58.9: from the FP32 logarithm k 2^-24 of the mantissa m by one Newton
// step on the exponential, log2 m = k 2^-24 + log2(m 2^(-k 2^-24)), the last argument 1 + d with |d| < 2^-21.
__device__ __forceinline__ Fix96 fix_log2(double x, const unsigned long long *tab)
{
  typedef unsigned long long u64;
  const u64 bits = (u64)__double_as_longlong(x);
  const u64 M = (bits << 11) | 0x8000000000000000ull;
  const float mf = __int_as_float(0x3f800000 | (int)((bits >> 29) & 0x7fffffu));
  int k = __float2int_rn(__log2f(mf) * 16777216.f);
  k = max(0, min(k, 0xffffff));
  const u64 P = fix_mulhi(M, fix_exp2(0ull - ((u64)k << 40), tab));  // 2^62 (1 + d), or 2^63 (1 + d) when k > 0
  const long long d = k ? (long long)(P - 0x8000000000000000ull) : (long long)(P - 0x4000000000000000ull) << 1;
  const int dh = (int)(d >> 11);
  const long long t = d - (((long long)dh * dh) >> 42);  // d - d^2 / 2, units of 2^-63
  const u64 at = (u64)(t < 0 ? -t : t) << 20;
  const u64 l = fix_mulhi(at, ((u64)kFixLog2e2 << 32) | kFixLog2e1) >> 18;  // times log2(e), units of 2^-64
  const Fix96 y = fix96((int)(bits >> 52) - 1023, (u64)k << 40);
  return t < 0 ? y - fix96(0, l) : y + fix96(0, l);
}

// y ln 2 as a double
__device__ __forceinline__ double fix96_ln(Fix96 y)
{
  typedef unsigned long long u64;
  const bool neg = y.n < 0;
  if (neg) y = Fix96{0u, 0u, 0} - y;
  // the leading 64 bits of |y|, past up to two zero words (selects, so that two logarithms can run interleaved)
  unsigned w2 = (unsigned)y.n, w1 = y.f1, w0 = y.f0;
  int e = 31;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const bool z = w2 == 0;
    w2 = z ? w1 : w2;
    w1 = z ? w0 : w1;
    w0 = z ? 0u : w0;
    e = z ? e - 32 : e;
  }
  const int c = __clz((int)w2);
  const u64 top = ((u64)__funnelshift_l(w1, w2, c) << 32) | __funnelshift_l(w0, w1, c);
  e -= c;
  u64 R = fix_mulhi(top, 0xb17217f7d1cf79acull);  // ln 2 2^64
  if (!(R >> 63)) {
    R <<= 1;
    --e;
  }
  const double v = w2 ? fix_to_double(R, e) : 0.;
  return neg ? -v : v;
}
__device__ __forceinline__ bool fix_normal(double x) { return (unsigned)(__double2hiint(x) - 0x00100000) < 0x7fe00000u; }

// ln x, absolute error below 2^-58 (and half an ulp); arguments that are not normal and positive go to log.
__device__ __forceinline__ double fix_log(double x, const unsigned long long *tab)
{
  if (!fix_normal(x)) return log(x);
  return fix96_ln(fix_log2(x, tab));
}

}  // namespace sfgb
