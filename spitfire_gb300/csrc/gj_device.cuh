// Inverse of a dense block by Gauss-Jordan elimination over several warps of a block, shared by the block-Thomas
// factorization (flamelet_kernels.cu) and the integrator's wide groups (integrate_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "fixed_point.cuh"

namespace sfgb {

// Inverse of the n x n row-major matrix in S (leading dimension ld, odd: rows then start in different banks) by
// Gauss-Jordan elimination with partial pivoting (G. H. Golub and C. F. Van Loan, "Matrix Computations", section 3.2;
// rows are not moved, the pivot order is recorded). Phase k maps the source buffer to the destination (S and D
// alternate): with pivot row p, ip = 1/S[p][k], m_p = ip and m_i = -S[i][k] ip otherwise,
//   D[i][j] = m_i S[p][j] + (i == p ? 0 : S[i][j])   (j != k),   D[i][k] = m_i.
// The other warps update the block while warp 0 forms column k+1 of D and, before the phase's barrier, chooses the
// next pivot among the unused rows (largest magnitude, lowest row on ties, as idamax) and its multipliers: one
// barrier per column. Returns the buffer Z holding the inverse permuted: inverse(r, c) = Z[piv[r]][pinv[c]], where
// pinv[piv[k]] = k. ws: 2n doubles. n <= 128. threads: a multiple of 32, at least 64; t: this thread; sync: their
// barrier. A pivot column of zeros gives 1/0 or, with ZERO_PIVOT, 0 in place of its reciprocal.
//
// Bound: n^2 FMAs per column at 76 cycles per warp FMA and scheduler, 46 us for n = 53 on one SM, against about 0.6 us
// of look-ahead per column. Every element takes one FP64 instruction: the pivot row and column k are cases of the
// same FMA by integer selects (as a select of two results the pivot row's product was formed for every element, which
// doubled the FP64 work: 108 us). 58 us with 384 threads, 64 with 256, 67 with 512 (n = 53, one block per SM).
template <bool ZERO_PIVOT, class Sync>
__device__ __forceinline__ double *gj_inverse(double *S, double *D, int n, int ld, int *piv, int *pinv, double *ws,
                                              int t, int threads, Sync sync)
{
  const int warp = t >> 5, lane = t & 31;
  const int stride = threads - 32;
  const int ut = t - 32;
  const int i0 = ut / n, j0 = ut - i0 * n, di = stride / n, dj = stride - di * n;
  unsigned used = 0;  // warp 0: bit s set when row lane + 32 s has been a pivot
  // warp 0: choose the pivot of column j from the lane-held column values v (row lane + 32 s) and publish it with its
  // multipliers for phase j. Magnitudes are compared as the integer bit patterns of |x|, high words first.
  auto choose = [&](int j, const double (&v)[4]) {
    unsigned h[4], bh = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const bool c = lane + 32 * s < n && !((used >> s) & 1u);
      h[s] = c ? ((unsigned)__double2hiint(v[s]) & 0x7fffffffu) + 1u : 0u;
      bh = max(bh, h[s]);
    }
    const unsigned mh = __reduce_max_sync(0xffffffffu, bh);
    unsigned bl = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (h[s] == mh) bl = max(bl, (unsigned)__double2loint(v[s]));
    const unsigned ml = __reduce_max_sync(0xffffffffu, bl);
    unsigned bi = n;
#pragma unroll
    for (int s = 3; s >= 0; --s)
      if (h[s] == mh && (unsigned)__double2loint(v[s]) == ml) bi = lane + 32 * s;
    const int bp = (int)__reduce_min_sync(0xffffffffu, bi);
    double pv = 0.;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (32 * s < n) {
        const double x = __shfl_sync(0xffffffffu, v[s], bp & 31);
        if ((bp >> 5) == s) pv = x;
      }
    }
    const bool zero = ZERO_PIVOT && (__double_as_longlong(pv) << 1) == 0;
    const double ip = zero ? 0. : fix_reciprocal(pv);
    double *f = ws + (j & 1) * n;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int i = lane + 32 * s;
      if (i < n) f[i] = i == bp ? ip : -(v[s] * ip);
    }
    if (lane == (bp & 31)) used |= 1u << (bp >> 5);
    if (lane == 0) {
      piv[j] = bp;
      pinv[bp] = j;
    }
  };
  if (warp == 0) {
    double v[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int i = lane + 32 * s;
      v[s] = i < n ? S[i * ld] : 0.;
    }
    choose(0, v);
  }
  sync();
  for (int k = 0; k < n; ++k) {
    const int p = piv[k], kn = k + 1;
    const double *mult = ws + (k & 1) * n;
    const double *Sp = S + (size_t)p * ld;
    if (warp == 0) {
      if (kn < n) {
        const double spj = Sp[kn];
        double v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int i = lane + 32 * s;
          v[s] = 0.;
          if (i < n) {
            const double a = S[i * ld + kn];
            v[s] = fma(mult[i], spj, i == p ? 0. : a);
            D[i * ld + kn] = v[s];
          }
        }
        choose(kn, v);
      }
    } else {
      int i = i0, j = j0;
      while (i < n) {
        const double m = mult[i];
        double a = S[i * ld + j], c = Sp[j];
        if (i == p) a = 0.;
        if (j == k) {
          a = m;
          c = 0.;
        }
        const double val = fma(m, c, a);
        if (j != kn) D[i * ld + j] = val;  // column k+1 is warp 0's
        i += di;
        j += dj;
        if (j >= n) {
          j -= n;
          ++i;
        }
      }
    }
    sync();
    double *x = S;
    S = D;
    D = x;
  }
  return S;
}

}  // namespace sfgb
