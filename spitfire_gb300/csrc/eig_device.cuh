// Largest real part of the eigenvalues of a small real nonsymmetric matrix, by one state group (a warp where there
// are many matrices, two or eight where there are about as many as SMs), in shared memory:
// Parlett-Reinsch balancing (diagonal similarity by powers of two, exact in floating point), Householder reduction
// to upper Hessenberg form, then the implicit double-shift (Francis) QR iteration with deflation on the active
// window only (eigenvalues, no Schur vectors). Published algorithms: B. N. Parlett and C. Reinsch, "Balancing a
// matrix for calculation of eigenvalues and eigenvectors", Numer. Math. 13 (1969); G. H. Golub and C. F. Van Loan,
// "Matrix Computations", sections 7.4-7.5 (Hessenberg reduction, Francis step, deflation, exceptional shifts).
//
// GB300 issues FP64 at a fixed cost per warp instruction whatever the number of active lanes, so the warp
// layout keeps lanes busy: column-parallel Hessenberg updates (no per-column reductions), reflectors in the
// tau form (one reciprocal) in the Hessenberg reduction, unit-scaled reflectors (one reciprocal square root) in
// the QR sweeps, and a lane-parallel deflation scan.
//
// Replaces the LAPACK dgeev call Griffon makes per flamelet Jacobian block for the pseudo-transient
// continuation time step (flamelet_kernels.cpp:1329-1341).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "chem_device.cuh"

namespace sfgb {

// x * 2^k for fac = 2^k, on the integer pipe where that is exact: a normal x whose product stays normal gets k added to
// its exponent field, a zero is unchanged; anything else (subnormal, infinite, NaN, leaving the normal range) is
// multiplied as before.
__device__ __forceinline__ double scale_pow2(double x, int k, double fac)
{
  const long long b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  if (e == 0 && (b & 0x7fffffffffffffffLL) == 0) return x;
  if (e == 0 || e == 0x7ff || e + k <= 0 || e + k >= 0x7ff) return x * fac;
  return __longlong_as_double(b + ((long long)k << 52));
}

// Sums of the magnitudes of column i and row i of A without the diagonal, n <= 64, one warp: the terms as integers on the
// scale of the largest (53 bits, the rest cut off), added by integer warp reductions in two halves. False where an exponent
// is near the ends of the range (or a sum is zero); c and r are then untouched.
__device__ __forceinline__ bool abs_sums(const double *A, int n, int i, int lane, double &c, double &r)
{
  unsigned long long b[2][2];
  unsigned hi[2] = {0u, 0u};
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int j = lane + 32 * s;
    const bool in = j < n && j != i;
    b[0][s] = in ? (unsigned long long)__double_as_longlong(A[j + i * n]) & 0x7fffffffffffffffull : 0ull;
    b[1][s] = in ? (unsigned long long)__double_as_longlong(A[i + j * n]) & 0x7fffffffffffffffull : 0ull;
#pragma unroll
    for (int q = 0; q < 2; ++q) hi[q] = max(hi[q], (unsigned)(b[q][s] >> 32));
  }
  int e[2];
  unsigned long long x[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) e[q] = (int)(__reduce_max_sync(0xffffffffu, hi[q]) >> 20);
  if (e[0] < 64 || e[1] < 64 || e[0] > 0x7b0 || e[1] > 0x7b0) return false;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    x[q] = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int ex = (int)(b[q][s] >> 52), sh = e[q] - ex;
      const unsigned long long m = (b[q][s] & 0xfffffffffffffull) | 0x10000000000000ull;
      x[q] += ex && sh < 64 ? m >> sh : 0ull;  // subnormals are below the last bit
    }
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)x[q] & 0x7ffffffu);
    const unsigned up = __reduce_add_sync(0xffffffffu, (unsigned)(x[q] >> 27));
    x[q] = lo + ((unsigned long long)up << 27);
    const int z = __clzll((long long)x[q]);
    (q ? r : c) = fix_to_double(x[q] << z, 63 - z + e[q] - 1075);
  }
  return true;
}

// Parlett-Reinsch balancing with radix 2 (scaling only): repeat until no row/column pair changes by more than
// 5%, at most `max_sweeps` sweeps. Column-major A, leading dimension n.
// GB300 issues FP64 at one warp instruction per 76 cycles per scheduler, so the scalings by powers of two (exact)
// run on the integer pipe: non-negative finite doubles order like their bit patterns, and a factor 4 or 1/4 on a
// normal value is a change of 2 in its exponent field; values near the ends of the exponent range take the FP64 form. The
// scalings themselves are exact. The sums of up to 64 rows are cut to 53 bits of their largest term (abs_sums), so that a
// choice of scaling can differ from the FP64 form's where a comparison ties within that cut.
// One warp, also where the matrix has several: a row/column pair is a serial step, and the exchange between warps cost more
// than it gained. The sums are integer sums (abs_sums) and a pair that needs no scaling (m = 0) is left at once: a 53 x 53
// block takes nine sweeps of 53 pairs, about 1700 cycles a pair in FP64 with two warps.
__device__ void warp_balance(double *A, int n, int max_sweeps = 32)
{
  const Group<32> g;
  const int lane = g.lane;
  constexpr long long kExp1 = 1LL << 52;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    bool changed = false;
    for (int i = 0; i < n; ++i) {
      double c = 0., r = 0.;
      if (n > 64 || !abs_sums(A, n, i, lane, c, r)) {
        for (int j = lane; j < n; j += 32)
          if (j != i) {
            c += fabs(A[j + i * n]);
            r += fabs(A[i + j * n]);
          }
        g.sum2(c, r, n);
      }
      // c, r >= 0: zero when the bit pattern is zero, not finite when the exponent field is all ones
      const long long cb = __double_as_longlong(c), rb = __double_as_longlong(r);
      const int ce = (int)(cb >> 52), re = (int)(rb >> 52);
      if (cb == 0 || rb == 0 || ce == 0x7ff || re == 0x7ff) continue;
      // the scaling f = 2^m: the smallest m >= 0 with c 4^m >= r / 2, else the m < 0 that brings c below 2 r
      int m = 0;
      const double c0 = c;
      if (ce > 4 && ce < 0x7f0 && re > 4 && re < 0x7f0) {
        long long cc = cb;
        const long long g1 = rb - kExp1, g2 = rb + kExp1;  // r / 2, 2 r
        for (int t = 0; t < 1100 && cc < g1; ++t) {
          cc += 2 * kExp1;
          ++m;
        }
        for (int t = 0; t < 1100 && cc >= g2; ++t) {
          cc -= 2 * kExp1;
          --m;
        }
        c = __longlong_as_double(cc);
      } else {
        double g = r * 0.5;
        for (int t = 0; t < 1100 && c < g; ++t) {
          c *= 4.;
          ++m;
        }
        g = r * 2.;
        for (int t = 0; t < 1100 && c >= g; ++t) {
          c *= 0.25;
          --m;
        }
      }
      if (m == 0) continue;  // nothing to scale
      const double s = c0 + r;
      const bool normal = m >= -1000 && m <= 1000;
      const double f = normal ? __longlong_as_double((long long)(1023 + m) << 52) : ldexp(1., m);
      const double fi = normal ? __longlong_as_double((long long)(1023 - m) << 52) : 1. / f;
      // (c + r) / f < 0.95 s, with (c + r) / f formed exactly on the exponent field where it stays normal
      const double t = c + r, lim = 0.95 * s;
      const int te = (int)(__double_as_longlong(t) >> 52);
      const bool fits = normal && te > 0 && te < 0x7ff && te - m > 0 && te - m < 0x7ff;
      const bool shrink = fits ? (__double_as_longlong(t) - (long long)m * kExp1) < __double_as_longlong(lim)
                               : (normal ? t * fi : t / f) < lim;
      if (shrink) {
        changed = true;
        for (int j = lane; j < n; j += 32) {
          if (normal) {
            A[i + j * n] = scale_pow2(A[i + j * n], -m, fi);
            A[j + i * n] = scale_pow2(A[j + i * n], m, f);
          } else {
            A[i + j * n] *= fi;
            A[j + i * n] *= f;
          }
        }
        g.sync();
      }
    }
    if (!changed) break;
  }
}

// Sufficient test that every eigenvalue of the n x n column-major A has real part below `cutoff`, by Gershgorin's
// theorem under the best diagonal scaling: if the comparison matrix M = diag(cutoff - a_ii) - |offdiag(A)| is a
// nonsingular M-matrix, some x > 0 has M x > 0, and then every Gershgorin disc of X^-1 A X (X = diag(x)) lies left
// of the cutoff. A Z-matrix is a nonsingular M-matrix iff its LU factorization without pivoting has positive
// pivots (all leading principal minors positive; A. Berman and R. J. Plemmons, "Nonnegative Matrices in the
// Mathematical Sciences", ch. 6). Each pivot must stay above 1e-10 of the diagonal entry it starts from, far above
// the rounding of the elimination, so a pass holds for the exact matrix. A is overwritten with M's partial
// factors; dg: n doubles of shared work. Lanes over rows (contiguous in column-major storage); a zero entry of
// the pivot row is skipped by the whole warp, which exploits the sparsity of chemistry Jacobians.
template <int G>
__device__ bool group_hmatrix_below(const Group<G> &g, double *A, int n, double cutoff, double *dg)
{
  const int lane = g.lane;
  constexpr int W = G > 64 ? 64 : G;  // lanes over rows; the columns are dealt to the parts of a larger group
  const int slot = lane % W, part = lane / W;
  bool ok = true;
  for (int e = lane; e < n * n; e += G) {
    const int c = e / n, r = e - c * n;
    const double a = A[e];
    if (r == c) {
      const double m = cutoff - a;
      A[e] = m;
      dg[r] = m;
      ok = ok && m > 0.;  // false for NaN too
    } else {
      A[e] = -fabs(a);
    }
  }
  if (g.max(ok ? 0. : 1.) != 0.) return false;
  g.sync();
  for (int k = 0; k < n; ++k) {
    const double p = A[k + k * n];
    if (!(p > 1e-10 * dg[k])) return false;  // the same value in every lane: a warp-uniform exit
    const double ip = fix_reciprocal(p);
    for (int i = k + 1 + slot; i < n; i += W) {
      const double l = A[i + k * n] * ip;
      for (int j = k + 1 + part; j < n; j += G / W) {
        const double mkj = A[k + j * n];
        if ((__double_as_longlong(mkj) << 1) != 0) A[i + j * n] -= l * mkj;
      }
    }
    g.sync();
  }
  return true;
}

// The same test for the unreduced upper Hessenberg block H[lo..hi, lo..hi] of a QR iterate: every eigenvalue of
// the block has real part below `cutoff` if its comparison matrix (diag(cutoff - h_ii), -|h_ij| elsewhere, zero
// below the subdiagonal) is a nonsingular M-matrix. A Hessenberg LU without pivoting eliminates one row per
// column, so the test keeps one row vector (r: hi + 1 doubles of shared work, lanes over columns) and costs
// O(m^2) for a block of m rows, against O(m^2) per double-shift QR sweep over the block.
template <int G>
__device__ bool group_hess_hmatrix_below(const Group<G> &g, const double *H, int n, int lo, int hi, double cutoff, double *r)
{
  const int lane = g.lane;
  for (int j = lo + lane; j <= hi; j += G) r[j] = j == lo ? cutoff - H[lo + lo * n] : -fabs(H[lo + j * n]);
  g.sync();
  for (int k = lo; k <= hi; ++k) {
    const double dgk = cutoff - H[k + k * n];
    const double p = r[k];
    if (!(dgk > 0.) || !(p > 1e-10 * dgk)) return false;  // the same values in every lane: a warp-uniform exit
    if (k == hi) break;
    const double l = -fabs(H[(k + 1) + k * n]) * fix_reciprocal(p);  // multiplier of row k + 1 (its only entry below the pivot)
    g.sync();
    for (int j = k + 1 + lane; j <= hi; j += G) {
      const double m = j == k + 1 ? cutoff - H[(k + 1) + (k + 1) * n] : -fabs(H[(k + 1) + j * n]);
      r[j] = m - l * r[j];
    }
    g.sync();
  }
  return true;
}

// Upper bound of the real parts of the eigenvalues by Gershgorin's theorem applied to rows and to columns.
template <int G>
__device__ double group_gershgorin_bound(const Group<G> &g, const double *A, int n)
{
  const int lane = g.lane;
  double br = -INFINITY, bc = -INFINITY;
  for (int i = lane; i < n; i += G) {
    double rs = 0., cs = 0.;
    for (int j = 0; j < n; ++j)
      if (j != i) {
        rs += fabs(A[i + j * n]);
        cs += fabs(A[j + i * n]);
      }
    br = fmax(br, A[i + i * n] + rs);
    bc = fmax(bc, A[i + i * n] + cs);
  }
  const double r = g.max(br, n), c = g.max(bc, n);
  return fmin(r, c);
}

// Reduce the n x n column-major A to upper Hessenberg form in place. v: n doubles; s: G doubles, sc: 8 doubles of shared
// work for a group of more than 64 threads. Such a group has 64 lanes over columns (rows), and the inner products and
// updates of a column are cut into G / 64 parts: FP64 instructions cost the same on each of an SM's four schedulers, and
// two warps use two of them. 144 points of
// 53 x 53, hardest point: 1.77 ms with two warps per point, 1.32 ms with eight and the balancing above.
template <int G>
__device__ void group_hessenberg(const Group<G> &g, double *A, int n, double *v, double *s, double *sc)
{
  constexpr int W = G > 64 ? 64 : G, P = G / W;
  const int lane = g.lane, slot = lane % W, part = lane / W;
  // x[base + i stride] -= tau (x . v) v over i = k+1 .. n-1 for the lines base = 0 .. lines-1 of this group
  auto reflect = [&](int k, int first, int base, int stride, double tau) {
    const int m = n - k - 1, a = k + 1 + m * part / P, e = k + 1 + m * (part + 1) / P;
    for (int j0 = first; j0 < n; j0 += W) {
      const int j = j0 + slot;
      double *x = A + (size_t)j * base;
      double d = 0.;
      if (j < n)
        for (int i = a; i < e; ++i) d += v[i] * x[i * stride];
      if (P > 1) {
        s[lane] = d;
        g.sync();
        d = s[slot];
#pragma unroll
        for (int q = 1; q < P; ++q) d += s[q * W + slot];
      }
      d *= tau;
      if (j < n)
        for (int i = a; i < e; ++i) x[i * stride] -= d * v[i];
      if (P > 1 && j0 + W < n) g.sync();
    }
  };
  for (int k = 0; k + 2 < n; ++k) {
    double tau = 0., alpha = 0.;
    if (P == 1 || lane < 32) {
      double ss = 0.;
      for (int i = k + 2 + (P > 1 ? lane & 31 : lane); i < n; i += P > 1 ? 32 : G) ss += A[i + k * n] * A[i + k * n];
      ss = P > 1 ? Group<32>().sum(ss) : g.sum(ss, n);
      if (ss != 0.) {  // else already zero below the subdiagonal
        const double x0 = A[(k + 1) + k * n];
        const double s2 = x0 * x0 + ss, nrm = s2 * fix_rsqrt(s2);
        alpha = -copysign(nrm, x0);
        tau = fix_reciprocal(nrm * (nrm + fabs(x0)));  // 2 / (u^T u) for u = x - alpha e1
        for (int i = k + 1 + lane; i < n; i += P > 1 ? 32 : G) v[i] = (i == k + 1) ? x0 - alpha : A[i + k * n];
      }
      if (P > 1 && lane == 0) {
        sc[4 * (k & 1)] = tau;
        sc[4 * (k & 1) + 1] = alpha;
      }
    }
    if (P > 1) {
      g.sync();
      tau = sc[4 * (k & 1)];
      alpha = sc[4 * (k & 1) + 1];
    }
    if (tau == 0. && alpha == 0.) continue;
    if (P == 1) g.sync();
    reflect(k, k + 1, n, 1, tau);  // left: A[k+1:, j] for the columns j > k; column k becomes alpha e1
    if (lane == 0) A[(k + 1) + k * n] = alpha;
    for (int i = k + 2 + lane; i < n; i += G) A[i + k * n] = 0.;
    g.sync();
    reflect(k, 0, 1, n, tau);      // right: A[i, k+1:] for all rows i
    g.sync();
  }
}

// Householder reflector P = I - v v^T mapping (x, y[, z]) to a multiple of e1: v = u / sqrt(beta) with
// u = (x + sign(x) ||.||, y, z) and beta = u^T u / 2 = ||.|| (||.|| + |x|), so |v|^2 = 2. Normalizing u by one
// reciprocal square root (instead of a square root and a reciprocal for tau = 1/beta) also drops the tau
// multiplication from every application; both square roots run on the integer pipes, which leaves ten FP64 instructions
// on the sweep's serial chain instead of 35. Returns false when (x, y, z) is zero (P = I).
template <int NR>
__device__ __forceinline__ bool house3(double x, double y, double z, double *v)
{
  const double nn = x * x + y * y + (NR == 3 ? z * z : 0.);
  if ((__double_as_longlong(nn) << 1) == 0) return false;
  const double nrm = nn * fix_rsqrt(nn);
  const double r = fix_rsqrt(nrm * (nrm + fabs(x)));
  v[0] = (x + copysign(nrm, x)) * r;
  v[1] = y * r;
  v[2] = NR == 3 ? z * r : 0.;
  return true;
}

// Apply P = I - v v^T (v of length NR <= 3) to rows r0..r0+NR-1 of H over columns c0..c1, and to columns
// r0..r0+NR-1 over rows c2..c3.
template <int NR, int G>
__device__ __forceinline__ void apply_reflector(const Group<G> &g, double *H, int n, const double *v, int r0, int c0, int c1, int c2,
                                                int c3)
{
  const int lane = g.lane;
  for (int j = c0 + lane; j <= c1; j += G) {
    double s = v[0] * H[r0 + j * n] + v[1] * H[(r0 + 1) + j * n];
    if (NR == 3) s += v[2] * H[(r0 + 2) + j * n];
    H[r0 + j * n] -= s * v[0];
    H[(r0 + 1) + j * n] -= s * v[1];
    if (NR == 3) H[(r0 + 2) + j * n] -= s * v[2];
  }
  g.sync();
  for (int i = c2 + lane; i <= c3; i += G) {
    double s = H[i + r0 * n] * v[0] + H[i + (r0 + 1) * n] * v[1];
    if (NR == 3) s += H[i + (r0 + 2) * n] * v[2];
    H[i + r0 * n] -= s * v[0];
    H[i + (r0 + 1) * n] -= s * v[1];
    if (NR == 3) H[i + (r0 + 2) * n] -= s * v[2];
  }
  g.sync();
}

// Start of the unreduced block ending at row hi: the largest lo <= hi with H[lo, lo-1] negligible (set to zero), or
// 0. Lanes test the subdiagonals in parallel, 32 rows at a time from the bottom.
template <int G>
__device__ __forceinline__ int group_find_lo(const Group<G> &g, double *H, int n, int hi)
{
  const int lane = g.lane & 31;  // every warp of the group finds the same row
  for (int top = hi; top > 0; top -= 32) {
    const int r = top - lane;  // candidate row, r >= 1
    bool neg = false;
    if (r >= 1) {
      const double sub = fabs(H[r + (r - 1) * n]);
      double s = fabs(H[(r - 1) + (r - 1) * n]) + fabs(H[r + r * n]);
      if (s == 0.) s = 1.;
      neg = sub <= 2.220446049250313e-16 * s;
    }
    const unsigned m = __ballot_sync(0xffffffffu, neg);
    if (m) {
      const int first = __ffs(m) - 1;  // lowest lane = largest row
      const int lo = top - first;
      if (g.lane == 0) H[lo + (lo - 1) * n] = 0.;
      g.sync();
      return lo;
    }
  }
  return 0;
}

// Shared doubles beside the n of `work`: partial sums, two scalars per parity, the result.
__host__ __device__ constexpr int eig_work_doubles(int G) { return G > 64 ? G + 8 + 2 : 0; }

// QR iteration of group_max_real_eig on the Hessenberg matrix A; work: n doubles.
template <int G>
__device__ bool group_qr_max_real(const Group<G> &g, double *A, int n, double *work, double *out_max, double cutoff)
{
  double *H = A;
  double vmax = -INFINITY;
  int hi = n - 1, iter = 0, total = 0;
  const int budget = 40 * n;
  bool ok = true;
  double u[3];
  while (hi >= 0) {
    if (total > budget) {
      ok = false;
      for (int i = 0; i <= hi; ++i) vmax = fmax(vmax, H[i + i * n]);
      break;
    }
    const int lo = hi > 0 ? group_find_lo<G>(g, H, n, hi) : 0;
    if (lo == hi) {
      vmax = fmax(vmax, H[hi + hi * n]);
      --hi;
      iter = 0;
      continue;
    }
    if (lo == hi - 1) {
      const double a = H[(hi - 1) + (hi - 1) * n], b = H[(hi - 1) + hi * n];
      const double c = H[hi + (hi - 1) * n], d = H[hi + hi * n];
      const double tr = 0.5 * (a + d), det = a * d - b * c;
      const double disc = tr * tr - det;
      vmax = fmax(vmax, disc >= 0. ? tr + sqrt(disc) : tr);
      hi -= 2;
      iter = 0;
      continue;
    }
    // the early exit: a block whose eigenvalues all lie left of the cutoff is done
    if (cutoff > -INFINITY && (iter & 1) && group_hess_hmatrix_below<G>(g, H, n, lo, hi, cutoff, work)) {
      hi = lo - 1;
      iter = 0;
      continue;
    }
    ++iter;
    ++total;
    // double shift from the trailing 2x2 block (exceptional shift after 10 and 20 stalled iterations)
    double s, t;
    if (iter == 10 || iter == 20) {
      const double w = fabs(H[hi + (hi - 1) * n]) + fabs(H[(hi - 1) + (hi - 2) * n]);
      s = 1.5 * w;
      t = w * w;
    } else {
      const int mm = hi - 1;
      s = H[mm + mm * n] + H[hi + hi * n];
      t = H[mm + mm * n] * H[hi + hi * n] - H[mm + hi * n] * H[hi + mm * n];
    }
    double x = H[lo + lo * n] * H[lo + lo * n] + H[lo + (lo + 1) * n] * H[(lo + 1) + lo * n] - s * H[lo + lo * n] + t;
    double y = H[(lo + 1) + lo * n] * (H[lo + lo * n] + H[(lo + 1) + (lo + 1) * n] - s);
    double z = H[(lo + 1) + lo * n] * H[(lo + 2) + (lo + 1) * n];
    if (G > 32) g.sync();  // every warp has read the scalars before any changes the matrix
    for (int k = lo - 1; k <= hi - 3; ++k) {
      if (house3<3>(x, y, z, u)) {
        const int c0 = k < lo ? lo : k;
        const int r1 = k + 4 < hi ? k + 4 : hi;
        apply_reflector<3, G>(g, H, n, u, k + 1, c0, hi, lo, r1);
      }
      x = H[(k + 2) + (k + 1) * n];
      y = H[(k + 3) + (k + 1) * n];
      if (k < hi - 3) z = H[(k + 4) + (k + 1) * n];
      if (G > 32) g.sync();
    }
    if (house3<2>(x, y, 0., u)) apply_reflector<2, G>(g, H, n, u, hi - 1, hi - 2, hi, lo, hi);
  }
  *out_max = vmax;
  return ok;
}

// Largest real part of the eigenvalues of the n x n matrix A (destroyed; A is balanced first). work: n +
// eig_work_doubles(G) doubles of shared memory. If cutoff is given and the balanced matrix's Gershgorin bound is <= cutoff, the function
// returns that bound instead of running QR (every eigenvalue is then known to have real part <= cutoff).
// With a cutoff the QR iteration also stops early: after every second sweep on an unreduced block, the block is
// tested with group_hess_hmatrix_below, and a block whose eigenvalues are all proven left of the cutoff is set aside
// without computing them. The returned maximum then covers only the eigenvalues computed, so it is exact whenever
// it exceeds the cutoff, and at most the cutoff otherwise, which is all max(lambda_max - cutoff, 0) needs.
// Returns false if the QR iteration did not converge within its budget (the largest real part of the diagonal
// found so far is returned then).
template <int G>
__device__ bool group_max_real_eig(const Group<G> &g, double *A, int n, double *work, double *out_max, double cutoff = -INFINITY)
{
  if (g.lane < 32) warp_balance(A, n);
  g.sync();
  const double gb = group_gershgorin_bound<G>(g, A, n);
  if (gb <= cutoff) {
    *out_max = gb;
    return true;
  }
  double *wide = work + n;
  group_hessenberg<G>(g, A, n, work, wide, wide + G);
  if constexpr (G <= 64) {
    return group_qr_max_real<G>(g, A, n, work, out_max, cutoff);
  } else {
    // the sweeps are a serial chain with a row and a column of work per step: the first two warps
    double *res = wide + G + 8;
    if (g.lane < 64) {
      Group<64> two(wide, 0);
      two.id = g.id + 8;  // a barrier of its own
      double m;
      const bool ok = group_qr_max_real<64>(two, A, n, work, &m, cutoff);
      if (g.lane == 0) {
        res[0] = m;
        res[1] = ok ? 1. : 0.;
      }
    }
    g.sync();
    *out_max = res[0];
    return res[1] != 0.;
  }
}

}  // namespace sfgb
