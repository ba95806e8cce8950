// Warp-level dense LU with partial pivoting and triangular solves on column-major matrices in shared memory
// (the factorization LAPACK dgetrf computes, with 0-based pivots), used by the batched Newton algebra, the adjoint's
// stage systems and the persistent integrator.
#pragma once
#include <cuda_runtime.h>

#include "gj_device.cuh"

namespace sfgb {

// Magnitudes as integer keys: finite non-negative values order like their bit patterns. The warp's largest |x| and the
// lowest index that has it (as idamax); a NaN orders above every number. none: this lane holds no value.
__device__ __forceinline__ int warp_argmax_abs(double x, int index, bool none)
{
  const unsigned h = none ? 0u : ((unsigned)__double2hiint(x) & 0x7fffffffu) + 1u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, h);
  const unsigned l = h == mh ? (unsigned)__double2loint(x) : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, l);
  return (int)__reduce_min_sync(0xffffffffu, h == mh && l == ml ? (unsigned)index : 0x7fffffffu);
}
__device__ __forceinline__ int warp_argmax_abs(float x, int index, bool none)
{
  const unsigned h = none ? 0u : ((unsigned)__float_as_int(x) & 0x7fffffffu) + 1u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, h);
  return (int)__reduce_min_sync(0xffffffffu, h == mh ? (unsigned)index : 0x7fffffffu);
}
__device__ __forceinline__ bool larger_abs(double a, double b)
{
  return ((unsigned long long)__double_as_longlong(a) << 1) > ((unsigned long long)__double_as_longlong(b) << 1);
}
__device__ __forceinline__ bool larger_abs(float a, float b)
{
  return ((unsigned)__float_as_int(a) << 1) > ((unsigned)__float_as_int(b) << 1);
}
__device__ __forceinline__ double lu_reciprocal(double p) { return fix_reciprocal(p); }
__device__ __forceinline__ float lu_reciprocal(float p) { return 1.f / p; }
// A reciprocal of full precision: neither infinite (of a subnormal pivot) nor itself subnormal.
__device__ __forceinline__ bool lu_normal(double r) { return (unsigned)(((__double2hiint(r) >> 20) & 0x7ff) - 1) < 2046u; }
__device__ __forceinline__ bool lu_normal(float r) { return (unsigned)(((__float_as_int(r) >> 23) & 0xff) - 1) < 254u; }

// A[i, j] -= A[i, k] A[k, j] for i, j > k. FP64: the elements are dealt to the lanes in column-major order, so that no
// FP64 instruction leaves lanes empty (an instruction costs the same with one lane as with 32); the position advances
// by 32 elements without a division. FP32: lanes over the rows of one column at a time, the multipliers in registers:
// more instructions with idle lanes, but on the FP32 pipe those cost a cycle each and the index arithmetic of the
// other form cost more than the update.
__device__ __forceinline__ void lu_trailing(double *A, int m, int ld, int k, int lane)
{
  const int r = m - k - 1;
  if (r <= 0) return;
  const int dj = 32 / r, di = 32 - dj * r;
  int jj = lane / r, ii = lane - jj * r;
  const double *lk = A + (size_t)k * ld + k + 1, *uk = A + (size_t)(k + 1) * ld + k;
  double *T = A + (size_t)(k + 1) * ld + k + 1;
  while (jj < r) {
    const int i0 = ii, j0 = jj;
    ii += di;
    jj += dj;
    if (ii >= r) {
      ii -= r;
      ++jj;
    }
    const bool two = jj < r;
    const int i1 = two ? ii : i0, j1 = two ? jj : j0;
    const double a0 = T[i0 + j0 * ld], l0 = lk[i0], u0 = uk[j0 * ld];
    const double a1 = T[i1 + j1 * ld], l1 = lk[i1], u1 = uk[j1 * ld];
    T[i0 + j0 * ld] = fma(-l0, u0, a0);
    if (two) T[i1 + j1 * ld] = fma(-l1, u1, a1);
    ii += di;
    jj += dj;
    if (ii >= r) {
      ii -= r;
      ++jj;
    }
  }
}

__device__ __forceinline__ void lu_trailing(float *A, int m, int ld, int k, int lane)
{
  for (int i = k + 1 + lane; i < m; i += 32) {
    const float l = A[i + k * ld];
    int j = k + 1;
    for (; j + 3 < m; j += 4) {
      float a[4], u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        u[q] = A[k + (j + q) * ld];
        a[q] = A[i + (j + q) * ld];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) A[i + (j + q) * ld] = fmaf(-l, u[q], a[q]);
    }
    for (; j < m; ++j) A[i + j * ld] = fmaf(-l, A[k + j * ld], A[i + j * ld]);
  }
}

// Right-looking LU with partial pivoting of an m x m column-major matrix (leading dimension ld) in shared memory, one
// warp. Returns info (0, or k+1 for an exactly zero pivot at step k). PERM false: piv holds LAPACK's interchanges
// (0-based). PERM true, for repeated solves: piv holds the final row permutation (piv[i]: the original row that ends
// in row i) and dinv the reciprocals of U's diagonal, so that a solve applies the permutation while loading its
// right-hand side and multiplies instead of dividing on its serial backward sweep.
template <bool PERM, typename F>
__device__ __forceinline__ int warp_lu_factor(F *A, int m, int ld, int *piv, F *dinv)
{
  const int lane = threadIdx.x & 31;
  if (PERM) {
    for (int i = lane; i < m; i += 32) piv[i] = i;
    __syncwarp();
  }
  int info = 0;
  for (int k = 0; k < m; ++k) {
    F best = (F)0;
    int at = -1;
    for (int i = k + lane; i < m; i += 32) {
      const F v = A[i + k * ld];
      if (at < 0 || larger_abs(v, best)) {
        best = v;
        at = i;
      }
    }
    const int bi = warp_argmax_abs(best, at, at < 0);
    if (!PERM && lane == 0) piv[k] = bi;
    if (bi != k) {
      if (PERM && lane == 0) {
        const int t = piv[k];
        piv[k] = piv[bi];
        piv[bi] = t;
      }
      for (int j = lane; j < m; j += 32) {
        const F t = A[k + j * ld];
        A[k + j * ld] = A[bi + j * ld];
        A[bi + j * ld] = t;
      }
    }
    __syncwarp();
    const F pv = A[k + k * ld];
    const F inv = lu_reciprocal(pv);
    if (PERM && lane == 0) dinv[k] = inv;
    if (pv == (F)0) {
      if (!info) info = k + 1;
      continue;
    }
    for (int i = k + 1 + lane; i < m; i += 32) A[i + k * ld] *= inv;
    __syncwarp();
    lu_trailing(A, m, ld, k, lane);
    __syncwarp();
  }
  return info;
}

template <typename F>
__device__ __forceinline__ int warp_lu_pd(F *A, int m, int *perm, F *dinv)
{
  return warp_lu_factor<true>(A, m, m, perm, dinv);
}

// Solve (LU) x = b with the factors of warp_lu_pd, x holding the permuted right-hand side (x[i] = b[perm[i]]).
template <typename F>
__device__ __forceinline__ void warp_lu_solve_pd(const F *LU, int m, const F *dinv, F *x)
{
  const int lane = threadIdx.x & 31;
  __syncwarp();
  for (int j = 0; j < m; ++j) {
    const F xj = x[j];
    for (int i = j + 1 + lane; i < m; i += 32) x[i] -= LU[i + j * m] * xj;
    __syncwarp();
  }
  for (int j = m - 1; j >= 0; --j) {
    const F xj = x[j] * dinv[j];
    for (int i = lane; i < j; i += 32) x[i] -= LU[i + j * m] * xj;
    __syncwarp();
    if (lane == 0) x[j] = xj;  // after the barrier: no lane still reads x[j]
  }
  __syncwarp();
}

// The triangular sweeps of warp_lu_solve_pd with row lane + 32 s of x in register s: a step's value travels by a shuffle
// instead of through shared memory behind a barrier, and the factors' columns are loaded ahead of it, so that a step waits
// for the shuffle and one FMA only. The register that holds the next step's value is updated first.
template <int R, typename F>
__device__ __forceinline__ void warp_lu_sweeps(const F *LU, int m, int lane, const F *dinv, F (&x)[R])
{
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int j1 = min(m, 32 * q + 32);
#pragma unroll 4
    for (int j = 32 * q; j < j1; ++j) {
      F l[R];
#pragma unroll
      for (int s = q; s < R; ++s) {
        const int i = lane + 32 * s;
        l[s] = i > j && i < m ? LU[i + j * m] : (F)0;
      }
      const F xj = __shfl_sync(0xffffffffu, x[q], j & 31);
#pragma unroll
      for (int s = q; s < R; ++s)
        if (lane + 32 * s > j) x[s] -= l[s] * xj;
    }
  }
#pragma unroll
  for (int q = R - 1; q >= 0; --q) {
    const F di = lane + 32 * q < m ? dinv[lane + 32 * q] : (F)0;
#pragma unroll 4
    for (int j = min(m, 32 * q + 32) - 1; j >= 32 * q; --j) {
      F l[R];
#pragma unroll
      for (int s = 0; s <= q; ++s) {
        const int i = lane + 32 * s;
        l[s] = i < j ? LU[i + j * m] : (F)0;
      }
      const F own = x[q] * di;  // the step's value in lane j
      const F xj = __shfl_sync(0xffffffffu, own, j & 31);
#pragma unroll
      for (int s = q; s >= 0; --s)
        if (lane + 32 * s < j) x[s] -= l[s] * xj;
      if (lane == (j & 31)) x[q] = own;
    }
  }
}

// warp_lu_solve_pd with x in registers, for m <= 32 R. The integrator keeps the form above: with this one its register
// spills cost more than the sweeps gained (1000 h2 reactors 199 -> 205 ms).
template <int R, typename F>
__device__ __forceinline__ void warp_lu_solve_regs(const F *LU, int m, const F *dinv, F *x)
{
  const int lane = threadIdx.x & 31;
  F r[R];
#pragma unroll
  for (int s = 0; s < R; ++s) r[s] = lane + 32 * s < m ? x[lane + 32 * s] : (F)0;
  warp_lu_sweeps<R>(LU, m, lane, dinv, r);
#pragma unroll
  for (int s = 0; s < R; ++s)
    if (lane + 32 * s < m) x[lane + 32 * s] = r[s];
  __syncwarp();
}

}  // namespace sfgb
