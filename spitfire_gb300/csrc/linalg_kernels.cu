// Batched dense Newton algebra: LU factorization of A = gamma_h * J - I with partial pivoting and the matching
// triangular solves, one warp per matrix.
//
// Replaces the scipy LAPACK calls of HomogeneousReactor (reactors.py:340-356): dgetrf on (prefactor*J - I) and
// dgetrs per Newton iteration. The FP32 variant factorizes the same matrix in single precision (FP32 pipe) and
// recovers FP64 accuracy in the solve by residual refinement r = b - A x with A in FP64.
#include <algorithm>

#include "sf_internal.h"
#include "warp_lu.cuh"

namespace sfgb {

namespace {

// Matrices per CTA: three warps, so that three CTAs with a 55 x 55 FP64 matrix (odd leading dimension: the row swaps and
// row reads then touch different banks) per warp fill an SM's shared memory.
constexpr int kWarpsPerCta = 3;

__host__ __device__ constexpr int lu_ld(int m) { return m | 1; }

// Shared memory of a factorization CTA
template <typename F>
size_t lu_smem(int m)
{
  return (size_t)kWarpsPerCta * ((size_t)m * lu_ld(m) * sizeof(F) + (size_t)m * 4);
}

// A = gamma h J - I (also to outA if given) and its LU factors, one warp per matrix, F = double or float. Bound for FP64:
// m^3 / 3 FMAs and a reciprocal per column, 1.05 ms for 8192 matrices of 54 x 54 at the FP64 issue rate.
template <typename F>
__global__ void __launch_bounds__(32 * kWarpsPerCta) lu_kernel(int n, int m, const double *J, const double *gh,
                                                               double *outA, F *outLU, int *piv, int *info)
{
  extern __shared__ __align__(16) unsigned char sm[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mm = m * m, ld = lu_ld(m);
  F *A = reinterpret_cast<F *>(sm) + (size_t)w * m * ld;
  int *pv = reinterpret_cast<int *>(reinterpret_cast<F *>(sm) + (size_t)kWarpsPerCta * m * ld) + w * m;
  const int dc = 32 / m, dr = 32 - dc * m, col0 = lane / m, row0 = lane - col0 * m;
  for (int s = blockIdx.x * kWarpsPerCta + w; s < n; s += gridDim.x * kWarpsPerCta) {
    const double g = gh[s];
    const double *Js = J + (size_t)s * mm;
    int row = row0, col = col0;
#pragma unroll 4
    for (int e = lane; e < mm; e += 32) {
      const double v = fma(g, Js[e], row == col ? -1. : 0.);
      A[row + col * ld] = (F)v;
      if (outA) outA[(size_t)s * mm + e] = v;
      row += dr;
      col += dc;
      if (row >= m) {
        row -= m;
        ++col;
      }
    }
    __syncwarp();
    const int inf = warp_lu_factor<false>(A, m, ld, pv, (F *)nullptr);
    row = row0;
    col = col0;
#pragma unroll 4
    for (int e = lane; e < mm; e += 32) {
      outLU[(size_t)s * mm + e] = A[row + col * ld];
      row += dr;
      col += dc;
      if (row >= m) {
        row -= m;
        ++col;
      }
    }
    for (int k = lane; k < m; k += 32) piv[(size_t)s * m + k] = pv[k];
    if (info && lane == 0) info[s] = inf;
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------------------------ solves
// One warp per system, its vectors in registers (element i in lane i % 32, register i / 32; R registers), the factors
// streamed from global memory a few columns ahead: every factor is used once per sweep, so staging it in shared memory
// only limited the warps per SM.
constexpr int kSolveWarps = 4;
constexpr int kAheadCols = 4;

template <int R, typename F>
__device__ __forceinline__ F reg_get(const F (&v)[R], int k)
{
  F out = __shfl_sync(0xffffffffu, v[0], k & 31);
#pragma unroll
  for (int s = 1; s < R; ++s) {
    const F t = __shfl_sync(0xffffffffu, v[s], k & 31);
    if ((k >> 5) == s) out = t;
  }
  return out;
}

// The row order that the interchanges of the factorization give: perm element i is the original row that ends in row i.
template <int R>
__device__ __forceinline__ void reg_permutation(const int *piv, int m, int lane, int (&perm)[R])
{
  int pv[R];
#pragma unroll
  for (int s = 0; s < R; ++s) {
    perm[s] = lane + 32 * s;
    pv[s] = perm[s] < m ? piv[perm[s]] : 0;
  }
  for (int k = 0; k < m; ++k) {
    const int p = reg_get<R>(pv, k);
    const int a = reg_get<R>(perm, k), b = reg_get<R>(perm, p);
#pragma unroll
    for (int s = 0; s < R; ++s) {
      if (lane + 32 * s == k) perm[s] = b;
      if (lane + 32 * s == p) perm[s] = a;
    }
  }
}

// A pivot kept for quotients by it as accurate as a division. FP64: its reciprocal in two parts, x (h + l) = fma(x, h, x l), one
// FP64 instruction beyond the product with a rounded reciprocal, whose rounding had made the solutions' errors up to 7 %
// larger (11 equations, root mean square over 64 systems). 16,384 solves of 53 equations: 285 us with the rounded
// reciprocal, 306 so, 376 with the quotient in fixed point, 708 with divisions. FP32: the reciprocal and the pivot, for one
// correction of the product. set: false where there is no such form (a reciprocal that is not a normal number: of a subnormal
// or zero pivot, or of one near the largest); the system is then solved by reg_lu_solve_dividing.
template <typename F>
struct Pivot;

template <>
struct Pivot<double> {
  double h, l;
  __device__ __forceinline__ bool set(double d)
  {
    h = lu_reciprocal(d);
    l = h * fma(-d, h, 1.);
    return lu_normal(h);
  }
  __device__ __forceinline__ double quotient(double x) const
  {
    const double t = x * l;
    // an infinite low part (of an infinite x, or where the quotient leaves the range) or a zero could have the other sign: -0
    // then, which changes no sum
    const unsigned a = (unsigned)__double2hiint(t) & 0x7fffffffu;
    return fma(x, h, (a | (unsigned)__double2loint(t)) != 0u && a < 0x7ff00000u ? t : -0.);
  }
};

template <>
struct Pivot<float> {
  float r, d;
  __device__ __forceinline__ bool set(float v)
  {
    d = v;
    r = lu_reciprocal(v);
    return lu_normal(r);
  }
  __device__ __forceinline__ float quotient(float x) const
  {
    const float q = x * r;
    const float c = fmaf(fmaf(-q, d, x), r, q);
    return ((unsigned)__float_as_int(q) & 0x7fffffffu) - 1u < 0x7f7fffffu ? c : q;  // zeros and infinities as they are
  }
};

template <int R, typename F>
__device__ __forceinline__ bool reg_pivots(const F *LU, int m, int lane, Pivot<F> (&rd)[R])
{
  bool odd = false;
#pragma unroll
  for (int s = 0; s < R; ++s) {
    const int i = lane + 32 * s;
    odd = !rd[s].set(i < m ? LU[(size_t)i * (m + 1)] : (F)1) || odd;
  }
  return __any_sync(0xffffffffu, odd);
}

template <int R, typename F>
__device__ __forceinline__ void load_columns(F (&c)[kAheadCols][R], const F *M, int m, int lane, int j, int step)
{
#pragma unroll
  for (int u = 0; u < kAheadCols; ++u) {
    const int jj = j + u * step;
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int i = lane + 32 * s;
      c[u][s] = jj >= 0 && jj < m && i < m ? M[i + (size_t)jj * m] : (F)0;
    }
  }
}

// x <- (LU)^-1 x with x in the factors' row order and rd U's diagonal.
template <int R, typename F>
__device__ __forceinline__ void reg_lu_solve(const F *LU, int m, int lane, const Pivot<F> (&rd)[R], F (&x)[R])
{
  F c[kAheadCols][R], nx[kAheadCols][R];
  load_columns<R>(c, LU, m, lane, 0, 1);
  for (int j0 = 0; j0 < m; j0 += kAheadCols) {
    load_columns<R>(nx, LU, m, lane, j0 + kAheadCols, 1);
#pragma unroll
    for (int u = 0; u < kAheadCols; ++u) {
      const int j = j0 + u;
      if (j < m) {
        const F xj = reg_get<R>(x, j);
#pragma unroll
        for (int s = 0; s < R; ++s)
          if (32 * s + 31 > j && lane + 32 * s > j) x[s] = fma(-c[u][s], xj, x[s]);
      }
    }
#pragma unroll
    for (int u = 0; u < kAheadCols; ++u)
#pragma unroll
      for (int s = 0; s < R; ++s) c[u][s] = nx[u][s];
  }
  load_columns<R>(c, LU, m, lane, m - 1, -1);
  for (int j0 = m - 1; j0 >= 0; j0 -= kAheadCols) {
    load_columns<R>(nx, LU, m, lane, j0 - kAheadCols, -1);
#pragma unroll
    for (int u = 0; u < kAheadCols; ++u) {
      const int j = j0 - u;
      if (j >= 0) {
        F xs = x[0];
        Pivot<F> rs = rd[0];
#pragma unroll
        for (int s = 1; s < R; ++s)
          if ((j >> 5) == s) {
            xs = x[s];
            rs = rd[s];
          }
        const F xj = __shfl_sync(0xffffffffu, rs.quotient(xs), j & 31);
#pragma unroll
        for (int s = 0; s < R; ++s) {
          if (32 * s < j && lane + 32 * s < j) x[s] = fma(-c[u][s], xj, x[s]);
          if (lane + 32 * s == j) x[s] = xj;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kAheadCols; ++u)
#pragma unroll
      for (int s = 0; s < R; ++s) c[u][s] = nx[u][s];
  }
}

// The same with a division per pivot and without columns held ahead, so that beside the sweeps above it needs no registers of
// its own (as a choice in every step of those, division cost them eight and a quarter of the FP32 solves' time).
template <int R, typename F>
__device__ __forceinline__ void reg_lu_solve_dividing(const F *LU, int m, int lane, F (&x)[R])
{
#pragma unroll 1
  for (int j = 0; j < m; ++j) {
    const F xj = reg_get<R>(x, j);
#pragma unroll
    for (int s = 0; s < R; ++s)
      if (lane + 32 * s > j && lane + 32 * s < m) x[s] = fma(-LU[lane + 32 * s + (size_t)j * m], xj, x[s]);
  }
#pragma unroll 1
  for (int j = m - 1; j >= 0; --j) {
    const F xj = reg_get<R>(x, j) / LU[(size_t)j * (m + 1)];
#pragma unroll
    for (int s = 0; s < R; ++s) {
      if (lane + 32 * s < j) x[s] = fma(-LU[lane + 32 * s + (size_t)j * m], xj, x[s]);
      if (lane + 32 * s == j) x[s] = xj;
    }
  }
}

template <int R>
__global__ void __launch_bounds__(32 * kSolveWarps) solve64_kernel(int n, int m, const double *LU, const int *piv,
                                                                   const double *b, double *x)
{
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int sys = blockIdx.x * kSolveWarps + w; sys < n; sys += gridDim.x * kSolveWarps) {
    const double *L = LU + (size_t)sys * m * m;
    int perm[R];
    reg_permutation<R>(piv + (size_t)sys * m, m, lane, perm);
    Pivot<double> rd[R];
    double xr[R];
    const bool odd = reg_pivots<R>(L, m, lane, rd);
#pragma unroll
    for (int s = 0; s < R; ++s) xr[s] = lane + 32 * s < m ? b[(size_t)sys * m + perm[s]] : 0.;
    if (odd)
      reg_lu_solve_dividing<R>(L, m, lane, xr);
    else
      reg_lu_solve<R>(L, m, lane, rd, xr);
#pragma unroll
    for (int s = 0; s < R; ++s)
      if (lane + 32 * s < m) x[(size_t)sys * m + lane + 32 * s] = xr[s];
  }
}

// FP32 triangular solves + FP64 residual refinement (r = b - A x, x += LU32^-1 r).
template <int R>
__global__ void __launch_bounds__(32 * kSolveWarps, R == 1 ? 8 : (R == 2 ? 5 : 4)) solve32_kernel(int n, int m, const double *A, const float *LU,
                                                                   const int *piv, int refine, const double *b,
                                                                   double *x)
{
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int sys = blockIdx.x * kSolveWarps + w; sys < n; sys += gridDim.x * kSolveWarps) {
    const float *L = LU + (size_t)sys * m * m;
    const double *As = A + (size_t)sys * m * m;
    int perm[R];
    reg_permutation<R>(piv + (size_t)sys * m, m, lane, perm);
    Pivot<float> rd[R];
    float r[R];
    const bool odd = reg_pivots<R>(L, m, lane, rd);
    double bs[R], xs[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
      bs[s] = lane + 32 * s < m ? b[(size_t)sys * m + lane + 32 * s] : 0.;
      r[s] = lane + 32 * s < m ? (float)b[(size_t)sys * m + perm[s]] : 0.f;
    }
    if (odd)
      reg_lu_solve_dividing<R>(L, m, lane, r);
    else
      reg_lu_solve<R>(L, m, lane, rd, r);
#pragma unroll
    for (int s = 0; s < R; ++s) xs[s] = (double)r[s];
    for (int it = 0; it < refine; ++it) {
      // residual in FP64, rows over lanes
      double res[R], c[kAheadCols][R], nx[kAheadCols][R];
#pragma unroll
      for (int s = 0; s < R; ++s) res[s] = bs[s];
      load_columns<R>(c, As, m, lane, 0, 1);
      for (int j0 = 0; j0 < m; j0 += kAheadCols) {
        load_columns<R>(nx, As, m, lane, j0 + kAheadCols, 1);
#pragma unroll
        for (int u = 0; u < kAheadCols; ++u)
          if (j0 + u < m) {
            const double xj = reg_get<R>(xs, j0 + u);
#pragma unroll
            for (int s = 0; s < R; ++s) res[s] = fma(-c[u][s], xj, res[s]);
          }
#pragma unroll
        for (int u = 0; u < kAheadCols; ++u)
#pragma unroll
          for (int s = 0; s < R; ++s) c[u][s] = nx[u][s];
      }
      // into the factors' row order: element perm[s] of the residual
      float rf[R];
#pragma unroll
      for (int s = 0; s < R; ++s) rf[s] = (float)res[s];
#pragma unroll
      for (int s = 0; s < R; ++s) {
        r[s] = __shfl_sync(0xffffffffu, rf[0], perm[s] & 31);
#pragma unroll
        for (int q = 1; q < R; ++q) {
          const float t = __shfl_sync(0xffffffffu, rf[q], perm[s] & 31);
          if ((perm[s] >> 5) == q) r[s] = t;
        }
      }
      if (odd)
        reg_lu_solve_dividing<R>(L, m, lane, r);
      else
        reg_lu_solve<R>(L, m, lane, rd, r);
#pragma unroll
      for (int s = 0; s < R; ++s) xs[s] += (double)r[s];
    }
#pragma unroll
    for (int s = 0; s < R; ++s)
      if (lane + 32 * s < m) x[(size_t)sys * m + lane + 32 * s] = xs[s];
  }
}

int grid_for(int n, int per_cta, int ctas_per_sm)
{
  int dev, nsm;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const long long need = ((long long)n + per_cta - 1) / per_cta;
  return (int)std::max<long long>(1, std::min<long long>(need, (long long)nsm * ctas_per_sm));
}

template <typename F>
int launch_lu(int n, int m, const double *J, const double *gamma_h, double *out_A, F *out_lu, int *out_piv,
              int *out_info, cudaStream_t st)
{
  const size_t smem = lu_smem<F>(m);
  try {
    ensure_dynamic_smem((const void *)lu_kernel<F>, smem);
  } catch (sf_error &e) {
    set_error(e.what());
    return e.code;
  }
  // as many CTAs as the shared memory holds (233,472 bytes per SM, 1 KB of it per CTA), at most 10
  const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(10, 233472 / (smem + 1024)));
  lu_kernel<F><<<grid_for(n, kWarpsPerCta, per_sm), 32 * kWarpsPerCta, smem, st>>>(n, m, J, gamma_h, out_A, out_lu,
                                                                                   out_piv, out_info);
  return SF_OK;
}

template <int R>
void launch_solve(int n, int m, const double *A, const void *lu, const int *piv, int precision, int refine,
                  const double *b, double *out_x, cudaStream_t st)
{
  // Several blocks per resident one (four to nine by the registers), so that a last wave that is part empty costs little: 16,384
  // FP32 systems of 53 x 53, five blocks resident, 380 us against 421 with eight blocks per SM.
  const int grid = grid_for(n, kSolveWarps, 16);
  if (precision == 0)
    solve64_kernel<R><<<grid, 32 * kSolveWarps, 0, st>>>(n, m, (const double *)lu, piv, b, out_x);
  else
    solve32_kernel<R><<<grid, 32 * kSolveWarps, 0, st>>>(n, m, A, (const float *)lu, piv, refine, b, out_x);
}

}  // namespace
}  // namespace sfgb

using namespace sfgb;

extern "C" {

int sf_newton_lu_batch(int n, int m, const double *J, const double *gamma_h, int precision, double *out_A,
                       void *out_lu, int *out_piv, int *out_info, void *stream)
{
  if (n < 0 || m < 1 || m > 80 || (n > 0 && (!J || !gamma_h || !out_lu || !out_piv))) {
    set_error("sf_newton_lu_batch: bad argument (1 <= m <= 80)");
    return SF_ERR_INVALID_ARGUMENT;
  }
  if (precision == 1 && !out_A) {
    set_error("sf_newton_lu_batch: precision 1 needs out_A for the refinement");
    return SF_ERR_INVALID_ARGUMENT;
  }
  if (n == 0) return SF_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == 0 || precision == 1) {
    const int rc = precision == 0 ? launch_lu<double>(n, m, J, gamma_h, out_A, (double *)out_lu, out_piv, out_info, st)
                                  : launch_lu<float>(n, m, J, gamma_h, out_A, (float *)out_lu, out_piv, out_info, st);
    if (rc != SF_OK) return rc;
  } else {
    set_error("sf_newton_lu_batch: precision must be 0 or 1");
    return SF_ERR_INVALID_ARGUMENT;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(cudaGetErrorString(e));
    return SF_ERR_CUDA;
  }
  return SF_OK;
}

int sf_newton_solve_batch(int n, int m, const double *A, const void *lu, const int *piv, int precision, int refine,
                          const double *b, double *out_x, void *stream)
{
  if (n < 0 || m < 1 || m > 80 || (n > 0 && (!lu || !piv || !b || !out_x))) {
    set_error("sf_newton_solve_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  if (n == 0) return SF_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == 0 || precision == 1) {
    if (precision == 1 && !A) {
      set_error("sf_newton_solve_batch: precision 1 needs A");
      return SF_ERR_INVALID_ARGUMENT;
    }
    if (m <= 32)
      launch_solve<1>(n, m, A, lu, piv, precision, refine, b, out_x, st);
    else if (m <= 64)
      launch_solve<2>(n, m, A, lu, piv, precision, refine, b, out_x, st);
    else
      launch_solve<3>(n, m, A, lu, piv, precision, refine, b, out_x, st);
  } else {
    set_error("sf_newton_solve_batch: precision must be 0 or 1");
    return SF_ERR_INVALID_ARGUMENT;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(cudaGetErrorString(e));
    return SF_ERR_CUDA;
  }
  return SF_OK;
}

}  // extern "C"
