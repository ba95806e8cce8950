// Device building blocks of the Griffon hot path on sm_103a.
//
// Execution model: one *state group* of G lanes evaluates one thermochemical state at a time: 8, 16 or 32 lanes of a warp, or
// 64, 128 or 256 threads of a block (and one lane, in the thread-per-state kernels).
// Lanes split species (thermodynamics, gathers by species) and reactions (rate evaluation), and a static gather
// program assembles Jacobian entries with one FP64 FMA per item. The packed mechanism is copied into shared
// memory once per CTA with a bulk-async (TMA) copy; every state group keeps its own scratch area in shared memory.
// Reference formulas: src/spitfire/griffon/src/thermodynamics_kernels.cpp, chemistry_kernels.cpp,
// rates_sensitivities_exact.cpp (file:line in comments below).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "exp_table.h"
#include "fixed_point.cuh"
#include "sf_mech.h"

namespace sfgb {

// -------------------------------------------------------------------------------------------- error reporting
// Device-side error word (one int per mechanism, allocated with it): kernels never trap; a failed bounded wait or
// an invalid input records a code there and the kernel returns. sf_device_status() (host) reads and clears it.
enum { DEVERR_BULK_TIMEOUT = 1, DEVERR_BAD_ARG = 2, DEVERR_WAIT_TIMEOUT = 3 };

__device__ __forceinline__ void report_error(int *status, int code)
{
  if (status) atomicCAS(status, 0, code);
}

// --------------------------------------------------------------------------------- bulk copy into shared memory
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Copy `bytes` (multiple of 16, both addresses 16-byte aligned) from global to shared memory through the TMA
// engine (cp.async.bulk) and wait for it on an mbarrier. The wait is bounded: on timeout the error word is set,
// a second bounded wait gives the copy a chance to land, and the function reports failure.
__device__ inline bool stage_to_smem(void *dst, const void *src, uint32_t bytes, uint64_t *bar, int *status)
{
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    constexpr uint32_t kChunk = 16384;
    for (uint32_t off = 0; off < bytes; off += kChunk) {
      const uint32_t n = bytes - off < kChunk ? bytes - off : kChunk;
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr((char *)dst + off)),
          "l"((const char *)src + off), "r"(n), "r"(smem_addr(bar))
          : "memory");
    }
  }
  bool done = false;
  for (int it = 0; it < (1 << 22) && !done; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(0)
        : "memory");
    done = ok != 0;
  }
  if (!done) {
    report_error(status, DEVERR_BULK_TIMEOUT);
    for (int it = 0; it < (1 << 22) && !done; ++it) {
      uint32_t ok;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(ok)
          : "r"(smem_addr(bar)), "r"(0)
          : "memory");
      done = ok != 0;
    }
  }
  __syncthreads();
  return done;
}

// ----------------------------------------------------------------------------------------------- state groups
// Sums over a group are formed together where the caller has several (sum2, sum4): on GB300 every FP64 instruction of
// a warp costs the same 64-76 cycles of its scheduler's FP64 unit however many lanes carry a value, and the
// transposed reduction below adds four 32-lane sums in 6 instructions instead of 20 (the first two exchanges leave
// each quarter of the lanes with one of the four sums).
//
// Group<G>, G <= 32: part of a warp. Group<G>, G = 64, 128 or 256: several warps of a block, for launches with too few
// states to give every scheduler of the GPU a warp of its own (below).
template <int G, bool WIDE = (G > 32)>
struct Group {
  static constexpr int kShared = 0;  // doubles of shared memory the group's reductions take
  int lane;       // 0..G-1
  unsigned mask;  // lanes of this group within the warp
  __device__ __forceinline__ Group(double * = nullptr, int = 0)
  {
    const int wl = threadIdx.x & 31;
    lane = wl & (G - 1);
    mask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (wl & ~(G - 1)));
  }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  // The sums take the number of leading lanes that hold a value (a wide group's other warps then add nothing).
  __device__ __forceinline__ double max(double v, int = G) const
  {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(mask, v, o, G));
    return v;
  }
  __device__ __forceinline__ double sum(double v, int = G, int = 0) const
  {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, G);
    return v;
  }
  __device__ __forceinline__ void sum2(double &a, double &b, int = G, int = 0) const
  {
    if (G == 1) return;
    constexpr int H = G > 1 ? G / 2 : 1;
    const bool up = (lane & H) != 0;
    double r = (up ? b : a) + __shfl_xor_sync(mask, up ? a : b, H, G);
#pragma unroll
    for (int o = H / 2; o > 0; o >>= 1) r += __shfl_xor_sync(mask, r, o, G);
    a = __shfl_sync(mask, r, 0, G);
    b = __shfl_sync(mask, r, H, G);
  }
  __device__ __forceinline__ void sum4(double &a, double &b, double &c, double &d, int = G) const
  {
    if (G < 4) {
      sum2(a, b);
      sum2(c, d);
      return;
    }
    constexpr int H = G / 2, Q = G > 2 ? G / 4 : 1;
    const bool up = (lane & H) != 0, uq = (lane & Q) != 0;
    const double x = (up ? b : a) + __shfl_xor_sync(mask, up ? a : b, H, G);
    const double y = (up ? d : c) + __shfl_xor_sync(mask, up ? c : d, H, G);
    double r = (uq ? y : x) + __shfl_xor_sync(mask, uq ? x : y, Q, G);
#pragma unroll
    for (int o = Q / 2; o > 0; o >>= 1) r += __shfl_xor_sync(mask, r, o, G);
    a = __shfl_sync(mask, r, 0, G);
    b = __shfl_sync(mask, r, H, G);
    c = __shfl_sync(mask, r, Q, G);
    d = __shfl_sync(mask, r, H + Q, G);
  }
  // reciprocals of three values that all lanes hold: one instruction sequence for all three where the group has lanes
  // to share it
  __device__ __forceinline__ void recip3(double a, double b, double c, double &ia, double &ib, double &ic) const
  {
    if (G < 4) {
      ia = fix_reciprocal(a);
      ib = fix_reciprocal(b);
      ic = fix_reciprocal(c);
      return;
    }
    const double r = fix_reciprocal(lane == 1 ? b : (lane == 2 ? c : a));
    ia = __shfl_sync(mask, r, 0, G);
    ib = __shfl_sync(mask, r, 1, G);
    ic = __shfl_sync(mask, r, G < 4 ? 0 : 2, G);
  }
};

// A state group of several whole warps of one block (G = 64, 128 or 256 threads). An SM's FP64 rate is shared by four
// schedulers and one warp can use only its own scheduler's quarter, so a launch whose states are fewer than about
// four per SM runs each of them on all four. Warps meet at the group's own named barrier; a reduction goes through
// shared memory, with two alternating buffers so that one barrier per reduction is enough (a thread reuses a buffer only
// after the next reduction's barrier, which every thread passes after its reads of this one).
template <int G>
struct Group<G, true> {
  static constexpr int W = G / 32;
  static constexpr int kScalars = 16;
  static constexpr int kShared = 2 * 4 * W + kScalars;
  int lane, warp, id;
  double *red, *scalars;
  mutable int flip;
  __device__ __forceinline__ Group(double *shared, int group_in_block)
      : lane(threadIdx.x % G), warp((threadIdx.x % G) >> 5), id(1 + group_in_block), red(shared),
        scalars(shared + 2 * 4 * W), flip(0)
  {
  }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(G) : "memory"); }
  // N values per warp published by its first lane; the warps that hold data are those of the lanes first .. first +
  // count - 1
  template <int N, class Op>
  __device__ __forceinline__ void combine(double (&v)[N], int count, int first, Op op) const
  {
    const int w0 = first >> 5, w1 = min(W, (first + count + 31) >> 5);
    double *buf = red + flip * 4 * W;
    flip ^= 1;
    if (warp >= w0 && warp < w1 && (lane & 31) == 0) {
#pragma unroll
      for (int j = 0; j < N; ++j) buf[4 * warp + j] = v[j];
    }
    sync();
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = buf[4 * w0 + j];
    for (int w = w0 + 1; w < w1; ++w) {
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = op(v[j], buf[4 * w + j]);
    }
  }
  __device__ __forceinline__ bool holds(int count, int first) const
  {
    return warp * 32 < first + count && warp * 32 + 31 >= first;
  }
  static __device__ __forceinline__ double add(double a, double b) { return a + b; }
  static __device__ __forceinline__ double larger(double a, double b) { return fmax(a, b); }
  __device__ __forceinline__ double max(double v, int count = G) const
  {
    if (holds(count, 0)) v = Group<32>().max(v);
    double t[1] = {v};
    combine(t, count, 0, larger);
    return t[0];
  }
  __device__ __forceinline__ double sum(double v, int count = G, int first = 0) const
  {
    if (holds(count, first)) v = Group<32>().sum(v);
    double t[1] = {v};
    combine(t, count, first, add);
    return t[0];
  }
  __device__ __forceinline__ void sum2(double &a, double &b, int count = G, int first = 0) const
  {
    // a warp whose lanes hold only zeros (as most do in the sums over third-body reactions) skips the exchange
    const bool any = ((__double_as_longlong(a) | __double_as_longlong(b)) << 1) != 0;
    if (holds(count, first) && __any_sync(0xffffffffu, any)) Group<32>().sum2(a, b);
    double t[2] = {a, b};
    combine(t, count, first, add);
    a = t[0];
    b = t[1];
  }
  __device__ __forceinline__ void sum4(double &a, double &b, double &c, double &d, int count = G) const
  {
    if (holds(count, 0)) Group<32>().sum4(a, b, c, d);
    double t[4] = {a, b, c, d};
    combine(t, count, 0, add);
    a = t[0];
    b = t[1];
    c = t[2];
    d = t[3];
  }
};

inline __host__ __device__ int wide_group_doubles(int G)
{
  return G == 256 ? Group<256>::kShared : (G == 128 ? Group<128>::kShared : (G == 64 ? Group<64>::kShared : 0));
}

struct Blob {
  const double *d;
  const int *i;
};

// Scratch of one state interleaved with the states of the other 31 lanes of its warp (thread-per-state kernels):
// element i of this lane's state lives at p[32 i], so the lanes of a warp touch one contiguous 256-byte row.
// The state-group kernels use a plain double * into their shared-memory area instead; the device code below is
// written for either.
struct ScrStrided {
  double *p;  // base + lane
  __device__ __forceinline__ double &operator[](int i) const { return p[(size_t)i << 5]; }
  __device__ __forceinline__ ScrStrided operator+(int o) const { return ScrStrided{p + ((size_t)o << 5)}; }
};

__device__ __forceinline__ Blob blob_at(const DevMech &m, const void *base)
{
  Blob b;
  b.d = (const double *)base;
  b.i = (const int *)((const char *)base + (size_t)m.blob_doubles * 8);
  return b;
}

// ----------------------------------------------------------------------------------------- thermodynamics
// One species at temperature T: cp (clamped outside [Tmin, Tmax]), h (linear extrapolation outside), dcp/dT
// (zero outside), Gibbs energy g and B = d(g/RT)/dT-like term of the reverse-rate sensitivity
// (thermodynamics_kernels.cpp:45-131, 183-260, 262-351; chemistry_kernels.cpp:56-97;
//  rates_sensitivities_exact.cpp:83-124).
struct SpeciesThermo {
  double cp, h, dcp, g, TdB;  // TdB: T times the B term
};

// Magnitude tests on temperatures as integers: non-negative doubles order like their bit patterns (and a negative one
// below every positive), so that a comparison does not take an FP64 instruction.
__device__ __forceinline__ bool le_bits(double a, double b) { return __double_as_longlong(a) <= __double_as_longlong(b); }

// The four temperature terms t_j = A_j T^j of a NASA7 polynomial (A_j the stored, scaled coefficients) serve g, h, cp
// and their derivatives together inside the polynomials' range: about 20 FP64 instructions per species for the
// right-hand side where three separate Horner forms took 45 and six FP64 comparisons. Outside the range, where cp is
// clamped and h extrapolated, the general form below runs.
__device__ __forceinline__ SpeciesThermo species_thermo(const DevMech &m, Blob b, int k, double T, double logT,
                                                        double invT, bool want_sens)
{
  SpeciesThermo s;
  const double *c = b.d + m.d_nasa + 15 * k;
  const double invmw = b.d[m.d_invmw + k];
  s.dcp = 0.;
  s.TdB = 0.;
  if (m.all_nasa7 || b.i[m.i_thermo + k] == 2) {
    const double tmin = b.d[m.d_tmin + k], tmax = b.d[m.d_tmax + k];
    const double *a = c + (le_bits(T, c[0]) ? 8 : 1);  // polynomial for g and B: chosen by Tmid only
    if (le_bits(tmin, T) && le_bits(T, tmax)) {
      const double T2 = T * T;
      const double t1 = a[1] * T, t2 = a[2] * T2, t3 = a[3] * (T2 * T), t4 = a[4] * (T2 * T2);
      s.g = fma(T, (a[0] - a[6]) - fma(a[0], logT, (t1 + t2) + (t3 + t4)), a[5]);
      const double hm = fma(T, fma(4., t4, fma(3., t3, fma(2., t2, a[0] + t1))), a[5]);
      s.h = invmw * hm;
      s.cp = invmw * fma(20., t4, fma(12., t3, fma(6., t2, fma(2., t1, a[0]))));
      if (want_sens) {
        s.dcp = invmw * invT * fma(80., t4, fma(36., t3, fma(12., t2, 2. * t1)));
        s.TdB = fma(hm, invT * m.invRu, -1.);
      }
      return s;
    }
    s.g = a[5] + T * (a[0] - a[6] - a[0] * logT - T * (a[1] + T * (a[2] + T * (a[3] + T * a[4]))));
    // cp / h on the clamped temperature (dcp/dT is zero outside the range)
    const double tt = fmin(fmax(T, tmin), tmax);
    const double *p = c + ((tt <= c[0]) ? 8 : 1);
    const double cpm = p[0] + tt * (2. * p[1] + tt * (6. * p[2] + tt * (12. * p[3] + 20. * tt * p[4])));
    s.cp = invmw * cpm;
    const double hm = p[5] + tt * (p[0] + tt * (p[1] + tt * (2. * p[2] + tt * (3. * p[3] + tt * 4. * p[4]))));
    s.h = invmw * (hm + cpm * (T - tt));
    if (want_sens)
      s.TdB = m.invRu * ((a[0] - m.Ru) + T * (a[1] + T * (2 * a[2] + T * (3 * a[3] + T * 4 * a[4]))) + a[5] * invT);
  } else {
    // constant cp: c = [T0, h0, s0, cp, log T0] (thermodynamics_kernels.cpp:60-63, chemistry_kernels.cpp:88-89)
    s.cp = invmw * c[3];
    s.h = invmw * (c[1] + c[3] * (T - c[0]));
    s.g = c[1] + c[3] * (T - c[0]) - T * (c[2] + c[3] * (logT - c[4]));
    if (want_sens) s.TdB = b.d[m.d_mw + k] * m.invRu * (c[3] - invT * (c[3] * c[0] - c[1])) - 1;
  }
  return s;
}

__device__ __forceinline__ double ipow(double x, int n)
{
  double r = 1.;
  for (int i = 0; i < n; ++i) r *= x;
  return r;
}

// ------------------------------------------------------------------------------- table-driven exponential
// e^x by Tang's table-driven method (P. T. P. Tang, "Table-driven implementation of the exponential function in
// IEEE floating-point arithmetic", ACM TOMS 15(2), 1989), written for FP64 throughput:
//   x = (64 m + j) ln2/64 + r, |r| <= ln2/128: N = 64 m + j is the nearest integer to x 64/ln2 (one FMA against
//   1.5 2^52, whose low word is then N), and r = (x - N L1) - N L2 with L1 + L2 = ln2/64 (the first FMA is exact:
//   x and N L1 are multiples of the ulp of L1, and |r| < 2^-7);
//   e^r - 1 = p(r), its Taylor polynomial of degree 6 (truncation below 3e-20 on |r| <= ln2/128);
//   e^x = 2^m (T_j + T_j p), T_j = 2^(j/64) as a head and a tail (the blob's table, 16-byte pairs), the power of two
//   applied to the exponent field while the result stays normal (|x| < 708), else by two exact factors.
// Against a 113-bit reference on 2M arguments over the whole range: at most 0.51 ulp for normal results (CUDA's exp:
// 0.86-0.88), 99.8 % correctly rounded; about 11.7 warp FP64 instructions per call against 15.0 for CUDA's exp
// (throughput loops on a GB300). NaN in, NaN out; beyond the range, 0 or +inf.
__device__ __forceinline__ double exp_parts(double x, double &r, int &N)
{
  const double tm = fma(x, kExpInvL, 0x1.8p52);
  N = __double2loint(tm);
  const double Nd = tm - 0x1.8p52;
  r = fma(-Nd, kExpL2, fma(-Nd, kExpL1, x));
  return Nd;
}

__device__ __forceinline__ double exp_finish(double x, double y, int N)
{
  const long long ax = __double_as_longlong(x) & 0x7fffffffffffffffll;
  if (ax < 0x4086200000000000ll)  // |x| < 708: the result is normal
    return __longlong_as_double(__double_as_longlong(y) + (long long)(N >> 6) * (1ll << 52));
  if (x != x) return x;
  if (x > 709.8) return __longlong_as_double(0x7ff0000000000000ll);
  if (x < -745.2) return 0.;
  const int m = N >> 6, m1 = m / 2, m2 = m - m1;  // both factors normal
  return y * __longlong_as_double((long long)(1023 + m1) << 52) * __longlong_as_double((long long)(1023 + m2) << 52);
}

__device__ __forceinline__ double tab_exp(double x, const double *tab)
{
  double r;
  int N;
  exp_parts(x, r, N);
  double q = fma(r, 1. / 720., 1. / 120.);
  q = fma(r, q, 1. / 24.);
  q = fma(r, q, 1. / 6.);
  q = fma(r, q, 0.5);
  const double p = fma(q, r * r, r);
  const double2 t = reinterpret_cast<const double2 *>(tab)[N & 63];
  return exp_finish(x, t.x + fma(t.x, p, t.y), N);
}

__device__ __forceinline__ double fix_exp(double x, const double *tab)
{
  if ((((unsigned)__double2hiint(x)) & 0x7fffffffu) >= 0x40862000u) return tab_exp(x, tab);  // |x| >= 708 or NaN
  int N;
  unsigned long long f;
  fix_reduce(x, N, f);
  return fix_to_double(fix_exp2(f, reinterpret_cast<const unsigned long long *>(tab + 128)), N);
}

// The species' contribution to the reverse constants, formed once per state: x = -g/RT as x log2(e) in fixed point
// (fraction in gm, integer part in gk). A state whose temperature is outside the fixed-point range keeps x itself.
template <class S>
__device__ __forceinline__ void store_gibbs_factor(S scr, const ScratchLayout &L, int i, double gRT, bool fixed)
{
  double x = -gRT;
  if (fixed) {
    int N;
    unsigned long long f;
    fix_reduce(x, N, f);
    if ((((unsigned)__double2hiint(x)) & 0x7fffffffu) >= 0x41300000u) {  // |x| >= 2^20: 0 or infinity in any product
      N = __double2hiint(x) < 0 ? -(1 << 20) : 1 << 20;
      f = 0;
    }
    x = __longlong_as_double((long long)f);
    scr[L.gk + i] = __hiloint2double(0, N);
  }
  scr[L.gm + i] = x;
}

// A small integer (a stoichiometric coefficient or a sum of them) as a double: from the blob's table when within
// -32..31 (a shared-memory load), else converted.
__device__ __forceinline__ double small_int(const double *table, int k)
{
  return (unsigned)(k + 32) < 64u ? table[k + 32] : (double)k;
}

// ------------------------------------------------------------------------------------------ reaction phase
// Per-state quantities every reaction needs.
struct StateCtx {
  double T, logT, invT, rho, invRho, mmw, ct;
  double port;  // p_ref / (R T)
  bool fixed;   // rate constants in fixed point: 16 < T < 65536 and the blob holds them
  unsigned long long l60, u68;  // log2 T 2^60, 2^68 / T
  int option;  // rates-sensitivity option: 0 / 2 exact, 1 without third-body/falloff derivatives
};

// Product of C_j^nu_j over a reactant/product list, with the factor of list position `at` differentiated with
// respect to its concentration (nu * C^(nu-1)); at < 0: no differentiation.
template <class SC>
__device__ __forceinline__ double mass_action(const int *lst, int n, const SC &C, int at)
{
  double v = 1.;
  for (int j = 0; j < n; ++j) {
    const int e = lst[j];
    const int s = e & 0xFFFF, nu = e >> 16;
    const double c = C[s];
    if (j == at)
      v *= nu * ipow(c, nu - 1);
    else
      v *= ipow(c, nu);
  }
  return v;
}

// One side of a reaction with at most three species: the rate R = k prod_i C_i^nu_i and, with JAC, its derivatives
// t_j = dR/dC_j of list position j. The products are shared: a side of two species with unit coefficients takes
// three multiplications for all three values, one of three species six.
struct Side3 {
  double R, t0, t1, t2;
  __device__ __forceinline__ double t(int j) const { return j == 0 ? t0 : (j == 1 ? t1 : t2); }
};

template <bool JAC, class SC>
__device__ __forceinline__ Side3 side3(const int *lst, int n, const SC &C, double k, const double *smallint)
{
  Side3 o;
  o.t1 = o.t2 = 0.;
  // position j: p_j = C_j^nu_j and kd_j = k nu_j C_j^(nu_j - 1)
  const int e0 = lst[0];
  double p0 = C[e0 & 0xFFFF], kd0 = k;
  const bool unit0 = (e0 >> 16) == 1;
  if (!unit0) {
    const double cm = ipow(p0, (e0 >> 16) - 1);
    p0 *= cm;
    kd0 *= small_int(smallint, e0 >> 16) * cm;
  }
  if (n == 1) {
    o.R = k * p0;
    o.t0 = kd0;
    return o;
  }
  const int e1 = lst[1];
  double p1 = C[e1 & 0xFFFF], kd1 = k;
  if ((e1 >> 16) != 1) {
    const double cm = ipow(p1, (e1 >> 16) - 1);
    p1 *= cm;
    kd1 *= small_int(smallint, e1 >> 16) * cm;
  }
  if (n == 2) {
    o.t0 = kd0 * p1;
    o.R = unit0 ? o.t0 * p0 : k * p0 * p1;
    if (JAC) o.t1 = kd1 * p0;
    return o;
  }
  const int e2 = lst[2];
  double p2 = C[e2 & 0xFFFF], kd2 = k;
  if ((e2 >> 16) != 1) {
    const double cm = ipow(p2, (e2 >> 16) - 1);
    p2 *= cm;
    kd2 *= small_int(smallint, e2 >> 16) * cm;
  }
  if (JAC) {
    o.t0 = kd0 * p1 * p2;
    o.t1 = kd1 * p0 * p2;
  }
  const double p01 = p0 * p1;
  o.t2 = kd2 * p01;
  o.R = (e2 >> 16) == 1 ? o.t2 * p2 : k * p01 * p2;
  return o;
}

// Special-order rate law (chemistry_kernels.cpp:316-325) and its Y derivative for order-list position `at`
// (rates_sensitivities_exact.cpp:177-261).
template <class SC>
__device__ __forceinline__ double special_orders(const DevMech &m, Blob b, int r, const SC &C, double rho, int at,
                                                 bool last_closure)
{
  const int o0 = b.i[m.i_ord_off + r], o1 = b.i[m.i_ord_off + r + 1];
  const double *invmw_d = b.d + m.d_invmw;
  double v = 1.;
  for (int j = o0; j < o1; ++j) {
    const int e = b.i[m.i_ord + j];
    const int s = e & 0xFFFF;
    const bool nz = (e >> 16) != 0;
    const double ord = b.d[m.d_ord + j];
    const double c = C[s];
    if (j - o0 == at) {
      if (last_closure)
        v *= ord * rho * invmw_d[s] * pow(fmax(c, 1.e-16), ord - 1.);
      else if (ord > 1)
        v *= ord * rho * invmw_d[s] * pow(fmax(c, 1.e-16), ord - 1.);
      else
        v *= ord * rho * invmw_d[s] / pow(fmax(c, 1.e-16), 1. - ord);
    } else if (nz) {
      v *= last_closure ? pow(c, ord) : pow(fmax(c, 0.), ord);
    }
  }
  return v;
}

// The fixed-point terms of a state: the logarithm of T (natural, and to base 2 in fixed point), 1/T.
__device__ __forceinline__ bool fixed_temperature(double T)
{
  return __double_as_longlong(T) > 0x4030000000000000ll && __double_as_longlong(T) < 0x40f0000000000000ll;
}
__device__ __forceinline__ double state_log(double T, const unsigned long long *tab, unsigned long long &l60)
{
  l60 = 0;
  if (!fixed_temperature(T)) return log(T);
  const Fix96 y = fix_log2(T, tab);
  l60 = ((unsigned long long)(unsigned)y.n << 60) | ((unsigned long long)y.f1 << 28) | (y.f0 >> 4);
  return fix96_ln(y);
}
__device__ __forceinline__ unsigned long long fixed_reciprocal(double invT)
{
  const unsigned long long bits = (unsigned long long)__double_as_longlong(invT);
  const int e = (int)(bits >> 52);  // 1007 to 1018 for T in range
  return ((bits & 0xfffffffffffffull) | 0x10000000000000ull) << ((e - 1007) & 15);
}

// log2 of an Arrhenius expression: w = (fraction of log2 A, b 2^58, (E/R) log2(e) 2^44) and the integer part of log2 A.
__device__ __forceinline__ Fix96 fixed_arrhenius(const double *w, int n, const StateCtx &s)
{
  Fix96 y = fix96(n, (unsigned long long)__double_as_longlong(w[0]));
  const long long bb = __double_as_longlong(w[1]), ee = __double_as_longlong(w[2]);
  if (bb) {
    const Fix96 p = fix_product<22>((unsigned long long)(bb < 0 ? -bb : bb), s.l60);  // 118 - 32 - 22 = 64
    y = bb < 0 ? y - p : y + p;
  }
  if (ee) {
    const Fix96 p = fix_product<16>((unsigned long long)(ee < 0 ? -ee : ee), s.u68);  // 112 - 32 - 16 = 64
    y = ee < 0 ? y + p : y - p;
  }
  return y;
}

// Forward rate constant of reaction r (chemistry_kernels.cpp:140-157) in FP64: states and reactions outside the
// fixed-point ranges.
static __device__ __noinline__ double forward_constant(const double *kc, const double *tab, double T, double logT, double invT,
                                                int kform)
{
  switch (kform) {
  case 0: return kc[0];
  case 1: return kc[0] * T;
  case 2: return kc[0] * (T * T);
  case 3: return kc[0] * invT;
  default: return kc[0] * fix_exp(fma(kc[1], logT, -(kc[2] * invT)), tab);
  }
}

// k e^x, with the power of two apart from the rest: e^x may lie outside the range of doubles where the product does not
static __device__ __noinline__ double times_exp(double k, double x, const unsigned long long *exp2tab)
{
  int N = x < 0. ? -(1 << 20) : 1 << 20;  // beyond 2^20: 0 or infinity times k
  unsigned long long f = 0;
  if (isnan(x)) return x;
  if (fabs(x) < 1048576.) fix_reduce(x, N, f);
  return scale_pow2(k * fix_to_double(fix_exp2(f, exp2tab), 0), N);
}

// k0 / kinf of falloff reaction f
__device__ __forceinline__ double falloff_ratio(const DevMech &m, const Blob &b, const StateCtx &s, int f)
{
  const int n = b.i[m.i_fixp + f];
  if (s.fixed && n != kFixNone)
    return fix96_exp2(fixed_arrhenius(b.d + m.d_fixp + 3 * f, n, s),
                      reinterpret_cast<const unsigned long long *>(b.d + m.d_exptab + 128));
  return forward_constant(b.d + m.d_kp + 3 * f, b.d + m.d_exptab, s.T, s.logT, s.invT, 4);
}

// F_cent of a Troe reaction and, with JAC, T dF_cent/dT. d_troe holds (a, -1/T3, -1/T1, T2).
template <bool JAC, bool PAIR>
__device__ __forceinline__ double troe_center(const DevMech &m, const Blob &b, const StateCtx &s, int f, int terms,
                                              double &Tdfc)
{
  const double *tr = b.d + m.d_troe + 4 * f;
  const double *tab = b.d + m.d_exptab;
  double fc = 0.;
  Tdfc = 0.;
  if constexpr (PAIR) {  // the three exponentials interleave where all arguments are in the fixed-point range
    const double x[3] = {s.T * tr[1], s.T * tr[2], -(s.invT * tr[3])};
    bool in = true;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      in = in && (!(terms >> k & 1) || (((unsigned)__double2hiint(x[k])) & 0x7fffffffu) < 0x40862000u);
    if (in) {
      double e[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        int N;
        unsigned long long f64;
        fix_reduce((terms >> k & 1) ? x[k] : 0., N, f64);
        e[k] = fix_to_double(fix_exp2(f64, reinterpret_cast<const unsigned long long *>(tab + 128)), N);
      }
      const double w[3] = {1. - tr[0], tr[0], 1.};
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (terms >> k & 1) {
          const double t = k == 2 ? e[k] : w[k] * e[k];
          fc += t;
          if (JAC) Tdfc = fma(k == 2 ? -x[k] : x[k], t, Tdfc);
        }
      return fc;
    }
  }
  if (terms & 1) {
    const double x = s.T * tr[1];
    const double e = (1. - tr[0]) * fix_exp(x, tab);
    fc += e;
    if (JAC) Tdfc = x * e;
  }
  if (terms & 2) {
    const double x = s.T * tr[2];
    const double e = tr[0] * fix_exp(x, tab);
    fc += e;
    if (JAC) Tdfc = fma(x, e, Tdfc);
  }
  if (terms & 4) {
    const double x = -(s.invT * tr[3]);
    const double e = fix_exp(x, tab);
    fc += e;
    if (JAC) Tdfc = fma(-x, e, Tdfc);
  }
  return fc;
}

// max(x, 1e-300), on the integer pipe
__device__ __forceinline__ double at_least_tiny(double x)
{
  return __double_as_longlong(x) < 0x01a56e1fc2f8f359ll ? 1.e-300 : x;
}

// Third-body concentration of reaction r: the default efficiency times the total plus the listed excesses.
template <bool PAIR, class SC>
__device__ __forceinline__ double third_body(const DevMech &m, const Blob &b, const StateCtx &s, int r, const SC &C)
{
  const int t0 = b.i[m.i_tb_off + r], t1 = b.i[m.i_tb_off + r + 1];
  double M = b.d[m.d_beff + r] * s.ct;
  if constexpr (PAIR) {
    for (int j = t0; j < t1; j += 4) {
      double e[4], c[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = j + k < t1;
        e[k] = in ? b.d[m.d_tbeff + j + k] : 0.;
        c[k] = in ? C[b.i[m.i_tb + j + k]] : 0.;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j + k < t1) M = fma(e[k], c[k], M);
    }
  } else {
    for (int j = t0; j < t1; ++j) M = fma(b.d[m.d_tbeff + j], C[b.i[m.i_tb + j]], M);
  }
  return M;
}

// Evaluate reaction r. Always writes its net rate q[r]; with JAC also
//   dqdrho = rho dq/drho, dqdT = T dq/dT, the sparse slots D_j = dq/dC_j (concentration C = rho Y / M), the dense
//   coefficients alpha, beta of dq/dY_k / rho = D_k / M_k + alpha u_k + beta.
// The kernels are bound by FP64 instructions, so the scaled forms were chosen for what they leave out: the factors 1/M,
// 1/rho and 1/T belong to a species or a state and are applied once there (1/M in the gather programs' coefficients),
// a reaction without a third body multiplies by no such factor, the products of a side are shared by its rate and
// derivatives (side3), and the product side carries its minus sign in the constant. About 45 FP64 instructions for
// a reversible 2+2 reaction with its derivatives (a third of them the exponential) where the form with every
// factor in place took 110.
// PAIR: rates of a wide group, whose few warps wait out the latency of one reaction at a time. The independent pieces of
// a falloff reaction (three exponentials, two logarithms, the third-body loads four at a time) are then interleaved:
// 4 % less for 300 integrated GRI reactors. Where several warps share a scheduler, or with the derivatives' registers, the
// same form was 1-2 % slower (right-hand sides and Jacobians of 4096 h2 states), so those keep one after another.
template <bool JAC, bool PAIR, class S>
__device__ __forceinline__ void eval_reaction(const DevMech &m, Blob b, const ScratchLayout &L, S scr,
                                              const StateCtx &s, int r)
{
  const int info = b.i[m.i_info + r];
  const int kind = (info >> RI_KIND_SHIFT) & 7;
  const bool rev = (info >> RI_REV_BIT) & 1;
  const bool has_ord = (info >> RI_ORD_BIT) & 1;
  const auto C = scr + L.C;
  const double *smallint = b.d + m.d_smallint;
  const double *kc = b.d + m.d_kf + 3 * r;
  const unsigned long long *exp2tab = reinterpret_cast<const unsigned long long *>(b.d + m.d_exptab + 128);
  const int kform = (info >> RI_KFORM_SHIFT) & 7;
  const int fixn = b.i[m.i_fixn + r];
  const bool fixed = s.fixed && fixn != kFixNone;
  Fix96 y;
  double kf;
  if (fixed) {
    y = fixed_arrhenius(b.d + m.d_fix + 3 * r, fixn, s);
    kf = kform == 0 ? kc[0] : fix96_exp2(y, exp2tab);
  } else {
    kf = forward_constant(kc, b.d + m.d_exptab, s.T, s.logT, s.invT, kform);
    y = fix96(0, 0);
  }
  const double Tdlogkf = fma(kc[2], s.invT, kc[1]);  // T d ln kf / dT
  // third-body / falloff factor (chemistry_kernels.cpp:158-314; rates_sensitivities_exact.cpp:826-1000); K = dCtbaf/dM
  double Ctbaf = 1., TdCdT = 0., K = 0., M = 0.;
  if (kind != 1) {
    M = third_body<PAIR>(m, b, s, r, C);
    if (kind == 2) {
      Ctbaf = M;
      K = 1.;
    } else {
      const int f = r - (m.nr - m.n_fall);
      const double *kp = b.d + m.d_kp + 3 * f;  // the ratio k0 / kinf as A, b, E/R
      const double kpf = falloff_ratio(m, b, s, f);
      const double pr = kpf * M;
      const double i1 = fix_reciprocal(1. + pr), hf = pr * i1;
      const double Tdlogk = fma(kp[2], s.invT, kp[1]);
      if (kind == 3) {
        Ctbaf = hf;
        if (JAC) {
          TdCdT = hf * i1 * Tdlogk;
          K = kpf * i1 * i1;
        }
      } else {
        double Tdfc;
        const double fc = troe_center<JAC, PAIR>(m, b, s, f, (info >> RI_TROE_SHIFT) & 7, Tdfc);
        constexpr double kLog10e = 0.43429448190325176;
        // Fc clamped at 1e-300 in the sensitivities (rates_sensitivities_exact.cpp:949-985), not in the rates
        // (chemistry_kernels.cpp:280-312): log10 F = log10 Fc / (1 + (a / bb)^2)
        const double prc = at_least_tiny(pr), fcc = JAC ? at_least_tiny(fc) : fc;
        double l10pr, lnfc;
        if (PAIR && fix_normal(prc) && fix_normal(fcc)) {  // the two logarithms interleave
          const double lnpr = fix96_ln(fix_log2(prc, exp2tab));
          lnfc = fix96_ln(fix_log2(fcc, exp2tab));
          l10pr = lnpr * kLog10e;
        } else {
          l10pr = fix_log(prc, exp2tab) * kLog10e;
          lnfc = fix_log(fcc, exp2tab);
        }
        const double l10fc = lnfc * kLog10e;
        const double a = l10pr - 0.67 * l10fc - 0.4;
        const double bb = 0.806 - 0.14 * l10pr - 1.1762 * l10fc;
        const double b2 = bb * bb;
        const double iq = fix_reciprocal(fma(a, a, b2));
        const double gt = b2 * iq;
        const double F = fix_exp(gt * lnfc, b.d + m.d_exptab);
        Ctbaf = F * hf;
        if (JAC) {
          const double dlfc = Tdfc * fix_reciprocal(fc);
          const double c1 = (-2. * kLog10e) * lnfc * (a * bb) * (iq * iq);
          const double p1 = fma(0.14, a, bb) * c1;
          const double TdlnF = fma(gt, dlfc, fma(p1, Tdlogk, -(c1 * (0.67 * bb - 1.1762 * a) * dlfc)));
          TdCdT = Ctbaf * fma(i1, Tdlogk, TdlnF);
          K = kpf * F * i1 * (p1 + i1);
        }
      }
    }
  }
  const bool orders = has_ord && !(JAC && s.option == 1);
  const int ro0 = b.i[m.i_reac_off + r], nre = b.i[m.i_reac_off + r + 1] - ro0;
  const int po0 = b.i[m.i_prod_off + r], npr = b.i[m.i_prod_off + r + 1] - po0;
  const int n0 = b.i[m.i_net_off + r], n1 = b.i[m.i_net_off + r + 1];
  const int *rl = b.i + m.i_reac + ro0;
  const int *pl = b.i + m.i_prod + po0;
  double Rf, nkr = 0., nRr = 0.;  // the reverse side carries its minus sign
  const int sums = b.i[m.i_sums + r];
  const int sum_nu = (int)(short)(sums & 0xFFFF);
  // lists of at most three entries (every reaction of common mechanisms) use the factored form
  const bool short_lists = !orders && (unsigned)(nre - 1) < 3u && (unsigned)(npr - 1) < 3u;
  Side3 fr, fp;
  fp.t0 = fp.t1 = fp.t2 = 0.;
  if (orders) {
    Rf = kf * special_orders(m, b, r, C, s.rho, -1, false);
  } else {
    if (short_lists) {
      fr = side3<JAC>(rl, nre, C, kf, smallint);
      Rf = fr.R;
    } else {
      Rf = kf * mass_action(rl, nre, C, -1);
    }
    // rates of a special-order reaction have no reverse part (chemistry_kernels.cpp:316-326)
    if (rev && !has_ord) {
      // kr = kf exp(sum_nu ln(p_ref/RT) - sum_i nu_i g_i/RT) (chemistry_kernels.cpp:327-341), as logarithms
      if (s.fixed) {
        if (sum_nu) {
          const Fix96 lp = fix96(m.log2_port_n, m.log2_port_f) - fix96((int)(s.l60 >> 60), s.l60 << 4);  // log2(p_ref/RT)
          for (int j = sum_nu < 0 ? -sum_nu : sum_nu; j > 0; --j) y = sum_nu > 0 ? y + lp : y - lp;
        }
        for (int j = n0; j < n1; ++j) {
          const int e = b.i[m.i_net + j];
          const int sp = e & 0xFFFF, nu = (e >> 16) - 128;
          const Fix96 g = fix96(__double2loint(scr[L.gk + sp]), (unsigned long long)__double_as_longlong(scr[L.gm + sp]));
          for (int q = nu < 0 ? -nu : nu; q > 0; --q) y = nu > 0 ? y + g : y - g;
        }
        if (fixed)
          nkr = -fix96_exp2(y, exp2tab);
        else  // 2^y may lie outside the range of doubles where its product with kf does not
          nkr = -scale_pow2(kf * fix_to_double(fix_exp2(((unsigned long long)y.f1 << 32) | y.f0, exp2tab), 0), y.n);
      } else {
        double x = sum_nu ? (double)sum_nu * log(s.port) : 0.;
        for (int j = n0; j < n1; ++j) {
          const int e = b.i[m.i_net + j];
          x += (double)((e >> 16) - 128) * scr[L.gm + (e & 0xFFFF)];
        }
        nkr = -times_exp(kf, x, exp2tab);
      }
      if (short_lists) {
        fp = side3<JAC>(pl, npr, C, nkr, smallint);
        nRr = fp.R;
      } else {
        nRr = nkr * mass_action(pl, npr, C, -1);
      }
    }
  }
  const double Rnet = Rf + nRr;
  const double q = kind == 1 ? Rnet : Rnet * Ctbaf;
  scr[L.q + r] = q;
  if (!JAC) return;

  const int snr = (sums >> 16) & 0xFF, snp = (sums >> 24) & 0xFF;
  double rdRdrho, TdRdT = Rnet * Tdlogkf;
  if (orders) {
    double sumo = 0.;
    const int o0 = b.i[m.i_ord_off + r], o1 = b.i[m.i_ord_off + r + 1];
    for (int j = o0; j < o1; ++j)
      if (b.i[m.i_ord + j] >> 16) sumo += b.d[m.d_ord + j];
    rdRdrho = Rf * sumo;
  } else {
    rdRdrho = snr == snp ? Rnet * small_int(smallint, snr)
                         : fma(nRr, small_int(smallint, snp), Rf * small_int(smallint, snr));
    if (rev && !has_ord) {
      double dKc = 0.;
      for (int j = n0; j < n1; ++j) {
        const int e = b.i[m.i_net + j];
        dKc = fma(small_int(smallint, (e >> 16) - 128), scr[L.dB + (e & 0xFFFF)], dKc);
      }
      TdRdT = fma(nRr, dKc, TdRdT);
    }
  }
  // d q / d Y_k / rho through the third-body concentration: Rnet K d M / d C_k
  double RK = 0.;
  if (kind != 1) {
    rdRdrho *= Ctbaf;
    TdRdT *= Ctbaf;
    if (s.option != 1) {
      RK = Rnet * K;
      rdRdrho = fma(RK, M, rdRdrho);  // rho dM/drho = M
      TdRdT = fma(Rnet, TdCdT, TdRdT);
    }
  }
  scr[L.dqdrho + r] = rdRdrho;
  scr[L.dqdT + r] = TdRdT;
  // sparse slots: D_j = d q / d C_k for the slot's species k
  const int ns = m.ns;
  const int s0 = b.i[m.i_slot_off + r], s1 = b.i[m.i_slot_off + r + 1];
  const int tb0 = b.i[m.i_tb_off + r];
  for (int j = s0; j < s1; ++j) {
    const int e = b.i[m.i_slot + j];
    const int rp = ((e >> 16) & 15) - 1, pp = ((e >> 20) & 15) - 1, tp = ((e >> 24) & 15) - 1;
    const int op = ((unsigned)e >> 28) - 1;
    double v = 0.;  // d (Rf - Rr) / d C_k
    if (orders) {
      if (op >= 0) {
        const int oe = b.i[m.i_ord + b.i[m.i_ord_off + r] + op];
        if (oe >> 16)
          v = kf * special_orders(m, b, r, C, s.rho, op, false) * s.invRho * b.d[m.d_mw + (e & 0xFFFF)];
      }
    } else if (short_lists) {
      if (rp >= 0) v = fr.t(rp);
      if (pp >= 0) v = rp >= 0 ? v + fp.t(pp) : fp.t(pp);
    } else {
      if (rp >= 0) v += kf * mass_action(rl, nre, C, rp);
      if (pp >= 0) v += nkr * mass_action(pl, npr, C, pp);
    }
    if (kind != 1) {
      v *= Ctbaf;
      if (tp >= 0) v = fma(RK, b.d[m.d_tbeff + tb0 + tp], v);
    }
    scr[L.D + j] = v;
  }
  const int di = b.i[m.i_dense + r];
  if (di >= 0) {
    // closure species ns-1 and third-body terms common to every Y column (all divided by rho)
    double closure = 0.;  // -d (Rf - Rr) / d C_{ns-1}
    if (orders) {
      const int o0 = b.i[m.i_ord_off + r], o1 = b.i[m.i_ord_off + r + 1];
      for (int j = o0; j < o1; ++j) {
        const int oe = b.i[m.i_ord + j];
        if ((oe & 0xFFFF) == ns - 1 && (oe >> 16))
          closure -= kf * special_orders(m, b, r, C, s.rho, j - o0, true) * s.invRho * b.d[m.d_mw + ns - 1];
      }
    } else {
      for (int j = 0; j < nre; ++j)
        if ((rl[j] & 0xFFFF) == ns - 1) closure -= short_lists ? fr.t(j) : kf * mass_action(rl, nre, C, j);
      if (rev && !has_ord)
        for (int j = 0; j < npr; ++j)
          if ((pl[j] & 0xFFFF) == ns - 1) closure -= short_lists ? fp.t(j) : nkr * mass_action(pl, npr, C, j);
    }
    double beta = closure;
    double alpha = 0.;
    if (kind != 1) {
      beta *= Ctbaf;
      if (s.option != 1) {
        const int t1 = b.i[m.i_tb_off + r + 1];
        for (int j = tb0; j < t1; ++j)
          if (b.i[m.i_tb + j] == ns - 1) beta -= RK * b.d[m.d_tbeff + j];
      }
      alpha = RK * b.d[m.d_beff + r];
    }
    beta *= b.d[m.d_invmw + ns - 1];
    scr[L.alpha + di] = alpha;
    scr[L.beta + di] = beta;
  }
}

// E_r = sum_i c_ir e_i of reaction r, for the temperature row: after the species gathers, in the place of q. The dense
// terms' share of the row's sums goes to Ea and Eb.
template <class S>
__device__ __forceinline__ void reaction_energy(const DevMech &m, const Blob &b, const ScratchLayout &L, S scr, int r,
                                                double &Ea, double &Eb)
{
  const int n0 = b.i[m.i_net_off + r], n1 = b.i[m.i_net_off + r + 1];
  double Er = 0.;
  for (int j = n0; j < n1; ++j) Er = fma(b.d[m.d_netc + j], scr[L.eh + (b.i[m.i_net + j] & 0xFFFF)], Er);
  scr[L.E + r] = Er;
  const int di = b.i[m.i_dense + r];
  if (di >= 0) {
    Ea = fma(Er, scr[L.alpha + di], Ea);
    Eb = fma(Er, scr[L.beta + di], Eb);
  }
}

// ------------------------------------------------------------------------------------------ gather programs
// Execute a gather program for one state: every lane runs prog.len items (see sf_mech.h). Scratch destinations are
// written to scratch, Jacobian ones passed to jw(row, col, value), their sums starting from scratch[qoff + row].
// Items are processed in batches of U (each lane's item count is padded to a multiple of GATHER_UNROLL): the
// operands of a whole batch are loaded before its FMAs, and the next batch's items while they run. This is sound
// because no program reads a scratch location that it writes (checked when the program is built), so no load
// can overtake a store it depends on.

// One lane per state reads its scratch from global memory and gains most from loads in flight; the lane groups
// (scratch in shared memory or L2) take half the batch, which keeps their larger kernels free of register spills.
__host__ __device__ constexpr int default_unroll(int G) { return G == 1 ? GATHER_UNROLL : GATHER_UNROLL / 2; }

template <int G, int U, class JW, class S>
__device__ __forceinline__ void run_items(const Group<G> &grp, const GatherItem *items, int len, S scr, int qoff, JW &jw)
{
  const int lane = grp.lane;
  static_assert(GATHER_UNROLL % U == 0, "batch must divide the program padding");
  const uint4 *it = reinterpret_cast<const uint4 *>(items) + lane;
  if (G <= 32) grp.sync();  // a wide group has its first items on their way while it waits for the scratch values
  uint4 x[U];
#pragma unroll
  for (int u = 0; u < U; ++u) x[u] = len > 0 ? __ldg(it + u * G) : make_uint4(0, 0, 0, IT_NOP);
  if (G > 32) grp.sync();
  double acc = 0.;
  for (int j = 0; j < len; j += U) {
    double a[U], bv[U], c0[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = __hiloint2double((int)x[u].y, (int)x[u].x);
      if (x[u].w & IT_PAIR) a[u] = scr[x[u].x];
      bv[u] = scr[x[u].z];
      c0[u] = 0.;
      if ((x[u].w & (IT_START | IT_JAC)) == (IT_START | IT_JAC)) c0[u] = scr[qoff + (x[u].w & IT_ROW_MASK)];
    }
    uint4 y[U];
    const bool more = j + U < len;
#pragma unroll
    for (int u = 0; u < U; ++u) y[u] = more ? __ldg(it + (j + U + u) * G) : make_uint4(0, 0, 0, IT_NOP);
    bool stop = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (x[u].w & IT_NOP) {
        stop = true;  // padding only follows a lane's last real item
      } else {
        acc = fma(a[u], bv[u], (x[u].w & IT_START) ? c0[u] : acc);
        if (x[u].w & IT_END) {
          if (x[u].w & IT_JAC)
            jw((int)(x[u].w & IT_ROW_MASK), (int)((x[u].w >> IT_COL_SHIFT) & IT_ROW_MASK), acc);
          else
            scr[x[u].w & IT_DST_MASK] = acc;
        }
      }
    }
    if (stop) break;
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = y[u];
  }
}

// A program and, where it has one, the second pass that adds the partial sums of its split entries; begins with a group
// barrier.
template <int G, int U = default_unroll(G), class JW, class S>
__device__ __forceinline__ void run_program(const DevProgram &prog, const Group<G> &grp, S scr, int qoff, JW &jw)
{
  run_items<G, U>(grp, prog.items, prog.len, scr, qoff, jw);
  if (prog.fix_len > 0) run_items<G, U>(grp, prog.fix_items, prog.fix_len, scr, qoff, jw);
}

struct NoJ {
  __device__ __forceinline__ void operator()(int, int, double) const {}
};

}  // namespace sfgb
