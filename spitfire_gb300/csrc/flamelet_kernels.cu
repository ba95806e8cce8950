// Flamelet kernels: the flamelet right-hand side (adiabatic or with heat loss) and its block-tridiagonal ("BTDDOD": block diagonal,
// diagonal off-diagonals) Jacobian for a batch of flamelets with different grids, and the block-Thomas algebra.
//
// Reference: src/spitfire/griffon/src/flamelet_kernels.cpp:31-90 (stencils, COO indices), :1039-1218
// (flamelet_rhs), :1220-1409 (flamelet_jacobian); src/btddod_matrix_kernels.cpp:19-465.
//
// Points of all flamelets are flattened: flamelet f owns interior points offsets_z[f] .. offsets_z[f+1]-1. One state
// group evaluates one point (isobaric chemistry via reactor_eval, then the mixture-fraction stencils). The
// block-Thomas factorization and solve are sequential in mixture fraction; they run from both ends of a flamelet
// toward its middle block, two CTAs per flamelet, parallel within each block.
#include "reactor_eval.cuh"
#include "sf_internal.h"
#include "eig_device.cuh"
#include "gj_device.cuh"

namespace sfgb {
namespace {

struct FlmParams {
  DevMech m;
  const void *blob;
  int *status;
  ScratchLayout L;
  Progs pg;
  int n_flamelets, n_points;
  const int *offz;        // device [nf+1]
  const long long *offv;  // device [nf+1]
  double pressure;
  const double *oxy, *fuel;  // [nf][ns]
  const double *cmajor, *csub, *csup, *mc, *nc, *chi;
  int eflux, vcp;
  const double *state;
  double *out_rhs;
  double *out_values;
  int scale_offset;
  int rates_option;
  double prefactor;
  const double *prefactors;  // device [nf] or null: each flamelet's own prefactor of scale_offset
  double *eflux_store;  // if set: the enthalpy-flux diagonal correction is stored here (per point) instead
  const int *active;    // device [nf] or null: flamelets with active[f] == 0 are skipped
  // nonadiabatic flamelets: convection / radiation temperature and coefficient per interior point (null: adiabatic)
  const double *Tconv, *hconv, *Trad, *hrad;
  int scaled_heat_loss;
  int groups_per_cta;
};

__device__ __forceinline__ int find_flamelet(const int *offz, int nf, int p)
{
  int lo = 0, hi = nf - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offz[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// cp of the mixture at a state [T, Y_0..Y_{ns-2}] (lanes over species, group reduction)
template <int G>
__device__ __forceinline__ double cp_of_state(const DevMech &m, const Blob &b, const Group<G> &grp, const double *st)
{
  const int ns = m.ns;
  const double T = st[0], logT = log(T), invT = 1. / T;
  double ys = 0., cp = 0.;
  for (int i = grp.lane; i < ns - 1; i += G) {
    const SpeciesThermo th = species_thermo(m, b, i, T, logT, invT, false);
    cp += st[1 + i] * th.cp;
    ys += st[1 + i];
  }
  grp.sum2(ys, cp, ns);
  const SpeciesThermo thn = species_thermo(m, b, ns - 1, T, logT, invT, false);
  return cp + (1. - ys) * thn.cp;
}

struct BlockWriter {
  double *blk;  // column-major ns x ns
  int ns;
  const double *cmaj;  // [ns] of this point
  int scale;
  double pref;
  __device__ __forceinline__ void operator()(int row, int col, double v) const
  {
    double x = v + (row == col ? cmaj[row] : 0.);
    if (scale) x = pref * x - (row == col ? 1. : 0.);
    blk[col * ns + row] = x;
  }
};

// Heat loss of a nonadiabatic flamelet point (flamelet_kernels.cpp:1121-1138, :1290-1320): the isobaric reactor's
// diathermal terms with unit surface-to-volume ratio and this point's convection (Tc, hc) and radiation (Tr, hr)
// parameters, q = hc (Tc - T) + hr sigma (Tr^4 - T^4) entering dT/dt as q / (rho cp). With use_scaled_heat_loss the
// coefficients are divided by (max T - Tc) and (max T^4 - Tr^4), max T over the flamelet's interior points (held
// constant in the Jacobian, as the reference does). The reference adds the Y-column terms in a loop that runs two
// columns past the end of its primitive Jacobian (flamelet_kernels.cpp:1316-1319); here they stop at the last Y
// column.
template <int G>
__device__ __forceinline__ void heat_loss_cfg(const FlmParams &p, const Group<G> &grp, int pt, int z0, int nzi,
                                              ReactorCfg &cfg)
{
  if (!p.Tconv) {
    cfg.heat = 0;
    return;
  }
  const double Tc = p.Tconv[pt], Tr = p.Trad[pt];
  double hc = p.hconv[pt], hr = p.hrad[pt];
  if (p.scaled_heat_loss) {
    double mx = -1.;
    for (int j = grp.lane; j < nzi; j += G) mx = fmax(mx, p.state[(size_t)(z0 + j) * p.m.ns]);
    mx = grp.max(mx);
    const double Tr4 = Tr * Tr * Tr * Tr;
    hc = hc / (mx - Tc);
    hr = hr / (mx * mx * mx * mx - Tr4);
  }
  cfg.heat = 2;
  cfg.Tc = Tc;
  cfg.hc = hc;
  cfg.Tr = Tr;
  cfg.eps = hr;
  cfg.SoV = 1.;
}

template <int G, bool JAC>
__global__ void __launch_bounds__(512, 1) flamelet_point_kernel(const FlmParams p)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint64_t bar;
  const DevMech &m = p.m;
  if (!stage_to_smem(smem, p.blob, m.blob_bytes, &bar, p.status)) return;
  const Blob b = blob_at(m, smem);
  const ScratchLayout &L = p.L;
  const int gid = threadIdx.x / G;
  // per group: Griffon scratch + ns doubles for the (unused) right-hand side of the Jacobian evaluation
  double *shared = reinterpret_cast<double *>(smem + m.blob_bytes) +
                   (size_t)gid * ((JAC ? L.total : L.total_rhs) + m.ns + 2 + Group<G>::kShared);
  double *scr = shared + Group<G>::kShared;
  const Group<G> grp(shared, gid);
  const int lane = grp.lane;
  const int ns = m.ns;
  ReactorCfg cfg{};
  cfg.configuration = 0;
  cfg.heat = 0;
  cfg.option = JAC ? p.rates_option : 0;
  NoJ noj;
  for (int pt = blockIdx.x * p.groups_per_cta + gid; pt < p.n_points; pt += gridDim.x * p.groups_per_cta) {
    const int f = find_flamelet(p.offz, p.n_flamelets, pt);
    const double pref = p.prefactors ? p.prefactors[f] : p.prefactor;
    if (p.active && !p.active[f]) continue;
    const int z0 = p.offz[f], nzi = p.offz[f + 1] - z0;
    const int iz = pt - z0;
    heat_loss_cfg<G>(p, grp, pt, z0, nzi, cfg);
    const double *st = p.state + (size_t)pt * ns;
    const double *oxy = p.oxy + (size_t)f * ns;
    const double *fuel = p.fuel + (size_t)f * ns;
    const double *sm1 = iz == 0 ? oxy : st - ns;
    const double *sp1 = iz == nzi - 1 ? fuel : st + ns;
    const double mcf = p.mc[pt], ncf = p.nc[pt], chi = p.chi[pt];
    if (!JAC) {
      double *out = p.out_rhs + (size_t)pt * ns;
      reactor_eval<G, false, default_unroll(G), false>(m, b, L, scr, grp, st, p.pressure, cfg, p.pg, out, noj);
      // enthalpy-flux and variable-cp terms of the temperature equation (flamelet_kernels.cpp:1141-1206)
      double cp = 0.;
      for (int i = lane; i < ns; i += G) cp += scr[L.y + i] * scr[L.cpv + i];
      cp = grp.sum(cp, ns);
      const double dTdZ = mcf * sm1[0] + ncf * sp1[0];
      double extra = 0.;
      if (p.eflux) {
        const double cpn = scr[L.cpv + ns - 1];
        double s = 0.;
        for (int j = lane; j < ns - 1; j += G) s += (scr[L.cpv + j] - cpn) * (mcf * sm1[1 + j] + ncf * sp1[1 + j]);
        s = grp.sum(s, ns);
        extra += 0.5 * chi / cp * dTdZ * s;
      }
      if (p.vcp) {
        const double cpm = cp_of_state<G>(m, b, grp, sm1);
        const double cpp = cp_of_state<G>(m, b, grp, sp1);
        extra += 0.5 * chi * (mcf * cpm + ncf * cpp) / cp * dTdZ;
      }
      grp.sync();
      // mixture-fraction diffusion (flamelet_kernels.cpp:1208-1217)
      const double *cma = p.cmajor + (size_t)pt * ns, *csb = p.csub + (size_t)pt * ns, *csp = p.csup + (size_t)pt * ns;
      for (int i = lane; i < ns; i += G) {
        double v = out[i] + (i == 0 ? extra : 0.);
        v += cma[i] * st[i] + csb[i] * sm1[i] + csp[i] * sp1[i];
        out[i] = v;
      }
      grp.sync();
    } else {
      // block of this point in the flamelet's BTDDOD value array
      double *vals = p.out_values + p.offv[f];
      double *blk = vals + (size_t)iz * ns * ns;
      BlockWriter bw{blk, ns, p.cmajor + (size_t)pt * ns, p.scale_offset, pref};
      double *rhs_tmp = scr + L.total;
      reactor_eval<G, true, default_unroll(G), false>(m, b, L, scr, grp, st, p.pressure, cfg, p.pg, rhs_tmp, bw);
      if (p.eflux) {
        // approximate diagonal correction of the enthalpy-flux term (flamelet_kernels.cpp:1350-1381)
        double cp = 0., cps = 0.;
        for (int i = lane; i < ns; i += G) {
          cp += scr[L.y + i] * scr[L.cpv + i];
          cps += scr[L.y + i] * scr[L.dcp + i];
        }
        grp.sum2(cp, cps, ns);
        const double cpm = cp_of_state<G>(m, b, grp, sm1);
        const double cpp = cp_of_state<G>(m, b, grp, sp1);
        const double dTdZ = mcf * sm1[0] + ncf * sp1[0];
        const double dcpdZ = mcf * cpm + ncf * cpp;
        const double f1 = 0.5 * chi / cp * dTdZ * dcpdZ;
        grp.sync();
        if (lane == 0) {
          const double corr = (p.scale_offset ? pref : 1.) * f1 / cp * cps;
          if (p.eflux_store)
            p.eflux_store[(size_t)pt * ns] = corr;
          else
            blk[0] -= corr;
        }
      } else if (p.eflux_store && lane == 0) {
        p.eflux_store[(size_t)pt * ns] = 0.;
      }
      // off-diagonals: sub row iz (iz >= 1) and super row iz (iz <= nzi-2) (flamelet_kernels.cpp:1383-1394)
      const long long sub_off = (long long)nzi * ns * ns, sup_off = sub_off + (long long)(nzi - 1) * ns;
      const double sc = p.scale_offset ? pref : 1.;
      for (int q = lane; q < ns; q += G) {
        if (iz >= 1) vals[sub_off + (long long)(iz - 1) * ns + q] = sc * p.csub[(size_t)pt * ns + q];
        if (iz <= nzi - 2) vals[sup_off + (long long)iz * ns + q] = sc * p.csup[(size_t)pt * ns + q];
      }
      grp.sync();
    }
  }
}

// Pseudo-time-step eigenvalue bound (flamelet_kernels.cpp:1329-1341): for each point, max(max Re(lambda) - d, 0)
// of the transformed isobaric chemistry block (the block before the diffusion diagonal and the enthalpy-flux
// correction are added), d the flamelet's diffusion term, written to all ns entries of the point; then the held-back
// enthalpy-flux correction is applied to the block. A warp, two or eight per point, the block in shared memory. The result is
// exactly 0 whenever every eigenvalue lies left of d; the scaled-Gershgorin (M-matrix) test proves that for a large
// share of the points at a small fraction of the QR iteration's cost, which then runs only for the rest.
inline __host__ __device__ size_t expeig_doubles(int G, int ns)
{
  return (size_t)ns * ns + 2 * ns + wide_group_doubles(G) + eig_work_doubles(G);
}

template <int G>
__global__ void __launch_bounds__(256) flamelet_expeig_kernel(int n_points, int nf, int ns, const int *offz, const long long *offv,
                                       double *values, const double *cmajor, double diffterm,
                                       const double *diffterm_f, const int *active, double *expeig, int *status,
                                       int *next_point)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int w = threadIdx.x / G;
  double *shared = reinterpret_cast<double *>(smem) + (size_t)w * expeig_doubles(G, ns);
  double *A = shared + Group<G>::kShared;
  const Group<G> g(shared, w);
  const int lane = g.lane;
  double *work = A + ns * ns;
  // points are taken dynamically (whether a point needs the QR iteration is known only once it is examined)
  for (;;) {
    int pt = 0;
    if (lane == 0) pt = atomicAdd(next_point, 1);
    if constexpr (G > 32) {
      if (lane == 0) g.scalars[0] = (double)pt;
      g.sync();
      pt = (int)g.scalars[0];
      g.sync();
    } else {
      pt = __shfl_sync(0xffffffffu, pt, 0);
    }
    if (pt >= n_points) break;
    const int f = find_flamelet(offz, nf, pt);
    if (active && !active[f]) continue;
    const int iz = pt - offz[f];
    const double d = diffterm_f ? diffterm_f[f] : diffterm;
    double *blk = values + offv[f] + (size_t)iz * ns * ns;
    auto load = [&]() {
      for (int e = lane; e < ns * ns; e += G) {
        const int col = e / ns, row = e - col * ns;
        A[e] = blk[e] - (row == col ? cmajor[(size_t)pt * ns + row] : 0.);
      }
      g.sync();
    };
    load();
    double mx = d;
    bool ok = true;
    if (!group_hmatrix_below<G>(g, A, ns, d, work)) {
      g.sync();
      load();
      ok = group_max_real_eig<G>(g, A, ns, work, &mx, d);
    }
    if (!ok && lane == 0) report_error(status, DEVERR_WAIT_TIMEOUT);
    const double corr = expeig[(size_t)pt * ns];
    g.sync();
    const double e = fmax(mx - d, 0.);
    for (int q = lane; q < ns; q += G) expeig[(size_t)pt * ns + q] = e;
    if (lane == 0) blk[0] -= corr;
    g.sync();
  }
}

// ------------------------------------------------------------------------------- block-Thomas (BTDDOD) algebra
// The reference factorization (btddod_matrix_kernels.cpp:19-80) eliminates downward from the first block:
// LU(D_0); for i >= 1: L_i = diag(sub_{i-1}) D_{i-1}^-1 (the reference solves D_{i-1} X = I with dgetrs),
// D_i <- D_i - L_i diag(sup_{i-1}), LU(D_i). Its chain of nzi dependent block steps is the critical path of a
// flamelet, so this factorization is twisted: with m = nzi/2, one CTA eliminates blocks 0..m-1 downward exactly as
// above, a second CTA eliminates blocks nzi-1..m+1 upward (T_{nzi-1} = D_{nzi-1}; U_i = diag(sup_{i-1}) T_i^-1;
// T_{i-1} = D_{i-1} - U_i diag(sub_{i-1})), and block m receives both: M = D_m - L_m diag(sup_{m-1})
// - U_{m+1} diag(sub_m). Same flops, half the chain, and as stable for these block-diagonally dominant matrices.
// Every eliminated block is inverted once (the multiplier blocks need the inverse anyway), by Gauss-Jordan
// elimination with one CTA barrier per column, and the inverse is what the solve applies.
// Storage: values block i holds the inverse of the eliminated block i; l_values block i holds L_i for
// 1 <= i <= m and U_i for m < i < nzi (block 0 unused).
constexpr int kFactorThreads = 384;  // 12 warps: warp 0 runs the pivot look-ahead, the others update the block

// Shared-memory bytes of the factorization kernels: two row-major blocks with an odd leading dimension, the
// elimination's multipliers, two index arrays.
inline size_t factor_smem_bytes(int ns)
{
  return (size_t)2 * ns * (ns | 1) * 8 + (size_t)2 * ns * 8 + (size_t)2 * ns * 4 + 16;
}

struct FactorShared {
  double *buf0, *buf1, *ws;
  int *piv, *pinv;
  int ld;
  __device__ FactorShared(unsigned char *smem, int ns) : ld(ns | 1)
  {
    buf0 = reinterpret_cast<double *>(smem);
    buf1 = buf0 + (size_t)ns * ld;
    ws = buf1 + (size_t)ns * ld;
    piv = reinterpret_cast<int *>(ws + 2 * ns);
    pinv = piv + ns;
  }
  __device__ __forceinline__ double *invert(double *S, double *D, int ns)
  {
    return gj_inverse<true>(S, D, ns, ld, piv, pinv, ws, threadIdx.x, kFactorThreads, [] { __syncthreads(); });
  }
};

constexpr int kAhead = 8;  // elements of the next block each thread holds: all of a block of up to 55 x 55

// One CTA per (flamelet, half): even CTAs eliminate blocks 0..m-1 downward, odd CTAs blocks nzi-1..m+1 upward.
// Each half ends with the multiplier block that feeds block m (L_m, or U_{m+1}); btddod_middle_kernel then forms
// and inverts block m.
__global__ void __launch_bounds__(kFactorThreads) btddod_factor_kernel(int nf, int ns, const int *offz,
                                                                       const long long *offv, double *values,
                                                                       double *lvals, int *perms, const int *active)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x >> 1;
  const bool down = (blockIdx.x & 1) == 0;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0, m = nb / 2;
  const int len = down ? m : nb - 1 - m;
  if (len <= 0) return;
  const int bs2 = ns * ns;
  double *vals = values + offv[f];
  double *lv = lvals + (size_t)z0 * bs2;
  int *pv = perms + (size_t)z0 * ns;
  const double *sub = vals + (size_t)nb * bs2;
  const double *sup = sub + (size_t)(nb - 1) * ns;
  FactorShared sh(smem, ns);
  double *cur = sh.buf0, *other = sh.buf1;  // cur: the block to invert (row-major)
  const int tid = threadIdx.x, nt = blockDim.x;
  {
    const double *D0 = vals + (size_t)(down ? 0 : nb - 1) * bs2;
    for (int e = tid; e < bs2; e += nt) {
      const int c = e / ns, r = e - c * ns;
      cur[r * sh.ld + c] = D0[e];
    }
  }
  __syncthreads();
  for (int t = 0; t < len; ++t) {
    const int i = down ? t : nb - 1 - t;
    // the next block of the chain is loaded while this one is eliminated
    const bool more = t + 1 < len;
    const double *Dn = vals + (size_t)(down ? i + 1 : i - 1) * bs2;
    double dn[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int e = tid + u * kFactorThreads;
      dn[u] = more && e < bs2 ? Dn[e] : 0.;
    }
    double *Z = sh.invert(cur, other, ns);
    double *nxt = Z == cur ? other : cur;  // the buffer the elimination no longer needs
    // multiplier: downward L_{i+1} = diag(sub_i) D_i^-1 at block i+1; upward U_i = diag(sup_{i-1}) T_i^-1 at block
    // i. Then the next block of the chain: D_{i+1} - L_{i+1} diag(sup_i), or D_{i-1} - U_i diag(sub_{i-1}).
    const double *rs = down ? sub + (size_t)i * ns : sup + (size_t)(i - 1) * ns;
    const double *cs = down ? sup + (size_t)i * ns : sub + (size_t)(i - 1) * ns;
    double *Di = vals + (size_t)i * bs2;
    double *Lm = lv + (size_t)(down ? i + 1 : i) * bs2;
    auto element = [&](int e, double next) {  // e: column-major index of the global arrays
      const int c = e / ns, r = e - c * ns;
      const double inv = Z[sh.piv[r] * sh.ld + sh.pinv[c]];
      Di[e] = inv;
      const double l = inv * rs[r];
      Lm[e] = l;
      if (more) nxt[r * sh.ld + c] = next + (-cs[c]) * l;
    };
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (tid + u * kFactorThreads < bs2) element(tid + u * kFactorThreads, dn[u]);
    for (int e = tid + kAhead * kFactorThreads; e < bs2; e += nt) element(e, more ? Dn[e] : 0.);
    for (int k = tid; k < ns; k += nt) pv[(size_t)i * ns + k] = sh.piv[k];
    __syncthreads();
    cur = nxt;
    other = Z;
  }
}

// Block m of each flamelet: M = D_m - L_m diag(sup_{m-1}) - U_{m+1} diag(sub_m) (terms present when m >= 1 and
// m + 1 < nzi), then its inverse. One CTA per flamelet, after btddod_factor_kernel.
__global__ void __launch_bounds__(kFactorThreads) btddod_middle_kernel(int nf, int ns, const int *offz,
                                                                       const long long *offv, double *values,
                                                                       const double *lvals, int *perms,
                                                                       const int *active)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0, m = nb / 2;
  const int bs2 = ns * ns;
  double *vals = values + offv[f];
  const double *lv = lvals + (size_t)z0 * bs2;
  const double *sub = vals + (size_t)nb * bs2;
  const double *sup = sub + (size_t)(nb - 1) * ns;
  FactorShared sh(smem, ns);
  double *Dm = vals + (size_t)m * bs2;
  const double *La = m >= 1 ? lv + (size_t)m * bs2 : nullptr;
  const double *Ub = m + 1 < nb ? lv + (size_t)(m + 1) * bs2 : nullptr;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < bs2; e += nt) {
    const int c = e / ns, r = e - c * ns;
    double v = Dm[e];
    if (La) v = v + (-sup[(size_t)(m - 1) * ns + c]) * La[e];
    if (Ub) v = v + (-sub[(size_t)m * ns + c]) * Ub[e];
    sh.buf0[r * sh.ld + c] = v;
  }
  __syncthreads();
  const double *Z = sh.invert(sh.buf0, sh.buf1, ns);
  for (int e = tid; e < bs2; e += nt) {
    const int c = e / ns, r = e - c * ns;
    Dm[e] = Z[sh.piv[r] * sh.ld + sh.pinv[c]];
  }
  int *pv = perms + (size_t)(z0 + m) * ns;
  for (int k = tid; k < ns; k += nt) pv[k] = sh.piv[k];
}

// Asynchronous 8-byte copies global -> shared by `threads` threads, t among them (cp.async, completion tracked by commit
// groups; no mbarrier wait is involved).
__device__ __forceinline__ void async_copy_doubles(double *dst, const double *src, int n, int t, int threads)
{
  for (int e = t; e < n; e += threads)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst + e)), "l"(src + e) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void async_wait_all_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A group of whole warps walks a chain of dependent block steps, each a matrix-vector product with a column-major ns x ns
// block staged in shared memory (the next one is copied while the current one is used, where two fit). A product's rows are
// dealt to the threads of whole warps and its columns cut into parts over the other warps: one warp alone takes two FP64
// instructions per column at 64 cycles each, 6.8 us a step for ns = 53; twelve take 9 per step.
constexpr int kSweepThreads = 384;
constexpr int kSmallSolveBlock = 32;    // blocks up to this size: both halves of a flamelet in one CTA,
constexpr int kSmallSolveThreads = 128; // on this many threads each

struct Sweep {
  double *b0, *b1, *part, *vec;
  int ns, bs2, rows, parts, p, r, c0, c1, t, threads, id;
  bool dbl;
  __device__ Sweep(unsigned char *smem, int ns_, bool dbl_, int t_, int threads_, int barrier)
      : ns(ns_), bs2(ns_ * ns_), t(t_), threads(threads_), id(barrier), dbl(dbl_)
  {
    b0 = reinterpret_cast<double *>(smem);
    b1 = dbl ? b0 + bs2 : b0;
    part = b1 + bs2;
    vec = part + threads;
    rows = (ns + 31) & ~31;
    parts = threads / rows;
    p = t / rows;
    r = t - p * rows;
    c0 = ns * p / parts;
    c1 = ns * (p + 1) / parts;
  }
  __host__ __device__ static size_t bytes(int ns, bool dbl, int threads = kSweepThreads)
  {
    return ((size_t)(dbl ? 2 : 1) * ns * ns + threads + ns) * 8;
  }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
  __device__ __forceinline__ double *slot(int k) const { return (k & 1) ? b1 : b0; }
  template <class Src>
  __device__ __forceinline__ void prime(int k, Src src) const
  {
    if (dbl) async_copy_doubles(slot(k), src(k), bs2, t, threads);
  }
  // The block of step k (steps k, k + step, ..., last are fetched in this order); ends with the barrier that also makes
  // the writes to vec visible.
  template <class Src>
  __device__ __forceinline__ const double *fetch(int k, int last, int step, Src src) const
  {
    if (dbl) {
      if (k != last) {
        async_copy_doubles(slot(k + step), src(k + step), bs2, t, threads);
        async_wait_all_but_one();
      } else {
        async_wait_all();
      }
    } else {
      async_copy_doubles(b0, src(k), bs2, t, threads);
      async_wait_all();
    }
    sync();
    return dbl ? slot(k) : b0;
  }
  // Row r of B vec, complete in the threads below ns.
  __device__ __forceinline__ double product(const double *B) const
  {
    double s = 0.;
    if (p < parts && r < ns)
      for (int c = c0; c < c1; ++c) s = fma(B[r + c * ns], vec[c], s);
    if (p > 0 && p < parts) part[t] = s;
    sync();
    if (t < ns)
      for (int q = 1; q < parts; ++q) s += part[q * rows + t];
    return s;
  }
};

// Solve with the twisted factors (the reference's btddod_matrix_kernels.cpp:82-119 sweeps, run from both ends), one half over
// blocks 0..m-1, the other over blocks nzi-1..m+1, m = nzi/2, in three parts:
//   1. sweeps toward block m: y_0 = b_0, y_i = b_i - L_i y_{i-1};   z_{nzi-1} = b_{nzi-1}, z_i = b_i - U_{i+1} z_{i+1}
//   2. the middle:            x_m = M^-1 (b_m - L_m y_{m-1} - U_{m+1} z_{m+1})
//   3. back substitution:     x_i = D_i^-1 (y_i - sup_i o x_{i+1}) for i < m;  x_i = T_i^-1 (z_i - sub_{i-1} o x_{i-1})
// y and z are parked in x until the back substitution overwrites them. The parts are launches of their own with a CTA per
// half; blocks of up to kSmallSolveBlock have steps so short that the two further launches cost more than the wider halves
// gain, so there one CTA takes the halves and all parts. 11 species: one flamelet of 30 blocks 50 us in three launches, 29 in
// one (40 with the two warps per flamelet before), eight of up to 95 blocks 122 and 80 (114), 64 of up to 126 156 and 107
// (155); 30 species, eight of up to 95 blocks: 118 in one (245).
__device__ __forceinline__ void solve_forward(const Sweep &sw, bool down, int nb, int m, const double *lv, const double *b,
                                              double *xs)
{
  const int len = down ? m : nb - 1 - m, ns = sw.ns, t = sw.t;
  if (len == 0) return;
  auto at = [&](int k) { return (size_t)(down ? k : nb - 1 - k) * ns; };
  auto src = [&](int k) { return lv + (size_t)(down ? k : nb - k) * sw.bs2; };
  if (len > 1) sw.prime(1, src);
  if (t < ns) xs[at(0) + t] = sw.vec[t] = b[at(0) + t];
  for (int k = 1; k < len; ++k) {
    const double *B = sw.fetch(k, len - 1, 1, src);
    const double s = sw.product(B);
    if (t < ns) xs[at(k) + t] = sw.vec[t] = b[at(k) + t] - s;
  }
}

__device__ __forceinline__ void solve_meet(const Sweep &sw, int nb, int m, const double *lv, const double *Dm, const double *b,
                                           double *xs)
{
  const int ns = sw.ns, t = sw.t;
  double v = t < ns ? b[(size_t)m * ns + t] : 0.;
  for (int side = 0; side < 2; ++side) {  // L_m y_{m-1}, then U_{m+1} z_{m+1}
    const int i = side == 0 ? m - 1 : m + 1;
    if (i < 0 || i >= nb) continue;
    if (t < ns) sw.vec[t] = xs[(size_t)i * ns + t];
    const double *B = sw.fetch(0, 0, 1, [&](int) { return lv + (size_t)(m + side) * sw.bs2; });
    v -= sw.product(B);
    sw.sync();
  }
  if (t < ns) sw.vec[t] = v;
  const double *B = sw.fetch(0, 0, 1, [&](int) { return Dm; });
  const double s = sw.product(B);
  if (t < ns) xs[(size_t)m * ns + t] = s;
}

__device__ __forceinline__ void solve_back(const Sweep &sw, bool down, int nb, int m, const double *vals, double *xs)
{
  const int len = down ? m : nb - 1 - m, ns = sw.ns, t = sw.t;
  if (len == 0) return;
  const double *sub = vals + (size_t)nb * sw.bs2;
  const double *sup = sub + (size_t)(nb - 1) * ns;
  auto blk = [&](int k) { return down ? k : nb - 1 - k; };
  auto src = [&](int k) { return vals + (size_t)blk(k) * sw.bs2; };
  sw.prime(len - 1, src);
  double xn = t < ns ? xs[(size_t)m * ns + t] : 0.;
  for (int k = len - 1; k >= 0; --k) {
    const int i = blk(k);
    const double *cpl = down ? sup + (size_t)i * ns : sub + (size_t)(i - 1) * ns;
    if (t < ns) sw.vec[t] = xs[(size_t)i * ns + t] - cpl[t] * xn;
    const double *B = sw.fetch(k, 0, -1, src);
    xn = sw.product(B);
    if (t < ns) xs[(size_t)i * ns + t] = xn;
  }
}

__global__ void __launch_bounds__(kSweepThreads) btddod_forward_kernel(int nf, int ns, const int *offz,
                                                                       const double *lvals, const double *rhs,
                                                                       double *x, const int *active, int double_buffer)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x >> 1;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0;
  const Sweep sw(smem, ns, double_buffer != 0, threadIdx.x, kSweepThreads, 0);
  solve_forward(sw, (blockIdx.x & 1) == 0, nb, nb / 2, lvals + (size_t)z0 * sw.bs2, rhs + (size_t)z0 * ns,
                x + (size_t)z0 * ns);
}

__global__ void __launch_bounds__(kSweepThreads) btddod_meet_kernel(int nf, int ns, const int *offz,
                                                                    const long long *offv, const double *values,
                                                                    const double *lvals, const double *rhs, double *x,
                                                                    const int *active)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0, m = nb / 2;
  const Sweep sw(smem, ns, false, threadIdx.x, kSweepThreads, 0);
  solve_meet(sw, nb, m, lvals + (size_t)z0 * sw.bs2, values + offv[f] + (size_t)m * sw.bs2, rhs + (size_t)z0 * ns,
             x + (size_t)z0 * ns);
}

__global__ void __launch_bounds__(kSweepThreads) btddod_back_kernel(int nf, int ns, const int *offz,
                                                                    const long long *offv, const double *values,
                                                                    double *x, const int *active, int double_buffer)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x >> 1;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0;
  const Sweep sw(smem, ns, double_buffer != 0, threadIdx.x, kSweepThreads, 0);
  solve_back(sw, (blockIdx.x & 1) == 0, nb, nb / 2, values + offv[f], x + (size_t)z0 * ns);
}

__global__ void __launch_bounds__(2 * kSmallSolveThreads) btddod_small_solve_kernel(int nf, int ns, const int *offz,
                                                                                    const long long *offv,
                                                                                    const double *values,
                                                                                    const double *lvals,
                                                                                    const double *rhs, double *x,
                                                                                    const int *active)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x;
  if (f >= nf || (active && !active[f])) return;
  const int half = threadIdx.x / kSmallSolveThreads, t = threadIdx.x - half * kSmallSolveThreads;
  const int z0 = offz[f], nb = offz[f + 1] - z0, m = nb / 2;
  unsigned char *own = smem + half * Sweep::bytes(ns, true, kSmallSolveThreads);
  const Sweep sw(own, ns, true, t, kSmallSolveThreads, 1 + half);
  const double *lv = lvals + (size_t)z0 * sw.bs2, *vals = values + offv[f], *b = rhs + (size_t)z0 * ns;
  double *xs = x + (size_t)z0 * ns;
  solve_forward(sw, half == 0, nb, m, lv, b, xs);
  __syncthreads();
  if (half == 0)
    solve_meet(Sweep(own, ns, false, t, kSmallSolveThreads, 1), nb, m, lv, vals + (size_t)m * sw.bs2, b, xs);
  __syncthreads();
  solve_back(sw, half == 0, nb, m, vals, xs);
}

// Block-triangular solves with the inverses of a block-diagonal factorization (btddod_matrix_kernels.cpp:386-428):
//   lower  x_0 = F_0 b_0,               x_i = F_i (b_i - sub_{i-1} o x_{i-1})
//   upper  x_{nb-1} = F_{nb-1} b_{nb-1}, x_i = F_i (b_i - sup_i o x_{i+1})
// One CTA per flamelet, of four warps for small blocks, whose few columns cost less than a barrier of twelve (one chain of 30
// blocks of 11 rows 27 us against 37, of 30 rows 37 against 45; one warp had taken 36 and 68); F_i are column-major
// inverses, [points][ns*ns].
__global__ void __launch_bounds__(kSweepThreads) btddod_triangle_solve_kernel(int nf, int ns, const int *offz,
                                                                              const long long *offv,
                                                                              const double *inverses,
                                                                              const double *values, const double *rhs,
                                                                              double *x, int upper, const int *active,
                                                                              int double_buffer)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int f = blockIdx.x;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0;
  const Sweep sw(smem, ns, double_buffer != 0, threadIdx.x, blockDim.x, 0);
  const double *sub = values + offv[f] + (size_t)nb * sw.bs2;
  const double *sup = sub + (size_t)(nb - 1) * ns;
  const double *b = rhs + (size_t)z0 * ns;
  double *xs = x + (size_t)z0 * ns;
  const int tid = threadIdx.x;
  auto blk = [&](int t) { return upper ? nb - 1 - t : t; };
  auto src = [&](int t) { return inverses + (size_t)(z0 + blk(t)) * sw.bs2; };
  sw.prime(0, src);
  double xp = 0.;
  for (int t = 0; t < nb; ++t) {
    const int i = blk(t);
    if (tid < ns) {
      double v = b[(size_t)i * ns + tid];
      if (t > 0) v -= (upper ? sup[(size_t)i * ns + tid] : sub[(size_t)(i - 1) * ns + tid]) * xp;
      sw.vec[tid] = v;
    }
    const double *F = sw.fetch(t, nb - 1, 1, src);
    xp = sw.product(F);
    if (tid < ns) xs[(size_t)i * ns + tid] = xp;
  }
}

// Inverse of every ns x ns column-major block of a list (btddod_matrix_kernels.cpp:364-373 factors each block of a
// block-diagonal matrix): one CTA per block, Gauss-Jordan with partial pivoting as in the block-Thomas
// factorization. pivots receives each block's pivot order.
__global__ void __launch_bounds__(kFactorThreads) blockdiag_inverse_kernel(int n_blocks, int ns, const double *blocks,
                                                                           double *out_inv, int *pivots)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int blkid = blockIdx.x;
  if (blkid >= n_blocks) return;
  const int bs2 = ns * ns;
  FactorShared sh(smem, ns);
  const double *A = blocks + (size_t)blkid * bs2;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < bs2; e += nt) {
    const int c = e / ns, r = e - c * ns;
    sh.buf0[r * sh.ld + c] = A[e];
  }
  __syncthreads();
  const double *Z = sh.invert(sh.buf0, sh.buf1, ns);
  double *O = out_inv + (size_t)blkid * bs2;
  for (int e = tid; e < bs2; e += nt) {
    const int c = e / ns, r = e - c * ns;
    O[e] = Z[sh.piv[r] * sh.ld + sh.pinv[c]];
  }
  for (int k = tid; k < ns; k += nt) pivots[(size_t)blkid * ns + k] = sh.piv[k];
}

// y_i = B_i x_i for every block of a list (btddod_matrix_kernels.cpp:167-177, and :375-384 with the inverses of a
// block-diagonal factorization): one thread per row.
__global__ void blockdiag_matvec_kernel(int n_blocks, int ns, const double *blocks, const double *x, double *y)
{
  const long long total = (long long)n_blocks * ns;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long bi = t / ns;
    const int r = (int)(t - bi * ns);
    const double *B = blocks + (size_t)bi * ns * ns;
    const double *xs = x + (size_t)bi * ns;
    double v = 0.;
    for (int c = 0; c < ns; ++c) v += B[r + c * ns] * xs[c];
    y[t] = v;
  }
}

// A <- matrix_scale*A + diag_scale*B over the BTDDOD values, B a block diagonal [points][ns*ns]
// (btddod_matrix_kernels.cpp:430-446): grid (chunks, flamelets), one value per thread per chunk step.
__global__ void btddod_scale_block_diag_kernel(int nf, int ns, const int *offz, const long long *offv, double *values,
                                               double ms, const double *bdiag, double ds, const int *active)
{
  const int f = blockIdx.y;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0;
  const long long bs2 = (long long)ns * ns;
  const long long ne = (long long)ns * (nb * ns + 2 * (nb - 1));
  double *vals = values + offv[f];
  const double *bd = bdiag + (size_t)z0 * bs2;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    double v = __dmul_rn(vals[e], ms);
    if (e < nb * bs2) v = __dadd_rn(v, __dmul_rn(bd[e], ds));
    vals[e] = v;
  }
}

// y = A x (btddod_matrix_kernels.cpp:121-160): one thread per row of every point of every flamelet.
__global__ void btddod_matvec_kernel(int n_points, int nf, int ns, const int *offz, const long long *offv,
                                     const double *values, const double *x, double *y, const int *active)
{
  const long long total = (long long)n_points * ns;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int pt = (int)(t / ns), r = (int)(t - (long long)pt * ns);
    const int f = find_flamelet(offz, nf, pt);
    if (active && !active[f]) continue;
    const int z0 = offz[f], nb = offz[f + 1] - z0, iz = pt - z0;
    const double *vals = values + offv[f];
    const double *D = vals + (size_t)iz * ns * ns;
    const double *xs = x + (size_t)z0 * ns;
    double v = 0.;
    for (int c = 0; c < ns; ++c) v += D[r + c * ns] * xs[(size_t)iz * ns + c];
    const double *sub = vals + (size_t)nb * ns * ns;
    const double *sup = sub + (size_t)(nb - 1) * ns;
    if (iz >= 1) v += sub[(size_t)(iz - 1) * ns + r] * xs[(size_t)(iz - 1) * ns + r];
    if (iz <= nb - 2) v += sup[(size_t)iz * ns + r] * xs[(size_t)(iz + 1) * ns + r];
    y[t] = v;
  }
}

// A <- matrix_scale*A + diag_scale*diag(d) (btddod_matrix_kernels.cpp:448-465): grid (chunks, flamelets), one
// value per thread per chunk step, the diagonal entries of the blocks getting the added term.
__global__ void btddod_scale_diag_kernel(int nf, int ns, const int *offz, const long long *offv, double *values,
                                         double ms, const double *diag, double ds, const int *active)
{
  const int f = blockIdx.y;
  if (f >= nf || (active && !active[f])) return;
  const int z0 = offz[f], nb = offz[f + 1] - z0;
  const long long bs2 = (long long)ns * ns;
  const long long ne = (long long)ns * (nb * ns + 2 * (nb - 1));
  double *vals = values + offv[f];
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    double v = __dmul_rn(vals[e], ms);
    if (e < nb * bs2) {
      const long long iz = e / bs2, rem = e - iz * bs2;
      if (rem % (ns + 1) == 0) v = __dadd_rn(v, __dmul_rn(ds, diag[(size_t)(z0 + iz) * ns + rem / (ns + 1)]));
    }
    vals[e] = v;
  }
}

int launch_points(HostMech &hm, FlmParams &p, bool jac, cudaStream_t st)
{
  int dev, smem_max, nsm;
  CUDA_THROW(cudaGetDevice(&dev));
  CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  CUDA_THROW(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const size_t scr_doubles = (size_t)(jac ? hm.sl.total : hm.sl.total_rhs) + hm.dm.ns + 2;
  const int G = fitting_group(hm.dm, default_group(hm.dm, jac, p.n_points, nsm, false), scr_doubles, smem_max);
  const auto &progs = hm.programs_for(G);
  p.m = hm.dm;
  p.blob = hm.d_blob;
  p.status = hm.d_status;
  p.L = hm.sl;
  p.pg.w = progs.progs[0];
  p.pg.full = progs.progs[1];
  p.pg.j = progs.progs[2];
  const int shared = wide_group_doubles(G);
  const size_t per = (scr_doubles + shared) * 8;
  const size_t avail = (size_t)smem_max - hm.dm.blob_bytes - 64;
  int groups = (int)std::min<size_t>(avail / per, 512 / G);
  if (groups < 1) throw sf_error(SF_ERR_UNSUPPORTED, "mechanism too large for the flamelet kernels");
  groups = balanced_groups(groups, p.n_points, nsm);
  p.groups_per_cta = groups;
  const size_t smem = hm.dm.blob_bytes + per * groups;
  void (*k)(const FlmParams);
  switch (G) {
  case 8: k = jac ? flamelet_point_kernel<8, true> : flamelet_point_kernel<8, false>; break;
  case 16: k = jac ? flamelet_point_kernel<16, true> : flamelet_point_kernel<16, false>; break;
  case 32: k = jac ? flamelet_point_kernel<32, true> : flamelet_point_kernel<32, false>; break;
  case 64: k = jac ? flamelet_point_kernel<64, true> : flamelet_point_kernel<64, false>; break;
  case 128: k = jac ? flamelet_point_kernel<128, true> : flamelet_point_kernel<128, false>; break;
  default: k = jac ? flamelet_point_kernel<256, true> : flamelet_point_kernel<256, false>; break;
  }
  ensure_dynamic_smem((const void *)k, smem);
  const int bps = std::max(1, (int)((size_t)smem_max / smem));
  const int grid = (int)std::max<long long>(1, std::min<long long>(((long long)p.n_points + groups - 1) / groups,
                                                                   (long long)nsm * bps));
  k<<<grid, groups * G, smem, st>>>(p);
  CUDA_THROW(cudaGetLastError());
  return SF_OK;
}

void fill(FlmParams &p, const sf_flamelet_batch *fb)
{
  if (!fb || fb->n_flamelets < 1 || !fb->offsets_z || !fb->offsets_v || !fb->offsets_z_host || !fb->oxy_state ||
      !fb->fuel_state || !fb->cmajor || !fb->csub || !fb->csup || !fb->mcoeff || !fb->ncoeff || !fb->chi)
    throw sf_error(SF_ERR_INVALID_ARGUMENT, "bad flamelet batch");
  p.n_flamelets = fb->n_flamelets;
  p.n_points = fb->offsets_z_host[fb->n_flamelets];
  for (int f = 0; f < fb->n_flamelets; ++f)
    if (fb->offsets_z_host[f + 1] - fb->offsets_z_host[f] < 2)
      throw sf_error(SF_ERR_INVALID_ARGUMENT, "every flamelet needs at least two interior points");
  p.offz = fb->offsets_z;
  p.offv = fb->offsets_v;
  p.pressure = fb->pressure;
  p.oxy = fb->oxy_state;
  p.fuel = fb->fuel_state;
  p.cmajor = fb->cmajor;
  p.csub = fb->csub;
  p.csup = fb->csup;
  p.mc = fb->mcoeff;
  p.nc = fb->ncoeff;
  p.chi = fb->chi;
  if (fb->T_convection || fb->h_convection || fb->T_radiation || fb->h_radiation) {
    if (!fb->T_convection || !fb->h_convection || !fb->T_radiation || !fb->h_radiation)
      throw sf_error(SF_ERR_INVALID_ARGUMENT, "nonadiabatic flamelets need all four heat-loss arrays");
    p.Tconv = fb->T_convection;
    p.hconv = fb->h_convection;
    p.Trad = fb->T_radiation;
    p.hrad = fb->h_radiation;
    p.scaled_heat_loss = fb->use_scaled_heat_loss ? 1 : 0;
  }
  p.eflux = fb->include_enthalpy_flux;
  p.vcp = fb->include_variable_cp;
  p.active = fb->active;
  p.prefactors = fb->prefactor;
}

template <class F>
int guarded(F f)
{
  try {
    return f();
  } catch (sf_error &e) {
    set_error(e.what());
    return e.code;
  }
}

int check_launch()
{
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(cudaGetErrorString(e));
    return SF_ERR_CUDA;
  }
  return SF_OK;
}

// Two staged blocks where they fit, else one
bool sweep_double_buffer(int ns, int smem_max)
{
  if (Sweep::bytes(ns, false) > (size_t)smem_max)
    throw sf_error(SF_ERR_UNSUPPORTED, "block size too large for the shared-memory block-Thomas solve");
  return Sweep::bytes(ns, true) <= (size_t)smem_max;
}

int launch_solve(int nf, int ns, const int *offz, const long long *offv, const double *values,
                 const double *l_values, const double *rhs, double *out_x, const int *active, cudaStream_t st)
{
  int dev, smem_max;
  CUDA_THROW(cudaGetDevice(&dev));
  CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if (ns <= kSmallSolveBlock) {
    const size_t smem = 2 * Sweep::bytes(ns, true, kSmallSolveThreads);
    ensure_dynamic_smem((const void *)btddod_small_solve_kernel, smem);
    btddod_small_solve_kernel<<<nf, 2 * kSmallSolveThreads, smem, st>>>(nf, ns, offz, offv, values, l_values, rhs, out_x,
                                                                        active);
    return check_launch();
  }
  const bool dbl = sweep_double_buffer(ns, smem_max);
  const size_t smem = Sweep::bytes(ns, dbl), smem1 = Sweep::bytes(ns, false);
  ensure_dynamic_smem((const void *)btddod_forward_kernel, smem);
  ensure_dynamic_smem((const void *)btddod_meet_kernel, smem1);
  ensure_dynamic_smem((const void *)btddod_back_kernel, smem);
  btddod_forward_kernel<<<2 * nf, kSweepThreads, smem, st>>>(nf, ns, offz, l_values, rhs, out_x, active, dbl);
  CUDA_THROW(cudaGetLastError());
  btddod_meet_kernel<<<nf, kSweepThreads, smem1, st>>>(nf, ns, offz, offv, values, l_values, rhs, out_x, active);
  CUDA_THROW(cudaGetLastError());
  btddod_back_kernel<<<2 * nf, kSweepThreads, smem, st>>>(nf, ns, offz, offv, values, out_x, active, dbl);
  return check_launch();
}

int launch_triangle(int nf, int ns, const int *offz, const long long *offv, const double *inverses,
                    const double *values, const double *rhs, double *out_x, int upper, const int *active,
                    cudaStream_t st)
{
  int dev, smem_max;
  CUDA_THROW(cudaGetDevice(&dev));
  CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const bool dbl = sweep_double_buffer(ns, smem_max);
  const size_t smem = Sweep::bytes(ns, dbl);
  ensure_dynamic_smem((const void *)btddod_triangle_solve_kernel, smem);
  const int threads = ns <= kSmallSolveBlock ? kSmallSolveThreads : kSweepThreads;
  btddod_triangle_solve_kernel<<<nf, threads, smem, st>>>(nf, ns, offz, offv, inverses, values, rhs, out_x, upper, active,
                                                          dbl);
  return check_launch();
}

}  // namespace
}  // namespace sfgb

using namespace sfgb;

extern "C" {

int sf_btddod_blockdiag_factor_batch(int n_blocks, int ns, const double *blocks, double *out_inverses,
                                     int *out_pivots, void *stream)
{
  if (n_blocks < 0 || ns < 1 || ns > 128 || (n_blocks > 0 && (!blocks || !out_inverses || !out_pivots))) {
    set_error("sf_btddod_blockdiag_factor_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  if (n_blocks == 0) return SF_OK;
  const size_t smem = factor_smem_bytes(ns);
  return guarded([&] {
    int dev, smem_max;
    CUDA_THROW(cudaGetDevice(&dev));
    CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (smem > (size_t)smem_max)
      throw sf_error(SF_ERR_UNSUPPORTED, "block size too large for the shared-memory block inverse");
    ensure_dynamic_smem((const void *)blockdiag_inverse_kernel, smem);
    blockdiag_inverse_kernel<<<n_blocks, kFactorThreads, smem, (cudaStream_t)stream>>>(n_blocks, ns, blocks,
                                                                                        out_inverses, out_pivots);
    return check_launch();
  });
}

int sf_btddod_blockdiag_matvec_batch(int n_blocks, int ns, const double *blocks, const double *x, double *out_y,
                                     void *stream)
{
  if (n_blocks < 0 || ns < 1 || (n_blocks > 0 && (!blocks || !x || !out_y))) {
    set_error("sf_btddod_blockdiag_matvec_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  if (n_blocks == 0) return SF_OK;
  const long long rows = (long long)n_blocks * ns;
  const int grid = (int)std::max<long long>(1, std::min<long long>((rows + 255) / 256, 152LL * 16));
  blockdiag_matvec_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(n_blocks, ns, blocks, x, out_y);
  return check_launch();
}

int sf_btddod_triangle_solve_batch(int nf, int ns, const int *offz, const long long *offv, const int *offz_host,
                                   const double *inverses, const double *values, const double *rhs, double *out_x,
                                   int upper, const int *active, void *stream)
{
  if (nf < 1 || ns < 1 || ns > 128 || !offz || !offv || !inverses || !values || !rhs || !out_x) {
    set_error("sf_btddod_triangle_solve_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  (void)offz_host;
  cudaStream_t st = (cudaStream_t)stream;
  const int up = upper ? 1 : 0;
  return guarded([&] {
    return launch_triangle(nf, ns, offz, offv, inverses, values, rhs, out_x, up, active, st);
  });
}

int sf_btddod_scale_and_add_block_diagonal_batch(int nf, int ns, const int *offz, const long long *offv,
                                                 const int *offz_host, double *values, double ms,
                                                 const double *block_diag, double ds, const int *active,
                                                 void *stream)
{
  if (nf < 1 || ns < 1 || nf > 65535 || !offz || !offv || !offz_host || !values || !block_diag) {
    set_error("sf_btddod_scale_and_add_block_diagonal_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  long long max_ne = 0;
  for (int f = 0; f < nf; ++f) {
    const long long nb = offz_host[f + 1] - offz_host[f];
    max_ne = std::max(max_ne, (long long)ns * (nb * ns + 2 * (nb - 1)));
  }
  const int chunks = (int)std::max<long long>(1, std::min<long long>((max_ne + 1023) / 1024, 1024));
  btddod_scale_block_diag_kernel<<<dim3(chunks, nf), 256, 0, (cudaStream_t)stream>>>(nf, ns, offz, offv, values, ms,
                                                                                     block_diag, ds, active);
  return check_launch();
}

int sf_flamelet_stencils(const sf_mech *mech, const double *dz, int nzi, const double *chi, const double *invLe,
                         double *cmaj, double *csub, double *csup, double *mc, double *nc)
{
  if (!mech || !dz || !chi || !invLe || !cmaj || !csub || !csup || !mc || !nc || nzi < 1) {
    set_error("sf_flamelet_stencils: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  const int ns = mech->m.dm.ns;
  for (int i = 0; i < nzi; ++i) {  // flamelet_kernels.cpp:31-48
    const double dzt = dz[i] + dz[i + 1];
    for (int l = 0; l < ns; ++l) {
      cmaj[i * ns + l] = -chi[1 + i] / (dz[i] * dz[i + 1]) * invLe[l];
      csub[i * ns + l] = chi[1 + i] / (dzt * dz[i]) * invLe[l];
      csup[i * ns + l] = chi[1 + i] / (dzt * dz[i + 1]) * invLe[l];
    }
    nc[i] = 1 / (dz[i] + dz[i + 1]);
    mc[i] = -nc[i];
  }
  return SF_OK;
}

int sf_flamelet_jac_indices(const sf_mech *mech, int nzi, int *rows, int *cols)
{
  if (!mech || !rows || !cols || nzi < 1) {
    set_error("sf_flamelet_jac_indices: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  const int ns = mech->m.dm.ns;
  int idx = 0;  // flamelet_kernels.cpp:50-90
  for (int iz = 0; iz < nzi; ++iz)
    for (int iq = 0; iq < ns; ++iq)
      for (int jq = 0; jq < ns; ++jq) {
        rows[idx] = iz * ns + jq;
        cols[idx] = iz * ns + iq;
        ++idx;
      }
  for (int iz = 1; iz < nzi; ++iz)
    for (int iq = 0; iq < ns; ++iq) {
      rows[idx] = iz * ns + iq;
      cols[idx] = iz * ns + iq - ns;
      ++idx;
    }
  for (int iz = 0; iz < nzi - 1; ++iz)
    for (int iq = 0; iq < ns; ++iq) {
      rows[idx] = iz * ns + iq;
      cols[idx] = iz * ns + iq + ns;
      ++idx;
    }
  return SF_OK;
}

int sf_flamelet_rhs_batch(const sf_mech *mech, const sf_flamelet_batch *fb, const double *state, double *out_rhs,
                          void *stream)
{
  return guarded([&] {
    if (!mech || !state || !out_rhs) throw sf_error(SF_ERR_INVALID_ARGUMENT, "bad argument");
    FlmParams p{};
    fill(p, fb);
    p.state = state;
    p.out_rhs = out_rhs;
    return launch_points(const_cast<HostMech &>(mech->m), p, false, (cudaStream_t)stream);
  });
}

size_t sf_flamelet_jac_workspace_size(const sf_mech *mech, int eigenvalues)
{
  return mech && eigenvalues ? 256 : 0;
}

int sf_flamelet_jac_batch(const sf_mech *mech, const sf_flamelet_batch *fb, const double *state, int rates_option,
                          int scale_and_offset, double prefactor, double diffterm, double *out_expeig,
                          double *out_values, void *workspace, size_t workspace_bytes, void *stream)
{
  return guarded([&] {
    if (!mech || !state || !out_values) throw sf_error(SF_ERR_INVALID_ARGUMENT, "bad argument");
    if (out_expeig && (!workspace || workspace_bytes < sf_flamelet_jac_workspace_size(mech, 1)))
      throw sf_error(SF_ERR_WORKSPACE, "eigenvalue bounds need the workspace sf_flamelet_jac_workspace_size reports");
    if (rates_option < 0 || rates_option > 2)
      throw sf_error(SF_ERR_INVALID_ARGUMENT, "rates option must be 0, 1 or 2");
    if (out_expeig && scale_and_offset)
      throw sf_error(SF_ERR_INVALID_ARGUMENT, "eigenvalue bounds need scale_and_offset = 0 (as flamelet.py calls it)");
    FlmParams p{};
    fill(p, fb);
    p.state = state;
    p.out_values = out_values;
    p.scale_offset = scale_and_offset;
    p.rates_option = rates_option;
    p.prefactor = prefactor;
    p.eflux_store = out_expeig;
    HostMech &hm = const_cast<HostMech &>(mech->m);
    cudaStream_t st = (cudaStream_t)stream;
    launch_points(hm, p, true, st);
    if (out_expeig) {
      const int ns = hm.dm.ns;
      int dev, smem_max, nsm;
      CUDA_THROW(cudaGetDevice(&dev));
      CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
      CUDA_THROW(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      // One point per SM: eight warps work on it (all four schedulers for the reduction to Hessenberg form); up to two
      // points per SM two warps each: every point has the FP64 unit of an SM, or half of it, to itself. With eight points
      // per block, 120 points had filled 15 SMs and taken 2.7 ms.
      int G = p.n_points <= nsm ? 256 : (p.n_points <= 2 * nsm ? 64 : 32);
      while (G > 32 && expeig_doubles(G, ns) * 8 > (size_t)smem_max) G = G == 256 ? 64 : 32;  // the largest blocks
      const size_t per = expeig_doubles(G, ns) * 8;
      int groups = (int)std::min<size_t>(G == 256 ? 1 : (G == 64 ? 2 : 8), (size_t)smem_max / per);
      if (groups < 1) throw sf_error(SF_ERR_UNSUPPORTED, "block too large for the eigenvalue kernel");
      groups = (int)std::max<long long>(1, std::min<long long>(groups, ((long long)p.n_points + nsm - 1) / nsm));
      const int threads = groups * G;
      auto kern = G == 256 ? flamelet_expeig_kernel<256> : (G == 64 ? flamelet_expeig_kernel<64> : flamelet_expeig_kernel<32>);
      ensure_dynamic_smem((const void *)kern, per * groups);
      int per_sm = 0;
      CUDA_THROW(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, per * groups));
      const int grid = (int)std::max<long long>(1, std::min<long long>((long long)nsm * std::max(1, per_sm),
                                                                       ((long long)p.n_points + groups - 1) / groups));
      // the points are handed out by an atomic counter in the caller's workspace, zeroed on the stream first
      int *counter = static_cast<int *>(workspace);
      CUDA_THROW(cudaMemsetAsync(counter, 0, sizeof(int), st));
      kern<<<grid, threads, per * groups, st>>>(p.n_points, p.n_flamelets, ns, p.offz, p.offv, out_values, p.cmajor,
                                                diffterm, fb->diffterm, fb->active, out_expeig, hm.d_status, counter);
      CUDA_THROW(cudaGetLastError());
    }
    return SF_OK;
  });
}

int sf_btddod_factor_batch(int nf, int ns, const int *offz, const long long *offv, const int *offz_host,
                           double *values, double *l_values, int *pivots, const int *active, void *stream)
{
  if (nf < 1 || ns < 1 || ns > 128 || !offz || !offv || !values || !l_values || !pivots) {
    set_error("sf_btddod_factor_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  (void)offz_host;
  const size_t smem = factor_smem_bytes(ns);
  return guarded([&] {
    int dev, smem_max;
    CUDA_THROW(cudaGetDevice(&dev));
    CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (smem > (size_t)smem_max)
      throw sf_error(SF_ERR_UNSUPPORTED, "block size too large for the shared-memory block-Thomas factorization");
    if ((long long)nf * 2 > 0x7fffffffLL) throw sf_error(SF_ERR_INVALID_ARGUMENT, "too many flamelets");
    int nsm;
    CUDA_THROW(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    // Each CTA is bound by its SM's FP64 unit. When every CTA can have an SM of its own, ask for more than half an
    // SM's shared memory so that no two CTAs share one (the block scheduler may otherwise pair them).
    const size_t smem_launch = 2LL * nf <= nsm ? std::max(smem, (size_t)smem_max / 2 + 1024) : smem;
    ensure_dynamic_smem((const void *)btddod_factor_kernel, smem_launch);
    ensure_dynamic_smem((const void *)btddod_middle_kernel, smem);
    cudaStream_t st = (cudaStream_t)stream;
    btddod_factor_kernel<<<2 * nf, kFactorThreads, smem_launch, st>>>(nf, ns, offz, offv, values, l_values, pivots,
                                                                      active);
    CUDA_THROW(cudaGetLastError());
    btddod_middle_kernel<<<nf, kFactorThreads, smem, st>>>(nf, ns, offz, offv, values, l_values, pivots, active);
    return check_launch();
  });
}

int sf_btddod_solve_batch(int nf, int ns, const int *offz, const long long *offv, const int *offz_host,
                          const double *values, const double *l_values, const int *pivots, const double *rhs,
                          double *out_x, const int *active, void *stream)
{
  if (nf < 1 || ns < 1 || ns > 128 || !offz || !offv || !values || !l_values || !pivots || !rhs || !out_x) {
    set_error("sf_btddod_solve_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  (void)offz_host;
  cudaStream_t st = (cudaStream_t)stream;
  return guarded([&] {
    if ((long long)nf * 2 > 0x7fffffffLL) throw sf_error(SF_ERR_INVALID_ARGUMENT, "too many flamelets");
    return launch_solve(nf, ns, offz, offv, values, l_values, rhs, out_x, active, st);
  });
}

int sf_btddod_matvec_batch(int nf, int ns, const int *offz, const long long *offv, const int *offz_host,
                           const double *values, const double *x, double *out_y, const int *active, void *stream)
{
  if (nf < 1 || ns < 1 || !offz || !offv || !offz_host || !values || !x || !out_y) {
    set_error("sf_btddod_matvec_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  const int npts = offz_host[nf];
  const long long rows = (long long)npts * ns;
  const int grid = (int)std::max<long long>(1, std::min<long long>((rows + 255) / 256, 152LL * 16));
  btddod_matvec_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(npts, nf, ns, offz, offv, values, x, out_y, active);
  return check_launch();
}

int sf_btddod_scale_and_add_diagonal_batch(int nf, int ns, const int *offz, const long long *offv,
                                           const int *offz_host, double *values, double ms, const double *diag,
                                           double ds, const int *active, void *stream)
{
  if (nf < 1 || ns < 1 || nf > 65535 || !offz || !offv || !offz_host || !values || !diag) {
    set_error("sf_btddod_scale_and_add_diagonal_batch: bad argument");
    return SF_ERR_INVALID_ARGUMENT;
  }
  long long max_ne = 0;
  for (int f = 0; f < nf; ++f) {
    const long long nb = offz_host[f + 1] - offz_host[f];
    max_ne = std::max(max_ne, (long long)ns * (nb * ns + 2 * (nb - 1)));
  }
  const int chunks = (int)std::max<long long>(1, std::min<long long>((max_ne + 1023) / 1024, 1024));
  btddod_scale_diag_kernel<<<dim3(chunks, nf), 256, 0, (cudaStream_t)stream>>>(nf, ns, offz, offv, values, ms, diag,
                                                                               ds, active);
  return check_launch();
}

}  // extern "C"
