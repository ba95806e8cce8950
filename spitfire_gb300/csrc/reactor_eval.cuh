// Per-state evaluation of the reactor right-hand side and analytical Jacobian by one state group, shared by the
// batched Jacobian kernel (chem_kernels.cu) and the persistent integrator (integrate_kernels.cu).
//
// Phases (group-synchronous):
//   P0  load the state; mixture molecular weight and density              (reduction over species)
//   P1  concentrations and species thermodynamics                         (lanes over species)
//   P2  reaction rates q_r and, for Jacobians, their derivatives           (lanes over reactions)
//   P3  species gathers w_i (and S_rho_i, S_T_i, P_i, Q_i)                 (gather program)
//   P4  right-hand side, rho/T columns, dense-term coefficients            (lanes over species)
//   P5  Y block of the Jacobian and T-row sums                             (gather program)
//   P6  T row of the Jacobian                                              (lanes over columns)
// Reference: isochoric_reactor_kernels.cpp:18-333, isobaric_reactor_kernels.cpp:19-343.
#pragma once
#include "chem_device.cuh"

namespace sfgb {

struct ReactorCfg {
  int configuration;  // 0 isobaric (q = [T, Y]), 1 isochoric (q = [rho, T, Y])
  int heat;           // 0 adiabatic, 1 isothermal, 2 diathermal
  int option;         // rates-sensitivity option
  double Tc, Tr, hc, eps, SoV;
  int open;           // mass exchange with a feed of temperature Tin, mass fractions yin[ns] (device), density
  double tau, rho_in, Tin;  // rho_in (isochoric), over the mixing time tau
  const double *yin;
};

struct Progs {
  DevProgram w, full, j;
};

struct SpeciesSums {
  double cpmix, cpsens;
};

// P1: concentrations and thermodynamics of every species; y must already be in scratch.
template <int G, bool JAC, class S>
__device__ __forceinline__ SpeciesSums prep_species(const DevMech &m, const Blob &b, const ScratchLayout &L,
                                                    S scr, const Group<G> &grp, const StateCtx &s,
                                                    bool isochoric, bool want_eh)
{
  const int ns = m.ns;
  double cpmix = 0., cpsens = 0.;
  // A wide group's first half takes the Gibbs factors and its second half the heat capacities and enthalpies: the
  // two parts need about the same number of FP64 instructions and one warp can issue only one every 64 cycles.
  constexpr int H = G > 32 ? G / 2 : G;
  const bool gibbs = G <= 32 || grp.lane < H, caloric = G <= 32 || grp.lane >= H;
  for (int i = grp.lane & (H - 1); i < ns; i += H) {
    const double yi = scr[L.y + i];
    const double invmw = b.d[m.d_invmw + i];
    const SpeciesThermo th = species_thermo(m, b, i, s.T, s.logT, s.invT, JAC);
    if (gibbs) {
      scr[L.C + i] = yi * s.rho * invmw;
      store_gibbs_factor(scr, L, i, th.g * (s.invT * m.invRu), s.fixed);
    }
    if (caloric) {
      if (want_eh) {
        scr[L.eh + i] = isochoric ? th.h - m.Ru * s.T * invmw : th.h;
        scr[L.cpv + i] = isochoric ? th.cp - m.Ru * invmw : th.cp;
        cpmix += yi * th.cp;
      } else {
        scr[L.eh + i] = 0.;
      }
      if (JAC) {
        scr[L.dB + i] = th.TdB;
        scr[L.dcp + i] = th.dcp;
        cpsens += yi * th.dcp;
      }
    }
  }
  SpeciesSums r{cpmix, cpsens};
  const int first = G <= 32 ? 0 : H, count = min(ns, H);
  if (JAC) {
    grp.sum2(r.cpmix, r.cpsens, count, first);
  } else {
    r.cpmix = grp.sum(r.cpmix, count, first);
  }
  if (G <= 32) grp.sync();  // a wide group's reduction has a barrier after the stores above
  return r;
}

// Scalars of a state: three reciprocals in one division sequence, everything else products. In a wide group the first
// warp forms them and the second one the logarithm, for all.
template <int G>
__device__ __forceinline__ StateCtx state_ctx(const DevMech &m, const Blob &b, const Group<G> &grp, double T,
                                              double rho, double sim, double pres, bool isochoric, int option)
{
  const unsigned long long *exp2tab = reinterpret_cast<const unsigned long long *>(b.d + m.d_exptab + 128);
  StateCtx s;
  s.T = T;
  s.option = option;
  auto scalars = [&](const auto &g) {
    double ix;  // 1 / rho isochoric, 1 / p isobaric
    g.recip3(T, sim, isochoric ? rho : pres, s.invT, s.mmw, ix);
    if (isochoric) {
      s.rho = rho;
      s.invRho = ix;
    } else {
      s.rho = pres * s.mmw * (s.invT * m.invRu);
      s.invRho = T * m.Ru * (sim * ix);
    }
    s.ct = s.rho * sim;
    s.port = m.pref * s.invT * m.invRu;
    s.u68 = fixed_reciprocal(s.invT);
  };
  s.fixed = m.fixed_rates && fixed_temperature(T);
  if constexpr (G <= 32) {
    s.logT = state_log(T, exp2tab, s.l60);
    scalars(grp);
  } else {
    double *sh = grp.scalars;
    if (grp.warp == 0) {
      scalars(Group<32>());
      if (grp.lane == 0) {
        sh[0] = s.invT;
        sh[1] = s.mmw;
        sh[2] = s.rho;
        sh[3] = s.invRho;
        sh[4] = s.ct;
        sh[5] = s.port;
        sh[6] = __longlong_as_double((long long)s.u68);
      }
    } else if (grp.warp == 1) {
      s.logT = state_log(T, exp2tab, s.l60);
      if (grp.lane == 32) {
        sh[7] = s.logT;
        sh[11] = __longlong_as_double((long long)s.l60);
      }
    }
    grp.sync();
    s.invT = sh[0];
    s.mmw = sh[1];
    s.rho = sh[2];
    s.invRho = sh[3];
    s.ct = sh[4];
    s.port = sh[5];
    s.u68 = (unsigned long long)__double_as_longlong(sh[6]);
    s.logT = sh[7];
    s.l60 = (unsigned long long)__double_as_longlong(sh[11]);
  }
  return s;
}

// The reactions of a group's lanes. In a wide group the last reactions in device order, the falloff ones, cost several
// times the others: the first warps take those in the first pass, and the last warps start the second.
template <int G, class F>
__device__ __forceinline__ void for_reactions(const Group<G> &grp, int nr, F f)
{
  if constexpr (G <= 32) {
    for (int r = grp.lane; r < nr; r += G) f(r);
  } else {
    for (int p = 0; p * G < nr; ++p) {
      const int r = nr - 1 - p * G - ((p & 1) ? G - 1 - grp.lane : grp.lane);
      if (r >= 0) f(r);
    }
  }
}

// P2 + P3: reaction rates (and derivatives) and the species gathers. energy: also the reactions' E (after the gathers,
// in the place of their rates) and (EA, EB), the T-row sums of the dense terms.
template <int G, bool JAC, int U = default_unroll(G), class S>
__device__ __forceinline__ double2 reactions_and_gathers(const DevMech &m, const Blob &b, const ScratchLayout &L,
                                                         S scr, const Group<G> &grp, const StateCtx &s,
                                                         const Progs &pg, bool energy)
{
  for_reactions<G>(grp, m.nr, [&](int r) { eval_reaction<JAC, (G > 32 && !JAC)>(m, b, L, scr, s, r); });
  NoJ noj;
  run_program<G, U>(JAC ? pg.full : pg.w, grp, scr, L.Q, noj);
  grp.sync();
  double EA = 0., EB = 0.;
  if (JAC && energy) {
    for_reactions<G>(grp, m.nr, [&](int r) { reaction_energy(m, b, L, scr, r, EA, EB); });
    grp.sum2(EA, EB);
  }
  return make_double2(EA, EB);
}

// Reactor right-hand side (and, with JAC, the analytical Jacobian) of the state qs (neq values, any memory space).
// rhs receives neq values; jset(row, col, value) receives every Jacobian entry exactly once.
// U: gather batch (loads in flight per lane); smaller batches use fewer registers. OPEN = false compiles the feed
// terms of open reactors out (c.open is then ignored).
template <int G, bool JAC, int U = default_unroll(G), bool OPEN = true, class JSet, class S>
__device__ void reactor_eval(const DevMech &m, const Blob &b, const ScratchLayout &L, S scr,
                             const Group<G> &grp, const double *qs, double pres, const ReactorCfg &c,
                             const Progs &pg, double *rhs, JSet &jset)
{
  const int ns = m.ns, lane = grp.lane;
  const bool isochoric = c.configuration == 1;
  const bool open_ = OPEN && c.open;
  const int neq = isochoric ? ns + 1 : ns;
  // ---------------- P0
  double T, rho = 0.;
  if (isochoric) {
    rho = qs[0];
    T = qs[1];
  } else {
    T = qs[0];
  }
  // the last mass fraction is 1 - sum y (extract_y, combustion_kernels.h:526-535), so 1 / mmw = sum y_i / M_i =
  // 1 / M_last + sum y_i u_i
  double sy = 0., sim = 0.;
  for (int i = lane; i < ns - 1; i += G) {
    const double yi = qs[(isochoric ? 2 : 1) + i];
    scr[L.y + i] = yi;
    sy += yi;
    sim = fma(yi, b.d[m.d_u + i], sim);
  }
  grp.sum2(sy, sim, ns - 1);
  if (lane == 0) scr[L.y + ns - 1] = 1. - sy;
  if (G <= 32) grp.sync();  // else the barrier in state_ctx
  sim += b.d[m.d_invmw + ns - 1];
  const StateCtx s = state_ctx<G>(m, b, grp, T, rho, sim, pres, isochoric, c.option);
  rho = s.rho;
  const double mmw = s.mmw;
  // ---------------- P1-P3
  const SpeciesSums sums = prep_species<G, JAC>(m, b, L, scr, grp, s, isochoric, true);
  const double cmix = isochoric ? sums.cpmix - m.Ru * sim : sums.cpmix;  // cv or cp
  const double invRho = s.invRho;
  double iC;
  if constexpr (G <= 32) {
    iC = fix_reciprocal(cmix);
  } else if (grp.warp == Group<G>::W / 2) {  // read after the reactions' barrier
    iC = fix_reciprocal(cmix);
    if ((lane & 31) == 0) grp.scalars[8] = iC;
  }
  const double2 E = reactions_and_gathers<G, JAC, U>(m, b, L, scr, grp, s, pg, true);
  const double EA = E.x, EB = E.y;
  if constexpr (G > 32) iC = grp.scalars[8];
  const double iRC = iC * invRho;
  const double cpsens = sums.cpsens;
  // feed of an open reactor (isochoric_reactor_kernels.cpp:39-154, isobaric_reactor_kernels.cpp:31-168):
  // fe = sum_i (e_i(Tin) - e_i(T)) yin_i (enthalpies when isobaric), fc = sum_i yin_i cv_i(T) (cp_i)
  double fe = 0., fc = 0.;
  if (open_) {
    const double Tin = c.Tin, lTin = log(Tin), iTin = 1. / Tin;
    for (int i = lane; i < ns; i += G) {
      const SpeciesThermo th = species_thermo(m, b, i, Tin, lTin, iTin, false);
      const double ein = isochoric ? th.h - m.Ru * Tin * b.d[m.d_invmw + i] : th.h;
      const double yi = c.yin[i];
      fe += (ein - scr[L.eh + i]) * yi;
      fc += yi * scr[L.cpv + i];
    }
    grp.sum2(fe, fc, ns);
  }
  // mass-exchange factor of the species and energy equations: rho_in / (tau rho) isochoric, 1 / tau isobaric
  const double itau = open_ ? 1. / c.tau : 0.;
  const double mfac = open_ ? (isochoric ? itau * c.rho_in * invRho : itau) : 0.;
  const double mrT = open_ ? fe * iC * mfac : 0.;  // feed term of the temperature equation

  // ---------------- P4: right-hand side and rho/T columns. The gathers hold rho S_rho and T S_T.
  double swe = 0., sre = 0., ste = 0., swc = 0.;
  for (int i = lane; i < ns; i += G) {
    const double e = scr[L.eh + i];
    swe += scr[L.w + i] * e;
    if (JAC) {
      sre += scr[L.Srho + i] * e;
      ste += scr[L.ST + i] * e;
      swc += scr[L.w + i] * scr[L.cpv + i];
    }
  }
  if (JAC)
    grp.sum4(swe, sre, ste, swc, ns);
  else
    swe = grp.sum(swe, ns);
  const double rhsT = -swe * iRC;
  double qheat = 0.;
  if (c.heat == 2)
    qheat = c.SoV * iRC * (c.hc * (c.Tc - T) + c.eps * 5.67e-8 * (c.Tr * c.Tr * c.Tr * c.Tr - T * T * T * T));
  const int tix = isochoric ? 1 : 0;  // index of T in the state
  for (int i = lane; i < ns - 1; i += G) {
    double v = scr[L.w + i] * invRho;
    if (open_) v += (c.yin[i] - scr[L.y + i]) * mfac;
    rhs[tix + 1 + i] = v;
  }
  if (lane == 0) {
    if (isochoric) rhs[0] = open_ ? (c.rho_in - rho) * itau : 0.;
    rhs[tix] = c.heat == 1 ? 0. : (open_ ? rhsT + qheat + mrT : rhsT + qheat);
  }
  if (!JAC) {
    grp.sync();
    return;
  }
  // primitive rho and T columns of the T row (chem_jac_isochoric / chem_jac_isobaric)
  const double JTrho = -invRho * fma(iRC, sre, rhsT);
  const double JTT = -iC * (invRho * fma(s.invT, ste, swc) + rhsT * cpsens);
  const double cpv_last = scr[L.cpv + ns - 1];
  if (isochoric) {
    const double ir2 = invRho * invRho, irt = invRho * s.invT;
    for (int i = lane; i < ns - 1; i += G) {
      double v = ir2 * (scr[L.Srho + i] - scr[L.w + i]);
      if (open_) v -= (c.yin[i] - scr[L.y + i]) * mfac * invRho;
      jset(2 + i, 0, v);
      jset(2 + i, 1, irt * scr[L.ST + i]);
    }
  } else {
    // isobaric transform (isobaric_reactor_kernels.cpp:319-343): T column = PJ_T - rho/T * PJ_rho, and the Y
    // columns get (-rho*mmw) * u_k * PJ_rho, folded into P; PJ_rho = (rho S_rho - w) / rho^2
    const double irt = invRho * s.invT, nmr = -(mmw * invRho);
    for (int i = lane; i < ns - 1; i += G) {
      const double d = scr[L.Srho + i] - scr[L.w + i];
      jset(1 + i, 0, irt * (scr[L.ST + i] - d));
      scr[L.P + i] = fma(nmr, d, scr[L.P + i]);
    }
  }
  for (int k = lane; k < ns; k += G) scr[L.trow + k] = 0.;

  // ---------------- P5: Y block (species rows/columns) and T-row sums; an open reactor's feed adds -mfac on the
  // diagonal (rho_in / (tau rho) isochoric, 1 / tau isobaric)
  {
    const int off = isochoric ? 2 : 1;
    const bool diag = open_;
    const double dyy = -mfac;
    auto yblock = [&](int row, int col, double v) {
      if (diag && row == col) v += dyy;
      jset(off + row, off + col, v);
    };
    run_program<G, U>(pg.j, grp, scr, L.Q, yblock);
  }
  grp.sync();

  // ---------------- P6: T row (and the zero rho row of the isochoric Jacobian). trow holds the sums over D = dq/dC.
  const double iso_heat = (c.heat == 1) ? 0. : 1.;
  const double fT = rhsT + mrT + qheat;  // every heat term of dT/dt varies with Y_k through the mixture's heat capacity
  if (isochoric) {
    for (int k = lane; k < ns - 1; k += G) {
      const double ts = fma(scr[L.trow + k], b.d[m.d_invmw + k], fma(b.d[m.d_u + k], EA, EB));
      const double v = -iC * fma(fT, scr[L.cpv + k] - cpv_last, ts);
      jset(1, 2 + k, v * iso_heat);
    }
    for (int k = lane; k < neq; k += G) jset(0, k, (k == 0 && open_) ? -itau : 0.);
    if (lane == 0) {
      double j10 = JTrho, j11 = JTT;
      if (open_) {
        j10 += -mrT * invRho;
        j11 += -iC * (itau * invRho * c.rho_in * fc + cpsens * mrT);
      }
      if (c.heat == 2) {
        j10 += -qheat * invRho;
        j11 += -iC * cpsens * qheat - c.SoV * iRC * (c.hc + 4. * c.eps * 5.67e-8 * T * T * T);
      }
      jset(1, 0, j10 * iso_heat);
      jset(1, 1, j11 * iso_heat);
    }
  } else {
    const double roT = rho * s.invT, nrm = -rho * mmw;
    double pjr = JTrho, pjt = JTT;
    if (open_) pjt += -iC * (cpsens * mrT + itau * fc);
    if (c.heat == 2) {
      pjr += -qheat * invRho;
      pjt += -iC * cpsens * qheat - c.SoV * iRC * (c.hc + 4. * c.eps * 5.67e-8 * T * T * T);
    }
    pjr *= iso_heat;
    pjt *= iso_heat;
    const double upj = nrm * pjr, niC = -iC * iso_heat;
    for (int k = lane; k < ns - 1; k += G) {
      const double u = b.d[m.d_u + k];
      const double ts = fma(scr[L.trow + k], b.d[m.d_invmw + k], fma(u, EA, EB));
      jset(0, 1 + k, fma(niC, fma(fT, scr[L.cpv + k] - cpv_last, ts), u * upj));
    }
    if (lane == 0) jset(0, 0, pjt - roT * pjr);
  }
  grp.sync();
}

}  // namespace sfgb
