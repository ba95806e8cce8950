// Host side of the mechanism: Griffon's finalize derivations, packing into the device blob, and the construction
// of the load-balanced gather programs used by the Jacobian kernels.
//
// Derivations restated from src/spitfire/griffon/src/chemistry_setup.cpp:
//   NASA7 storage scaled by R and 1/2, 1/6, 1/12, 1/20          (:102-130)
//   third-body efficiencies stored as eff - default               (:406-419)
//   net stoichiometry over species in ascending index order       (:459-541), 2 <= n_net <= 8 enforced
//   dense/sparse sensitivity classification                       (:543-602)
//   rate-constant temperature form and Troe term flags            (:670-730)
#include "sf_internal.h"
#include "exp_table.h"

#include <algorithm>
#include <cmath>
#include <deque>
#include <functional>
#include <map>
#include <numeric>
#include <queue>
#include <stdexcept>
#include <string>

namespace sfgb {

static int pack_sp(int s, int hi) { return (s & 0xFFFF) | (hi << 16); }

namespace {
typedef unsigned long long u64;
typedef unsigned __int128 u128;

// log2(x) = n + f 2^-64 of a positive normal x, in integers (the same on every host) within 2^-59: x = 2^e m with m in
// [2^-1/2, 2^1/2), ln m = 2 atanh(z), z = (m - 1) / (m + 1), |z| < 0.172.
void fixed_log2_of(double x, int *n, u64 *f)
{
  int e;
  double m = std::frexp(x, &e);  // [0.5, 1)
  if (m < 0.70710678118654752) { m *= 2.; --e; }
  const bool below = m < 1.;
  const u64 one = 1ull << 53, mi = (u64)std::ldexp(m, 53);
  const u64 num = below ? one - mi : mi - one, den = one + mi;
  const u64 z = (u64)(((u128)num << 64) / den);
  const u64 z2 = (u64)(((u128)z * z) >> 64);
  u128 sum = z;
  u64 term = z;
  for (int k = 3; term; k += 2) {
    term = (u64)(((u128)term * z2) >> 64);
    sum += term / k;
  }
  // log2 m = 2 sum log2(e): log2(e) 2^63 rounded
  const u64 l2e63 = ((u64)kFixLog2e2 << 32) | kFixLog2e1;
  const u64 l = (u64)((sum * l2e63) >> 62);  // |log2 m| < 1/2 in units of 2^-64
  *n = e;
  *f = l;
  if (below && l) {
    *f = 0ull - l;
    --*n;
  }
}

// Fixed-point form of A T^b exp(-c/T): false where it has none (A not positive, b or c too large). The signed words hold
// |b| 2^58 up to 32 and |c| log2(e) 2^44 up to 2^19 / log2(e) = 363,408 K.
bool fixed_arrhenius_of(const double *k, double *w, int *n)
{
  if (!(k[0] > 1e-300 && k[0] < 1e300) || !(std::abs(k[1]) < 31.) || !(std::abs(k[2]) < 3.6e5)) return false;
  u64 f;
  fixed_log2_of(k[0], n, &f);
  const long long b = (long long)std::ldexp(k[1], 58);
  // |c| log2(e) 2^44 from the 53-bit mantissa of c and log2(e) 2^63
  int e;
  const u64 mi = (u64)std::ldexp(std::frexp(std::abs(k[2]), &e), 53);  // |c| = mi 2^(e - 53)
  const u64 l2e63 = ((u64)kFixLog2e2 << 32) | kFixLog2e1;
  const int sh = 53 - e + 63 - 44;  // mi l2e63 2^-sh
  const u128 prod = (u128)mi * l2e63;
  const u128 rounded = sh < 128 ? (prod + (((u128)1 << sh) >> 1)) >> sh : 0;
  if (rounded >> 63) return false;
  long long c = (long long)rounded;
  if (k[2] < 0.) c = -c;
  std::memcpy(&w[0], &f, 8);
  std::memcpy(&w[1], &b, 8);
  std::memcpy(&w[2], &c, 8);
  return true;
}

// The forward constant that a reaction's temperature form means: forms 0 to 3 have b = 0, 1, 2, -1 and no E, whatever the
// last digits of the b and E that selected them.
std::array<double, 3> form_constant(const HRxn &x)
{
  static const double form_b[4] = {0., 1., 2., -1.};
  if (x.kform == 4) return {x.kf[0], x.kf[1], x.kf[2]};
  return {x.kf[0], form_b[x.kform], 0.};
}
}  // namespace

HostMech::~HostMech()
{
  if (d_items) cudaFree(d_items);
  if (d_blob) cudaFree(d_blob);
  if (d_status) cudaFree(d_status);
  for (cudaEvent_t e : events) cudaEventDestroy(e);
  if (copy_stream) cudaStreamDestroy(copy_stream);
}

void HostMech::build(const sf_mech_desc *d)
{
  const int ns = d->n_species, nr = d->n_reactions;
  if (ns < 2 || ns > kMaxSpecies) throw sf_error(SF_ERR_INVALID_ARGUMENT, "n_species must be in [2, 1024]");
  if (nr < 0) throw sf_error(SF_ERR_INVALID_ARGUMENT, "n_reactions < 0");
  DevMech &m = dm;
  m = DevMech{};
  m.ns = ns;
  m.nr = nr;
  m.Ru = d->gas_constant;
  m.invRu = 1. / d->gas_constant;
  m.pref = d->ref_pressure;

  // ---------------- species
  invmw.resize(ns);
  mw.assign(d->molecular_weights, d->molecular_weights + ns);
  for (int i = 0; i < ns; ++i) invmw[i] = 1. / mw[i];
  std::vector<double> nasa(ns * 15, 0.), tmin(ns), tmax(ns);
  std::vector<int> thermo(ns);
  m.all_nasa7 = 1;
  for (int k = 0; k < ns; ++k) {
    const double *t = d->thermo_coefs + 20 * k;
    double *c = &nasa[15 * k];
    thermo[k] = d->thermo_kind[k];
    if (thermo[k] == SF_THERMO_NASA7) {
      tmin[k] = t[0];
      tmax[k] = t[2];
      c[0] = t[1];
      for (int j = 0; j < 7; ++j) c[1 + j] = t[10 + j] * m.Ru;
      for (int j = 0; j < 7; ++j) c[8 + j] = t[3 + j] * m.Ru;
      c[2] /= 2.; c[3] /= 6.; c[4] /= 12.; c[5] /= 20.;
      c[9] /= 2.; c[10] /= 6.; c[11] /= 12.; c[12] /= 20.;
    } else if (thermo[k] == SF_THERMO_CONST) {
      m.all_nasa7 = 0;
      tmin[k] = t[0];
      tmax[k] = t[1];
      c[0] = t[2]; c[1] = t[3]; c[2] = t[4]; c[3] = t[5];
      c[4] = std::log(t[2]);
    } else {
      throw sf_error(SF_ERR_UNSUPPORTED, "NASA9 thermodynamics is not supported by the GPU kernels");
    }
  }

  // ---------------- reactions
  rx.clear();
  rx.resize(nr);
  int n_fall = 0, n_dense = 0;
  for (int r = 0; r < nr; ++r) {
    HRxn &x = rx[r];
    x.kind = d->rxn_kind[r];
    if (x.kind < SF_RXN_SIMPLE || x.kind > SF_RXN_TROE)
      throw sf_error(SF_ERR_MECHANISM, "reaction " + std::to_string(r) + ": unknown kind");
    x.reversible = d->rxn_reversible[r] != 0;
    for (int j = 0; j < 3; ++j) x.kf[j] = d->rxn_kfwd[3 * r + j];
    if (x.kind >= SF_RXN_LINDEMANN) {
      for (int j = 0; j < 3; ++j) x.kp[j] = d->rxn_kflf[3 * r + j];
      x.fall = n_fall++;
    }
    if (x.kind == SF_RXN_TROE)
      for (int j = 0; j < 4; ++j) x.troe[j] = d->rxn_troe[4 * r + j];
    x.beff = x.kind != SF_RXN_SIMPLE ? d->rxn_default_eff[r] : 0.;
    for (int i = d->reac_offsets[r]; i < d->reac_offsets[r + 1]; ++i) {
      x.reac.push_back(d->reac_species[i]);
      x.reac_nu.push_back(d->reac_stoich[i]);
    }
    for (int i = d->prod_offsets[r]; i < d->prod_offsets[r + 1]; ++i) {
      x.prod.push_back(d->prod_species[i]);
      x.prod_nu.push_back(d->prod_stoich[i]);
    }
    if (x.kind != SF_RXN_SIMPLE)
      for (int i = d->eff_offsets[r]; i < d->eff_offsets[r + 1]; ++i) {
        const int s = d->eff_species[i];
        x.tb.push_back(s);
        x.tbeff.push_back(d->eff_values[i] - x.beff);
      }
    if (d->order_offsets && d->order_offsets[r + 1] > d->order_offsets[r]) {
      x.has_orders = true;
      for (int i = d->order_offsets[r]; i < d->order_offsets[r + 1]; ++i) {
        x.ord.push_back(d->order_species[i]);
        x.ord_val.push_back(d->order_values[i]);
      }
    }
    for (const auto *v : {&x.reac, &x.prod, &x.tb, &x.ord})
      for (int s : *v)
        if (s < 0 || s >= ns) throw sf_error(SF_ERR_MECHANISM, "reaction " + std::to_string(r) + ": bad species index");
    std::map<int, int> net;
    x.sum_nu = 0;
    for (size_t i = 0; i < x.reac.size(); ++i) { net[x.reac[i]] += x.reac_nu[i]; x.sum_nu += x.reac_nu[i]; }
    for (size_t i = 0; i < x.prod.size(); ++i) { net[x.prod[i]] -= x.prod_nu[i]; x.sum_nu -= x.prod_nu[i]; }
    for (auto &kv : net)
      if (kv.second != 0) { x.net.push_back(kv.first); x.net_nu.push_back(kv.second); }
    if (x.net.size() < 2 || x.net.size() > (size_t)kMaxNet)
      throw sf_error(SF_ERR_MECHANISM, "reaction " + std::to_string(r) + ": bad number of net reacting species (n < 2 or n > 8)");
    x.sum_reac_nu = 0;
    for (int v : x.reac_nu) x.sum_reac_nu += std::abs(v);
    x.sum_prod_nu = 0;
    for (int v : x.prod_nu) x.sum_prod_nu += std::abs(v);
    // coefficients and their sums are read through the device's table of small integers
    if (x.sum_reac_nu > 127 || x.sum_prod_nu > 127)
      throw sf_error(SF_ERR_MECHANISM, "reaction " + std::to_string(r) + ": stoichiometric coefficients above 127");
    if (std::abs(x.kf[2]) < 1.e-6) {
      if (std::abs(x.kf[1]) < 1.e-6) x.kform = 0;
      else if (std::abs(x.kf[1] - 1) < 1.e-6) x.kform = 1;
      else if (std::abs(x.kf[1] - 2) < 1.e-6) x.kform = 2;
      else if (std::abs(x.kf[1] + 1) < 1.e-6) x.kform = 3;
      else x.kform = 4;
    } else x.kform = 4;
    if (x.kind == SF_RXN_TROE) {
      x.troe_terms = (std::abs(x.troe[1]) > 1.e-8 ? 1 : 0) | (std::abs(x.troe[2]) > 1.e-8 ? 2 : 0) |
                     (std::abs(x.troe[3]) > 1.e-8 ? 4 : 0);
      if (!x.troe_terms) throw sf_error(SF_ERR_MECHANISM, "no troe terms flagged for evaluation");
    }
    // Jacobian slots: every species other than the last whose Y column receives a sparse contribution from this
    // reaction (reactants, products, third bodies, special-order species). The closure species ns-1 contributes
    // a constant to every column (beta), third-body/falloff reactions a term proportional to u_s (alpha).
    auto pos = [](const std::vector<int> &v, int s) {
      for (size_t i = 0; i < v.size(); ++i) if (v[i] == s) return (int)i;
      return -1;
    };
    std::vector<int> slots;
    for (const auto *v : {&x.reac, &x.prod, &x.tb, &x.ord})
      for (int s : *v)
        if (s != ns - 1 && std::find(slots.begin(), slots.end(), s) == slots.end()) slots.push_back(s);
    std::sort(slots.begin(), slots.end());
    x.slots.clear();
    for (int s : slots) {
      const int rp = pos(x.reac, s);
      const int pp = pos(x.prod, s);
      const int tp = pos(x.tb, s);
      const int op = pos(x.ord, s);
      if (rp < 0 && pp < 0 && tp < 0 && op < 0) continue;
      x.slots.push_back(s | ((rp + 1) << 16) | ((pp + 1) << 20) | ((tp + 1) << 24) | ((op + 1) << 28));
    }
    bool last_involved = false;
    for (const auto *v : {&x.reac, &x.prod, &x.tb, &x.ord})
      for (int s : *v) if (s == ns - 1) last_involved = true;
    x.dense = (x.kind != SF_RXN_SIMPLE) || last_involved;
    x.dense_idx = x.dense ? n_dense++ : -1;
  }
  // Device order: reactions grouped by kind and, within a kind, by the form of their forward constant (those without an
  // exponential first), the lengths of their sides and their number of Jacobian slots (stable). Lanes of a state
  // group take reactions in strides of the group width, so the lanes of a pass then mostly take the same paths and
  // run the slot loop about as many times. Per-reaction outputs map back through i_orig.
  std::vector<int> order(nr);
  std::iota(order.begin(), order.end(), 0);
  auto key = [&](int r) {
    const HRxn &x = rx[r];
    return std::array<int, 6>{x.kind, x.kform == 4 ? 1 : 0, x.reversible ? 0 : 1, (int)x.reac.size(),
                              (int)x.prod.size(), (int)x.slots.size()};
  };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key(a) < key(b); });
  {
    std::vector<HRxn> sorted(nr);
    for (int k = 0; k < nr; ++k) sorted[k] = std::move(rx[order[k]]);
    rx = std::move(sorted);
    n_fall = 0;
    n_dense = 0;
    for (HRxn &x : rx) {
      x.fall = x.kind >= SF_RXN_LINDEMANN ? n_fall++ : -1;
      x.dense_idx = x.dense ? n_dense++ : -1;
    }
  }
  orig_index = order;
  m.n_fall = n_fall;
  m.n_dense = n_dense;

  // ---------------- pack the blob
  std::vector<double> D;
  std::vector<int> I;
  auto dsec = [&](int n) { const int o = (int)D.size(); D.resize(D.size() + std::max(n, 0), 0.); return o; };
  auto isec = [&](int n) { const int o = (int)I.size(); I.resize(I.size() + std::max(n, 0), 0); return o; };
  m.d_nasa = dsec(15 * ns);
  std::copy(nasa.begin(), nasa.end(), D.begin() + m.d_nasa);
  m.d_tmin = dsec(ns);
  m.d_tmax = dsec(ns);
  m.d_invmw = dsec(ns);
  m.d_mw = dsec(ns);
  m.d_u = dsec(ns);
  for (int i = 0; i < ns; ++i) {
    D[m.d_tmin + i] = tmin[i];
    D[m.d_tmax + i] = tmax[i];
    D[m.d_invmw + i] = invmw[i];
    D[m.d_mw + i] = mw[i];
    D[m.d_u + i] = invmw[i] - invmw[ns - 1];
  }
  m.d_kf = dsec(3 * nr);
  m.d_kp = dsec(3 * n_fall);
  m.d_troe = dsec(4 * n_fall);
  m.d_beff = dsec(nr);
  for (int r = 0; r < nr; ++r) {
    const HRxn &x = rx[r];
    for (int j = 0; j < 3; ++j) D[m.d_kf + 3 * r + j] = x.kf[j];
    if (x.fall >= 0) {
      const std::array<double, 3> kf = form_constant(x);
      D[m.d_kp + 3 * x.fall] = x.kp[0] / kf[0];
      for (int j = 1; j < 3; ++j) D[m.d_kp + 3 * x.fall + j] = x.kp[j] - kf[j];
      const double tr[4] = {x.troe[0], -1. / x.troe[1], -1. / x.troe[2], x.troe[3]};
      for (int j = 0; j < 4; ++j) D[m.d_troe + 4 * x.fall + j] = tr[j];
    }
    D[m.d_beff + r] = x.beff;
  }
  int ntb = 0, nnet = 0, nord = 0, nslot = 0, nreac = 0, nprod = 0;
  for (const auto &x : rx) {
    ntb += (int)x.tb.size(); nnet += (int)x.net.size(); nord += (int)x.ord.size(); nslot += (int)x.slots.size();
    nreac += (int)x.reac.size(); nprod += (int)x.prod.size();
  }
  m.n_slots = nslot;
  m.n_net_total = nnet;
  m.d_tbeff = dsec(ntb);
  m.d_netc = dsec(nnet);
  m.d_ord = dsec(nord);
  m.d_smallint = dsec(64);
  for (int k = 0; k < 64; ++k) D[m.d_smallint + k] = k - 32;
  while (D.size() % 2) D.push_back(0.);  // 16-byte boundary: the table is read as (head, tail) pairs
  m.d_exptab = dsec(128 + 256);
  std::copy(kExpTable, kExpTable + 128, D.begin() + m.d_exptab);
  std::memcpy(&D[m.d_exptab + 128], kFixExpTable, sizeof kFixExpTable);
  m.i_info = isec(nr);
  m.i_orig = isec(nr);
  for (int r = 0; r < nr; ++r) I[m.i_orig + r] = orig_index[r];
  m.i_sums = isec(nr);
  m.i_dense = isec(nr);
  m.i_reac_off = isec(nr + 1); m.i_reac = isec(nreac);
  m.i_prod_off = isec(nr + 1); m.i_prod = isec(nprod);
  m.i_net_off = isec(nr + 1); m.i_net = isec(nnet);
  m.i_tb_off = isec(nr + 1); m.i_tb = isec(ntb);
  m.i_ord_off = isec(nr + 1); m.i_ord = isec(nord);
  m.i_slot_off = isec(nr + 1); m.i_slot = isec(nslot);
  m.i_thermo = isec(ns);
  for (int i = 0; i < ns; ++i) I[m.i_thermo + i] = thermo[i];
  int cr = 0, cp = 0, cn = 0, ct = 0, co = 0, cs = 0;
  net_entry_of.assign(nr, std::vector<int>());
  slot_entry_of.assign(nr, std::vector<int>());
  for (int r = 0; r < nr; ++r) {
    const HRxn &x = rx[r];
    I[m.i_info + r] = (x.kind << RI_KIND_SHIFT) | (x.kform << RI_KFORM_SHIFT) | (x.troe_terms << RI_TROE_SHIFT) |
                      (x.reversible ? 1 << RI_REV_BIT : 0) | (x.has_orders ? 1 << RI_ORD_BIT : 0) |
                      (x.dense ? 1 << RI_DENSE_BIT : 0);
    I[m.i_sums + r] = (x.sum_nu & 0xFFFF) | ((x.sum_reac_nu & 0xFF) << 16) | ((x.sum_prod_nu & 0xFF) << 24);
    I[m.i_dense + r] = x.dense_idx;
    I[m.i_reac_off + r] = cr;
    for (size_t i = 0; i < x.reac.size(); ++i) I[m.i_reac + cr++] = pack_sp(x.reac[i], x.reac_nu[i]);
    I[m.i_prod_off + r] = cp;
    for (size_t i = 0; i < x.prod.size(); ++i) I[m.i_prod + cp++] = pack_sp(x.prod[i], x.prod_nu[i]);
    I[m.i_net_off + r] = cn;
    for (size_t i = 0; i < x.net.size(); ++i) {
      I[m.i_net + cn] = pack_sp(x.net[i], x.net_nu[i] + 128);
      D[m.d_netc + cn] = -x.net_nu[i] * mw[x.net[i]];
      net_entry_of[r].push_back(cn);
      ++cn;
    }
    I[m.i_tb_off + r] = ct;
    for (size_t i = 0; i < x.tb.size(); ++i) {
      I[m.i_tb + ct] = x.tb[i];
      D[m.d_tbeff + ct] = x.tbeff[i];
      ++ct;
    }
    I[m.i_ord_off + r] = co;
    for (size_t i = 0; i < x.ord.size(); ++i) {
      I[m.i_ord + co] = pack_sp(x.ord[i], std::abs(x.ord_val[i]) > 1.e-12 ? 1 : 0);
      D[m.d_ord + co] = x.ord_val[i];
      ++co;
    }
    I[m.i_slot_off + r] = cs;
    for (size_t i = 0; i < x.slots.size(); ++i) {
      I[m.i_slot + cs] = x.slots[i];
      slot_entry_of[r].push_back(cs);
      ++cs;
    }
  }
  I[m.i_reac_off + nr] = cr; I[m.i_prod_off + nr] = cp; I[m.i_net_off + nr] = cn;
  I[m.i_tb_off + nr] = ct; I[m.i_ord_off + nr] = co; I[m.i_slot_off + nr] = cs;
  // ---------------- scratch layout (RHS-only path uses the prefix up to total_rhs)
  ScratchLayout &L = sl;
  int o = 0;
  auto take = [&](int n) { const int r = o; o += (n + 1) & ~1; return r; };
  L.y = take(ns); L.C = take(ns); L.eh = take(ns); L.cpv = take(ns); L.w = take(ns);
  L.gm = take(ns); L.gk = take(ns);
  L.q = take(nr);
  L.total_rhs = o;
  L.dB = take(ns); L.dcp = take(ns); L.P = take(ns); L.Q = take(ns);
  L.dqdrho = take(nr); L.dqdT = take(nr);
  // arrays that take the place of dead ones: C and dB after the reactions, S_rho after the rho column, q after the
  // species gathers
  L.Srho = L.C; L.ST = L.dB; L.trow = L.Srho; L.E = L.q;
  L.alpha = take(n_dense); L.beta = take(n_dense);
  L.D = take(nslot);
  L.total = o;

  // ---------------- fixed-point rate constants, 28 bytes per reaction and falloff ratio: left out (the rates are then formed
  // in FP64) where some kernel's narrowest group fits a block's shared memory only without them, and where the Gibbs energies
  // or the reference concentration are no finite numbers, which a fixed-point word cannot hold
  CUDA_THROW(cudaGetDevice(&device));
  {
    int smem_max;
    CUDA_THROW(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    std::vector<size_t> need = {0, (size_t)L.total_rhs, (size_t)L.total, (size_t)L.total_rhs + ns + 3, (size_t)L.total + ns + 2};
    for (int neq : {ns, ns + 1})
      for (int place = 0; place <= 2; ++place)
        for (int prec = 0; prec <= 1; ++prec)
          need.push_back(integrate_warp_doubles(*this, neq, prec, place >= 1, place == 2, true));
    const size_t base = D.size() * 8 + I.size() * 4 + 32, fix = (size_t)28 * (nr + n_fall);
    m.fixed_rates = 1;
    for (size_t n : need)
      if (base + 8 * n + 64 <= (size_t)smem_max && base + fix + 8 * n + 64 > (size_t)smem_max) m.fixed_rates = 0;
    for (double c : nasa)
      if (!std::isfinite(c)) m.fixed_rates = 0;
    if (!std::isnormal(m.pref / m.Ru) || !(m.pref / m.Ru > 0.)) m.fixed_rates = 0;
  }
  if (m.fixed_rates) {
    fixed_log2_of(m.pref / m.Ru, &m.log2_port_n, &m.log2_port_f);
    m.d_fix = dsec(3 * nr);
    m.d_fixp = dsec(3 * n_fall);
    m.i_fixn = isec(nr);
    m.i_fixp = isec(n_fall);
    for (int r = 0; r < nr; ++r) {
      const int f = rx[r].fall;
      if (!fixed_arrhenius_of(form_constant(rx[r]).data(), &D[m.d_fix + 3 * r], &I[m.i_fixn + r])) I[m.i_fixn + r] = kFixNone;
      if (f >= 0 && !fixed_arrhenius_of(&D[m.d_kp + 3 * f], &D[m.d_fixp + 3 * f], &I[m.i_fixp + f])) I[m.i_fixp + f] = kFixNone;
    }
  }
  while (D.size() % 2) D.push_back(0.);  // 16-byte boundary for the int section
  while (I.size() % 4) I.push_back(0);   // 16-byte total
  m.blob_doubles = (int)D.size();
  m.blob_ints = (int)I.size();
  m.blob_bytes = m.blob_doubles * 8 + m.blob_ints * 4;
  host_dbl = D;
  host_int = I;

  // ---------------- upload
  CUDA_THROW(cudaMalloc(&d_blob, m.blob_bytes));
  std::vector<unsigned char> bytes(m.blob_bytes);
  std::memcpy(bytes.data(), D.data(), D.size() * 8);
  std::memcpy(bytes.data() + D.size() * 8, I.data(), I.size() * 4);
  CUDA_THROW(cudaMemcpy(d_blob, bytes.data(), m.blob_bytes, cudaMemcpyHostToDevice));
  CUDA_THROW(cudaMalloc(&d_status, 16));
  CUDA_THROW(cudaMemset(d_status, 0, 16));
  // every gather program the kernels use, built here so that no evaluation call builds or allocates one
  build_programs();
}

const HostMech::Programs &HostMech::programs_for(int G) const
{
  auto it = programs.find(G);
  if (it == programs.end()) throw sf_error(SF_ERR_INVALID_ARGUMENT, "no gather program for this lane width");
  return it->second;
}

void ensure_dynamic_smem(const void *kernel, size_t bytes)
{
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> set;
  int dev;
  CUDA_THROW(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  size_t &cur = set[{kernel, dev}];
  if (bytes <= cur) return;
  CUDA_THROW(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  cur = bytes;
}

// ------------------------------------------------------------------------------------------ gather programs
namespace {
struct Item {
  double c;
  uint32_t ref;
  int pair;  // >= 0: scratch index of the coefficient
};
struct Entry {
  std::vector<Item> items;
  uint32_t dst;  // IT_JAC | row | col << IT_COL_SHIFT, or a scratch index
};

typedef std::vector<const Entry *> EntryList;

// The device runner loads operands ahead of the stores of earlier items, so a program must never read a scratch
// location that it writes (as a destination or through an entry's initial value).
void check_no_read_after_write(const EntryList &entries, int qoff, int scratch)
{
  std::vector<char> written(scratch, 0);
  for (const Entry *e : entries)
    if (!(e->dst & IT_JAC)) written[e->dst] = 1;
  bool bad = false;
  for (const Entry *e : entries) {
    if (e->dst & IT_JAC) bad |= written[qoff + (e->dst & IT_ROW_MASK)] != 0;
    for (const Item &it : e->items) bad |= written[it.ref] || (it.pair >= 0 && written[it.pair]);
  }
  if (bad) throw sf_error(SF_ERR_MECHANISM, "internal: gather program reads what it writes");
}

// Assignment of entries to G lanes and the interleaved item array, each lane's items padded with no-ops to a
// multiple of the device runner's batch. G > 1: longest-processing-time assignment (balanced lanes). G = 1 (one
// lane per state): entries in destination order, Jacobian entries column-major, so that each thread writes its
// Jacobian block sequentially through memory.
std::vector<GatherItem> schedule(const EntryList &entries, int G, int qoff, int scratch, int *len_out)
{
  check_no_read_after_write(entries, qoff, scratch);
  std::vector<int> order(entries.size());
  std::iota(order.begin(), order.end(), 0);
  if (G == 1) {
    auto key = [&](int e) {
      const uint32_t d = entries[e]->dst;
      const uint64_t jac = (d & IT_JAC) ? 0 : 1;  // the Jacobian first
      return jac << 32 | (d & IT_DST_MASK);       // col << 13 | row: column-major
    };
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key(a) < key(b); });
  } else {
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return entries[a]->items.size() > entries[b]->items.size(); });
  }
  std::vector<std::vector<int>> lane(G);
  std::vector<size_t> load(G, 0);
  typedef std::pair<size_t, int> Load;  // (items, lane): the least loaded lane, the lowest on ties
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> least;
  for (int l = 0; l < G; ++l) least.push({0, l});
  for (int e : order) {
    if (entries[e]->items.empty()) continue;
    const int best = least.top().second;
    least.pop();
    lane[best].push_back(e);
    load[best] += entries[e]->items.size();
    least.push({load[best], best});
  }
  size_t len = 0;
  for (int l = 0; l < G; ++l) len = std::max(len, load[l]);
  len = (len + GATHER_UNROLL - 1) / GATHER_UNROLL * GATHER_UNROLL;
  std::vector<GatherItem> out(len * G, GatherItem{0., 0, IT_NOP});
  for (int l = 0; l < G; ++l) {
    size_t j = 0;
    for (int e : lane[l]) {
      const Entry &E = *entries[e];
      for (size_t k = 0; k < E.items.size(); ++k, ++j) {
        const Item &x = E.items[k];
        GatherItem it{x.c, x.ref, E.dst};
        if (x.pair >= 0) {
          const uint64_t bits = (uint32_t)x.pair;
          std::memcpy(&it.c, &bits, 8);
          it.ctl |= IT_PAIR;
        }
        if (k == 0) it.ctl |= IT_START;
        if (k + 1 == E.items.size()) it.ctl |= IT_END;
        out[j * G + l] = it;
      }
    }
  }
  *len_out = (int)len;
  return out;
}

// Entries longer than a lane's share are cut into parts of about that share, which sum into the scratch slots
// part .. part + cap - 1 and are added up by the entries put into `fix`. (GRI-3.0's species rates on 32 lanes: 137
// items for H against a share of 39.) A Jacobian entry's first item, u_k P_i on top of Q_i, stays in its fix entry.
// own holds the entries made here.
EntryList split_entries(const std::vector<Entry> &entries, int G, int part, int cap, std::deque<Entry> *own, EntryList *fix)
{
  EntryList out;
  out.reserve(entries.size());
  if (G == 1) {
    for (const Entry &e : entries) out.push_back(&e);
    return out;
  }
  size_t total = 0;
  for (const Entry &e : entries) total += e.items.size();
  for (size_t share = std::max<size_t>(4, (total + G - 1) / G);; share += (share + 3) / 4) {
    out.clear();
    fix->clear();
    own->clear();
    int used = 0;
    for (const Entry &e : entries) {
      const size_t keep = (e.dst & IT_JAC) ? 1 : 0, n = e.items.size() - std::min(keep, e.items.size());
      if (e.items.size() <= share + share / 8) {
        out.push_back(&e);
        continue;
      }
      const size_t parts = (n + share - 1) / share;
      Entry f{{e.items.begin(), e.items.begin() + keep}, e.dst};
      for (size_t p = 0; p < parts; ++p) {
        const size_t a = keep + n * p / parts, b = keep + n * (p + 1) / parts;
        own->push_back(Entry{{e.items.begin() + a, e.items.begin() + b}, (uint32_t)(part + used)});
        out.push_back(&own->back());
        f.items.push_back(Item{1., (uint32_t)(part + used), -1});
        ++used;
      }
      own->push_back(std::move(f));
      fix->push_back(&own->back());
    }
    if (used <= cap) return out;
  }
}
}  // namespace

void HostMech::build_programs()
{
  const int ns = dm.ns, nr = dm.nr;
  const ScratchLayout &L = sl;
  // species -> list of (reaction, coefficient of its rate) in increasing reaction order
  std::vector<std::vector<std::pair<int, double>>> by_species(ns);
  for (int r = 0; r < nr; ++r)
    for (size_t i = 0; i < rx[r].net.size(); ++i)
      by_species[rx[r].net[i]].push_back({r, host_dbl[dm.d_netc + net_entry_of[r][i]]});
  std::vector<Entry> E[4];
  auto item = [](double c, int ref) { return Item{c, (uint32_t)ref, -1}; };
  // program 0: production rates only  w_i = sum_r c_ir q_r
  for (int i = 0; i < ns; ++i) {
    Entry e{{}, (uint32_t)(L.w + i)};
    for (auto &re : by_species[i]) e.items.push_back(item(re.second, L.q + re.first));
    E[0].push_back(e);
  }
  // program 1: w, S_rho, S_T, P, Q for all species
  for (int i = 0; i < ns; ++i) {
    Entry ew{{}, (uint32_t)(L.w + i)}, er{{}, (uint32_t)(L.Srho + i)}, et{{}, (uint32_t)(L.ST + i)},
        ep{{}, (uint32_t)(L.P + i)}, eq{{}, (uint32_t)(L.Q + i)};
    for (auto &re : by_species[i]) {
      const double c = re.second;
      ew.items.push_back(item(c, L.q + re.first));
      er.items.push_back(item(c, L.dqdrho + re.first));
      et.items.push_back(item(c, L.dqdT + re.first));
      const int di = rx[re.first].dense_idx;
      if (di >= 0) {
        ep.items.push_back(item(c, L.alpha + di));
        eq.items.push_back(item(c, L.beta + di));
      }
    }
    for (Entry *e : {&ew, &er, &et, &ep, &eq}) E[1].push_back(*e);
  }
  // an entry with no contributions (an inert species) is written as zero
  for (int k = 0; k < 2; ++k)
    for (Entry &e : E[k])
      if (e.items.empty()) e.items.push_back(item(0., L.y));
  // program 2: the Y block (rows/cols 0..ns-2) and the T-row sums; program 3: every species row (the (ns+1)^2
  // sensitivity block of prod_rates_primitive_sensitivities)
  {
    std::vector<std::vector<std::vector<std::pair<double, int>>>> contrib(ns);  // [row][col] -> (coefficient, slot)
    for (int i = 0; i < ns; ++i) contrib[i].resize(ns - 1);
    std::vector<std::vector<std::pair<int, int>>> tcontrib(ns - 1);  // [col] -> (reaction, slot)
    for (int r = 0; r < nr; ++r) {
      const HRxn &x = rx[r];
      for (size_t j = 0; j < x.slots.size(); ++j) {
        const int k = x.slots[j] & 0xFFFF;
        tcontrib[k].push_back({r, slot_entry_of[r][j]});
        for (size_t i = 0; i < x.net.size(); ++i)
          contrib[x.net[i]][k].push_back({host_dbl[dm.d_netc + net_entry_of[r][i]] * invmw[k], slot_entry_of[r][j]});
      }
    }
    for (int variant = 2; variant <= 3; ++variant) {
      const int nrows = variant == 2 ? ns - 1 : ns;
      for (int i = 0; i < nrows; ++i)
        for (int k = 0; k < ns - 1; ++k) {
          Entry e{{}, IT_JAC | (uint32_t)i | ((uint32_t)k << IT_COL_SHIFT)};
          e.items.push_back(item(host_dbl[dm.d_u + k], L.P + i));
          for (auto &c : contrib[i][k]) e.items.push_back(item(c.first, L.D + c.second));
          E[variant].push_back(e);
        }
      if (variant == 2)
        for (int k = 0; k < ns - 1; ++k) {
          Entry e{{}, (uint32_t)(L.trow + k)};
          for (auto &c : tcontrib[k]) e.items.push_back(Item{0., (uint32_t)(L.D + c.second), L.E + c.first});
          E[variant].push_back(e);
        }
    }
  }
  // every program's items in one device array: offsets until it exists
  std::vector<GatherItem> all;
  auto add = [&](const EntryList &entries, int G, int *len) {
    const std::vector<GatherItem> items = schedule(entries, G, L.Q, L.total, len);
    const size_t at = all.size();
    all.insert(all.end(), items.begin(), items.end());
    return at;
  };
  std::vector<std::pair<const GatherItem **, size_t>> places;
  for (int G : {1, 8, 16, 32, 64, 128, 256}) {
    Programs &P = programs[G];
    for (int k = 0; k < 4; ++k) {
      // partial sums: the Gibbs factors are dead after the reactions, dqdrho and dqdT after the species gathers
      const int part = k < 2 ? L.gm : L.dqdrho, cap = k < 2 ? L.q - L.gm : L.alpha - L.dqdrho;
      std::deque<Entry> own;
      EntryList fix;
      const EntryList main = split_entries(E[k], G, part, cap, &own, &fix);
      places.push_back({&P.progs[k].items, add(main, G, &P.progs[k].len)});
      P.progs[k].fix_items = nullptr;
      P.progs[k].fix_len = 0;
      if (!fix.empty()) places.push_back({&P.progs[k].fix_items, add(fix, G, &P.progs[k].fix_len)});
    }
  }
  CUDA_THROW(cudaMalloc(&d_items, std::max<size_t>(all.size(), 1) * sizeof(GatherItem)));
  if (!all.empty()) CUDA_THROW(cudaMemcpy(d_items, all.data(), all.size() * sizeof(GatherItem), cudaMemcpyHostToDevice));
  for (auto &p : places) *p.first = d_items + p.second;
}

}  // namespace sfgb
