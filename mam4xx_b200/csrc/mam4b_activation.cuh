// mam4b_activation.cuh -- aerosol activation of a cell, the per-cell part
// of the droplet-nucleation process (src/mam4xx/ndrop.hpp): the modes'
// number, volume and hygroscopicity from the interstitial mixing ratios
// (loadaer :244-331, get_aer_mmr_sum :116-155, get_aer_num :157-181), and
// the Abdul-Razzak & Ghan activated number and mass fractions for a given
// updraft (activate_modal :509-697 with maxsat :183-242), as
// get_activate_frac (:699-765) composes them. A consumer of the state the
// microphysics step produces.
#pragma once

#include "mam4b_physics.cuh"

namespace mam4b {
namespace act {

// species-type data of get_e3sm_parameters (ndrop.hpp:44-114): the type of
// species s of mode m (1-based) and each type's density and hygroscopicity
MAM4B_HD constexpr int spectype(int m, int s) {
  constexpr int t[4][7] = {{1, 4, 5, 6, 8, 7, 9}, {1, 5, 7, 9, 0, 0, 0},
                           {8, 7, 1, 6, 4, 5, 9}, {4, 6, 9, 0, 0, 0, 0}};
  return t[m][s];
}
MAM4B_HD constexpr double type_dens(int t) {
  constexpr double d[9] = {0.1770000000E+04, 0.0, 0.0, 0.1000000000E+04, 0.1000000000E+04,
                           0.1700000000E+04, 0.1900000000E+04, 0.2600000000E+04,
                           0.1601000000E+04};
  return d[t - 1];
}
MAM4B_HD constexpr double type_hygro(int t) {
  constexpr double h[9] = {0.5070000000E+00, 0.0, 0.0, 0.1000000083E-09, 0.1400000000E+00,
                           0.1000000013E-09, 0.1160000000E+01, 0.6800000000E-01,
                           0.1000000015E+00};
  return h[t - 1];
}

// mam4 physical constants (mam4_constants.hpp:33-123)
constexpr double kRGas = 6.022214076e23 * 1.380649e-23;  // J/K/mol
constexpr double kRAir = kRGas / 0.028966;
constexpr double kRH2o = kRGas / 0.018016;
constexpr double kLatvap = 2.501e6;
constexpr double kCpAir = 1.00464e3;
constexpr double kGravity = 9.80616;
constexpr double kRhoH2o = 1.0e3;
constexpr double kT0 = 273.0;
constexpr double kP0 = 1013.25e2;
constexpr double kSurften = 0.076;

MAM4B_HD double pow10(double x) {
#ifdef __CUDA_ARCH__
  return exp10(x);
#else
  return pow(10.0, x);
#endif
}

// saturation specific humidity with the water-ice transition below 0 C
// (wv_sat_svp_trans, wv_sat_methods.hpp:139-164; ndrop::qsat,
// ndrop.hpp:450-471); it = 1 / t
MAM4B_HD double qsat_trans(double t, double it, double p) {
  const double ttrice = 20.0, tmelt = 273.15;
  double es = 0.0;
  if (t >= (tmelt - ttrice)) {
    const double tboil = 373.16, r = tboil * it;
    const double hot = pow10(fma(-11.344 / tboil, t, 11.344)) - 1.0;
    const double cold = pow10(-3.49149 * (r - 1.0)) - 1.0;
    double e = fma(-7.90298, r - 1.0, 5.02808 * log10(r));
    e = fma(-1.3816e-7, hot, e);
    e = fma(8.1328e-3, cold, e);
    es = pow10(e) * (1013.246 * 100.0);
  }
  if (t < tmelt) {
    const double h2otrip = 273.16, r = h2otrip * it;
    double e = fma(-9.09718, r - 1.0, -3.56654 * log10(r));
    e = fma(0.876793, fma(-1.0 / h2otrip, t, 1.0), e);
    const double esice = pow10(e) * (6.1071 * 100.0);
    const double weight = (tmelt - t) < ttrice ? (tmelt - t) * (1.0 / ttrice) : 1.0;
    es = fma(weight, esice, (1.0 - weight) * es);
  }
  const double epsilo = 0.018016 / 0.028966;
  const double omeps = 1.0 - epsilo;
  return ((p - es) <= 0.0) ? 1.0 : epsilo * es / fma(-omeps, es, p);
}

// ln of the modes' geometric standard deviations (the widths of K::sig)
MAM4B_HD constexpr double ln_sig(int m) {
  constexpr double t[NMODE] = {0.5877866649021191, 0.47000362924573563, 0.5877866649021191, 0.4700036441468979};
  return t[m];
}

// One cell: ai the 25 interstitial populations (kg/kg, #/kg), air density
// [kg/m3] at the level the aerosol is loaded from and at the cell, updraft
// w [m/s], temperature. out: fn[4], fm[4], fluxn[4], fluxm[4],
// flux_fullact (all zero when there is no accumulation-mode aerosol or no
// updraft, the cases where activate_modal returns without writing; the
// return value is false then).
//
// Bound by issuing the instructions of eight erf, five logs and the powers of
// the saturation pressure (62 % of the issue slots). Written as the reference
// has it, with 25 divisions by densities, a power for each 3/2 and the
// critical supersaturations' roots taken and squared again, the warps waited
// for instructions most of all: 8,191 x 80 cells took 0.180 ms, now 0.101,
// in 17 stores and 28 loads a cell (0.037 ms at least). The competition of the
// modes is in the squares: with s_m^2 = smc^2 the critical supersaturation's,
//   smc^2 = 4 aten^3 pi exp(4.5 ln^2 sigma) n / (20.25 hygroscopic volume),
//   (smc / sqrt(eta + 3 zeta))^(3/2) = sqrt(q) sqrt(sqrt(q)), q = smc^2 / (eta + 3 zeta),
//   ln(smc / smax) = (ln smc^2 + ln sum) / 2, smax = 1 / sqrt(sum).
MAM4B_HD bool activate_cell(const StepConsts &C, const double (&ai)[NPOP], double rho_load,
                            double rho, double w, double tair, double (&out)[17]) {
#pragma unroll
  for (int k = 0; k < 17; ++k)
    out[k] = 0.0;
  // loadaer (phase 1, no cloud-borne part): volume vol, hygroscopic volume
  // hv of a mode in the air, number
  double na[NMODE], vol[NMODE], hv[NMODE];
  bool hygroscopic[NMODE];
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    double vs = 0.0, hs = 0.0;
#pragma unroll
    for (int s = 0; s < K::nspec(m); ++s) {
      const int t = spectype(m, s);
      const double q = dmax(ai[K::spec0(m) + s] + 0.0, 0.0);
      vs = fma(q, 1.0 / type_dens(t), vs);
      hs = fma(q, type_hygro(t) / type_dens(t), hs);
    }
    const bool some = vs > 1.0e-30;
    vol[m] = some ? vs * rho_load : 0.0;
    hv[m] = some ? hs * rho_load : 0.0;
    hygroscopic[m] = some && hs > 1.0e-10 * vs;
    const double nraw = (ai[K::numslot(m)] + 0.0) * rho_load;
    na[m] = bound(vol[m] * C.n2v_min[m], vol[m] * C.n2v_max[m], nraw);
  }
  // activate_modal with wmaxf = 10
  if (na[0] < 1.0e-20 || w <= 0.0)
    return false;
  const double wmaxf = 10.0;
  const double twothird = 2.0 / 3.0;
  const double aten = 2.0 * (0.018016 * 1e3) * kSurften / ((kRGas * 1e3) * kT0 * kRhoH2o);
  const double it = 1.0 / tair;
  const double pres = kRAir * rho * tair;
  const double qs = qsat_trans(tair, it, pres);
  const double rqs = rho * qs, lvr = kLatvap / kRH2o * it;  // L / (Rv T)
  const double dqsdt = lvr * it * qs;
  const double alpha = kGravity * it * (lvr * (1.0 / kCpAir) - 1.0 / kRAir);
  const double gamma = fma(kLatvap / kCpAir, dqsdt, 1.0) / rqs;
  const double diff0 = 0.211e-4 * (kP0 / pres) * exp(1.94 * log(tair * (1.0 / kT0)));
  const double conduct0 = (5.69 + 0.017 * (tair - kT0)) * (4.186e2 * 1.0e-5);
  // 1 / gtherm
  const double rgth =
      kRhoH2o / (diff0 * rqs) + kLatvap * kRhoH2o * it / conduct0 * (lvr - 1.0);
  const double gtherm = 1.0 / rgth, sgth = sqrt(gtherm);
  const double bg = 2.0 * K::pi * kRhoH2o * gtherm * gamma * sgth;  // beta sqrt(gtherm)
  const double alw = alpha * w, salw = sqrt(alw);
  const double etafac1 = alw * salw;
  const double zeta = twothird * aten * salw * (rgth * sgth);
  double smc2[NMODE], eta[NMODE];
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    const double exp45 = exp(4.5 * ln_sig(m) * ln_sig(m));
    if (vol[m] > 1.0e-39 && na[m] > 1.0e-39) {
      eta[m] = etafac1 / (na[m] * bg);
      smc2[m] = hygroscopic[m]
                    ? (4.0 * aten * aten * aten * K::pi * exp45 / 20.25) * na[m] / hv[m]
                    : 1.0e4;
    } else {
      const double aw = alpha * wmaxf;
      eta[m] = etafac1 * (1.0e10 / (aw * sqrt(aw)));
      smc2[m] = 1.0;
    }
  }
  // maximum supersaturation of competing modes (maxsat, ndrop.hpp:183-242),
  // as its power -2
  const double small = 1e-20, mid = 1e5, big = 1.0 / small;
  bool weak = true;
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    weak = weak && (zeta > mid * eta[m] || smc2[m] > mid * eta[m]);
  double sum = 0.0;
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    const double f1 = 0.5 * exp(2.5 * (ln_sig(m) * ln_sig(m)));
    const double f2 = 1.0 + 0.25 * ln_sig(m);
    if (eta[m] > small) {
      const double r = zeta / eta[m];
      const double q = smc2[m] / fma(3.0, zeta, eta[m]), sq = sqrt(q);
      sum += fma(f1 * r, sqrt(r), f2 * sq * sqrt(sq)) / smc2[m];
    } else {
      sum = big;
    }
  }
  if (weak)
    sum = big * big;
  const double lnsum = log(sum);
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    const double sq2 = 1.4142135623730951;
    const double an = (log(smc2[m]) + lnsum) * (0.5 * twothird / (sq2 * ln_sig(m)));
    out[m] = 0.5 * (1.0 - erf(an));
    const double am = an - 1.5 * sq2 * ln_sig(m);
    out[4 + m] = 0.5 * (1.0 - erf(am));
    out[8 + m] = out[m] * w;
    out[12 + m] = out[4 + m] * w;
  }
  out[16] = w;
  return true;
}

}  // namespace act
}  // namespace mam4b
