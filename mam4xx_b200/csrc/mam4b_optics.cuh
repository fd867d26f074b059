// mam4b_optics.cuh -- longwave aerosol optics of a cell,
// mam4::modal_aero_opt::modal_aero_lw_k (src/mam4xx/modal_aero_opt.hpp:
// 879-989): dry and wet mode sizes (calcsize and water uptake, as the
// microphysics step computes them), then for every mode and longwave band
// the volume-mixed complex refractive index of the species and water
// (calc_refin_complex :329-410), a bilinear interpolation of the
// Chebyshev coefficients of specific absorption over the refractive-index
// table (binterp / compute_factors :412-508), their evaluation at the
// mode's surface radius (modal_size_parameters / calc_parameterized
// :192-258) and the layer's absorption optical depth.
#pragma once

#include "mam4b_activation.cuh"
#include "mam4b_physics.cuh"

namespace mam4b {
namespace opt {

constexpr int kLwBands = 16, kSwBands = 14, kNcoef = 5, kPrefr = 7, kPrefi = 10;
constexpr int kSwDiagBand = 9;  // visible band of the optical-depth diagnostic

// The tables of one band as the band kernels read them, packed on the host
// and staged whole in shared memory (doubles):
//  * species and water refractive indices as (real, imaginary) pairs, the
//    species' divided by their densities (a pair then multiplies a mass),
//    21 species in mode order, then water;
//  * per mode and refractive-index grid its running maximum, padded with
//    infinity to the length of a binary search (the reference takes the first
//    point above the index, which is the first running maximum above it in a
//    grid of any order), and the points with the reciprocals of their spacings
//    (zero where the reference does not interpolate: the last point, equal
//    points);
//  * per mode the coefficient tables, one run of kNode doubles per grid point
//    with the Chebyshev coefficients of that point next to each other (the
//    first one halved, as the sum takes it), so that a thread reads a corner
//    of its bracket with 16-byte loads.
constexpr int kSpecies = 21, kRePad = 8, kImPad = 16;
constexpr int kBandWater = 2 * kSpecies;
constexpr int kBandGrids = kBandWater + 2;
constexpr int kSearchRe = 0, kSearchIm = kRePad, kPointsRe = kRePad + kImPad,
              kPointsIm = kPointsRe + 2 * kPrefr, kGridDoubles = kPointsIm + 2 * kPrefi;
constexpr int kBandNodes = kBandGrids + NMODE * kGridDoubles;
// doubles per grid point: longwave absorption; shortwave extinction,
// absorption, asymmetry. The stride (48 and 144 bytes) spreads points over
// the banks: eight lanes reading 16 bytes of eight points whose numbers
// differ modulo 8 do not conflict.
constexpr int kLwNode = 6, kSwNode = 18;
constexpr int band_doubles(int node) { return kBandNodes + NMODE * kPrefr * kPrefi * node; }
constexpr int kLwBandDoubles = band_doubles(kLwNode), kSwBandDoubles = band_doubles(kSwNode);
// number of the first species of mode m among the 21
MAM4B_HD constexpr int species0(int m) { return K::spec0(m) - m; }

// Packs band b: specref [bands][types][2], water [bands][2], grids
// [4][bands][7 or 10], tabs coefficient tables [4][bands][5][7][10] each.
inline void pack_band(const double *specref, int ntypes, const double *water, const double *refr,
                      const double *refi, const double *const *tabs, int ntab, int node, int bands,
                      int b, double *out) {
  for (int i = 0; i < band_doubles(node); ++i)
    out[i] = 0.0;
  for (int m = 0; m < NMODE; ++m)
    for (int s = 0; s < K::nspec(m); ++s) {
      const int type = act::spectype(m, s);
      for (int k = 0; k < 2; ++k)
        out[2 * (species0(m) + s) + k] =
            specref[2 * ((size_t)b * ntypes + type - 1) + k] / act::type_dens(type);
    }
  for (int k = 0; k < 2; ++k)
    out[kBandWater + k] = water[2 * b + k];
  for (int m = 0; m < NMODE; ++m) {
    double *g = out + kBandGrids + m * kGridDoubles;
    auto grid = [&](const double *v, int n, int pad, double *search, double *points) {
      double top = -HUGE_VAL;
      for (int i = 0; i < pad; ++i) {
        if (i < n)
          top = v[i] > top ? v[i] : top;
        search[i] = i < n ? top : HUGE_VAL;
      }
      for (int i = 0; i < n; ++i) {
        const double dx = i + 1 < n ? v[i + 1] - v[i] : 0.0;
        points[2 * i] = v[i];
        points[2 * i + 1] = fabs(dx) > 1.e-20 ? 1.0 / dx : 0.0;
      }
    };
    grid(refr + ((size_t)m * bands + b) * kPrefr, kPrefr, kRePad, g + kSearchRe, g + kPointsRe);
    grid(refi + ((size_t)m * bands + b) * kPrefi, kPrefi, kImPad, g + kSearchIm, g + kPointsIm);
    double *nd = out + kBandNodes + (size_t)m * kPrefr * kPrefi * node;
    for (int q = 0; q < ntab; ++q)
      for (int c = 0; c < kNcoef; ++c)
        for (int i = 0; i < kPrefr * kPrefi; ++i)
          nd[(size_t)i * node + q * kNcoef + c] =
              tabs[q][(((size_t)m * bands + b) * kNcoef + c) * kPrefr * kPrefi + i] *
              (c == 0 ? 0.5 : 1.0);
  }
}

// species volumes of mode m over their masses
MAM4B_HD constexpr double inv_type_dens(int m, int s) { return 1.0 / act::type_dens(act::spectype(m, s)); }

// What the bands take of a mode: the Chebyshev argument, the water volume
// and the reciprocal and thousandfold of the wet volume (calc_refin_complex
// :329-410, calc_parameterized's factor 1000).
struct ModeOptics {
  double xrad, water, inv_wet, wet1000;
};
template <int M>
MAM4B_HD ModeOptics mode_optics(const double (&sp)[7], double logradsurf, double qaerwat,
                                bool shortwave) {
  const double xrmin = log(0.01e-6), xrmax = log(25.e-6);
  ModeOptics o;
  const double xrad = bound(xrmin, xrmax, logradsurf);
  o.xrad = (2.0 * xrad - xrmax - xrmin) / (xrmax - xrmin);
  double dry = 0.0;
#pragma unroll
  for (int s = 0; s < K::nspec(M); ++s)
    dry = fma(sp[s], inv_type_dens(M, s), dry);
  o.water = qaerwat / 1.0e3;
  double wet = o.water + dry;
  if (o.water < 0.0) {
    o.water = 0.0;
    wet = dry;
  }
  // the shortwave bounds the divisor below, the longwave skips the division
  o.inv_wet = shortwave ? 1.0 / dmax(wet, 1.e-40) : wet > 1.e-40 ? 1.0 / wet : 1.0;
  o.wet1000 = wet * 1.0e3;
  if (shortwave && dry < 0.0 && dry > -1.e-16)
    o.inv_wet = o.wet1000 = 0.0;  // no_optics()
  return o;
}
// A shortwave mode that contributes nothing: its dry volume is slightly below
// zero (what advection leaves of an empty mode), where the reference returns
// before any arithmetic. The divisor of its refractive index would be the
// bound 1e-40, the index as large as the volume times 1e40, the fit extrapolated
// to that beyond exp's range, and infinity times the zero volume not a number.
// The reciprocal of a volume is zero for no other finite one.
MAM4B_HD bool no_optics(const ModeOptics &o) { return o.inv_wet == 0.0 && o.wet1000 == 0.0; }

#ifdef __CUDACC__
// Bracket of ref in a grid of N points (pack_band): the point before the
// first one above ref (0 if that is the first, the last if there is none) and
// the fraction (compute_factors).
template <int N>
__device__ __forceinline__ int bracket(const double *search, const double *points, double ref,
                                       double &t) {
  int i = 0;
  if constexpr (N > 8)
    i = !(ref < search[7]) ? 8 : 0;
  i += !(ref < search[i + 3]) ? 4 : 0;
  i += !(ref < search[i + 1]) ? 2 : 0;
  i += !(ref < search[i]) ? 1 : 0;  // running maxima not above ref
  i = max(min(i, N) - 1, 0);
  const double2 p = reinterpret_cast<const double2 *>(points)[i];
  t = p.y != 0.0 ? (ref - p.x) * p.y : 0.0;
  return i;
}

// Mode M in the staged band: its refractive index (volume mixing of species
// and water) and the NQ tables bilinear in it, each a Chebyshev sum at the
// mode's radius (binterp :412-508, calc_parameterized :192-258), the sums
// taken at the bracket's corners.
template <int M, int NQ, int NODE>
__device__ __forceinline__ void mode_fit(const double *s, const double (&sp)[7],
                                         const ModeOptics &o, double (&fit)[NQ]) {
  const double2 *pairs = reinterpret_cast<const double2 *>(s);
  const double2 w = pairs[kBandWater / 2];
  double re = o.water * w.x, im = o.water * w.y;
#pragma unroll
  for (int k = 0; k < K::nspec(M); ++k) {
    const double2 v = pairs[species0(M) + k];
    re = fma(sp[k], v.x, re);
    im = fma(sp[k], v.y, im);
  }
  re *= o.inv_wet;
  im = fabs(im * o.inv_wet);
  const double *g = s + kBandGrids + M * kGridDoubles;
  double t, u;
  const int i = bracket<kPrefr>(g + kSearchRe, g + kPointsRe, re, t);
  const int j = bracket<kPrefi>(g + kSearchIm, g + kPointsIm, im, u);
  const double tu = t * u, tuc = t - tu, tcu = u - tu, tcuc = 1.0 - tuc - u;
  double cheb[kNcoef];
  cheb[0] = 1.0;
  cheb[1] = o.xrad;
#pragma unroll
  for (int c = 2; c < kNcoef; ++c)
    cheb[c] = fma(2.0 * o.xrad, cheb[c - 1], -cheb[c - 2]);
  const double *node = s + kBandNodes + (M * kPrefr * kPrefi + i * kPrefi + j) * NODE;
  const int di = i + 1 < kPrefr ? kPrefi * NODE : 0, dj = j + 1 < kPrefi ? NODE : 0;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    fit[q] = 0.0;
#pragma unroll
  for (int corner = 0; corner < 4; ++corner) {
    const double2 *p = reinterpret_cast<const double2 *>(
        node + (corner == 1 || corner == 2 ? di : 0) + (corner >= 2 ? dj : 0));
    const double wgt = corner == 0 ? tcuc : corner == 1 ? tuc : corner == 2 ? tu : tcu;
    double v[NQ * kNcoef + 1];
#pragma unroll
    for (int k = 0; k < (NQ * kNcoef + 1) / 2; ++k) {
      const double2 x = p[k];
      v[2 * k] = x.x;
      v[2 * k + 1] = x.y;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double d = v[q * kNcoef];
#pragma unroll
      for (int c = 1; c < kNcoef; ++c)
        d = fma(cheb[c], v[q * kNcoef + c], d);
      fit[q] = fma(wgt, d, fit[q]);
    }
  }
}
#endif

}  // namespace opt
}  // namespace mam4b

// ---- radiation-facing optics: the tropopause and the volcanic (CMIP6)
// stratospheric aerosol, aero_rad_props (src/mam4xx/aero_rad_props.hpp).
namespace mam4b {
namespace rad {

// R/cp of dry air and -g/R_dry (tropopause.hpp:17-30, mam4_constants.hpp)
constexpr double kRgas = 6.022214076e23 * 1.380649e-23;
constexpr double kKap = ((kRgas * 1e3) / (0.028966 * 1e3)) / 1.00464e3;
constexpr double kFaktor = -9.80616 / (kRgas / 0.028966);
constexpr double kKa1 = kKap - 1.0;

MAM4B_HD double p_kappa(double p) { return pow(p, kKap); }

// lapse rate and mean temperature between two levels in p^kappa (pk_up,
// pk_down; get_dtdz, tropopause.hpp:34-55)
MAM4B_HD void lapse_rate(double pm, double pmk, double pk_up, double pk_down, double t_up,
                         double t_down, double &dtdz, double &tm) {
  const double a1 = (t_up - t_down) / (pk_up - pk_down);
  const double b1 = t_down - a1 * pk_down;
  tm = a1 * pmk + b1;
  const double dtdp = a1 * kKap * (pow(pm, kKa1));
  dtdz = kFaktor * dtdp * pm / tm;
}

// The lapse-rate quantities of the layer between levels k - 1 and k
// (k >= 1): mean p^kappa, mean pressure, dT/dz and mean temperature, as
// twmo computes them for its scan (tropopause.hpp:114-119, 124-129,
// 171-188); the same values wherever the scan asks for them.
struct LapsePair {
  double pmk, pm, dtdz, tm;
};
template <class ColT, class ColP>
MAM4B_HD LapsePair lapse_pair(const ColT &temp, const ColP &, int k, double pk_up,
                              double pk_down) {
  LapsePair q;
  q.pmk = 0.5 * (pk_up + pk_down);
  q.pm = pow(q.pmk, (1.0 / kKap));
  lapse_rate(q.pm, q.pmk, pk_up, pk_down, temp(k - 1), temp(k), q.dtdz, q.tm);
  return q;
}
template <class ColT, class ColP>
MAM4B_HD LapsePair lapse_pair(const ColT &temp, const ColP &pmid, int k) {
  return lapse_pair(temp, pmid, k, p_kappa(pmid(k - 1)), p_kappa(pmid(k)));
}

// WMO lapse-rate tropopause of a column (twmo, Reichler et al. 2003;
// tropopause.hpp:81-204) from its layers' lapse-rate quantities pair(k),
// k = 1 .. nlev-1: scanning up from the surface, the first layer where the
// lapse rate falls below 2 K/km, between 75 and 450 hPa, and stays below
// it on average over the 2 km above. Returns its pressure, or -99 when
// there is none.
template <class Pairs>
MAM4B_HD double twmo_from_pairs(const Pairs &pair, int nlev) {
  const double gam = -0.002, plimu = 45000, pliml = 7500, deltaz = 2000.0;
  LapsePair cur = pair(nlev - 1);
  for (int k = nlev - 2; k >= 1; --k) {
    const double pmk0 = cur.pmk, dtdz0 = cur.dtdz;
    cur = pair(k);
    const double pmk = cur.pmk, pm = cur.pm, dtdz = cur.dtdz, tm = cur.tm;
    if (dtdz <= gam || pm > plimu)
      continue;
    double ptph;
    if (dtdz0 < gam) {
      const double ag = (dtdz - dtdz0) / (pmk - pmk0);
      const double bg = dtdz0 - (ag * pmk0);
      ptph = exp(log((gam - bg) / ag) / kKap);
    } else {
      ptph = pm;
    }
    if (ptph < pliml || ptph > plimu)
      continue;
    const double p2km = ptph + deltaz * (pm / tm) * kFaktor;
    double asum = 0.0;
    int icount = 0;
    for (int j = k; j >= 1; --j) {
      const LapsePair up = pair(j);
      if (up.pm > ptph)
        continue;
      if (up.pm < p2km)
        return ptph;  // the layer above stays stable: tropopause found
      asum += up.dtdz;
      icount++;
      const double aquer = asum / double(icount);
      if (aquer <= gam)
        break;  // not stable enough above: try the next level up
    }
  }
  return -99.0;
}

// tropopause_twmo's level search (tropopause.hpp:222-231) for tropopause
// pressure tp: the level k in [2, nlev-1], scanning up, whose upper
// interface pressure pint(k) lies at or below tp; 0 when tp is not
// positive or no level qualifies.
template <class ColI>
MAM4B_HD int tropopause_level_at(double tp, const ColI &pint, int nlev) {
  if (tp > 0) {
    for (int k = nlev - 1; k > 1; --k)
      if (tp >= pint(k))
        return k;
  }
  return 0;
}

// tropopause_twmo (tropopause.hpp:210-233) of one column, serially.
template <class ColT, class ColP, class ColI>
MAM4B_HD int tropopause_level(const ColT &temp, const ColP &pmid, const ColI &pint, int nlev) {
  auto pair = [&](int k) { return lapse_pair(temp, pmid, k); };
  return tropopause_level_at(twmo_from_pairs(pair, nlev), pint, nlev);
}

}  // namespace rad
}  // namespace mam4b
