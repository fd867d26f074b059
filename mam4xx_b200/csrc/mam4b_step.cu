// mam4b_step.cu -- sm_100a kernels and the C ABI (include/mam4b.h) of the
// B200-native MAM4 microphysics step.
//
// The step (calcsize -> water uptake -> amicphys) is a pipeline of kernels
// (StepArgs) whose threads own a cell, a mode or a mode pair of a cell, or an
// SOA loop; inputs, outputs and hand-off are structure-of-arrays fields, so
// each load/store instruction of a warp touches 32 consecutive doubles. Cells
// are independent; the two modes of a block of the front stage exchange a few
// values through shared memory. The coagulation correction tables are read
// through L1.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "../../include/mam4b.h"
#include "mam4b_physics.cuh"
#include "mam4b_physics_mixed.cuh"
#include "mam4b_adjoint.cuh"
#include "mam4b_process.cuh"
#include "mam4b_setsox.cuh"
#include "mam4b_gaschem.cuh"
#include "mam4b_activation.cuh"
#include "mam4b_dropmix.cuh"
#include "mam4b_optics.cuh"

namespace mam4b {

// ------------------------------------------------------- device constants
__constant__ StepConsts c_k;

#define COAG_TABLE_QUALIFIER __device__ const
#include "coag_tables.inc"
#undef COAG_TABLE_QUALIFIER

struct StepArgs {
  const double *in[MAM4B_NIN];
  const double *pblh;
  double *out[MAM4B_NOUT];
  double *diag[MAM4B_NDIAG];
  unsigned *flags;
  long long ncell;
  int nlev;
  double dt;
  int do_cond, do_rename, do_newnuc, do_coag, optaa;
  unsigned nmono;
  // SOA solver hand-off (see soa_kernel): per-cell loop state, the list of
  // queued cells, the solver's order and counters (CNT_*)
  double *soa;       // [SOA_FIELDS][ncell]
  double *hand;      // [H_FIELDS][ncell]
  int *done;         // [ncell]: cells that pre_kernel<.., FUSE> finished
  int *order;        // [ncell]: cells in solver order, long loops from the
                     // front, short ones from the back
  double *aux;       // [AUX_FIELDS][ncell], indexed by cell (front and mode kernels)
  unsigned *counters;
  int *npass;        // [ncell] or null: passes of each cell's loop (adjoint only)
  int mixed;         // the mode/pair stages ran in FP32 (MAM4B_MIXED, _FAST)
  double long_steps;    // a loop is long (soa_kernel runs it first) when its
                        // first sub-step is shorter than dt / long_steps
  int quads;            // long loops run four lanes to a loop (soa_long_loops)
  double inline_scale;  // pre_kernel<.., FUSE>: cells whose first SOA sub-step
                        // is at least 1/inline_scale of the step finish in pre
};

// The step runs as a pipeline of six kernels when condensation is on:
// front_kernel runs calcsize, the humidity of
// water uptake, the subarea set-up and the cloudy subarea, and leaves the
// clear subarea at its SOA condensation loop in scratch (cloudy
// cells finish there); mode_kernel and pair_kernel compute water uptake,
// uptake rates and coagulation coefficients; pre_kernel adds the uptake
// rates and orders the loops; soa_kernel runs them with per-lane work
// stealing; post_kernel finishes the queued cells from the hand-off and the
// loop result. With process tendencies the front stage stores some of them
// and post_diag_kernel the others. With chemistry, which runs between
// calcsize's update and the subareas, front_kernel's work is that of
// chem_size_kernel, chem_cell_kernel and chem_subarea_kernel. Without
// condensation full_kernel or chem_step_kernel runs each cell start to end in
// one thread.
enum { SOA_G = 0, SOA_A = 1, SOA_OPOA = 5, SOA_UPTK = 9, SOA_G0 = 13, SOA_FIELDS = 14 };
// per-cell values from the first two stages for the later ones:
// relative humidity for water uptake, H2SO4 diffusivity and mean free path,
// per-particle H2SO4 uptake rate of each mode
// and the 12 coagulation coefficients (coag_all_coefs order)
enum { AUX_RH = 0, AUX_GDIFF = 1, AUX_FPATH = 2, AUX_RATE = 3, AUX_COAG = 7, AUX_FIELDS = 19 };
// with chemistry, until pair_kernel fills the coagulation rows: cloud-borne SO4
// of modes 1-3 after cloud chemistry; SOAG and H2SO4 before it and after it
enum { AUX_CHEM_SO4 = AUX_COAG, AUX_CHEM_GAS = AUX_COAG + 3 };
// queue counters: long and short loops in the order list, short and long
// loops handed to the solver, and to the adjoint's
enum { CNT_TAKEN = 0, CNT_LONG = 1, CNT_SHORT = 2, CNT_TAKEN_ADJ = 3, CNT_TAKEN_LONG = 4,
       CNT_TAKEN_ADJ_LONG = 5, CNT_WORDS = 8 };
// Cells with a cloud fraction above this are cloudy throughout: they have no
// clear subarea and no SOA loop.
constexpr double kCloudy = 0.999;

// ----------------------------------------------------- per-cell amicphys
__device__ __forceinline__ constexpr int pop_to_i31(int p) { return 6 + p; }
// amicphys tracer index of the number of mode m (mam4_amicphys.hpp:36)
__device__ __forceinline__ constexpr int num_i31(int m) {
  return m == 0 ? 13 : m == 1 ? 18 : m == 2 ? 26 : 30;
}

// Process tendencies of a grid cell, in the 31-tracer order ([process
// 0..3][tracer], then cloud-borne renaming [tracer]), straight to the
// caller's arrays, which may be absent. Every one is a single term, but that
// renaming in a partly cloudy cell is the clear subarea's plus the cloudy
// one's, which was stored first (`joined`). Increments come in amicphys
// units over the step: volume mixing ratio times unit (the unit factor of
// the species), scaled by the subarea's fraction.
struct Diag {
  const StepArgs &a;
  long long c;
  bool joined;
  __device__ __forceinline__ Diag(const StepArgs &a_, long long c_) : a(a_), c(c_), joined(false) {}
  // increment v of a population of species x (number: x < 0)
  __device__ __forceinline__ double rate(int x, double v) const {
    return (0.0 + v) / ((x == 0 || x == 2 ? K::fcvt_aer(0) : 1.0) * a.dt);
  }
  __device__ __forceinline__ void put(int k, int i, double t) const {
    double *d = a.diag[k * 31 + i];
    if (d)
      d[c] = k == 1 && joined ? (0.0 + t) + d[c] : 0.0 + t;
  }
};

// Zeros to the fields that a cell leaves without a term: bit i of fields[k] is
// tracer i of process k.
__device__ __forceinline__ void diag_zeros(const StepArgs &a, long long c,
                                           const unsigned (&fields)[NQTEND + 1]) {
#pragma unroll 1
  for (int k = 0; k <= NQTEND; ++k)
#pragma unroll 1
    for (int i = 0; i < 31; ++i)
      if (((fields[k] >> i) & 1u) && a.diag[31 * k + i])
        a.diag[31 * k + i][c] = 0.0;
}

// Hand-off of a cell with a clear subarea from the first stage to the later
// ones: one double per field and cell.
enum {
  H_GAS1 = 0,      // H2SO4 of the clear subarea at the loop
  H_POP = 1,       // 25 numbers/masses of the clear subarea at the loop
  H_UPTK = 26,     // 4 H2SO4 uptake rates
  H_NETPROD = 30,  // H2SO4 net production of other processes
  H_SV_SO4 = 31,   // aitken SO4 and SOA before condensation
  H_SV_SOA = 32,
  H_DGN_PC = 33,   // dry diameter of the primary-carbon mode
  H_RELHUM = 34,   // relative humidity of the clear subarea
  H_CI = 35,       // 25 interstitial contributions of the cloudy subarea
  H_CG = 60,       // 2 gas contributions of the cloudy subarea (SOAG, H2SO4)
  H_SOAG0 = 62,    // SOA gas at the start of the loop (read by the adjoint)
  H_FIELDS = 63
};
// (The outgoing cloud-borne grid means are final once the subareas are set up:
// the clear subarea does not change them. front_out writes their tendencies, so
// they are not handed off.)

// Clear subarea, mam_amicphys_1subarea (mam4_amicphys.hpp:1127-1697), part 1:
// optaa-2 production split and H2SO4 uptake rates from the per-particle
// rates `rate` (uptake_rates). Returns the SOAG uptake rates for the SOA
// loop.
template <bool DIAG>
__device__ __forceinline__ void clear_prefix(const StepArgs &a, double deltat, double temp,
                                             double pmid, const double (&rate)[NMODE],
                                             const double (&qgas1)[2], Sub &s, ClearMid &cm,
                                             double (&uptk0)[NMODE]) {
  const double aircon = pmid / (8314.46759100000 * temp);
  cm.netprod1 = 0.0;
  if (a.do_cond && a.optaa == 2) {
    cm.netprod1 = (s.gas[1] - qgas1[1]) / deltat;
    s.gas[1] = (cm.netprod1 >= 0) ? qgas1[1] : 0;
  }
  if (!a.do_cond)
    return;
  cm.gas_sv[0] = s.gas[0];
  cm.gas_sv[1] = s.gas[1];
  cm.sv_so4_ait = s.aer[1][1];
  cm.sv_soa_ait = s.aer[0][1];
  if (DIAG) {
#pragma unroll
    for (int x = 0; x < NAER; ++x)
#pragma unroll
      for (int m = 0; m < NMODE; ++m)
        cm.sv_all[x][m] = s.aer[x][m];
  }
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    cm.uptk1[n] = rate[n] * (s.num[n] * aircon);
    uptk0[n] = cm.uptk1[n] * 0.81;
  }
}

// Part 2, after the SOA loop: H2SO4 update, renaming, nucleation,
// coagulation, aging. With DIAG the per-process increments go to dg, scaled
// by afrac. With PRECOAG, cc_pre (stride cc_stride)
// holds the 12 coagulation coefficients of the cell (coag_all_coefs) and
// dgn_awet/wetdens are not read.
template <bool DIAG, bool PRECOAG>
__device__ __forceinline__ void clear_suffix(const StepArgs &a, double deltat, double temp,
                                             double pmid, double zmid, double pblh,
                                             double relhum, double dgn_a_pc,
                                             const double (&dgn_awet)[NMODE],
                                             const double (&wetdens)[NMODE], const ClearMid &cm,
                                             Sub &s, Diag *dg, double afrac,
                                             const double *cc_pre, size_t cc_stride) {
  const StepConsts &C = c_k;
  const double aircon = pmid / (8314.46759100000 * temp);
  const double dtsub = (double)(int)(deltat / 1);
  double qgas_avg1 = s.gas[1];
  double uptkrate_h2so4 = 0.0;
  // the primary-carbon mode holds no SO4/SOA before condensation, so its
  // condensation gains are its values after it
  double cond_so4_pc = 0.0, cond_soa_pc = 0.0;
  double dcond[NAER][NMODE], dcoag[NAER][NMODE], dncond[NMODE], dncoag[NMODE];
  if (DIAG) {
#pragma unroll
    for (int x = 0; x < NAER; ++x)
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        dcond[x][m] = 0.0;
        dcoag[x][m] = 0.0;
      }
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      dncond[m] = 0.0;
      dncoag[m] = 0.0;
    }
  }
  double grow[NAER];
#pragma unroll
  for (int x = 0; x < NAER; ++x)
    grow[x] = 0.0;

  if (a.do_cond) {
#pragma unroll
    for (int n = 0; n < NMODE; ++n)
      uptkrate_h2so4 += cm.uptk1[n];
    h2so4_update(dtsub, cm.netprod1, s, cm.uptk1, qgas_avg1);
    // growth of the aitken mode by condensation: only SO4 and SOA change
    grow[1] = s.aer[1][1] - cm.sv_so4_ait;
    grow[0] = s.aer[0][1] - cm.sv_soa_ait;
    cond_so4_pc = s.aer[1][3] - 0.0;
    cond_soa_pc = s.aer[0][3] - 0.0;
    if (DIAG) {
#pragma unroll
      for (int x = 0; x < NAER; ++x)
#pragma unroll
        for (int m = 0; m < NMODE; ++m)
          dcond[x][m] = s.aer[x][m] - cm.sv_all[x][m];
      // gas increment of condensation (mam4_amicphys.hpp:1434-1438)
      dg->put(0, 5, ((0.0 + (s.gas[0] - (cm.gas_sv[0] + 0.0 * dtsub))) / (C.fcvt_soag * a.dt)) * afrac);
      dg->put(0, 2, dg->rate(-1, s.gas[1] - (cm.gas_sv[1] + cm.netprod1 * dtsub)) * afrac);
    }
  }

  // -------------------------------------------------------- renaming
  if (a.do_rename) {
    double nsv[NMODE], asv[NAER][NMODE];
    if (DIAG) {
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        nsv[m] = s.num[m];
#pragma unroll
        for (int x = 0; x < NAER; ++x)
          asv[x][m] = s.aer[x][m];
      }
    }
    const double zero7[NAER] = {0, 0, 0, 0, 0, 0, 0};
    rename_subarea<false>(C, s, s, grow, zero7);
    if (DIAG) {
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        dg->put(1, num_i31(m), dg->rate(-1, s.num[m] - nsv[m]) * afrac);
#pragma unroll
        for (int x = 0; x < NAER; ++x) {
          const int slot = K::aer_slot(x, m);
          if (slot >= 0)
            dg->put(1, pop_to_i31(slot), dg->rate(x, s.aer[x][m] - asv[x][m]) * afrac);
        }
      }
    }
  }

  // ------------------------------------------------------ nucleation
  if (a.do_newnuc) {
    const double g1 = s.gas[1], n1 = s.num[1], a1 = s.aer[1][1];
    nucleation(C, dtsub, temp, pmid, zmid, pblh, relhum, uptkrate_h2so4, qgas_avg1, s);
    if (DIAG) {
      dg->put(2, 2, dg->rate(-1, s.gas[1] - g1) * afrac);
      dg->put(2, 18, dg->rate(-1, s.num[1] - n1) * afrac);
      dg->put(2, 14, dg->rate(1, s.aer[1][1] - a1) * afrac);
    }
  }

  // ----------------------------------------------------- coagulation
  double coag_in[NAER];
  if (a.do_coag) {
    double nsv[NMODE], asv[NAER][NMODE];
    if (DIAG) {
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        nsv[m] = s.num[m];
#pragma unroll
        for (int x = 0; x < NAER; ++x)
          asv[x][m] = s.aer[x][m];
      }
    }
    double cc[12];
    if (PRECOAG) {
      // coefficients from pair_kernel
#pragma unroll
      for (int k = 0; k < 12; ++k)
        cc[k] = cc_pre[k * cc_stride];
    } else {
      const CoagTables T = {kCoagBm0ij, kCoagBm3i, kCoagBm0};
      coag_all_coefs(C, T, temp, pmid, aircon, dgn_awet, wetdens, cc);
    }
    coagulation(dtsub, cc, s, coag_in);
    if (DIAG) {
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        dncoag[m] = s.num[m] - nsv[m];
#pragma unroll
        for (int x = 0; x < NAER; ++x)
          dcoag[x][m] = s.aer[x][m] - asv[x][m];
      }
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        dg->put(3, num_i31(m), dg->rate(-1, dncoag[m]) * afrac);
#pragma unroll
        for (int x = 0; x < NAER; ++x) {
          const int slot = K::aer_slot(x, m);
          if (slot >= 0)
            dg->put(3, pop_to_i31(slot), dg->rate(x, dcoag[x][m]) * afrac);
        }
      }
    }
  } else {
#pragma unroll
    for (int x = 0; x < NAER; ++x)
      coag_in[x] = 0.0;
  }

  // ----------------------------------------------------------- aging
  if (DIAG) {
    aging(C, a.nmono, dgn_a_pc, s, dncond, dncoag, dcond, dcoag, coag_in);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      if (a.do_cond)
        dg->put(0, num_i31(m), dg->rate(-1, dncond[m]) * afrac);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0 && a.do_cond)
          dg->put(0, pop_to_i31(slot), dg->rate(x, dcond[x][m]) * afrac);
      }
    }
  } else {
    // Only the primary-carbon condensation gains of SO4/SOA enter the aging
    // fraction; the other increments are bookkeeping for diagnostics.
    double dn_c[NMODE] = {0, 0, 0, 0}, dn_g[NMODE] = {0, 0, 0, 0};
    double dc[NAER][NMODE], dq[NAER][NMODE];
#pragma unroll
    for (int x = 0; x < NAER; ++x)
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        dc[x][m] = 0.0;
        dq[x][m] = 0.0;
      }
    dc[1][3] = cond_so4_pc;
    dc[0][3] = cond_soa_pc;
    aging(C, a.nmono, dgn_a_pc, s, dn_c, dn_g, dc, dq, coag_in);
  }
}

// Whole clear subarea in one thread: part 1, the SOA loop inline, part 2.
// Returns the SOA sub-step count.
template <bool DIAG>
__device__ __forceinline__ int clear_subarea(const StepArgs &a, double deltat, double temp,
                                             double pmid, double zmid, double pblh,
                                             double relhum, const double (&dgn_a)[NMODE],
                                             const double (&dgn_awet)[NMODE],
                                             const double (&wetdens)[NMODE],
                                             const double (&qgas1)[2], Sub &s, Diag *dg,
                                             double afrac) {
  ClearMid cm;
  double uptk0[NMODE], rate[NMODE] = {0, 0, 0, 0};
  if (a.do_cond) {
    double gas_diffus, freepath;
    h2so4_diffusivity(temp, pmid, gas_diffus, freepath);
    uptake_rates(c_k, gas_diffus, freepath, dgn_awet, rate);
  }
  clear_prefix<DIAG>(a, deltat, temp, pmid, rate, qgas1, s, cm, uptk0);
  int niter = 0;
  if (a.do_cond)
    niter = soa_exchange((double)(int)(deltat / 1), temp, pmid, s, uptk0);
  clear_suffix<DIAG, false>(a, deltat, temp, pmid, zmid, pblh, relhum, dgn_a[3], dgn_awet, wetdens, cm, s,
                     dg, afrac, nullptr, 0);
  return niter;
}

// Tendencies of the 25 cloud-borne populations from their outgoing grid
// means oc (vmr) and incoming values ac (mmr).
__device__ __forceinline__ void store_cloudborne(const StepArgs &a, long long c,
                                                 const double (&oc)[NPOP],
                                                 const double (&ac)[NPOP]) {
  const StepConsts &C = c_k;
  const double dt = a.dt;
  double *const *out = a.out;
#pragma unroll
  for (int p = 0; p < NPOP; ++p)
    out[MAM4B_OUT_TEND + 27 + p][c] = (oc[p] * C.to_mmr[2 + p] - ac[p]) / dt;
}

// Tendencies of the gases and the 25 interstitial populations. The changes are
// formed first: the group of quotients then holds nothing but them
// (post_kernel with the division alone 0.54 ms on 16,384 x 72 cells, now 0.44).
__device__ __forceinline__ void store_interstitial(const StepArgs &a, long long c, double o_h2so4,
                                                   double o_soag, const double (&oi)[NPOP],
                                                   double h2so4, double soag,
                                                   const double (&ai)[NPOP]) {
  const StepConsts &C = c_k;
  const double dt = a.dt;
  double *const *out = a.out;
  double change[NPOP + 2];
  change[0] = o_h2so4 * C.to_mmr[0] - h2so4;
  change[1] = o_soag * C.to_mmr[1] - soag;
#pragma unroll
  for (int p = 0; p < NPOP; ++p)
    change[2 + p] = oi[p] * C.to_mmr[2 + p] - ai[p];
  with_quotients([&](auto &q) {
    const Divisor per_dt = q.divisor(dt);
#pragma unroll
    for (int k = 0; k < NPOP + 2; ++k)
      out[MAM4B_OUT_TEND + k][c] = q.under(per_dt, change[k]);
  });
}

__device__ __forceinline__ void store_outputs(const StepArgs &a, long long c, double o_h2so4,
                                              double o_soag, const double (&oi)[NPOP],
                                              const double (&oc)[NPOP], double h2so4, double soag,
                                              const double (&ai)[NPOP], const double (&ac)[NPOP]) {
  store_interstitial(a, c, o_h2so4, o_soag, oi, h2so4, soag, ai);
  store_cloudborne(a, c, oc, ac);
}

// Per-cell state after calcsize and water uptake (modal_aero_calcsize_sub,
// modal_aero_water_uptake_dr), in amicphys units where amicphys reads it.
struct Front {
  double temp, pmid, zm, qv, cld, h2so4, soag, pblh;
  double ai[NPOP], ac[NPOP];          // populations as passed in (mmr)
  double dgn_a[NMODE], dgn_awet[NMODE], wetdens[NMODE];
  double qi[NPOP], qc[NPOP];          // after the calcsize update (vmr)
  double g_h2so4, g_soag;             // gases (vmr)
  double relhumgcm;
};

// Relative humidity of the cell as amicphys diagnoses it
// (mam4_amicphys.hpp:2199-2205)
__device__ __forceinline__ double relhum_gcm(double qv, double temp, double pmid) {
  const double epsqs = 0.018016 / 0.028966;
  const double tc = temp - 273.15;
  const double ew = 610.94 * exp(17.625 * tc / (234.04 + tc));
  const double ev_sat = 1.00071 * exp(4.5e-8 * pmid) * ew;
  const double qv_sat = epsqs * ev_sat / (pmid - (1 - epsqs) * ev_sat);
  return dmax(0.0, dmin(1.0, qv / qv_sat));
}

// Loads the cell, checks it, runs calcsize and water uptake, writes the
// size outputs and prepares the amicphys inputs: the part of
// modal_aero_amicphys_intr (mam4_amicphys.hpp:2120-2260) before the
// subarea loop, with q_pregaschem = q_precldchem = qq and
// qqcw_precldchem = qqcw.
__device__ __forceinline__ void cell_front(const StepArgs &a, const long long c, Front &f) {
  const StepConsts &C = c_k;
  f.temp = __ldg(a.in[MAM4B_IN_T] + c);
  f.pmid = __ldg(a.in[MAM4B_IN_P] + c);
  f.zm = __ldg(a.in[MAM4B_IN_ZM] + c);
  f.qv = __ldg(a.in[MAM4B_IN_QV] + c);
  f.cld = __ldg(a.in[MAM4B_IN_CLD] + c);
  f.h2so4 = __ldg(a.in[MAM4B_IN_H2SO4] + c);
  f.soag = __ldg(a.in[MAM4B_IN_SOAG] + c);
  f.pblh = __ldg(a.pblh + c / a.nlev);
  const double dt = a.dt;
#pragma unroll
  for (int p = 0; p < NPOP; ++p) {
    f.ai[p] = __ldg(a.in[MAM4B_IN_AER_I + p] + c);
    f.ac[p] = __ldg(a.in[MAM4B_IN_AER_C + p] + c);
  }
  {
    double chk = f.temp + f.pmid + f.zm + f.qv + f.cld + f.h2so4 + f.soag + f.pblh;
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      chk += f.ai[p] + f.ac[p];
    if (!isfinite(chk))
      atomicOr(a.flags, MAM4B_FLAG_NONFINITE_INPUT);
  }
  double pt_i[NPOP], pt_c[NPOP];
  calcsize(C, f.ai, f.ac, dt, f.dgn_a, pt_i, pt_c);
  double wetdens_wu[NMODE];
  double qaerwat[NMODE];
  water_uptake(C, f.ai, f.qv, f.temp, f.pmid, f.cld, f.dgn_a, f.dgn_awet, qaerwat, wetdens_wu);
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    a.out[MAM4B_OUT_DGN_A + m][c] = f.dgn_a[m];
    a.out[MAM4B_OUT_DGN_AWET + m][c] = f.dgn_awet[m];
    a.out[MAM4B_OUT_WETDENS + m][c] = wetdens_wu[m];
    a.out[MAM4B_OUT_QAERWAT + m][c] = qaerwat[m];
  }
  // calcsize tendencies applied for one step, then amicphys units
#pragma unroll
  for (int p = 0; p < NPOP; ++p) {
    f.qi[p] = dmax(0.0, dmax(0.0, f.ai[p] + pt_i[p] * dt) * C.to_vmr[2 + p]);
    f.qc[p] = dmax(0.0, dmax(0.0, f.ac[p] + pt_c[p] * dt) * C.to_vmr[2 + p]);
  }
  f.g_h2so4 = dmax(0.0, f.h2so4 * C.to_vmr[0]);
  f.g_soag = dmax(0.0, f.soag * C.to_vmr[1]);
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    f.wetdens[m] = dmax(1000.0, wetdens_wu[m]);
  f.relhumgcm = relhum_gcm(f.qv, f.temp, f.pmid);
}

// Renaming of a cloudy (sub)area, interstitial si and cloud-borne sc,
// weighted by f; adds the renaming diagnostics when DIAG.
template <bool DIAG>
__device__ __forceinline__ void cloudy_rename(const StepArgs &a, Sub &si, Sub &sc, double f,
                                              Diag *dg) {
  const StepConsts &C = c_k;
  si.gas[0] = si.gas[1] = sc.gas[0] = sc.gas[1] = 0.0;
  double nsv_i[NMODE], nsv_c[NMODE], asv_i[NAER][NMODE], asv_c[NAER][NMODE];
  if (DIAG) {
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      nsv_i[m] = si.num[m];
      nsv_c[m] = sc.num[m];
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        asv_i[x][m] = si.aer[x][m];
        asv_c[x][m] = sc.aer[x][m];
      }
    }
  }
  if (a.do_rename) {
    const double zero7[NAER] = {0, 0, 0, 0, 0, 0, 0};
    rename_subarea<true>(C, si, sc, zero7, zero7);
  }
  if (DIAG && a.do_rename) {
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      const int ln = num_i31(m);
      dg->put(1, ln, dg->rate(-1, si.num[m] - nsv_i[m]) * f);
      dg->put(NQTEND, ln, dg->rate(-1, sc.num[m] - nsv_c[m]) * f);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0) {
          dg->put(1, pop_to_i31(slot), dg->rate(x, si.aer[x][m] - asv_i[x][m]) * f);
          dg->put(NQTEND, pop_to_i31(slot), dg->rate(x, sc.aer[x][m] - asv_c[x][m]) * f);
        }
      }
    }
  }
}

// Cloudy grid cell (cloud fraction > 0.999): renaming only.
template <bool DIAG>
__device__ __forceinline__ void cloudy_cell(const StepArgs &a, const Front &f, double &o_h2so4,
                                            double &o_soag, double (&oi)[NPOP],
                                            double (&oc)[NPOP], Diag *dg) {
  Sub si, sc;
  load_sub_plain(si, f.qi);
  load_sub_plain(sc, f.qc);
  const double w = 1.0;
  cloudy_rename<DIAG>(a, si, sc, w, dg);
  o_soag = dmax(0.0, 0.0 + f.g_soag * w);
  o_h2so4 = dmax(0.0, 0.0 + f.g_h2so4 * w);
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    oi[K::numslot(m)] = dmax(0.0, 0.0 + (si.num[m] / 1.0) * w);
    oc[K::numslot(m)] = 0.0 + (sc.num[m] / 1.0) * w;
#pragma unroll
    for (int x = 0; x < NAER; ++x) {
      const int slot = K::aer_slot(x, m);
      if (slot >= 0) {
        oi[slot] = dmax(0.0, 0.0 + (si.aer[x][m] / K::fcvt_aer(x)) * w);
        oc[slot] = 0.0 + (sc.aer[x][m] / K::fcvt_aer(x)) * w;
      }
    }
  }
}

// Partly cloudy grid cell, set-up of both subareas and the cloudy one
// (jsub 2, renaming only): the clear subarea's incoming state s, its gases
// and relative humidity, and the cloudy subarea's contributions to the
// grid means (ci interstitial, cg gases SOAG/H2SO4, oc cloud-borne).
// Partition factors: get_partition_factors (mam4_amicphys.hpp:414-449).
template <bool DIAG>
__device__ __forceinline__ void partly_cloudy_setup(const StepArgs &a, const Front &f, Sub &s,
                                                    double (&gcl)[2], double &rhc,
                                                    double (&ci)[NPOP], double (&cg)[2],
                                                    double (&oc)[NPOP], Diag *dg) {
  const StepConsts &C = c_k;
  const double fcldy = f.cld, fclea = 1.0 - fcldy;
  double fn_c[NMODE], fn_y[NMODE], fm_c[NMODE], fm_y[NMODE];
  auto part = [&](double q_i, double q_c, double &fc, double &fy) {
    const double cldbrn_cldy = q_c / fcldy;
    const double intrst_cldy = dmax(0.0, ((q_i + q_c) - cldbrn_cldy));
    const double intrst_clea = (q_i - fcldy * intrst_cldy) / fclea;
    double r = dmax(1.e-35, intrst_clea * fclea) / dmax(1.e-35, q_i);
    r = dmax(0.0, dmin(1.0, r));
    fc = r / fclea;
    fy = (1 - r) / fcldy;
  };
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    part(f.qi[K::numslot(m)], f.qc[K::numslot(m)], fn_c[m], fn_y[m]);
    double si_ = 0.0, sc_ = 0.0;
#pragma unroll
    for (int k = 0; k < K::nspec(m); ++k) {
      si_ = si_ + f.qi[K::spec0(m) + k];
      sc_ = sc_ + f.qc[K::spec0(m) + k];
    }
    part(si_, sc_, fm_c[m], fm_y[m]);
  }
  // gases: clear keeps the grid mean, cloudy gets the remainder
  double gcy[2];
  gcl[0] = f.g_soag;
  gcl[1] = f.g_h2so4;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    gcy[g] = (gcl[g] - fclea * gcl[g]) / fcldy;
    if (gcy[g] < 0) {
      gcy[g] = 0;
      gcl[g] = gcl[g] / fclea;
    }
  }
  rhc = bound(0.0, 1.0, (f.relhumgcm - fcldy) / fclea);
  {
    Sub si, sc;
    load_sub(si, f.qi, fn_y, fm_y);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      sc.num[m] = (f.qc[K::numslot(m)] / fcldy) * 1;
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        sc.aer[x][m] = (slot >= 0) ? (f.qc[slot] / fcldy) * K::fcvt_aer(x) : 0.0;
      }
    }
    cloudy_rename<DIAG>(a, si, sc, fcldy, dg);
    cg[0] = gcy[0] * fcldy;
    cg[1] = gcy[1] * fcldy;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      ci[K::numslot(m)] = (si.num[m] / 1.0) * fcldy;
      oc[K::numslot(m)] = (0.0 + 0.0 * fclea) + (sc.num[m] / 1.0) * fcldy;
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0) {
          ci[slot] = (si.aer[x][m] / K::fcvt_aer(x)) * fcldy;
          oc[slot] = (0.0 + 0.0 * fclea) + (sc.aer[x][m] / K::fcvt_aer(x)) * fcldy;
        }
      }
    }
  }
  load_sub(s, f.qi, fn_c, fm_c);
  s.gas[0] = gcl[0] * C.fcvt_soag;
  s.gas[1] = gcl[1] * 1.0;
}

// One grid cell start to end in one thread (modal_aero_amicphys_intr,
// mam4_amicphys.hpp:2120-2376): the diagnostics path, and the whole step
// when condensation is off (no SOA loop to pipeline).
template <bool DIAG>
__device__ __forceinline__ void cell_step(const StepArgs &a, const long long c) {
  const StepConsts &C = c_k;
  Front f;
  cell_front(a, c, f);
  const double dt = a.dt;
  Diag dgv(a, c);
  Diag *dg = DIAG ? &dgv : nullptr;
  if (DIAG)
    diag_zeros(a, c, {~0u, ~0u, ~0u, ~0u, ~0u});
  // outgoing grid-cell means (amicphys units): gases, interstitial, cloud
  double o_h2so4, o_soag, oi[NPOP], oc[NPOP];
  const double fsoag = C.fcvt_soag;
  const bool map_gas = a.do_cond || a.do_newnuc;
  const double qgas1[2] = {f.g_soag * fsoag, f.g_h2so4 * 1.0};

  if (f.cld > kCloudy) {
    cloudy_cell<DIAG>(a, f, o_h2so4, o_soag, oi, oc, dg);
  } else if (f.cld < 1.0e-5) {
    // clear grid cell: the subarea is the grid mean
    Sub s;
    load_sub_plain(s, f.qi);
    s.gas[0] = f.g_soag * fsoag;
    s.gas[1] = f.g_h2so4 * 1.0;
    const int niter = clear_subarea<DIAG>(a, dt, f.temp, f.pmid, f.zm, f.pblh, f.relhumgcm,
                                                f.dgn_a, f.dgn_awet, f.wetdens, qgas1, s, dg, 1.0);
    if (niter > 1000)
      atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
    const double w = 1.0 - 0.0;
    o_soag = dmax(0.0, 0.0 + (map_gas ? s.gas[0] / fsoag : f.g_soag) * w);
    o_h2so4 = dmax(0.0, 0.0 + (map_gas ? s.gas[1] / 1.0 : f.g_h2so4) * w);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] = dmax(0.0, 0.0 + (s.num[m] / 1.0) * w);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0)
          oi[slot] = dmax(0.0, 0.0 + (s.aer[x][m] / K::fcvt_aer(x)) * w);
      }
    }
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      oc[p] = f.qc[p];
  } else {
    // partly cloudy grid cell: cloudy subarea first (its contributions are
    // added after the clear subarea's, as in the reference's jsub order)
    const double fclea = 1.0 - f.cld;
    Sub s;
    double gcl[2], rhc, ci[NPOP], cg[2];
    partly_cloudy_setup<DIAG>(a, f, s, gcl, rhc, ci, cg, oc, dg);
    dgv.joined = true;
    const int niter = clear_subarea<DIAG>(a, dt, f.temp, f.pmid, f.zm, f.pblh, rhc, f.dgn_a,
                                                f.dgn_awet, f.wetdens, qgas1, s, dg, fclea);
    if (niter > 1000)
      atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
    o_soag = dmax(0.0, (0.0 + (map_gas ? s.gas[0] / fsoag : gcl[0]) * fclea) + cg[0]);
    o_h2so4 = dmax(0.0, (0.0 + (map_gas ? s.gas[1] / 1.0 : gcl[1]) * fclea) + cg[1]);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] = dmax(0.0, (0.0 + (s.num[m] / 1.0) * fclea) + ci[K::numslot(m)]);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0)
          oi[slot] = dmax(0.0, (0.0 + (s.aer[x][m] / K::fcvt_aer(x)) * fclea) + ci[slot]);
      }
    }
  }

  store_outputs(a, c, o_h2so4, o_soag, oi, oc, f.h2so4, f.soag, f.ai, f.ac);
}

// ---- the step with the chemistry that precedes amicphys, one thread per
// cell: calcsize and water uptake, the calcsize update, then gas-phase
// chemistry (gas_phase_chemistry.hpp:40) and aqueous chemistry
// (mo_setsox.hpp:944) on the cell's 31 tracers, then amicphys with the three
// states the chemistry leaves: before gas chemistry (q_pregaschem), before
// cloud chemistry (q_precldchem, qqcw_precldchem) and after it (qq, qqcw).
struct ChemArgs {
  const double *in;  // [MAM4B_CHEM_NIN][ld]
  double *out;       // [MAM4B_CHEM_NOUT][ld]
  size_t ld;
};

// amicphys-unit states before the chemistry, clipped at zero as amicphys
// clips its inputs (mam4_amicphys.hpp:2258-2267)
struct ChemPre {
  double g1[2];               // SOAG, H2SO4 before gas chemistry
  double g2[2];               // SOAG, H2SO4 before cloud chemistry
  double qi2[NPOP], qc2[NPOP];  // populations before cloud chemistry
};

// Renaming in a cloudy (sub)area whose populations grew by cloud chemistry:
// the growth increments of the aitken mode are the change from the
// before-cloud-chemistry state (mam4_amicphys.hpp:1440-1455; no
// condensation in a cloudy subarea).
__device__ __forceinline__ void cloudy_rename_grown(const StepArgs &a, Sub &si, Sub &sc,
                                                    const Sub &si2, const Sub &sc2) {
  const StepConsts &C = c_k;
  si.gas[0] = si.gas[1] = sc.gas[0] = sc.gas[1] = 0.0;
  if (!a.do_rename)
    return;
  double gi[NAER], gc[NAER];
#pragma unroll
  for (int x = 0; x < NAER; ++x) {
    gi[x] = (si.aer[x][1] - si2.aer[x][1]) / 1 + 0.0;
    gc[x] = (sc.aer[x][1] - sc2.aer[x][1]) / 1;
  }
  rename_subarea<true>(C, si, sc, gi, gc);
}

// Cloudy grid cell (cloud fraction > 0.999) after chemistry.
__device__ __forceinline__ void cloudy_cell_chem(const StepArgs &a, const Front &f,
                                                 const ChemPre &cp, double &o_h2so4,
                                                 double &o_soag, double (&oi)[NPOP],
                                                 double (&oc)[NPOP]) {
  Sub si, sc;
  load_sub_plain(si, f.qi);
  load_sub_plain(sc, f.qc);
  {
    Sub si2, sc2;
    load_sub_plain(si2, cp.qi2);
    load_sub_plain(sc2, cp.qc2);
    cloudy_rename_grown(a, si, sc, si2, sc2);
  }
  const double w = 1.0;
  o_soag = dmax(0.0, 0.0 + f.g_soag * w);
  o_h2so4 = dmax(0.0, 0.0 + f.g_h2so4 * w);
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    oi[K::numslot(m)] = dmax(0.0, 0.0 + (si.num[m] / 1.0) * w);
    oc[K::numslot(m)] = 0.0 + (sc.num[m] / 1.0) * w;
#pragma unroll
    for (int x = 0; x < NAER; ++x) {
      const int slot = K::aer_slot(x, m);
      if (slot >= 0) {
        oi[slot] = dmax(0.0, 0.0 + (si.aer[x][m] / K::fcvt_aer(x)) * w);
        oc[slot] = 0.0 + (sc.aer[x][m] / K::fcvt_aer(x)) * w;
      }
    }
  }
}

// Partly cloudy grid cell after chemistry (set_subarea_gases_and_aerosols,
// mam4_amicphys.hpp:679-911): the interstitial partition factors come from
// the before-cloud-chemistry state and split both it and the current one;
// gases keep their before-cloud-chemistry value in the clear subarea and
// the cloudy subarea takes the remainder of the current grid mean
// (compute_qsub_from_gcm_and_qsub_of_other_subarea, :367-408).
__device__ __forceinline__ void partly_cloudy_setup_chem(const StepArgs &a, const Front &f,
                                                         const ChemPre &cp, Sub &s,
                                                         double (&gcl)[2], double &rhc,
                                                         double (&ci)[NPOP], double (&cg)[2],
                                                         double (&oc)[NPOP]) {
  const StepConsts &C = c_k;
  const double fcldy = f.cld, fclea = 1.0 - fcldy;
  double fn_c[NMODE], fn_y[NMODE], fm_c[NMODE], fm_y[NMODE];
  auto part = [&](double q_i, double q_c, double &fc, double &fy) {
    const double cldbrn_cldy = q_c / fcldy;
    const double intrst_cldy = dmax(0.0, ((q_i + q_c) - cldbrn_cldy));
    const double intrst_clea = (q_i - fcldy * intrst_cldy) / fclea;
    double r = dmax(1.e-35, intrst_clea * fclea) / dmax(1.e-35, q_i);
    r = dmax(0.0, dmin(1.0, r));
    fc = r / fclea;
    fy = (1 - r) / fcldy;
  };
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    part(cp.qi2[K::numslot(m)], cp.qc2[K::numslot(m)], fn_c[m], fn_y[m]);
    double si_ = 0.0, sc_ = 0.0;
#pragma unroll
    for (int k = 0; k < K::nspec(m); ++k) {
      si_ = si_ + cp.qi2[K::spec0(m) + k];
      sc_ = sc_ + cp.qc2[K::spec0(m) + k];
    }
    part(si_, sc_, fm_c[m], fm_y[m]);
  }
  const double g3[2] = {f.g_soag, f.g_h2so4};
  double gcy[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    gcl[g] = cp.g2[g];
    gcy[g] = (g3[g] - fclea * gcl[g]) / fcldy;
    if (gcy[g] < 0) {
      gcy[g] = 0;
      gcl[g] = g3[g] / fclea;
    }
  }
  rhc = bound(0.0, 1.0, (f.relhumgcm - fcldy) / fclea);
  {
    Sub si, sc, si2, sc2;
    load_sub(si, f.qi, fn_y, fm_y);
    load_sub(si2, cp.qi2, fn_y, fm_y);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      sc.num[m] = (f.qc[K::numslot(m)] / fcldy) * 1;
      sc2.num[m] = (cp.qc2[K::numslot(m)] / fcldy) * 1;
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        sc.aer[x][m] = (slot >= 0) ? (f.qc[slot] / fcldy) * K::fcvt_aer(x) : 0.0;
        sc2.aer[x][m] = (slot >= 0) ? (cp.qc2[slot] / fcldy) * K::fcvt_aer(x) : 0.0;
      }
    }
    cloudy_rename_grown(a, si, sc, si2, sc2);
    cg[0] = gcy[0] * fcldy;
    cg[1] = gcy[1] * fcldy;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      ci[K::numslot(m)] = (si.num[m] / 1.0) * fcldy;
      oc[K::numslot(m)] = (0.0 + 0.0 * fclea) + (sc.num[m] / 1.0) * fcldy;
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0) {
          ci[slot] = (si.aer[x][m] / K::fcvt_aer(x)) * fcldy;
          oc[slot] = (0.0 + 0.0 * fclea) + (sc.aer[x][m] / K::fcvt_aer(x)) * fcldy;
        }
      }
    }
  }
  load_sub(s, f.qi, fn_c, fm_c);
  s.gas[0] = gcl[0] * C.fcvt_soag;
  s.gas[1] = gcl[1] * 1.0;
}

// amicphys tracer index of the gas-chemistry gases O3, H2O2, SO2, DMS
__device__ __forceinline__ constexpr int chem_gas_i31(int g) { return g < 2 ? g : g + 1; }

// The chemistry of a cell between calcsize and amicphys: gas-phase
// chemistry of the gases and of the interstitial populations qi(p), then
// aqueous chemistry, on the cell's 31 tracers in vmr (qq, qqcw). before() is
// called between the two; it sets the cloud-borne populations. The four
// chemistry gases' tendencies are written.
template <class Qi, class Before>
__device__ __forceinline__ void chemistry(const StepArgs &a, const ChemArgs &ch,
                                          const long long c, double temp, double pmid, double cld,
                                          double h2so4, double soag, const Qi &qi,
                                          double (&qq)[31], double (&qqcw)[31],
                                          const Before &before) {
  const StepConsts &C = c_k;
  const double dt = a.dt;
  auto CIN = [&](int k) { return __ldg(ch.in + (size_t)k * ch.ld + c); };
  auto start = [&](int t) {
    if (t >= 6)
      return qi(t - 6);
    if (t == 2 || t == 5)
      return t == 2 ? h2so4 * C.to_vmr[0] : soag * C.to_vmr[1];
    return CIN(MAM4B_CHEM_IN_O3 + (t < 2 ? t : t - 1)) * (K::mw_dry_air / K::adv_mass(t));
  };
#pragma unroll
  for (int t = 0; t < 6; ++t)
    qqcw[t] = 0.0;
  {  // gas-phase chemistry
    double ext[gch::kExt], inv[gch::kInv];
#pragma unroll
    for (int e = 0; e < gch::kExt; ++e)
      ext[e] = CIN(MAM4B_CHEM_IN_EXTFRC + e);
#pragma unroll
    for (int i = 0; i < gch::kInv; ++i)
      inv[i] = CIN(MAM4B_CHEM_IN_INV + i);
    const double *het_c = ch.in + (size_t)MAM4B_CHEM_IN_HET * ch.ld + c;
    const size_t ld = ch.ld;
    auto het = [het_c, ld](int t) { return __ldg(het_c + (size_t)t * ld); };
    gch::gas_chemistry_from(temp, dt, CIN(MAM4B_CHEM_IN_PHOTO), ext, inv, het, start, qq);
  }
  before();
  {  // cloud chemistry; the total air density is the invariant density of air
    double dso4[3], dh2so4[3];
    sox::setsox_cell(dt, pmid, temp, CIN(MAM4B_CHEM_IN_LWC), cld,
                     CIN(MAM4B_CHEM_IN_CLDNUM), CIN(MAM4B_CHEM_IN_INV + 0), qq, qqcw, dso4,
                     dh2so4);
  }
  // the gases amicphys does not map keep the chemistry's result
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int i = chem_gas_i31(g);
    ch.out[(size_t)(MAM4B_CHEM_OUT_TEND + g) * ch.ld + c] =
        (qq[i] * (K::adv_mass(i) / K::mw_dry_air) - CIN(MAM4B_CHEM_IN_O3 + g)) / dt;
  }
}

// chemistry() of a cell in one thread: cp receives the states before each
// part, f the state after both (clipped, as amicphys reads it).
__device__ __forceinline__ void run_chemistry(const StepArgs &a, const ChemArgs &ch,
                                              const long long c, Front &f, ChemPre &cp) {
  double qq[31], qqcw[31];
  cp.g1[0] = f.g_soag;
  cp.g1[1] = f.g_h2so4;
  auto qi = [&](int p) { return f.qi[p]; };
  chemistry(a, ch, c, f.temp, f.pmid, f.cld, f.h2so4, f.soag, qi, qq, qqcw, [&] {
    cp.g2[0] = dmax(0.0, qq[5]);
    cp.g2[1] = dmax(0.0, qq[2]);
#pragma unroll
    for (int p = 0; p < NPOP; ++p) {
      qqcw[6 + p] = f.qc[p];
      cp.qi2[p] = dmax(0.0, qq[6 + p]);
      cp.qc2[p] = dmax(0.0, qqcw[6 + p]);
    }
  });
  f.g_soag = dmax(0.0, qq[5]);
  f.g_h2so4 = dmax(0.0, qq[2]);
#pragma unroll
  for (int p = 0; p < NPOP; ++p) {
    f.qi[p] = dmax(0.0, qq[6 + p]);
    f.qc[p] = dmax(0.0, qqcw[6 + p]);
  }
}

// chemistry() of a cell between chem_size_kernel and chem_subarea_kernel, on
// the populations in the hand-off. Aqueous chemistry changes of them but the
// cloud-borne SO4; the states before it and after it differ in no other.
__device__ __forceinline__ void chem_cell(const StepArgs &a, const ChemArgs &ch,
                                          const long long c) {
  const size_t n = (size_t)a.ncell;
  double *hi = a.hand + H_POP * n + c, *hc = a.hand + H_CI * n + c;
  double *aux = a.aux + c;
  double qq[31], qqcw[31];
  auto qi = [&](int p) { return hi[p * n]; };
  chemistry(a, ch, c, __ldg(a.in[MAM4B_IN_T] + c), __ldg(a.in[MAM4B_IN_P] + c),
            __ldg(a.in[MAM4B_IN_CLD] + c), __ldg(a.in[MAM4B_IN_H2SO4] + c),
            __ldg(a.in[MAM4B_IN_SOAG] + c), qi, qq, qqcw, [&] {
#pragma unroll
              for (int p = 0; p < NPOP; ++p) {
                hi[p * n] = dmax(0.0, qq[6 + p]);
                qqcw[6 + p] = hc[p * n];
              }
              aux[AUX_CHEM_GAS * n] = dmax(0.0, qq[5]);
              aux[(AUX_CHEM_GAS + 1) * n] = dmax(0.0, qq[2]);
            });
  aux[(AUX_CHEM_GAS + 2) * n] = dmax(0.0, qq[5]);
  aux[(AUX_CHEM_GAS + 3) * n] = dmax(0.0, qq[2]);
#pragma unroll
  for (int m = 0; m < 3; ++m)
    aux[(AUX_CHEM_SO4 + m) * n] = dmax(0.0, qqcw[sox::so4_cw(m)]);
}

// The per-particle H2SO4 uptake rate of mode M of cell c as the FP64 step
// computes it: FP64 water uptake of the mode from the cell's inputs, the
// calcsize dry diameter and the relative humidity of the size stage, then
// uptake_rate_mode. The mixed step (FP32 rates from the mode stage) uses
// it where a decision of the SOA loop sits at its threshold, so that the
// decision is the FP64 step's.
template <int M>
__device__ double rate_fp64_mode(const StepArgs &a, const long long c) {
  const StepConsts &C = c_k;
  const size_t n = (size_t)a.ncell;
  double sp[7];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    sp[s] = (s < K::nspec(M)) ? __ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0;
  double dgn_awet, qaerwat, wetdens;
  water_uptake_mode<M>(C, sp, a.aux[AUX_RH * n + c], a.out[MAM4B_OUT_DGN_A + M][c], dgn_awet,
                       qaerwat, wetdens);
  return uptake_rate_mode(C, M, a.aux[AUX_GDIFF * n + c], a.aux[AUX_FPATH * n + c], dgn_awet);
}
__device__ __forceinline__ double rate_fp64(const StepArgs &a, const long long c, int m) {
  switch (m) {
  case 0: return rate_fp64_mode<0>(a, c);
  case 1: return rate_fp64_mode<1>(a, c);
  case 2: return rate_fp64_mode<2>(a, c);
  default: return rate_fp64_mode<3>(a, c);
  }
}

// The SOA loop skips a mode, and zeroes its SOA, when its uptake rate is
// not above 1e-15 (gasaerexch_soaexch.hpp:189-193). With FP32 rates
// (relative error well below 1e-5) a rate within 1e-4 of that threshold may
// fall on the other side of it than the FP64 step's, so such modes take
// the FP64 rate instead (a few cells in 10^4).
__device__ __forceinline__ bool at_soa_threshold(double uptk0) {
  return fabs(uptk0 - 1.0e-15) <= 1.0e-4 * 1.0e-15;
}

// Appends cell c's SOA loop to the solver's order list, one append per warp;
// first_rate: the loop time over its first sub-step, times 0.05.
__device__ __forceinline__ void append_loop(const StepArgs &a, long long c, double first_rate) {
  const bool long_loop = first_rate > 0.05 * a.long_steps;
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  const unsigned m_long = __ballot_sync(m, long_loop), m_short = m & ~m_long;
  unsigned b_long = 0, b_short = 0;
  if (lane == leader) {
    if (m_long)
      b_long = atomicAdd(&a.counters[CNT_LONG], (unsigned)__popc(m_long));
    if (m_short)
      b_short = atomicAdd(&a.counters[CNT_SHORT], (unsigned)__popc(m_short));
  }
  b_long = __shfl_sync(m, b_long, leader);
  b_short = __shfl_sync(m, b_short, leader);
  const unsigned below = (1u << lane) - 1;
  if (long_loop)
    a.order[b_long + __popc(m_long & below)] = (int)c;
  else
    a.order[a.ncell - 1 - (b_short + __popc(m_short & below))] = (int)c;
}

template <int SOA, class State>
__device__ __forceinline__ bool soa_pass(State &st, bool fast);

// Second half of a cell after its SOA loop: the rest of the clear subarea
// (H2SO4 update, renaming, nucleation, coagulation with the coefficients of
// pair_kernel, aging), recombination with the cloudy subarea's
// contributions (ci, cg; partly cloudy cells), tendencies of the gases and
// interstitial populations (the cloud-borne ones are written by front_out). s
// holds the clear subarea with the loop's result, cm the values saved before
// condensation. src supplies the values read late (src.ci(p), cg(g), ai(p),
// h2so4(), soag()), from the hand-off and the inputs: reading them only when
// needed keeps them out of registers during the suffix.
template <bool DIAG, class Src>
__device__ __forceinline__ void cell_finish(const StepArgs &a, const long long c, double temp,
                                            double pmid, double zm, double cld, double pblh,
                                            double relhum, double dgn_pc, Sub &s, ClearMid &cm,
                                            const Src &src) {
  const StepConsts &C = c_k;
  const size_t n = (size_t)a.ncell;
  const double dt = a.dt;
  // wet sizes enter the suffix only through the coagulation coefficients,
  // which pair_kernel computed
  const double unused[NMODE] = {0, 0, 0, 0};
  Diag dgv(a, c);
  dgv.joined = !(cld < 1.0e-5);
  clear_suffix<DIAG, true>(a, dt, temp, pmid, zm, pblh, relhum, dgn_pc, unused, unused, cm, s,
                           &dgv, dgv.joined ? 1.0 - cld : 1.0, a.aux + AUX_COAG * n + c, n);
  // recombination (form_gcm_of_gases_and_aerosols_from_subareas)
  double o_h2so4, o_soag, oi[NPOP];
  double po[NPOP];
  sub_to_pop(s, po);
  double org[2][NMODE];  // SOA and POM in grid-cell units
  with_quotients([&](auto &q) {
    constexpr Divisor organic = constant_divisor(K::fcvt_aer(0));
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      org[0][m] = q.under(organic, s.aer[0][m]);
      org[1][m] = q.under(organic, s.aer[2][m]);
    }
  });
  if (cld < 1.0e-5) {
    const double f = 1.0 - 0.0;
    o_soag = dmax(0.0, 0.0 + (s.gas[0] / C.fcvt_soag) * f);
    o_h2so4 = dmax(0.0, 0.0 + (s.gas[1] / 1.0) * f);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] = dmax(0.0, 0.0 + (po[K::numslot(m)] / 1.0) * f);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int sl = K::aer_slot(x, m);
        if (sl >= 0)
          oi[sl] = dmax(0.0, 0.0 + (x == 0 ? org[0][m] : x == 2 ? org[1][m] : po[sl]) * f);
      }
    }
  } else {
    const double fclea = 1.0 - cld;
    o_soag = dmax(0.0, (0.0 + (s.gas[0] / C.fcvt_soag) * fclea) + src.cg(0));
    o_h2so4 = dmax(0.0, (0.0 + (s.gas[1] / 1.0) * fclea) + src.cg(1));
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] =
          dmax(0.0, (0.0 + (po[K::numslot(m)] / 1.0) * fclea) + src.ci(K::numslot(m)));
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int sl = K::aer_slot(x, m);
        if (sl >= 0)
          oi[sl] = dmax(0.0, (0.0 + (x == 0 ? org[0][m] : x == 2 ? org[1][m] : po[sl]) * fclea) + src.ci(sl));
      }
    }
  }
  double ai[NPOP];
#pragma unroll
  for (int p = 0; p < NPOP; ++p)
    ai[p] = src.ai(p);
  store_interstitial(a, c, o_h2so4, o_soag, oi, src.h2so4(), src.soag(), ai);
}

// cell_finish's late inputs read from the hand-off and the cell's inputs
// (post_kernel)
struct FinishLoads {
  const StepArgs &a;
  long long c;
  const double *h;
  size_t n;
  __device__ double ci(int p) const { return h[(H_CI + p) * n]; }
  __device__ double cg(int g) const { return h[(H_CG + g) * n]; }
  __device__ double ai(int p) const { return __ldg(a.in[MAM4B_IN_AER_I + p] + c); }
  __device__ double h2so4() const { return __ldg(a.in[MAM4B_IN_H2SO4] + c); }
  __device__ double soag() const { return __ldg(a.in[MAM4B_IN_SOAG] + c); }
};

// Second half of a cell with a clear subarea: the state at the SOA loop
// (hand-off), the loop's result (solver), then cell_finish.
template <bool DIAG = false>
__device__ __forceinline__ void cell_post(const StepArgs &a, const long long c) {
  const size_t n = (size_t)a.ncell;
  const double cld = __ldg(a.in[MAM4B_IN_CLD] + c);
  if (cld > kCloudy)
    return;
  const double temp = __ldg(a.in[MAM4B_IN_T] + c);
  const double pmid = __ldg(a.in[MAM4B_IN_P] + c);
  const double zm = __ldg(a.in[MAM4B_IN_ZM] + c);
  const double pblh = __ldg(a.pblh + c / a.nlev);
  const double *h = a.hand + c;
  const double *q = a.soa + c;
  Sub s;
  {
    double pop[NPOP];
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      pop[p] = h[(H_POP + p) * n];
    pop_to_sub(pop, s);
  }
  s.gas[0] = q[SOA_G * n];
  s.gas[1] = h[H_GAS1 * n];
#pragma unroll
  for (int k = 0; k < NMODE; ++k)
    s.aer[0][k] = q[(SOA_A + k) * n];
  ClearMid cm;
  cm.netprod1 = h[H_NETPROD * n];
  cm.sv_so4_ait = h[H_SV_SO4 * n];
  cm.sv_soa_ait = h[H_SV_SOA * n];
#pragma unroll
  for (int k = 0; k < NMODE; ++k)
    cm.uptk1[k] = h[(H_UPTK + k) * n];
  if (DIAG) {
    cm.gas_sv[0] = h[H_SOAG0 * n];
    cm.gas_sv[1] = s.gas[1];
#pragma unroll
    for (int m = 0; m < NMODE; ++m)
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        cm.sv_all[x][m] = slot >= 0 ? h[(H_POP + slot) * n] : 0.0;
      }
  }
  const FinishLoads src{a, c, h, n};
  cell_finish<DIAG>(a, c, temp, pmid, zm, cld, pblh, h[H_RELHUM * n], h[H_DGN_PC * n], s, cm, src);
}

template <bool DIAG>
__global__ void __launch_bounds__(128) full_kernel(const __grid_constant__ StepArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.ncell)
    cell_step<DIAG>(a, c);
}

// The step with chemistry start to end in one thread (process switches
// without condensation: no SOA loop to pipeline).
__device__ __forceinline__ void cell_step_chem(const StepArgs &a, const ChemArgs &ch,
                                               const long long c) {
  const StepConsts &C = c_k;
  Front f;
  cell_front(a, c, f);
  const double dt = a.dt;
  ChemPre cp;
  run_chemistry(a, ch, c, f, cp);
  double o_h2so4, o_soag, oi[NPOP], oc[NPOP];
  const double fsoag = C.fcvt_soag;
  const bool map_gas = a.do_cond || a.do_newnuc;
  const double qgas1[2] = {cp.g1[0] * fsoag, cp.g1[1] * 1.0};
  if (f.cld > kCloudy) {
    cloudy_cell_chem(a, f, cp, o_h2so4, o_soag, oi, oc);
  } else if (f.cld < 1.0e-5) {
    Sub s;
    load_sub_plain(s, f.qi);
    s.gas[0] = f.g_soag * fsoag;
    s.gas[1] = f.g_h2so4 * 1.0;
    const int niter = clear_subarea<false>(a, dt, f.temp, f.pmid, f.zm, f.pblh, f.relhumgcm,
                                           f.dgn_a, f.dgn_awet, f.wetdens, qgas1, s, nullptr,
                                           1.0);
    if (niter > 1000)
      atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
    const double w = 1.0 - 0.0;
    o_soag = dmax(0.0, 0.0 + (map_gas ? s.gas[0] / fsoag : f.g_soag) * w);
    o_h2so4 = dmax(0.0, 0.0 + (map_gas ? s.gas[1] / 1.0 : f.g_h2so4) * w);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] = dmax(0.0, 0.0 + (s.num[m] / 1.0) * w);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0)
          oi[slot] = dmax(0.0, 0.0 + (s.aer[x][m] / K::fcvt_aer(x)) * w);
      }
    }
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      oc[p] = f.qc[p];
  } else {
    const double fclea = 1.0 - f.cld;
    Sub s;
    double gcl[2], rhc, ci[NPOP], cg[2];
    partly_cloudy_setup_chem(a, f, cp, s, gcl, rhc, ci, cg, oc);
    const int niter = clear_subarea<false>(a, dt, f.temp, f.pmid, f.zm, f.pblh, rhc, f.dgn_a,
                                           f.dgn_awet, f.wetdens, qgas1, s, nullptr, fclea);
    if (niter > 1000)
      atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
    o_soag = dmax(0.0, (0.0 + (map_gas ? s.gas[0] / fsoag : gcl[0]) * fclea) + cg[0]);
    o_h2so4 = dmax(0.0, (0.0 + (map_gas ? s.gas[1] / 1.0 : gcl[1]) * fclea) + cg[1]);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      oi[K::numslot(m)] = dmax(0.0, (0.0 + (s.num[m] / 1.0) * fclea) + ci[K::numslot(m)]);
#pragma unroll
      for (int x = 0; x < NAER; ++x) {
        const int slot = K::aer_slot(x, m);
        if (slot >= 0)
          oi[slot] = dmax(0.0, (0.0 + (s.aer[x][m] / K::fcvt_aer(x)) * fclea) + ci[slot]);
      }
    }
  }
  store_outputs(a, c, o_h2so4, o_soag, oi, oc, f.h2so4, f.soag, f.ai, f.ac);
}

__global__ void __launch_bounds__(128) chem_step_kernel(const __grid_constant__ StepArgs a,
                                                        const __grid_constant__ ChemArgs ch) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.ncell)
    cell_step_chem(a, ch, c);
}

// Launch shapes of the pipeline kernels. Each whole-cell kernel is compiled
// once per register cap (__maxnreg__; a lower cap lets more warps reside on
// an SM, at the price of spills) and takes its block size and the number
// of cells each thread steps (a grid-stride loop) at launch; the values are
// chosen per device by mam4b_autotune (include/mam4b.h). The arithmetic is
// the same in every variant, so their results are bit for bit equal.
// Register caps compiled:
//   front_kernel 255, 128, 96; pre_kernel and post_kernel 255, 168, 128;
//   soa_kernel 64, 96, 128.

// Stage 1, one thread per (cell, mode): a block holds two modes of
// blockDim.x / 2 cells, accumulation and aitken (blockIdx.y 0) or coarse and
// primary carbon, a warp one of them. Everything up to the SOA loop of a
// cell treats its modes apart but for the aitken <-> accumulation exchange
// of calcsize and renaming, which pass a few values through shared memory
// (XF_*); the cell's own scalars go to the accumulation mode, which waits
// for renaming, and to primary carbon, which has the fewest species. A whole
// cell in one thread needs more than 255 registers and keeps 7.6 warps per
// SM resident. The mode is a run-time value, its tables (c_modes) in
// constant memory: with one copy of the code per mode the warps of an SM
// fetch four times the instructions, and waiting for them takes two thirds
// of the time.
enum {
  XF_DV_I = 0,    // accumulation, aitken: dry volumes, numbers
  XF_DV_C = 2,
  XF_N_I = 4,
  XF_N_C = 6,
  XF_NOXF_I = 8,  // accumulation: volumes without an aitken counterpart
  XF_NOXF_C = 9,
  XF_COMMON = 10,  // common species [accumulation, aitken][interstitial, cloud-borne][4]
  XF_RN_I = 26,    // rename: number and 4 species moved
  XF_RN_C = 31,
  XF_FIELDS = 36
};
struct ModeTables {
  int nspec[NMODE], spec0[NMODE], numslot[NMODE];
  double dmin[NMODE], dmax[NMODE], dnom[NMODE];
  double fcvt[NMODE][7];
  // position of species s among the four that the aitken and accumulation
  // modes share (SO4, SOA, NaCl, MOM), -1: none
  int common[NMODE][7];
  int soa[NMODE], pom[NMODE];  // position of SOA and POM in the mode, -1: none
};
constexpr ModeTables make_mode_tables() {
  ModeTables t = {};
  for (int m = 0; m < NMODE; ++m) {
    constexpr int nspec[NMODE] = {7, 4, 7, 3}, spec0[NMODE] = {0, 8, 13, 21},
                  num[NMODE] = {7, 12, 20, 24};
    constexpr int spec[NMODE][7] = {{1, 2, 0, 3, 5, 4, 6},
                                    {1, 0, 4, 6, -1, -1, -1},
                                    {5, 4, 1, 3, 2, 0, 6},
                                    {2, 3, 6, -1, -1, -1, -1}};
    t.nspec[m] = nspec[m];
    t.spec0[m] = spec0[m];
    t.numslot[m] = num[m];
    t.soa[m] = t.pom[m] = -1;
    constexpr double dmin[NMODE] = {5.35e-8, 8.7e-9, 1e-6, 1e-8},
                     dmax[NMODE] = {4.4e-7, 5.2e-8, 4e-6, 1e-7},
                     dnom[NMODE] = {1.1e-7, 2.6e-8, 2e-6, 5e-8};
    t.dmin[m] = dmin[m];
    t.dmax[m] = dmax[m];
    t.dnom[m] = dnom[m];
    for (int s = 0; s < 7; ++s) {
      const int x = spec[m][s];
      t.fcvt[m][s] = x == 0 || x == 2 ? 8.000000000000000E-002 : 1.0;
      t.common[m][s] =
          m > 1 ? -1 : x == 1 ? 0 : x == 0 ? 1 : x == 4 ? 2 : x == 6 ? 3 : -1;
      if (x == 0)
        t.soa[m] = s;
      if (x == 2)
        t.pom[m] = s;
    }
  }
  return t;
}
__constant__ ModeTables c_modes = make_mode_tables();
struct FrontMode {
  int m, ns, s0, num;           // mode, its species count, first slot, number slot
  double ai[7], ac[7], ni, nc;  // the mode's inputs (zero beyond its species)
  double pn_i, pn_c;            // number tendencies of calcsize
  double num_i, num_c, dv_i, dv_c;
  double si[7], sc[7], sni, snc;  // cloudy subarea
};

__device__ __forceinline__ FrontMode front_mode_of(int m) {
  FrontMode f;
  f.m = m;
  f.ns = c_modes.nspec[m];
  f.s0 = c_modes.spec0[m];
  f.num = c_modes.numslot[m];
  return f;
}

__device__ __forceinline__ void front_load(const StepArgs &a, long long c, double adj_inv,
                                           FrontMode &f, double *x, int stride) {
  const StepConsts &C = c_k;
  const int m = f.m;
#pragma unroll
  for (int s = 0; s < 7; ++s) {
    f.ai[s] = f.ac[s] = 0.0;
    if (s < f.ns) {
      f.ai[s] = __ldg(a.in[MAM4B_IN_AER_I + f.s0 + s] + c);
      f.ac[s] = __ldg(a.in[MAM4B_IN_AER_C + f.s0 + s] + c);
    }
  }
  f.ni = __ldg(a.in[MAM4B_IN_AER_I + f.num] + c);
  f.nc = __ldg(a.in[MAM4B_IN_AER_C + f.num] + c);
  f.dv_i = f.dv_c = 0.0;
  double chk = f.ni + f.nc;
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (s < f.ns) {
      f.dv_i += dmax(0.0, f.ai[s]) * C.inv_density[m][s];
      f.dv_c += dmax(0.0, f.ac[s]) * C.inv_density[m][s];
      chk += f.ai[s] + f.ac[s];
    }
  if (!isfinite(chk))
    atomicOr(a.flags, MAM4B_FLAG_NONFINITE_INPUT);
  f.num_i = f.ni < 0 ? 0.0 : f.ni;
  f.num_c = f.nc < 0 ? 0.0 : f.nc;
  f.pn_i = f.pn_c = 0.0;
  if (m >= 2) {
    adjust_num_sizes(f.dv_i, f.dv_c, f.ni, f.nc, a.dt, C.n2v_min[m], C.n2v_max[m], adj_inv,
                     f.num_i, f.num_c, f.pn_i, f.pn_c);
    return;
  }
  x[(XF_DV_I + m) * stride] = f.dv_i;
  x[(XF_DV_C + m) * stride] = f.dv_c;
  x[(XF_N_I + m) * stride] = f.num_i;
  x[(XF_N_C + m) * stride] = f.num_c;
  if (m == 0) {
    AitAccTotals v;
    accumulation_noxf(C, f.ai[1], f.ai[3], f.ai[4], f.ac[1], f.ac[3], f.ac[4], v);
    x[XF_NOXF_I * stride] = v.noxf_i;
    x[XF_NOXF_C * stride] = v.noxf_c;
  }
#pragma unroll
  for (int s = 0; s < 7; ++s) {
    const int k = c_modes.common[m][s];
    if (k >= 0) {
      x[(XF_COMMON + 8 * m + k) * stride] = f.ai[s];
      x[(XF_COMMON + 8 * m + 4 + k) * stride] = f.ac[s];
    }
  }
}

// Partition factor pair of get_partition_factors (mam4_amicphys.hpp:414-449)
template <class Quotients>
__device__ __forceinline__ void partition(Quotients &q, double q_i, double q_c, double fcldy,
                                          const Divisor &dy, const Divisor &dc, double fclea,
                                          double &fc, double &fy) {
  const double cldbrn_cldy = q.under(dy, q_c);
  const double intrst_cldy = dmax(0.0, ((q_i + q_c) - cldbrn_cldy));
  const double intrst_clea = q.under(dc, q_i - fcldy * intrst_cldy);
  double r = q.quot(dmax(1.e-35, intrst_clea * fclea), dmax(1.e-35, q_i));
  r = dmax(0.0, dmin(1.0, r));
  fc = q.under(dc, r);
  fy = q.under(dy, 1 - r);
}

// The mode's calcsize: its dry diameter (an output) and its populations after
// the calcsize update, in amicphys units.
__device__ __forceinline__ void front_sizes(const StepArgs &a, long long c, double cld,
                                            double adj_inv, FrontMode &f, const double *x,
                                            int stride, double (&qi)[7], double (&qc)[7],
                                            double &qni, double &qnc) {
  const StepConsts &C = c_k;
  const int m = f.m;
  const size_t n = (size_t)a.ncell;
  const double dt = a.dt;
  {
    // volume and number of the dry diameter, and their size bounds
    double drv = f.dv_i, num = f.num_i, lo = C.n2v_lo_wide[m], hi = C.n2v_hi_wide[m];
    AitAccExchange e;
    e.ait2acc = e.acc2ait = false;
    if (m < 2) {
      AitAccTotals t;
      t.dv_i_acc = x[XF_DV_I * stride];
      t.dv_i_ait = x[(XF_DV_I + 1) * stride];
      t.dv_c_acc = x[XF_DV_C * stride];
      t.dv_c_ait = x[(XF_DV_C + 1) * stride];
      t.n_i_acc = x[XF_N_I * stride];
      t.n_i_ait = x[(XF_N_I + 1) * stride];
      t.n_c_acc = x[XF_N_C * stride];
      t.n_c_ait = x[(XF_N_C + 1) * stride];
      t.noxf_i = x[XF_NOXF_I * stride];
      t.noxf_c = x[XF_NOXF_C * stride];
      e = aitken_accumulation_exchange(C, t, adj_inv);
      if (e.ait2acc || e.acc2ait) {
        // number and volume that leave the aitken mode
        const double ndi = (e.xt00 - e.xt10) * dt;
        const double vdi =
            (t.dv_i_ait * e.xv_ait2acc - (t.dv_i_acc - e.noxf_i) * e.xv_acc2ait) * dt;
        drv = dmax(0.0, m == 1 ? t.dv_i_ait - vdi : t.dv_i_acc + vdi);
        num = dmax(0.0, m == 1 ? t.n_i_ait - ndi : t.n_i_acc + ndi);
        lo = C.n2v_min[m];
        hi = C.n2v_max[m];
      }
      // calcsize adds the transfers one after the other, each with its sign
      if (e.ait2acc) {
        f.pn_i += m == 1 ? -e.xt00 : e.xt00;
        f.pn_c += m == 1 ? -e.xt01 : e.xt01;
      }
      if (e.acc2ait) {
        f.pn_i += m == 1 ? e.xt10 : -e.xt10;
        f.pn_c += m == 1 ? e.xt11 : -e.xt11;
      }
    }
    const double dgn = size_after_transfer(drv, num, lo, hi, c_modes.dmax[m], c_modes.dmin[m],
                                           c_modes.dnom[m], C.diam_fac[m]);
    a.out[MAM4B_OUT_DGN_A + m][c] = dgn;
    if (m == 3 && !(cld > kCloudy))
      a.hand[H_DGN_PC * n + c] = dgn;
#pragma unroll
    for (int s = 0; s < 7; ++s) {
      if (s >= f.ns)
        continue;
      double pi = 0.0, pc = 0.0;
      const int k = c_modes.common[m][s];
      if (k >= 0 && e.ait2acc) {
        const double xi = dmax(0.0, x[(XF_COMMON + 8 + k) * stride]) * e.xv_ait2acc;
        const double xc = dmax(0.0, x[(XF_COMMON + 12 + k) * stride]) * e.xv_ait2acc;
        pi += m == 1 ? -xi : xi;
        pc += m == 1 ? -xc : xc;
      }
      if (k >= 0 && e.acc2ait) {
        const double xi = dmax(0.0, x[(XF_COMMON + k) * stride]) * e.xv_acc2ait;
        const double xc = dmax(0.0, x[(XF_COMMON + 4 + k) * stride]) * e.xv_acc2ait;
        pi += m == 1 ? xi : -xi;
        pc += m == 1 ? xc : -xc;
      }
      qi[s] = dmax(0.0, dmax(0.0, f.ai[s] + pi * dt) * C.to_vmr[2 + f.s0 + s]);
      qc[s] = dmax(0.0, dmax(0.0, f.ac[s] + pc * dt) * C.to_vmr[2 + f.s0 + s]);
    }
    qni = dmax(0.0, dmax(0.0, f.ni + f.pn_i * dt) * C.to_vmr[2 + f.num]);
    qnc = dmax(0.0, dmax(0.0, f.nc + f.pn_c * dt) * C.to_vmr[2 + f.num]);
  }
}

// The mode's populations split between the subareas: the clear subarea at
// the SOA loop (into the hand-off; cells that are not cloudy) and the cloudy
// subarea before renaming. The aitken mode renames and leaves what moves in
// x; the accumulation mode takes it in front_out. With CHEM the populations
// are those before cloud chemistry, which changes but the cloud-borne SO4, to
// so4: the split is that of the values before, renaming counts the change of
// the aitken mode as growth.
template <bool DIAG, bool CHEM>
__device__ __forceinline__ void front_subareas(const StepArgs &a, long long c, double cld,
                                               FrontMode &f, double *x, int stride,
                                               const double (&qi)[7], double (&qc)[7],
                                               const double qni, const double qnc,
                                               const double so4) {
  const StepConsts &C = c_k;
  const int m = f.m;
  const size_t n = (size_t)a.ncell;
  const bool cloudy = cld > kCloudy, clear = cld < 1.0e-5;
  // subarea factors: clear (number, mass), cloudy interstitial (number,
  // mass); a clear or cloudy cell is its only subarea
  double fn_c = 1.0, fm_c = 1.0, fn_y = 1.0, fm_y = 1.0;
  // cloud-borne amounts of the cloudy subarea (of the cell when clear): with
  // CHEM the SO4 after cloud chemistry, whose change counts as growth
  const double fcldy = cld, fclea = 1.0 - fcldy;
  double ti = 0.0, tc = 0.0, grow = 0.0;
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (s < f.ns) {
      ti = ti + qi[s];
      tc = tc + qc[s];
    }
  const double so4_0 = qc[0];
  if (CHEM) {
    if (m < 2)
      qc[0] = so4;
    else if (m == 2)
      qc[2] = so4;
  }
  if (clear) {
#pragma unroll
    for (int s = 0; s < 7; ++s)
      f.sc[s] = qc[s];
    f.snc = qnc;
  } else {
    with_quotients([&](auto &q) {
      const Divisor dy = q.divisor(cloudy ? 1.0 : fcldy);
      if (!cloudy) {
        const Divisor dc = q.divisor(fclea);
        partition(q, qni, qnc, fcldy, dy, dc, fclea, fn_c, fn_y);
        partition(q, ti, tc, fcldy, dy, dc, fclea, fm_c, fm_y);
      }
      if (CHEM && m < 2)
        grow = q.under(dy, so4) * 1.0 - q.under(dy, so4_0) * 1.0;
#pragma unroll
      for (int s = 0; s < 7; ++s)
        if (s < f.ns)
          f.sc[s] = q.under(dy, qc[s]) * c_modes.fcvt[m][s];
      f.snc = q.under(dy, qnc) * 1;
    });
  }
  if (!cloudy) {
    // the clear subarea at the SOA loop (times one in a clear cell)
    double *h = a.hand + c;
    double soa = 0.0, pom = 0.0;
#pragma unroll
    for (int s = 0; s < 7; ++s) {
      if (s >= f.ns)
        continue;
      const double q = (qi[s] * fm_c) * c_modes.fcvt[m][s];
      h[(H_POP + f.s0 + s) * n] = q;
      if (s == c_modes.soa[m])
        soa = q;
      if (s == c_modes.pom[m])
        pom = q;
    }
    h[(H_POP + f.num) * n] = (qni * fn_c) * 1;
    if (m == 1) {
      h[H_SV_SO4 * n] = (qi[0] * fm_c) * 1;
      h[H_SV_SOA * n] = soa;
    }
    a.soa[(SOA_A + m) * n + c] = soa;
    a.soa[(SOA_OPOA + m) * n + c] = 0.0 + (m == 3 ? 0.0 : 0.1) * dmax(pom, 0.0);
  }
  // interstitial amounts of the cloudy subarea
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (s < f.ns)
      f.si[s] = (qi[s] * fm_y) * c_modes.fcvt[m][s];
  f.sni = (qni * fn_y) * 1;
  if (m == 1 && !clear) {
    // renaming (rename_subarea<true>): aitken volumes in AeroId order SOA,
    // SO4, NaCl, MOM
    double xn = 0.0, xv = 0.0;
    bool renamed = false;
    if (a.do_rename) {
      constexpr int order[4] = {1, 0, 2, 3};
      double ti = 0.0, tc = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        ti += f.si[order[k]] * K::mass_2_vol(K::mode_spec(1, order[k]));
        tc += f.sc[order[k]] * K::mass_2_vol(K::mode_spec(1, order[k]));
      }
      const double td = CHEM ? grow * K::mass_2_vol(1) : 0.0;
      renamed = rename_fractions<true>(C, ti - 0.0, 0.0, tc - td, td, f.sni, f.snc, xn, xv);
    }
    double mn_i = 0.0, mn_c = 0.0, mi[4] = {0, 0, 0, 0}, mc[4] = {0, 0, 0, 0};
    if constexpr (DIAG)
      if (a.do_rename) {
        const double w = cloudy ? 1.0 : cld;
        auto lost = [](double v, double by, bool yes) { return yes ? (v - by) - v : v - v; };
        const Diag dg(a, c);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const int x = k < 4 ? K::mode_spec(1, k < 4 ? k : 0) : -1;
          const int i = pop_to_i31(k < 4 ? K::spec0(1) + k : K::numslot(1));
          const double vi = k < 4 ? f.si[k < 4 ? k : 0] : f.sni;
          const double vc = k < 4 ? f.sc[k < 4 ? k : 0] : f.snc;
          const double part = k < 4 ? xv : xn;
          dg.put(1, i, dg.rate(x, lost(vi, vi * part, renamed)) * w);
          dg.put(NQTEND, i, dg.rate(x, lost(vc, vc * part, renamed)) * w);
        }
      }
    if (renamed) {
      mn_i = f.sni * xn;
      mn_c = f.snc * xn;
      f.sni -= mn_i;
      f.snc -= mn_c;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        mi[k] = f.si[k] * xv;
        mc[k] = f.sc[k] * xv;
        f.si[k] -= mi[k];
        f.sc[k] -= mc[k];
      }
    }
    x[XF_RN_I * stride] = mn_i;
    x[XF_RN_C * stride] = mn_c;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[(XF_RN_I + 1 + k) * stride] = mi[k];
      x[(XF_RN_C + 1 + k) * stride] = mc[k];
    }
  }
}

// The process tendencies of renaming in cloud that front_subareas did not store
// (it stores the aitken mode's); zero for the cloud-borne populations of a
// clear cell.
__device__ __forceinline__ void front_rename_diag(const StepArgs &a, long long c, double cld,
                                                  const FrontMode &f, const double *x,
                                                  int stride) {
  const bool clear = cld < 1.0e-5;
  if (f.m == 1 && !clear && a.do_rename)
    return;
  const double w = cld > kCloudy ? 1.0 : cld;
  const Diag dg(a, c);
#pragma unroll
  for (int s = 0; s <= 7; ++s) {
    if (s >= f.ns && s < 7)
      continue;
    const int i = pop_to_i31(s == 7 ? f.num : f.s0 + (s < 7 ? s : 0));
    double ti = 0.0, tc = 0.0;
    if (!clear && a.do_rename) {
      const int k = s == 7 ? -1 : c_modes.common[f.m][s < 7 ? s : 0];
      const double vi = s == 7 ? f.sni : f.si[s < 7 ? s : 0];
      const double vc = s == 7 ? f.snc : f.sc[s < 7 ? s : 0];
      const bool gains = f.m == 0 && (s == 7 || k >= 0);
      ti = (gains ? vi + x[(XF_RN_I + 1 + k) * stride] : vi) - vi;
      tc = (gains ? vc + x[(XF_RN_C + 1 + k) * stride] : vc) - vc;
      const bool org = s < 7 && c_modes.fcvt[f.m][s < 7 ? s : 0] != 1.0;
      ti = dg.rate(org ? 0 : -1, ti) * w;
      tc = dg.rate(org ? 0 : -1, tc) * w;
    }
    if (!clear)
      dg.put(1, i, ti);
    dg.put(NQTEND, i, tc);
  }
}

// What leaves the stage after renaming: cloud-borne tendencies; the
// interstitial tendencies of a cloudy cell, or the cloudy subarea's
// contributions to the grid means of a partly cloudy one.
template <bool DIAG>
__device__ __forceinline__ void front_out(const StepArgs &a, long long c, double cld,
                                          FrontMode &f, const double *x, int stride) {
  const StepConsts &C = c_k;
  const int m = f.m;
  const size_t n = (size_t)a.ncell;
  const bool cloudy = cld > kCloudy, clear = cld < 1.0e-5;
  double *h = a.hand + c;
  constexpr Divisor organic = constant_divisor(K::fcvt_aer(0));
  static_assert(K::fcvt_aer(0) == K::fcvt_aer(2), "SOA and POM share their unit factor");
  const double w = cloudy ? 1.0 : cld;
  if constexpr (DIAG)
    front_rename_diag(a, c, cld, f, x, stride);
  if (m == 0 && !clear) {
    f.sni += x[XF_RN_I * stride];
    f.snc += x[XF_RN_C * stride];
  }
  with_quotients([&](auto &q) {
    const Divisor dt = q.divisor(a.dt);
#pragma unroll
    for (int s = 0; s <= 7; ++s) {
      if (s >= f.ns && s < 7)
        continue;
      const bool number = s == 7;
      const int p = number ? f.num : f.s0 + s;
      double vi = number ? f.sni : f.si[s < 7 ? s : 0], vc = number ? f.snc : f.sc[s < 7 ? s : 0];
      const double ac = number ? f.nc : f.ac[s < 7 ? s : 0];
      if (!number && !clear) {
        const int k = c_modes.common[m][s < 7 ? s : 0];
        if (m == 0 && k >= 0) {
          vi += x[(XF_RN_I + 1 + k) * stride];
          vc += x[(XF_RN_C + 1 + k) * stride];
        }
        if (c_modes.fcvt[m][s < 7 ? s : 0] != 1.0) {
          vi = q.under(organic, vi);
          vc = q.under(organic, vc);
        }
      }
      const double oc = clear ? vc : 0.0 + vc * w;
      a.out[MAM4B_OUT_TEND + 27 + p][c] = q.under(dt, oc * C.to_mmr[2 + p] - ac);
      if (cloudy) {
        const double ai = __ldg(a.in[MAM4B_IN_AER_I + p] + c);
        a.out[MAM4B_OUT_TEND + 2 + p][c] =
            q.under(dt, dmax(0.0, 0.0 + vi * w) * C.to_mmr[2 + p] - ai);
      } else if (!clear) {
        h[(H_CI + p) * n] = vi * w;
      }
    }
  });
}

// The cell's scalars for the mode stage: humidity of water uptake, H2SO4
// diffusivity and mean free path.
__device__ __forceinline__ void front_uptake(const StepArgs &a, long long c, double cld) {
  const size_t n = (size_t)a.ncell;
  const double temp = __ldg(a.in[MAM4B_IN_T] + c), pmid = __ldg(a.in[MAM4B_IN_P] + c);
  a.aux[AUX_RH * n + c] = water_uptake_rh(__ldg(a.in[MAM4B_IN_QV] + c), temp, pmid, cld);
  double gd, fp;
  h2so4_diffusivity(temp, pmid, gd, fp);
  a.aux[AUX_GDIFF * n + c] = gd;
  a.aux[AUX_FPATH * n + c] = fp;
}
// The cell's gases: gases and relative humidity of the clear subarea
// (clear_prefix) and the equilibrium SOA gas for the SOA loop, or the gas
// tendencies of a cloudy cell.
template <bool CHEM>
__device__ __forceinline__ void front_gases(const StepArgs &a, long long c, double cld) {
  const StepConsts &C = c_k;
  const size_t n = (size_t)a.ncell;
  const double temp = __ldg(a.in[MAM4B_IN_T] + c), pmid = __ldg(a.in[MAM4B_IN_P] + c);
  const double qv = __ldg(a.in[MAM4B_IN_QV] + c);
  const double h2so4 = __ldg(a.in[MAM4B_IN_H2SO4] + c), soag = __ldg(a.in[MAM4B_IN_SOAG] + c);
  {
    const double chk = temp + pmid + __ldg(a.in[MAM4B_IN_ZM] + c) + qv + cld + h2so4 + soag +
                       __ldg(a.pblh + c / a.nlev);
    if (!isfinite(chk))
      atomicOr(a.flags, MAM4B_FLAG_NONFINITE_INPUT);
  }
  const double dt = a.dt;
  double g_h2so4 = dmax(0.0, h2so4 * C.to_vmr[0]), g_soag = dmax(0.0, soag * C.to_vmr[1]);
  const double qgas1 = g_h2so4 * 1.0;  // before chemistry
  // the clear subarea's gases: the grid mean before cloud chemistry
  double gcl[2] = {g_soag, g_h2so4};
  if (CHEM) {
    const double *g = a.aux + AUX_CHEM_GAS * n + c;
    gcl[0] = g[0];
    gcl[1] = g[n];
    g_soag = g[2 * n];
    g_h2so4 = g[3 * n];
  }
  if (cld > kCloudy) {
    const double w = 1.0;
    a.out[MAM4B_OUT_TEND + 0][c] =
        (dmax(0.0, 0.0 + g_h2so4 * w) * C.to_mmr[0] - h2so4) / dt;
    a.out[MAM4B_OUT_TEND + 1][c] = (dmax(0.0, 0.0 + g_soag * w) * C.to_mmr[1] - soag) / dt;
    return;
  }
  double rh = relhum_gcm(qv, temp, pmid);
  double *h = a.hand + c;
  if (CHEM && cld < 1.0e-5) {
    gcl[0] = g_soag;
    gcl[1] = g_h2so4;
  }
  if (!(cld < 1.0e-5)) {
    // gases: clear keeps the grid mean, cloudy gets the remainder
    const double fcldy = cld, fclea = 1.0 - fcldy;
    const double mean[2] = {g_soag, g_h2so4};
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      double gcy = (mean[g] - fclea * gcl[g]) / fcldy;
      if (gcy < 0) {
        gcy = 0;
        gcl[g] = mean[g] / fclea;
      }
      h[(H_CG + g) * n] = gcy * fcldy;
    }
    rh = bound(0.0, 1.0, (rh - fcldy) / fclea);
  }
  const double gas0 = gcl[0] * C.fcvt_soag;
  double gas1 = gcl[1] * 1.0, netprod = 0.0;
  if (a.optaa == 2) {
    netprod = (gas1 - qgas1) / dt;
    gas1 = (netprod >= 0) ? qgas1 : 0;
  }
  h[H_GAS1 * n] = gas1;
  h[H_NETPROD * n] = netprod;
  h[H_RELHUM * n] = rh;
  h[H_SOAG0 * n] = gas0;
  a.soa[SOA_G * n + c] = gas0;
  a.soa[SOA_G0 * n + c] = soa_equilibrium_gas(temp, pmid);
}

// LOOP: grid-stride loop over groups of cells (cells_per_thread > 1).
// Dynamic shared memory: XF_FIELDS doubles per cell.
template <int R, bool LOOP, bool DIAG = false>
__global__ void __maxnreg__(R) front_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ double s_x[];
  const int cells = blockDim.x / 2;
  const int k = threadIdx.x % cells;
  double *x = s_x + k;
  FrontMode f = front_mode_of(2 * blockIdx.y + threadIdx.x / cells);
  const double adj_inv = safe_denominator(dmax(86400.0, a.dt));
  for (long long c = blockIdx.x * (long long)cells + k; c - k < a.ncell;
       c += gridDim.x * (long long)cells) {
    const bool valid = c < a.ncell;
    const double cld = valid ? __ldg(a.in[MAM4B_IN_CLD] + c) : 0.0;
    if (valid)
      front_load(a, c, adj_inv, f, x, cells);
    if (blockIdx.y == 0)
      __syncthreads();
    if (valid) {
      double qi[7], qc[7], qni, qnc;
      front_sizes(a, c, cld, adj_inv, f, x, cells, qi, qc, qni, qnc);
      front_subareas<DIAG, false>(a, c, cld, f, x, cells, qi, qc, qni, qnc, 0.0);
      if (f.m == 3)
        front_uptake(a, c, cld);
      if (f.m == 0)
        front_gases<false>(a, c, cld);
    }
    if (blockIdx.y == 0)
      __syncthreads();
    if (valid)
      front_out<DIAG>(a, c, cld, f, x, cells);
    if constexpr (!LOOP)
      break;
    if (blockIdx.y == 0)
      __syncthreads();  // before the next cells' values overwrite these
  }
}

// The block's cells c = blockIdx.x * blockDim.x + threadIdx.x regrouped so
// that those with `first` fill warps of their own (cell order kept within
// each group; blocks of whole warps, at most 256 threads): cells below the
// crystallisation humidity, whose water uptake needs no Kohler solve, cells
// with cloud water. wanted: the cell takes part; returns the thread's cell,
// -1 for none.
__device__ __forceinline__ long long group_cells(bool wanted, bool first) {
  __shared__ int s_perm[256];
  __shared__ unsigned s_cnt[8][2];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, nw = blockDim.x >> 5;
  first = wanted && first;
  const unsigned bd = __ballot_sync(0xffffffffu, first);
  const unsigned bo = __ballot_sync(0xffffffffu, wanted && !first);
  if (lane == 0) {
    s_cnt[w][0] = __popc(bd);
    s_cnt[w][1] = __popc(bo);
  }
  __syncthreads();
  unsigned before_d = 0, before_o = 0, total_d = 0, total = 0;
  for (int k = 0; k < nw; ++k) {
    if (k < w) {
      before_d += s_cnt[k][0];
      before_o += s_cnt[k][1];
    }
    total_d += s_cnt[k][0];
    total += s_cnt[k][0] + s_cnt[k][1];
  }
  if (wanted) {
    const unsigned below = (1u << lane) - 1u;
    s_perm[first ? before_d + __popc(bd & below) : total_d + before_o + __popc(bo & below)] = t;
  }
  __syncthreads();
  return (unsigned)t < total ? (long long)blockIdx.x * blockDim.x + s_perm[t] : -1;
}

// ---- the front of the step with chemistry in three launches: calcsize per
// (cell, mode), as front_kernel's first part; the chemistry per cell; the
// subareas per (cell, mode), as its second. The populations pass between
// them in the hand-off rows that the second fills (interstitial H_POP,
// cloud-borne H_CI), SO4 after cloud chemistry and the gases in the rows that
// pair_kernel fills later. In one thread per cell this took 254 registers
// (7.7 warps per SM) and 1.40 ms for 8,192 x 72 cells, against 0.20, 0.34 and
// 0.25 ms; the second is bound by the latency of its 100 loads a cell and of
// the pH's bisection (three blocks per SM hide more of it than two, 0.40 ms,
// or four), the others by FP64 latency.
__global__ void __launch_bounds__(128, 5) chem_size_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ double s_x[];
  const int cells = blockDim.x / 2;
  const int k = threadIdx.x % cells;
  double *x = s_x + k;
  FrontMode f = front_mode_of(2 * blockIdx.y + threadIdx.x / cells);
  const double adj_inv = safe_denominator(dmax(86400.0, a.dt));
  const long long c = blockIdx.x * (long long)cells + k;
  const bool valid = c < a.ncell;
  if (valid)
    front_load(a, c, adj_inv, f, x, cells);
  if (blockIdx.y == 0)
    __syncthreads();
  if (!valid)
    return;
  const double cld = __ldg(a.in[MAM4B_IN_CLD] + c);
  double qi[7], qc[7], qni, qnc;
  front_sizes(a, c, cld, adj_inv, f, x, cells, qi, qc, qni, qnc);
  const size_t n = (size_t)a.ncell;
  double *hi = a.hand + H_POP * n + c, *hc = a.hand + H_CI * n + c;
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (s < f.ns) {
      hi[(f.s0 + s) * n] = qi[s];
      hc[(f.s0 + s) * n] = qc[s];
    }
  hi[f.num * n] = qni;
  hc[f.num * n] = qnc;
  if (f.m == 3)
    front_uptake(a, c, cld);
}

// The cells with cloud water, whose pH is found by bisection, fill warps of
// their own.
__global__ void __launch_bounds__(256, 3) chem_cell_kernel(const __grid_constant__ StepArgs a,
                                                           const __grid_constant__ ChemArgs ch) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = c < a.ncell;
  c = group_cells(valid, valid && __ldg(a.in[MAM4B_IN_CLD] + c) > 0.0 &&
                                   __ldg(ch.in + (size_t)MAM4B_CHEM_IN_LWC * ch.ld + c) > 0.0);
  if (c >= 0)
    chem_cell(a, ch, c);
}

__global__ void __launch_bounds__(128, 5) chem_subarea_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ double s_x[];
  const int cells = blockDim.x / 2;
  const int k = threadIdx.x % cells;
  double *x = s_x + k;
  FrontMode f = front_mode_of(2 * blockIdx.y + threadIdx.x / cells);
  const long long c = blockIdx.x * (long long)cells + k;
  const bool valid = c < a.ncell;
  const double cld = valid ? __ldg(a.in[MAM4B_IN_CLD] + c) : 0.0;
  if (valid) {
    const size_t n = (size_t)a.ncell;
    const double *hi = a.hand + H_POP * n + c, *hc = a.hand + H_CI * n + c;
    double qi[7], qc[7];
#pragma unroll
    for (int s = 0; s < 7; ++s) {
      f.ac[s] = qi[s] = qc[s] = 0.0;
      if (s < f.ns) {
        qi[s] = hi[(f.s0 + s) * n];
        qc[s] = hc[(f.s0 + s) * n];
        f.ac[s] = __ldg(a.in[MAM4B_IN_AER_C + f.s0 + s] + c);
      }
    }
    f.nc = __ldg(a.in[MAM4B_IN_AER_C + f.num] + c);
    const double so4 = f.m < 3 ? a.aux[(AUX_CHEM_SO4 + f.m) * n + c] : 0.0;
    front_subareas<false, true>(a, c, cld, f, x, cells, qi, qc, hi[f.num * n], hc[f.num * n], so4);
    if (f.m == 3)
      front_gases<true>(a, c, cld);
  }
  if (blockIdx.y == 0)
    __syncthreads();
  if (valid)
    front_out<false>(a, c, cld, f, x, cells);
}

// Stage 2, one thread per (cell, mode): water uptake of the mode (Kohler
// equilibrium, wet size, water, wet density; outputs) and its per-particle
// H2SO4 uptake rate. The modes are independent here, and a thread holds
// one mode's state only, so many more warps are resident than in a
// whole-cell thread.
// With MIXED the mode's arithmetic is single precision (mam4b::f32).
template <int M, bool MIXED>
__device__ __forceinline__ void mode_work(const StepArgs &a, const long long c) {
  const StepConsts &C = c_k;
  const size_t n = (size_t)a.ncell;
  if constexpr (MIXED) {
    float sp[7];
#pragma unroll
    for (int s = 0; s < 7; ++s)
      sp[s] = (s < K::nspec(M)) ? (float)__ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0f;
    float dgn_awet, qaerwat, wetdens;
    f32::water_uptake_mode<M>(C, sp, a.aux[AUX_RH * n + c],
                              (float)a.out[MAM4B_OUT_DGN_A + M][c], dgn_awet, qaerwat, wetdens);
    a.out[MAM4B_OUT_DGN_AWET + M][c] = dgn_awet;
    a.out[MAM4B_OUT_WETDENS + M][c] = wetdens;
    a.out[MAM4B_OUT_QAERWAT + M][c] = qaerwat;
    a.aux[(AUX_RATE + M) * n + c] = f32::uptake_rate_mode(
        C, M, (float)a.aux[AUX_GDIFF * n + c], (float)a.aux[AUX_FPATH * n + c], dgn_awet);
    return;
  }
  double sp[7];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    sp[s] = (s < K::nspec(M)) ? __ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0;
  const double dgn_a = a.out[MAM4B_OUT_DGN_A + M][c];
  double dgn_awet, qaerwat, wetdens;
  water_uptake_mode<M>(C, sp, a.aux[AUX_RH * n + c], dgn_a, dgn_awet, qaerwat, wetdens);
  a.out[MAM4B_OUT_DGN_AWET + M][c] = dgn_awet;
  a.out[MAM4B_OUT_WETDENS + M][c] = wetdens;
  a.out[MAM4B_OUT_QAERWAT + M][c] = qaerwat;
  a.aux[(AUX_RATE + M) * n + c] =
      uptake_rate_mode(C, M, a.aux[AUX_GDIFF * n + c], a.aux[AUX_FPATH * n + c], dgn_awet);
}

template <bool MIXED>
__global__ void mode_kernel(const __grid_constant__ StepArgs a) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (!MIXED) {
    const bool valid = c < a.ncell;
    c = group_cells(valid, valid && a.aux[AUX_RH * (size_t)a.ncell + c] < K::rh_cryst);
    if (c < 0)
      return;
  }
  if (c >= a.ncell)
    return;
  switch (blockIdx.y) {
  case 0: mode_work<0, MIXED>(a, c); break;
  case 1: mode_work<1, MIXED>(a, c); break;
  case 2: mode_work<2, MIXED>(a, c); break;
  default: mode_work<3, MIXED>(a, c); break;
  }
}

// Stage 3, one thread per (cell, mode pair): the Brownian coagulation
// coefficients of the pair (getcoags, coagulation.hpp:651-817) from the wet
// sizes and densities of stage 2; they do not depend on what condensation
// changes, so the post kernel only applies them.
template <bool MIXED>
__global__ void pair_kernel(const __grid_constant__ StepArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const StepConsts &C = c_k;
  const int p = blockIdx.y;
  const int sm = coag_src(p), dm = coag_dst(p);
  const double temp = __ldg(a.in[MAM4B_IN_T] + c);
  const double pmid = __ldg(a.in[MAM4B_IN_P] + c);
  const double aircon = pmid / (8314.46759100000 * temp);
  const double dens_s = dmax(1000.0, a.out[MAM4B_OUT_WETDENS + sm][c]);
  const double dens_d = dmax(1000.0, a.out[MAM4B_OUT_WETDENS + dm][c]);
  const CoagTables T = {kCoagBm0ij, kCoagBm3i, kCoagBm0};
  double bij0, bij3, bii0, bjj0;
  // the FP32 coefficients unless the correction-table index (round() of
  // 2 ln(dg_dst / dg_src) / ln 2, coagulation.hpp:715-717) sits within 1e-3
  // of a rounding boundary, where FP32 might round the other way
  bool fp32 = MIXED;
  if constexpr (MIXED) {
    const double r = a.out[MAM4B_OUT_DGN_AWET + dm][c] / a.out[MAM4B_OUT_DGN_AWET + sm][c];
    const double xr = log(r) / log(sqrt(2.0));
    fp32 = fabs(xr - floor(xr) - 0.5) > 1.0e-3;
  }
  if (fp32) {
    float f0, f3, fi, fj;
    f32::coag_pair_coefs(C, T, p, (float)temp, (float)pmid, (float)aircon,
                         (float)a.out[MAM4B_OUT_DGN_AWET + sm][c],
                         (float)a.out[MAM4B_OUT_DGN_AWET + dm][c], (float)dens_s, (float)dens_d,
                         f0, f3, fi, fj);
    bij0 = f0;
    bij3 = f3;
    bii0 = fi;
    bjj0 = fj;
  } else {
    coag_pair_coefs(C, T, p, temp, pmid, aircon, a.out[MAM4B_OUT_DGN_AWET + sm][c],
                    a.out[MAM4B_OUT_DGN_AWET + dm][c], dens_s, dens_d, bij0, bij3, bii0, bjj0);
  }
  const size_t n = (size_t)a.ncell;
  double *cc = a.aux + AUX_COAG * n + c;
  cc[p * n] = bij0;
  cc[(3 + p) * n] = bij3;
  cc[(6 + p) * n] = bii0;
  cc[(9 + p) * n] = bjj0;
}

// Stage 4, one thread per cell: the uptake rates of the clear subarea from
// the per-particle rates of the mode stage, and the solver's order of the
// loops. With MIXED a mode at the threshold of the SOA loop takes the FP64
// rate. FUSE: cells with short SOA loops finish here
// (StepArgs::inline_scale).
template <bool MIXED, bool FUSE>
__device__ __forceinline__ void pre_cell(const StepArgs &a, const long long c) {
  const size_t n = (size_t)a.ncell;
  if (__ldg(a.in[MAM4B_IN_CLD] + c) > kCloudy) {
    if constexpr (FUSE)
      a.done[c] = 1;
    return;
  }
  const double temp = __ldg(a.in[MAM4B_IN_T] + c), pmid = __ldg(a.in[MAM4B_IN_P] + c);
  const double aircon = pmid / (8314.46759100000 * temp);
  double *h = a.hand + c, *q = a.soa + c;
  SoaState st;
#pragma unroll
  for (int k = 0; k < NMODE; ++k) {
    const double num = h[(H_POP + K::numslot(k)) * n];
    double uptk1 = a.aux[(AUX_RATE + k) * n + c] * (num * aircon);
    st.uptk[k] = uptk1 * 0.81;
    if constexpr (MIXED) {
      if (at_soa_threshold(st.uptk[k])) {
        uptk1 = rate_fp64(a, c, k) * (num * aircon);
        st.uptk[k] = uptk1 * 0.81;
      }
    }
    h[(H_UPTK + k) * n] = uptk1;
    q[(SOA_UPTK + k) * n] = st.uptk[k];
  }
  st.g = q[SOA_G * n];
#pragma unroll
  for (int k = 0; k < NMODE; ++k) {
    st.a[k] = q[(SOA_A + k) * n];
    st.opoa[k] = q[(SOA_OPOA + k) * n];
  }
  st.g0 = q[SOA_G0 * n];
  st.dtfull = (double)(int)(a.dt / 1);
  const double first_rate = soa_first_rate(st) * st.dtfull;
  if constexpr (FUSE) {
    // a short loop (first sub-step at least 1/inline_scale of the step)
    // runs here, and its cell finishes, with the arithmetic of the solver
    // and post kernels
    const bool here = first_rate <= 0.05 * a.inline_scale;
    a.done[c] = here;
    if (here) {
      st.tcur = 0.0;
      st.niter = 0;
      const bool fast = soa_begin(st);
      while (soa_pass<MIXED ? 1 : 0>(st, fast)) {
      }
      if (st.niter > 1000)
        atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
      q[SOA_G * n] = st.g;
#pragma unroll
      for (int k = 0; k < NMODE; ++k)
        q[(SOA_A + k) * n] = st.a[k];
      cell_post(a, c);
      return;
    }
  }
  append_loop(a, c, first_rate);
}

template <int R, bool MIXED, bool FUSE>
__global__ void __maxnreg__(R) pre_kernel(const __grid_constant__ StepArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.ncell)
    pre_cell<MIXED, FUSE>(a, c);
}

// (the 128-register cap, 4 blocks of 128 per SM with a few hundred bytes
// spilled to L1, was 2 % faster than the unconstrained 231-register build)
template <int R, bool LOOP>
__global__ void __maxnreg__(R) post_kernel(const __grid_constant__ StepArgs a) {
  const long long c0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool fused = a.inline_scale > 0.0;
  if constexpr (LOOP) {
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 1
    for (long long c = c0; c < a.ncell; c += stride)
      if (!fused || !a.done[c])
        cell_post(a, c);
  } else if (c0 < a.ncell && (!fused || !a.done[c0])) {
    cell_post(a, c0);
  }
}

// The post stage with process tendencies. The front stage has stored those
// of renaming in cloud (processes 1 and 4 of the populations). Bound by the
// latency of the suffix and of some hundred stores a cell, as post_kernel;
// 128 registers keep 16 warps per SM.
__global__ void __launch_bounds__(128, 4) post_diag_kernel(const __grid_constant__ StepArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const double cld = __ldg(a.in[MAM4B_IN_CLD] + c);
  const bool cloudy = cld > kCloudy;
  constexpr unsigned all = 0x7fffffffu, gases = 0x3fu, mapped = 1u << 2 | 1u << 5;
  constexpr unsigned nucleated = 1u << 2 | 1u << 14 | 1u << 18;
  const bool keep_rename = a.do_rename || !(cld < 1.0e-5);
  diag_zeros(a, c,
             {cloudy ? all : gases & ~mapped, keep_rename ? gases : all,
              cloudy || !a.do_newnuc ? all : all & ~nucleated, cloudy || !a.do_coag ? all : gases,
              gases});
  cell_post<true>(a, c);
}

// SOA sub-stepping of the queued cells.
constexpr int kSoaBlock = 256;
template <int SOA, class State>
__device__ __forceinline__ bool soa_pass(State &st, bool fast) {
  if constexpr (SOA == 0)
    return soa_step(st, fast);
  else if constexpr (SOA == 1)
    return f32::soa_step_mx(st);
  else
    return f32::soa_step(st);
}

// One loop on four lanes, one mode each (lanes 4 k + mode of a warp): the
// values of the loop state that belong to a mode are the lane's, the others
// are the same on the four lanes. A pass is the arithmetic of soa_step
// (SOA 0), f32::soa_step_mx (1) or f32::soa_step (2), value by value: the
// sums over the modes are taken by every lane in mode order, a skipped
// mode adding nothing. What it changes is the length of the chain: a
// thread that owns a whole loop issues four modes' divisions one after the
// other, so a loop of 1,000 passes, which nothing else can shorten, takes
// four times as long.
template <class T>
struct SoaQuad {
  T g, a, opoa, uptk, g0;
  double tcur, dtfull;
  int niter;
};
template <class T>
struct ModeVals {
  T v[NMODE];
};
template <class T>
__device__ __forceinline__ ModeVals<T> of_modes(T x, int base) {
  ModeVals<T> r;
#pragma unroll
  for (int n = 0; n < NMODE; ++n)
    r.v[n] = __shfl_sync(0xffffffffu, x, base + n);
  return r;
}
// The pass itself, by all lanes of a warp together; lanes of loops that
// have ended (or of no loop) take part with no uptake and no SOA. Skipped
// modes are cleared (soa_clear_skipped) before the first pass.
template <bool FAST>
__device__ __forceinline__ void soa_quad_fp64(SoaQuad<double> &st, int base) {
  auto quot = [](double x, double y) { return FAST ? quot_in_range(x, y) : x / y; };
  const double g = dmax(st.g, 0.0), a = dmax(st.a, 0.0);
  double sat = quot(st.g0, dmax(st.opoa + a, 1.0e-20));
  const double g_star = sat * a;
  const double part = st.uptk * fabs(quot(g - g_star, dmax(g, dmax(g_star, 1.0e-20))));
  const ModeVals<double> all_a = of_modes(a, base), all_part = of_modes(part, base);
  double tot = g, tmpb = 0.0;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    tot += all_a.v[n];
    tmpb += all_part.v[n];
  }
  const double tmpa = dmax(0.0, tmpb), dtmax = st.dtfull - st.tcur;
  const bool last = dtmax * tmpa <= 0.05;
  const double dtcur = last ? dtmax : quot(0.05, tmpa);
  st.tcur = last ? st.dtfull : st.tcur + dtcur;
  const double beta = dtcur * st.uptk, del_g = g - g_star;
  if (del_g > 0.0)
    sat = quot(st.g0, dmax(st.opoa + (a + beta * del_g), 1.0e-20));
  const double den = 1.0 + beta * sat;
  const Divisor d(den);
  auto over_den = [&](double x) { return FAST ? d.under(x) : x / den; };
  const ModeVals<double> all_qa = of_modes(over_den(a), base),
                         all_qb = of_modes(over_den(beta), base);
  double ta = 0.0, tb = 0.0;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    ta += all_qa.v[n];
    tb += all_qb.v[n];
  }
  st.g = dmax(0.0, quot(tot - ta, 1.0 + tb));
  st.a = over_den(a + beta * st.g);
}
// fast: the lane's own parameters allow quot_in_range (soa_params_moderate);
// one form for the whole warp, whose lanes exchange values
__device__ __forceinline__ void soa_quad_pass(SoaQuad<double> &st, bool fast, int base,
                                              std::integral_constant<int, 0>) {
  if (__all_sync(0xffffffffu, fast && zero_or_moderate(st.g) && zero_or_moderate(st.a)))
    soa_quad_fp64<true>(st, base);
  else
    soa_quad_fp64<false>(st, base);
}
__device__ __forceinline__ void soa_quad_pass(SoaQuad<double> &st, bool, int base,
                                              std::integral_constant<int, 1>) {
  const double g = dmax(st.g, 0.0);
  const double a = dmax(st.a, 0.0), uptk = st.uptk;
  double sat = st.g0 * f32::mx::rcp(dmax(st.opoa + a, 1.0e-20));
  const double g_star = sat * a;
  const double aphi = fabs((g - g_star) * f32::mx::rcp(dmax(g, dmax(g_star, 1.0e-20))));
  const ModeVals<double> all_a = of_modes(a, base), all_phi = of_modes(aphi, base),
                         all_u = of_modes(uptk, base);
  double tot = g, tmpb = 0.0;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    tot += all_a.v[n];
    tmpb = __fma_rn(all_u.v[n], all_phi.v[n], tmpb);
  }
  const double tmpa = dmax(0.0, tmpb);
  const double dtmax = st.dtfull - st.tcur;
  double dtcur;
  if (dtmax * tmpa <= 0.05) {
    dtcur = dtmax;
    st.tcur = st.dtfull;
  } else {
    dtcur = 0.05 * f32::mx::rcp(tmpa);
    st.tcur += dtcur;
  }
  const double beta = dtcur * uptk, del_g = g - g_star;
  if (del_g > 0.0)
    sat = st.g0 * f32::mx::rcp(dmax(st.opoa + __fma_rn(beta, del_g, a), 1.0e-20));
  const double r = f32::mx::rcp(__fma_rn(beta, sat, 1.0));
  const ModeVals<double> all_r = of_modes(r, base);
  double ta = 0.0, tb = 0.0;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    ta = __fma_rn(all_a.v[n], all_r.v[n], ta);
    tb = __fma_rn(dtcur * all_u.v[n], all_r.v[n], tb);
  }
  st.g = dmax(0.0, (tot - ta) * f32::mx::rcp(1.0 + tb));
  st.a = __fma_rn(beta, st.g, a) * r;
}
__device__ __forceinline__ void soa_quad_pass(SoaQuad<float> &st, bool, int base,
                                              std::integral_constant<int, 2>) {
  using f32::fmx;
  const float g = fmx(st.g, 0.0f);
  const float a = fmx(st.a, 0.0f), uptk = st.uptk;
  float sat = __fdividef(st.g0, fmx(st.opoa + a, 1.0e-20f));
  const float g_star = sat * a;
  const float phi = __fdividef(g - g_star, fmx(g, fmx(g_star, 1.0e-20f)));
  const ModeVals<float> all_a = of_modes(a, base),
                        all_part = of_modes(uptk * fabsf(phi), base);
  float tot = g, tmpb = 0.0f;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    tot += all_a.v[n];
    tmpb += all_part.v[n];
  }
  const double dtmax = st.dtfull - st.tcur;
  float dtcur;
  if (dtmax * (double)tmpb <= 0.05) {
    dtcur = (float)dtmax;
    st.tcur = st.dtfull;
  } else {
    dtcur = __fdividef(0.05f, tmpb);
    st.tcur += (double)dtcur;
  }
  const float beta = dtcur * uptk, del_g = g - g_star;
  if (del_g > 0.0f)
    sat = __fdividef(st.g0, fmx(st.opoa + (a + beta * del_g), 1.0e-20f));
  const float den = __fdividef(1.0f, 1.0f + beta * sat);
  const ModeVals<float> all_ta = of_modes(a * den, base), all_tb = of_modes(beta * den, base);
  float ta = 0.0f, tb = 0.0f;
#pragma unroll
  for (int n = 0; n < NMODE; ++n) {
    ta += all_ta.v[n];
    tb += all_tb.v[n];
  }
  st.g = fmx(0.0f, __fdividef(tot - ta, 1.0f + tb));
  st.a = (a + beta * st.g) * den;
}

// soa_begin for one lane: clears a skipped mode and returns whether the
// lane's parameters allow quot_in_range.
template <class T>
__device__ __forceinline__ bool soa_quad_begin(SoaQuad<T> &st) {
  if (!(st.uptk > (T)1.0e-15) && 0.0 < st.dtfull - 1.0e-3)
    st.uptk = st.a = st.opoa = (T)0.0;
  return zero_or_moderate(st.g0) && st.g0 != (T)0.0 && zero_or_moderate(st.dtfull) &&
         zero_or_moderate(st.opoa) && zero_or_moderate(st.uptk);
}

// The long loops of the queue, four lanes to a loop, with work stealing as
// in soa_kernel (eight loops per warp).
template <int SOA, class T>
__device__ __forceinline__ void soa_long_loops(const StepArgs &a) {
  const unsigned nlong = a.counters[CNT_LONG];
  const int lane = threadIdx.x & 31, mode = lane & 3, base = lane & ~3;
  const size_t n = (size_t)a.ncell;
  SoaQuad<T> st = {};
  unsigned slot = 0;
  bool active = false, want = nlong > 0, fast = true;
  while (true) {
    const unsigned need = __ballot_sync(0xffffffffu, want);
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned first = 0;
      if (lane == leader)
        first = atomicAdd(&a.counters[CNT_TAKEN_LONG], (unsigned)__popc(need) / 4u);
      first = __shfl_sync(0xffffffffu, first, leader);
      if (want) {
        const unsigned t = first + __popc(need & ((1u << base) - 1)) / 4u;
        want = false;
        if (t < nlong) {
          slot = (unsigned)a.order[t];
          const double *q = a.soa + slot;
          st.g = q[SOA_G * n];
          st.a = q[(SOA_A + mode) * n];
          st.opoa = q[(SOA_OPOA + mode) * n];
          st.uptk = q[(SOA_UPTK + mode) * n];
          st.g0 = q[SOA_G0 * n];
          st.tcur = 0.0;
          st.dtfull = (double)(int)(a.dt / 1);
          st.niter = 0;
          fast = soa_quad_begin(st);
          active = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, active))
      return;
    // passes until a loop of the warp ends
    bool more;
    while (true) {
      more = active && soa_more(st);
      if (__any_sync(0xffffffffu, active && !more))
        break;
      soa_quad_pass(st, fast, base, std::integral_constant<int, SOA>());
    }
    if (active && !more) {
      double *q = a.soa + slot;
      if (mode == 0) {
        q[SOA_G * n] = st.g;
        if (st.niter > 1000)
          atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
        if (a.npass)
          a.npass[slot] = st.niter > 1000 ? 1000 : st.niter;
      }
      q[(SOA_A + mode) * n] = st.a;
      active = false;
      want = true;
      fast = true;
      st.g = st.a = st.uptk = (T)0.0;
    }
    if (more)
      --st.niter;  // counted again when this pass runs
  }
}

// Persistent warps. The long loops of the queue (StepArgs::long_steps) run
// first, four lanes to a loop; then every lane owns one short loop and, as
// soon as that loop ends, takes the next queued cell (one atomic per warp
// for all lanes that need work), so a warp never idles behind one cell.
// SOA: 0 the FP64 loop (soa_step), 1 FP64 state with FP32 step control
// (f32::soa_step_mx, MAM4B_MIXED), 2 the FP32 loop (f32::soa_step,
// MAM4B_MIXED_FAST).
// Launched with any block size that is a multiple of 32 and one grid of
// persistent blocks (SMs x blocks per SM).
template <int SOA, int R>
__global__ void __maxnreg__(R) soa_kernel(const __grid_constant__ StepArgs a) {
  constexpr bool F32 = SOA == 2;
  if (a.quads)
    soa_long_loops<SOA, typename std::conditional<F32, float, double>::type>(a);
  using State = typename std::conditional<F32, f32::SoaStateF, SoaState>::type;
  // the loops left, long ones first
  const unsigned nlong = a.quads ? 0 : a.counters[CNT_LONG];
  const unsigned ntask = nlong + a.counters[CNT_SHORT];
  const int lane = threadIdx.x & 31;
  const size_t n = (size_t)a.ncell;
  State st;
  unsigned slot = 0;
  bool active = false, want = true, fast = false;
  while (true) {
    const unsigned need = __ballot_sync(0xffffffffu, want);
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned base = 0;
      if (lane == leader)
        base = atomicAdd(&a.counters[CNT_TAKEN], (unsigned)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (want) {
        const unsigned t = base + __popc(need & ((1u << lane) - 1));
        want = false;
        if (t < ntask) {
          slot = (unsigned)(t < nlong ? a.order[t] : a.order[a.ncell - 1 - (t - nlong)]);
          const double *q = a.soa + slot;
          st.g = q[SOA_G * n];
#pragma unroll
          for (int k = 0; k < NMODE; ++k) {
            st.a[k] = q[(SOA_A + k) * n];
            st.opoa[k] = q[(SOA_OPOA + k) * n];
            st.uptk[k] = q[(SOA_UPTK + k) * n];
          }
          st.g0 = q[SOA_G0 * n];
          st.tcur = 0.0;
          st.dtfull = (double)(int)(a.dt / 1);
          st.niter = 0;
          if constexpr (SOA != 2)
            fast = soa_begin(st);
          active = true;
        }
      }
    }
    if (!__any_sync(0xffffffffu, active))
      break;
    // passes until a loop of the warp ends
    bool ran;
    do {
      ran = active && soa_pass<SOA>(st, fast);
    } while (!__any_sync(0xffffffffu, active && !ran));
    if (active && !ran) {
      double *q = a.soa + slot;
      q[SOA_G * n] = st.g;
#pragma unroll
      for (int k = 0; k < NMODE; ++k)
        q[(SOA_A + k) * n] = st.a[k];
      if (st.niter > 1000)
        atomicOr(a.flags, MAM4B_FLAG_SOA_NITER_LIMIT);
      if (a.npass)
        a.npass[slot] = st.niter > 1000 ? 1000 : st.niter;
      active = false;
      want = true;
    }
  }
}

// ============================================================ adjoint
// Reverse-mode adjoint of the FP64 step: in_bar = (d out / d in)^T out_bar
// per cell. Persistent threads; each runs one cell's forward sweep (state
// at process boundaries in local memory, the SOA loop's state every
// adj::kSoaCheck passes in its own slice of `ck`, laid out
// [checkpoint][component][thread] so a warp's accesses are coalesced) and
// then its reverse sweep.
struct AdjArgs {
  const double *in;    // [MAM4B_NIN][ld]
  const double *pblh;  // [ncol]
  const double *ybar;  // [MAM4B_NOUT][ld]
  double *xbar;        // [MAM4B_NIN][ld]
  size_t ld;
  long long ncell;
  int nlev;
  double dt;
  adj::AdjCfg cfg;
  double *ck;          // [6 * kSoaCkMax][nthreads]
};

__global__ void __launch_bounds__(128) adjoint_kernel(const __grid_constant__ AdjArgs a) {
  const size_t nthreads = (size_t)gridDim.x * blockDim.x;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const CoagTables T = {kCoagBm0ij, kCoagBm3i, kCoagBm0};
  double *ck = a.ck + tid;
  for (long long c = (long long)tid; c < a.ncell; c += (long long)nthreads) {
    double x[MAM4B_NIN], yb[MAM4B_NOUT], y[MAM4B_NOUT], xb[MAM4B_NIN];
#pragma unroll
    for (int f = 0; f < MAM4B_NIN; ++f)
      x[f] = __ldg(a.in + (size_t)f * a.ld + c);
#pragma unroll
    for (int f = 0; f < MAM4B_NOUT; ++f)
      yb[f] = __ldg(a.ybar + (size_t)f * a.ld + c);
    const double pblh = __ldg(a.pblh + c / a.nlev);
    int niter;
    adj::cell_adjoint(c_k, T, a.cfg, x, pblh, a.dt, ck, nthreads, yb, y, xb, niter);
#pragma unroll
    for (int f = 0; f < MAM4B_NIN; ++f)
      a.xbar[(size_t)f * a.ld + c] = xb[f];
  }
}

// ---- pipelined adjoint (condensation on): after the forward pipeline,
// adj_post_kernel reverses each queued cell's suffix (H2SO4 update,
// renaming, nucleation, coagulation, aging, recombination) from the
// hand-off, adj_soa_kernel reverses the SOA loops with the same work
// stealing as the forward solver, and adj_pre_kernel recomputes each cell's
// front and reverses it. Cotangents pass through cell-indexed scratch.
enum {
  AB_SB = 0,        // 29: subarea state after the loop: num[4], aer[1..6][4], gas[1]
  AB_NETPROD = 29,
  AB_UPTK1 = 30,    // 4
  AB_SV_SO4 = 34,
  AB_SV_SOA = 35,
  AB_DGN_PC = 36,
  AB_RH_SUB = 37,
  AB_T = 38,
  AB_DGN_AWET = 39,  // 4
  AB_WETDENS = 43,   // 4
  AB_CI = 47,        // 25
  AB_CG = 72,        // 2
  AB_FIELDS = 74
};
enum { LB_G = 0, LB_A = 1, LB_OPOA = 5, LB_UPTK = 9, LB_G0 = 13, LB_FIELDS = 14 };

struct AdjPipeArgs {
  StepArgs s;           // the forward pipeline's arguments and scratch
  const double *ybar;   // [MAM4B_NOUT][ld]
  double *xbar;         // [MAM4B_NIN][ld]
  size_t ld;
  double *abar;         // [AB_FIELDS][ncell]
  double *lbar;         // [LB_FIELDS][ncell]
  double *ck;           // SOA states [6 adj_soa_slots(CK)][nthreads of adj_soa_kernel]
  unsigned *bins;       // [2 kPassBins]: loops per pass count, start offsets
  adj::AdjCfg cfg;
};

// sb slot j (0..28) <-> Sub components other than the SOA ones
MAM4B_HD double &sb_ref(Sub &b, int j) {
  if (j < 4)
    return b.num[j];
  if (j < 28)
    return b.aer[1 + (j - 4) / 4][(j - 4) % 4];
  return b.gas[1];
}

// whether cell c has a clear subarea and with it an SOA loop
__device__ __forceinline__ bool has_loop(const StepArgs &a, long long c) {
  return !(__ldg(a.in[MAM4B_IN_CLD] + c) > kCloudy);
}

__global__ void __launch_bounds__(128, 4) adj_post_kernel(const __grid_constant__ AdjPipeArgs p) {
  const StepArgs &a = p.s;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell || !has_loop(a, c))
    return;
  const StepConsts &C = c_k;
  const CoagTables T = {kCoagBm0ij, kCoagBm3i, kCoagBm0};
  const size_t n = (size_t)a.ncell;
  const double temp = __ldg(a.in[MAM4B_IN_T] + c);
  const double pmid = __ldg(a.in[MAM4B_IN_P] + c);
  const double zm = __ldg(a.in[MAM4B_IN_ZM] + c);
  const double cld = __ldg(a.in[MAM4B_IN_CLD] + c);
  const double pblh = __ldg(a.pblh + c / a.nlev);
  const double *h = a.hand + c;
  double *q = a.soa + c;
  adj::SuffixIn in;
  {
    double pop[NPOP];
#pragma unroll
    for (int k = 0; k < NPOP; ++k)
      pop[k] = h[(H_POP + k) * n];
    pop_to_sub(pop, in.s_soa);
  }
  in.s_soa.gas[0] = q[SOA_G * n];
  in.s_soa.gas[1] = h[H_GAS1 * n];
#pragma unroll
  for (int k = 0; k < NMODE; ++k)
    in.s_soa.aer[0][k] = q[(SOA_A + k) * n];
  in.cm.netprod1 = h[H_NETPROD * n];
  in.cm.sv_so4_ait = h[H_SV_SO4 * n];
  in.cm.sv_soa_ait = h[H_SV_SOA * n];
#pragma unroll
  for (int k = 0; k < NMODE; ++k)
    in.cm.uptk1[k] = h[(H_UPTK + k) * n];
  in.dgn_pc = h[H_DGN_PC * n];
  in.rh_sub = h[H_RELHUM * n];
#pragma unroll
  for (int k = 0; k < 12; ++k)
    in.cc[k] = a.aux[(AUX_COAG + k) * n + c];
  in.partly = !(cld < 1.0e-5);
  in.fclea = 1.0 - cld;
#pragma unroll
  for (int k = 0; k < NPOP; ++k)
    in.ci[k] = in.partly ? h[(H_CI + k) * n] : 0.0;
  in.cg[0] = in.partly ? h[H_CG * n] : 0.0;
  in.cg[1] = in.partly ? h[(H_CG + 1) * n] : 0.0;
  adj::SuffixStates st;
  adj::suffix_states(C, p.cfg, temp, pmid, zm, pblh, a.dt, in, st);
  double ybt[MAM4B_NUM_PROG];
#pragma unroll
  for (int k = 0; k < MAM4B_NUM_PROG; ++k)
    ybt[k] = __ldg(p.ybar + (size_t)(MAM4B_OUT_TEND + k) * p.ld + c);
  adj::SuffixBar sb;
  adj::suffix_rev(C, p.cfg, temp, pmid, zm, pblh, a.dt, in, st, ybt, sb);
  double dgn_awet[NMODE], wetdens[NMODE], dgn_awetb[NMODE] = {0, 0, 0, 0},
                                           wetdensb[NMODE] = {0, 0, 0, 0};
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    dgn_awet[m] = a.out[MAM4B_OUT_DGN_AWET + m][c];
    wetdens[m] = dmax(1000.0, a.out[MAM4B_OUT_WETDENS + m][c]);
  }
  double tb = sb.tb;
  if (p.cfg.do_coag)
    adj::coef_rev(C, T, temp, pmid, dgn_awet, wetdens, sb.ccb, tb, dgn_awetb, wetdensb);
  // loop-end cotangents for the solver's reverse
  q[SOA_G * n] = sb.sb.gas[0];
#pragma unroll
  for (int k = 0; k < NMODE; ++k)
    q[(SOA_A + k) * n] = sb.sb.aer[0][k];
  double *ab = p.abar + c;
#pragma unroll
  for (int j = 0; j < 29; ++j)
    ab[(AB_SB + j) * n] = sb_ref(sb.sb, j);
  ab[AB_NETPROD * n] = sb.netprodb;
#pragma unroll
  for (int k = 0; k < NMODE; ++k) {
    ab[(AB_UPTK1 + k) * n] = sb.uptk1b[k];
    ab[(AB_DGN_AWET + k) * n] = dgn_awetb[k];
    ab[(AB_WETDENS + k) * n] = wetdensb[k];
  }
  ab[AB_SV_SO4 * n] = sb.sv_so4b;
  ab[AB_SV_SOA * n] = sb.sv_soab;
  ab[AB_DGN_PC * n] = sb.dgn_pcb;
  ab[AB_RH_SUB * n] = sb.rh_subb;
  ab[AB_T * n] = tb;
#pragma unroll
  for (int k = 0; k < NPOP; ++k)
    ab[(AB_CI + k) * n] = sb.cib[k];
  ab[AB_CG * n] = sb.cgb[0];
  ab[(AB_CG + 1) * n] = sb.cgb[1];
}

// The SOA loops are reversed in order of decreasing pass count, so that the
// 32 loops of a warp take the same number of passes and run in step:
// adj_hist_kernel counts the loops per pass count (npass, written by
// soa_kernel), adj_scan_kernel turns the counts into start offsets (most
// passes first) and adj_sort_kernel writes the cells in that order over the
// forward solver's order list, which is free once soa_kernel has run.
constexpr int kPassBins = 1001;  // pass counts 0..1000

__global__ void __launch_bounds__(256) adj_hist_kernel(const __grid_constant__ AdjPipeArgs p) {
  __shared__ unsigned h[kPassBins];
  for (int i = threadIdx.x; i < kPassBins; i += blockDim.x)
    h[i] = 0;
  __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < p.s.ncell; c += stride)
    if (has_loop(p.s, c))
      atomicAdd(&h[1000 - p.s.npass[c]], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < kPassBins; i += blockDim.x)
    if (h[i])
      atomicAdd(&p.bins[i], h[i]);
}

__global__ void __launch_bounds__(1024) adj_scan_kernel(const __grid_constant__ AdjPipeArgs p) {
  // exclusive scan of kPassBins counts, one block: each thread sums its
  // run of bins, the runs' totals are scanned in shared memory
  __shared__ unsigned tot[1024];
  constexpr int per = (kPassBins + 1023) / 1024;
  const int i0 = threadIdx.x * per;
  unsigned sum = 0;
  for (int i = i0; i < i0 + per && i < kPassBins; ++i)
    sum += p.bins[i];
  tot[threadIdx.x] = sum;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const unsigned v = threadIdx.x >= (unsigned)d ? tot[threadIdx.x - d] : 0u;
    __syncthreads();
    tot[threadIdx.x] += v;
    __syncthreads();
  }
  unsigned off = tot[threadIdx.x] - sum;
  for (int i = i0; i < i0 + per && i < kPassBins; ++i) {
    const unsigned c = p.bins[i];
    p.bins[kPassBins + i] = off;
    off += c;
  }
}

__global__ void __launch_bounds__(256) adj_sort_kernel(const __grid_constant__ AdjPipeArgs p) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < p.s.ncell; c += stride)
    if (has_loop(p.s, c))
      p.s.order[atomicAdd(&p.bins[kPassBins + 1000 - p.s.npass[c]], 1u)] = (int)c;
}

// Reverse of the SOA loops. Warps take 32 loops at a time from the sorted
// order list (one atomic per warp); every lane runs its loop forward,
// keeping the state (g, a[4], tcur) before passes in its own column of
// p.ck ([6 * index + component][thread]: the lanes of a warp are at the
// same pass, so a warp's stores and loads are coalesced), then the reverse
// passes, last to first, starting from the loop-end cotangents left by
// adj_post_kernel. CK = 1 stores the state before every pass (1,001 states
// per thread). CK > 1 keeps a checkpoint every CK passes (the states
// before passes 0, CK, 2 CK, ...: ceil(1001 / CK) per thread) and reverses
// the loop block by block: it recomputes the block's states from its
// checkpoint into a CK-state slice of the thread's column, then reverses
// the block's passes from them. Both give the same gradient bit for bit
// (the recomputed passes are the forward's arithmetic on the same state);
// CK > 1 needs about 1/CK of the memory and recomputes up to CK - 1 passes
// per block. The forward loop is the step's: soa_step (FP64), or with FAST
// f32::soa_step_mx (the mixed-precision adjoint); the reverse of a pass is
// adj::soa_pass_rev. Long loops of small batches (StepArgs::quads) go first,
// four lanes to a loop (adj_long_loops). 2 blocks per SM (128 registers,
// some spilled to L1): the extra warps hide more FP64 latency than the
// unconstrained 255-register build (10 % faster).
constexpr int kAdjSoaStates = 1001;  // states before passes 0..1000 (passes <= 1000)
// states kept per solver thread: checkpoints plus, with CK > 1, one block
__host__ __device__ constexpr int adj_soa_slots(int ck) {
  return ck == 1 ? kAdjSoaStates : (kAdjSoaStates + ck - 1) / ck + ck;
}
// rows of a thread's column of p.ck that adj_long_loops uses: one SOA value
// per pass, and g or tcur of every other pass
constexpr int kAdjQuadRows = kAdjSoaStates + (kAdjSoaStates + 1) / 2;
static_assert(kAdjQuadRows <= 6 * adj_soa_slots(4), "the quads' states fit either form's columns");

template <bool FAST>
__device__ __forceinline__ bool adj_soa_pass(SoaState &st, bool fast) {
  if constexpr (FAST)
    return f32::soa_step_mx(st);
  else
    return soa_step(st, fast);
}

// The loops of at least kAdjLongPasses passes (the head of the sorted order
// list), eight per warp and four lanes each, with the state before every
// pass kept in the four lanes' columns: row i of a lane its mode's SOA
// before pass i, rows kAdjSoaStates + i / 2 of lanes 2 (i % 2) and 2 (i % 2)
// + 1 g and tcur. The chain of a 1,000-pass loop, forward and reverse, is
// what bounds a small batch. Where the line lies hardly matters: 32, 64 and 150
// passes took 7.50, 7.43 and 7.30 ms on 4,096 x 72 cells, 2.92, 2.94 and 2.95
// on 512 x 72.
constexpr int kAdjLongPasses = 64;
template <bool FAST>
__device__ __forceinline__ void adj_long_loops(const AdjPipeArgs &p, unsigned nlong) {
  const StepArgs &a = p.s;
  const int lane = threadIdx.x & 31, mode = lane & 3, base = lane & ~3;
  const size_t n = (size_t)a.ncell;
  const size_t nthreads = (size_t)gridDim.x * blockDim.x;
  double *own = p.ck + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double *group = own - mode;
  auto pair_row = [&](int i) {
    return group + (size_t)(kAdjSoaStates + (i >> 1)) * nthreads + 2 * (i & 1);
  };
  while (true) {
    unsigned first = 0;
    if (lane == 0)
      first = atomicAdd(&a.counters[CNT_TAKEN_ADJ_LONG], 8u);
    first = __shfl_sync(0xffffffffu, first, 0);
    if (first >= nlong)
      return;
    const unsigned t = first + lane / 4;
    const bool valid = t < nlong;
    const unsigned slot = (unsigned)a.order[valid ? t : nlong - 1];
    const double *h = a.hand + slot;
    const double *q = a.soa + slot;
    constexpr int kSoaSlot[NMODE] = {K::aer_slot(0, 0), K::aer_slot(0, 1), K::aer_slot(0, 2), -1};
    const int soa_slot = mode == 0 ? kSoaSlot[0] : mode == 1 ? kSoaSlot[1] : kSoaSlot[2];
    SoaQuad<double> st;
    st.g = h[H_SOAG0 * n];
    st.a = mode < 3 ? h[(H_POP + soa_slot) * n] : 0.0;
    st.opoa = q[(SOA_OPOA + mode) * n];
    st.uptk = q[(SOA_UPTK + mode) * n];
    st.g0 = q[SOA_G0 * n];
    st.tcur = 0.0;
    st.dtfull = (double)(int)(a.dt / 1);
    st.niter = 0;
    const bool fast = soa_quad_begin(st);
    const SoaQuad<double> init = st;
    int k = 0;
    bool go = valid;
    while (true) {
      if (go) {
        own[(size_t)k * nthreads] = st.a;
        if (mode < 2)
          pair_row(k)[mode] = mode == 0 ? st.g : st.tcur;
        go = soa_more(st);
      }
      if (!__any_sync(0xffffffffu, go))
        break;
      soa_quad_pass(st, fast, base, std::integral_constant<int, FAST ? 1 : 0>());
      k += go;
    }
    __syncwarp();  // the group reads g and tcur where its other lanes stored them
    adj::LoopState<1> x;
    x.opoa[0] = init.opoa;
    x.uptk[0] = init.uptk;
    x.g0 = init.g0;
    x.dtfull = init.dtfull;
    adj::LoopBar<1> b;
    b.g = q[SOA_G * n];
    // a pass leaves a skipped mode no SOA, so nothing passes back through it
    b.a[0] = k == 0 || init.uptk > 1.0e-15 ? q[(SOA_A + mode) * n] : 0.0;
    b.tcur = b.opoa[0] = b.uptk[0] = b.g0 = 0.0;
    for (int i = __reduce_max_sync(0xffffffffu, k) - 1; i >= 0; --i) {
      const int j = min(i, max(k - 1, 0));  // loops with fewer passes wait
      x.a[0] = own[(size_t)j * nthreads];
      x.g = pair_row(j)[0];
      x.tcur = pair_row(j)[1];
      adj::LoopBar<1> nb = b;
      adj::soa_pass_rev(x, nb);
      if (i < k)
        b = nb;
    }
    if (valid) {
      double *lb = p.lbar + slot;
      if (mode == 0) {
        lb[LB_G * n] = b.g;
        lb[LB_G0 * n] = b.g0;
      }
      lb[(LB_A + mode) * n] = b.a[0];
      lb[(LB_OPOA + mode) * n] = b.opoa[0];
      lb[(LB_UPTK + mode) * n] = b.uptk[0];
    }
    __syncwarp();  // before the next loops' states overwrite these
  }
}

template <int CK, bool FAST>
__global__ void __launch_bounds__(kSoaBlock, 2) adj_soa_kernel(const __grid_constant__ AdjPipeArgs p) {
  const StepArgs &a = p.s;
  const unsigned ntask = a.counters[CNT_LONG] + a.counters[CNT_SHORT];
  // loops of at least kAdjLongPasses passes: where adj_sort_kernel left off
  // in their last bin
  const unsigned nlong = a.quads ? p.bins[kPassBins + 1000 - kAdjLongPasses] : 0u;
  adj_long_loops<FAST>(p, nlong);
  const int lane = threadIdx.x & 31;
  const size_t n = (size_t)a.ncell;
  const size_t nthreads = (size_t)gridDim.x * blockDim.x;
  double *ck = p.ck + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto put = [&](int idx, const SoaState &x) {
    double *e = ck + (size_t)6 * idx * nthreads;
    e[0] = x.g;
#pragma unroll
    for (int j = 0; j < NMODE; ++j)
      e[(1 + j) * nthreads] = x.a[j];
    e[5 * nthreads] = x.tcur;
  };
  auto get = [&](int idx, auto &x) {
    const double *e = ck + (size_t)6 * idx * nthreads;
    x.g = e[0];
#pragma unroll
    for (int j = 0; j < NMODE; ++j)
      x.a[j] = e[(1 + j) * nthreads];
    x.tcur = e[5 * nthreads];
  };
  while (true) {
    unsigned base = 0;
    if (lane == 0)
      base = nlong + atomicAdd(&a.counters[CNT_TAKEN_ADJ], 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= ntask)
      break;
    const unsigned t = base + lane;
    if (t >= ntask)
      continue;
    const unsigned slot = (unsigned)a.order[t];
    const double *h = a.hand + slot;
    const double *q = a.soa + slot;
    SoaState st;
    st.g = h[H_SOAG0 * n];
    {
      double pop[NPOP];
#pragma unroll
      for (int j = 0; j < NPOP; ++j)
        pop[j] = h[(H_POP + j) * n];
      Sub s0;
      pop_to_sub(pop, s0);
#pragma unroll
      for (int j = 0; j < NMODE; ++j)
        st.a[j] = s0.aer[0][j];
    }
#pragma unroll
    for (int j = 0; j < NMODE; ++j) {
      st.opoa[j] = q[(SOA_OPOA + j) * n];
      st.uptk[j] = q[(SOA_UPTK + j) * n];
    }
    st.g0 = q[SOA_G0 * n];
    st.tcur = 0.0;
    st.dtfull = (double)(int)(a.dt / 1);
    st.niter = 0;
    const bool fast = soa_begin(st);
    // forward: k passes (the states before passes 0..k-1 are reversed)
    int k = 0;
    while (true) {
      if (CK == 1 || k % CK == 0)
        put(k / CK, st);
      if (!adj_soa_pass<FAST>(st, fast))
        break;
      ++k;
    }
    adj::LoopState<NMODE> x;
    adj::LoopBar<NMODE> b;
    b.g = q[SOA_G * n];
#pragma unroll
    for (int j = 0; j < NMODE; ++j) {
      x.opoa[j] = st.opoa[j];
      x.uptk[j] = st.uptk[j];
      b.a[j] = k == 0 || st.uptk[j] > 1.0e-15 ? q[(SOA_A + j) * n] : 0.0;
      b.opoa[j] = 0.0;
      b.uptk[j] = 0.0;
    }
    x.g0 = st.g0;
    x.dtfull = st.dtfull;
    b.tcur = 0.0;
    b.g0 = 0.0;
    if constexpr (CK == 1) {
      while (k > 0) {
        --k;
        get(k, x);
        adj::soa_pass_rev(x, b);
      }
    } else {
      constexpr int kBlock = (kAdjSoaStates + CK - 1) / CK;  // first state of the block slice
      for (int b0 = k > 0 ? ((k - 1) / CK) * CK : -1; b0 >= 0; b0 -= CK) {
        const int nb = min(CK, k - b0);  // passes b0 .. b0 + nb - 1
        get(b0 / CK, st);
        // these passes all continued in the forward (niter only caps it)
        st.niter = 0;
        put(kBlock, st);
        for (int j = 1; j < nb; ++j) {
          adj_soa_pass<FAST>(st, fast);
          put(kBlock + j, st);
        }
        for (int j = nb - 1; j >= 0; --j) {
          get(kBlock + j, x);
          adj::soa_pass_rev(x, b);
        }
      }
    }
    double *lb = p.lbar + slot;
    lb[LB_G * n] = b.g;
#pragma unroll
    for (int j = 0; j < NMODE; ++j) {
      lb[(LB_A + j) * n] = b.a[j];
      lb[(LB_OPOA + j) * n] = b.opoa[j];
      lb[(LB_UPTK + j) * n] = b.uptk[j];
    }
    lb[LB_G0 * n] = b.g0;
  }
}

// The whole-cell reverse kernels (adj_post, adj_pre, adj_fin) run 4 blocks
// of 128 per SM (128 registers, their tapes in L1-cached local memory):
// 2.8 ms faster in total than unconstrained at 255 registers.
//
// Reverse of each cell's front (and of cloudy cells entirely), up to the
// water uptake: the front's forward sweep takes water uptake, diffusivity
// and uptake rates from the forward pipeline (out rows, aux), the
// reverse leaves the partial input cotangents in xbar and the cotangents
// of the water uptake's and calcsize's outputs in abar (FT_* fields, over
// the suffix cotangents it has read).
enum { FT_PT_IB = 0, FT_PT_CB = 25, FT_DGN_AB = 50, FT_DGN_AWETB = 54, FT_QAERWATB = 58,
       FT_WETDENS_WUB = 62, FT_RHB = 66, FT_FIELDS = 70 };
static_assert(FT_FIELDS <= AB_FIELDS, "front hand-off must fit in abar");

__global__ void __launch_bounds__(128, 4) adj_pre_kernel(const __grid_constant__ AdjPipeArgs p) {
  const StepArgs &a = p.s;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const size_t n = (size_t)a.ncell;
  double x[MAM4B_NIN], yb[MAM4B_NOUT], y[MAM4B_NOUT], xb[MAM4B_NIN];
#pragma unroll
  for (int f = 0; f < MAM4B_NIN; ++f)
    x[f] = __ldg(a.in[f] + c);
#pragma unroll
  for (int f = 0; f < MAM4B_NOUT; ++f)
    yb[f] = __ldg(p.ybar + (size_t)f * p.ld + c);
  adj::FrontKnown kn;
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    kn.dgn_awet[m] = a.out[MAM4B_OUT_DGN_AWET + m][c];
    kn.wetdens_wu[m] = a.out[MAM4B_OUT_WETDENS + m][c];
    kn.qaerwat[m] = a.out[MAM4B_OUT_QAERWAT + m][c];
    kn.rate[m] = a.aux[(AUX_RATE + m) * n + c];
  }
  kn.rh_wu = a.aux[AUX_RH * n + c];
  kn.gd = a.aux[AUX_GDIFF * n + c];
  kn.fp = a.aux[AUX_FPATH * n + c];
  adj::FrontTape ft;
  adj::front_forward<true>(c_k, p.cfg, x, a.dt, ft, y, &kn);
  const double zero4[NMODE] = {0, 0, 0, 0};
  adj::FrontTail tl;
  if (ft.cat == 1) {
    adj::front_rev_head(c_k, p.cfg, x, a.dt, ft, nullptr, nullptr, yb, zero4, zero4, 0.0, xb, tl);
  } else {
    const double *ab = p.abar + c;
    const double *lbp = p.lbar + c;
    adj::SuffixBar sb;
    adj::sub_zero(sb.sb);
#pragma unroll
    for (int j = 0; j < 29; ++j)
      sb_ref(sb.sb, j) = ab[(AB_SB + j) * n];
    sb.netprodb = ab[AB_NETPROD * n];
    double dgn_awetb[NMODE], wetdensb[NMODE];
#pragma unroll
    for (int k = 0; k < NMODE; ++k) {
      sb.uptk1b[k] = ab[(AB_UPTK1 + k) * n];
      dgn_awetb[k] = ab[(AB_DGN_AWET + k) * n];
      wetdensb[k] = ab[(AB_WETDENS + k) * n];
    }
    sb.sv_so4b = ab[AB_SV_SO4 * n];
    sb.sv_soab = ab[AB_SV_SOA * n];
    sb.dgn_pcb = ab[AB_DGN_PC * n];
    sb.rh_subb = ab[AB_RH_SUB * n];
    sb.tb = 0.0;
#pragma unroll
    for (int k = 0; k < NPOP; ++k)
      sb.cib[k] = ab[(AB_CI + k) * n];
    sb.cgb[0] = ab[AB_CG * n];
    sb.cgb[1] = ab[(AB_CG + 1) * n];
    adj::SoaBar lb;
    lb.g = lbp[LB_G * n];
#pragma unroll
    for (int k = 0; k < NMODE; ++k) {
      lb.a[k] = lbp[(LB_A + k) * n];
      lb.opoa[k] = lbp[(LB_OPOA + k) * n];
      lb.uptk[k] = lbp[(LB_UPTK + k) * n];
    }
    lb.g0 = lbp[LB_G0 * n];
    lb.tcur = 0.0;
    adj::front_rev_head(c_k, p.cfg, x, a.dt, ft, &sb, &lb, yb, dgn_awetb, wetdensb,
                        ab[AB_T * n], xb, tl);
  }
#pragma unroll
  for (int f = 0; f < MAM4B_NIN; ++f)
    p.xbar[(size_t)f * p.ld + c] = xb[f];
  double *ft_out = p.abar + c;
#pragma unroll
  for (int k = 0; k < NPOP; ++k) {
    ft_out[(FT_PT_IB + k) * n] = tl.pt_ib[k];
    ft_out[(FT_PT_CB + k) * n] = tl.pt_cb[k];
  }
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    ft_out[(FT_DGN_AB + m) * n] = tl.dgn_ab[m];
    ft_out[(FT_DGN_AWETB + m) * n] = tl.dgn_awetb[m];
    ft_out[(FT_QAERWATB + m) * n] = tl.qaerwatb[m];
    ft_out[(FT_WETDENS_WUB + m) * n] = tl.wetdens_wub[m];
  }
}

// Reverse of the water uptake, one thread per (cell, mode) as in the
// forward's mode_kernel: adds the species' cotangents to xbar, updates the
// mode's dry-diameter cotangent and leaves the RH cotangent in abar.
template <int M>
__device__ __forceinline__ void adj_mode_work(const AdjPipeArgs &p, long long c) {
  const StepArgs &a = p.s;
  const size_t n = (size_t)a.ncell;
  double sp[7], spb[7];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    sp[s] = (s < K::nspec(M)) ? __ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0;
  double *ft = p.abar + c;
  double dgn_ab = ft[(FT_DGN_AB + M) * n];
  const double r = adj::front_rev_mode<M>(
      c_k, sp, a.aux[AUX_RH * n + c], a.out[MAM4B_OUT_DGN_A + M][c], ft[(FT_DGN_AWETB + M) * n],
      ft[(FT_QAERWATB + M) * n], ft[(FT_WETDENS_WUB + M) * n], spb, dgn_ab);
  ft[(FT_DGN_AB + M) * n] = dgn_ab;
  ft[(FT_RHB + M) * n] = r;
#pragma unroll
  for (int s = 0; s < K::nspec(M); ++s)
    p.xbar[(size_t)(MAM4B_IN_AER_I + K::spec0(M) + s) * p.ld + c] += spb[s];
}

// Cells regrouped within the block as in mode_kernel: those below the
// crystallisation humidity (no Kohler reverse) fill warps of their own.
// Launched with 128 threads per block.
__global__ void __launch_bounds__(128) adj_mode_kernel(const __grid_constant__ AdjPipeArgs p) {
  const StepArgs &a = p.s;
  const long long c0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = c0 < a.ncell;
  const long long c =
      group_cells(valid, valid && a.aux[AUX_RH * (size_t)a.ncell + c0] < K::rh_cryst);
  if (c < 0)
    return;
  switch (blockIdx.y) {
  case 0: adj_mode_work<0>(p, c); break;
  case 1: adj_mode_work<1>(p, c); break;
  case 2: adj_mode_work<2>(p, c); break;
  default: adj_mode_work<3>(p, c); break;
  }
}

// Last part of the reverse, per cell: RH of water uptake and calcsize. Bound by
// the traffic of its spills: two blocks per SM with 255 registers took 0.265 ms
// for 4,096 x 72 cells, four with 128 registers 0.32.
__global__ void __launch_bounds__(128, 2) adj_fin_kernel(const __grid_constant__ AdjPipeArgs p) {
  const StepArgs &a = p.s;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const size_t n = (size_t)a.ncell;
  double ai[NPOP], ac[NPOP], aib[NPOP], acb[NPOP];
  double *xbc = p.xbar + c;
#pragma unroll
  for (int k = 0; k < NPOP; ++k) {
    ai[k] = __ldg(a.in[MAM4B_IN_AER_I + k] + c);
    ac[k] = __ldg(a.in[MAM4B_IN_AER_C + k] + c);
    aib[k] = xbc[(size_t)(MAM4B_IN_AER_I + k) * p.ld];
    acb[k] = xbc[(size_t)(MAM4B_IN_AER_C + k) * p.ld];
  }
  double tb = xbc[(size_t)MAM4B_IN_T * p.ld], qvb = xbc[(size_t)MAM4B_IN_QV * p.ld];
  const double *ft = p.abar + c;
  adj::FrontTail tl;
#pragma unroll
  for (int k = 0; k < NPOP; ++k) {
    tl.pt_ib[k] = ft[(FT_PT_IB + k) * n];
    tl.pt_cb[k] = ft[(FT_PT_CB + k) * n];
  }
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    tl.dgn_ab[m] = ft[(FT_DGN_AB + m) * n];
  double rh_wub = 0.0;
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    rh_wub += ft[(FT_RHB + m) * n];
  adj::front_rev_tail(c_k, ai, ac, __ldg(a.in[MAM4B_IN_QV] + c), __ldg(a.in[MAM4B_IN_T] + c),
                      __ldg(a.in[MAM4B_IN_P] + c), __ldg(a.in[MAM4B_IN_CLD] + c), a.dt, tl, rh_wub,
                      aib, acb, tb, qvb);
  xbc[(size_t)MAM4B_IN_T * p.ld] = tb;
  xbc[(size_t)MAM4B_IN_QV * p.ld] = qvb;
#pragma unroll
  for (int k = 0; k < NPOP; ++k) {
    xbc[(size_t)(MAM4B_IN_AER_I + k) * p.ld] = aib[k];
    xbc[(size_t)(MAM4B_IN_AER_C + k) * p.ld] = acb[k];
  }
}

// ====================================================== derived constants
// Evaluated once per device by a one-thread kernel, with the same
// expressions the reference evaluates inline (and the same math library the
// kernel uses), then copied into constant memory.
__host__ __device__ static double h_vol_from_diam(double d, double sig) {
  return (d * d * d) * exp(4.5 * (log(sig) * log(sig))) * K::pi_sixth;
}

__host__ __device__ static StepConsts make_consts() {
  StepConsts C = {};
  for (int m = 0; m < NMODE; ++m) {
    C.n2v_nom[m] = 1.0 / h_vol_from_diam(K::dnom(m), K::sig(m));
    C.n2v_min[m] = 1.0 / h_vol_from_diam(K::dmax(m), K::sig(m));
    C.n2v_max[m] = 1.0 / h_vol_from_diam(K::dmin(m), K::sig(m));
    for (int s = 0; s < K::nspec(m); ++s)
      C.inv_density[m][s] = 1.0 / K::aero_dens(K::mode_spec(m, s));
    C.log_sig[m] = log(K::sig(m));
    C.diam_fac[m] = exp(-1.5 * sq(C.log_sig[m]));
    C.exp45[m] = exp(4.5 * sq(C.log_sig[m]));
    C.coag[m].e01 = exp(0.125 * C.log_sig[m] * C.log_sig[m]);
    C.coag[m].e04 = pow(C.coag[m].e01, 4.0);
    C.coag[m].e36 = exp(4.5 * C.log_sig[m] * C.log_sig[m]);
    C.coag[m].dlgsqt2 = 1.0 / log(sqrt(2.0));
    C.coag[m].row = (int)dmax(1.0, dmin(10.0, round(4.0 * (K::sig(m) - 0.75)))) - 1;
    C.n2v_lo_wide[m] = C.n2v_min[m];
    C.n2v_hi_wide[m] = C.n2v_max[m];
  }
  C.n2v_lo_wide[1] /= 1.0e6;
  C.n2v_hi_wide[0] *= 1.0e6;
  // unit factors: H2SO4 (tracer 2), SOAG (tracer 5), populations 6..30
  auto is_num = [](int i31) { return i31 == 13 || i31 == 18 || i31 == 26 || i31 == 30; };
  const int tr[2] = {2, 5};
  for (int k = 0; k < NPOP + 2; ++k) {
    const int i31 = k < 2 ? tr[k] : 6 + (k - 2);
    C.to_vmr[k] = is_num(i31) ? K::mw_dry_air : K::mw_dry_air / K::adv_mass(i31);
    C.to_mmr[k] = is_num(i31) ? 1.0 / K::mw_dry_air : K::adv_mass(i31) / K::mw_dry_air;
  }
  C.fcvt_soag = K::adv_mass(5) / 150;
  // renaming pair aitken -> accumulation (rename.hpp:393-476)
  {
    const double alnsg = log(K::sig(1));
    C.rn_fac = sqrt(0.5) / alnsg;
    C.rn_v2n_lo_rlx = 1.0 / h_vol_from_diam(K::dmin(1), K::sig(1)) * 27.0;
    C.rn_v2n_hi_rlx = 1.0 / h_vol_from_diam(K::dmax(1), K::sig(1)) / 27.0;
    C.rn_ln_tail_fac = 3.0 * (alnsg * alnsg);
    const double alnsg_d = log(K::sig(0));
    const double cutoff = sqrt(K::dnom(1) * exp(1.5 * (alnsg * alnsg)) * K::dnom(0) *
                               exp(1.5 * (alnsg_d * alnsg_d)));
    C.rn_ln_cutoff = log(cutoff);
    C.rn_threshold = 0.99 * cutoff;
  }
  // nucleation size bounds (mam4_amicphys.hpp:990-1008)
  C.nuc_dplom = exp(0.67 * log(K::dmin(1)) + 0.33 * log(K::dnom(1)));
  {
    const double tmpa = 1770.0 * K::pi / 6.0;
    C.nuc_mass1p_lo = tmpa * (pow(C.nuc_dplom, 3.0));
    C.nuc_mass1p_hi = tmpa * (pow(K::dmax(1), 3.0));
  }
  // aging (aging.hpp:82-150)
  {
    const double mw_soa = 150 / 1000.0, mw_so4 = 115 / 1000.0;
    C.so4_vol = mw_so4 * 1000.0 / 1770.0;
    const double soa_vol = mw_soa * 1000.0 / 1000.0;
    C.soa_fac_eqvhyg = soa_vol * 0.14000000000000001 / 0.50700000000000001;
    const double l = log(K::sig(3));
    C.aging_fac_volsfc = exp(2.5 * (l * l));
  }
  C.geomean_ait_acc = sqrt(C.n2v_nom[1]) * sqrt(C.n2v_nom[0]);
  C.hystfac = 1.0 / dmax(1.0e-5, (K::rh_deliq - K::rh_cryst));
  C.kohler_aa = 2.0e4 * 18.0 * 76.0 / (8.3e7 * 273.0 * 1.0);
  return C;
}

__global__ void init_consts_kernel(StepConsts *out) { *out = make_consts(); }

// ============================================ scratch of the no-alloc step
// mam4b_step_slab_noalloc keeps the pipeline's working memory in this one
// array instead of context allocations: SOA loop state [SOA_FIELDS][ncell],
// hand-off [H_FIELDS][ncell], queue and solver order ([ncell] ints each),
// per-cell values of the size and mode kernels [AUX_FIELDS][ncell], and a
// 256-byte tail with the queue counters and a spare flag word. Host code must not pass the
// name g_noalloc_scratch to a kernel (on the host it is a stand-in, not a
// device address); it uses the address from cudaGetSymbolAddress.
constexpr size_t kNoAllocCells = MAM4B_NOALLOC_MAX_CELLS;
constexpr size_t kNoAllocSoa = 0;
constexpr size_t kNoAllocHand = kNoAllocSoa + (size_t)SOA_FIELDS * kNoAllocCells;
constexpr size_t kNoAllocDone = kNoAllocHand + (size_t)H_FIELDS * kNoAllocCells;
constexpr size_t kNoAllocOrder = kNoAllocDone + kNoAllocCells / 2;
constexpr size_t kNoAllocAux = kNoAllocOrder + kNoAllocCells / 2;
constexpr size_t kNoAllocTail = kNoAllocAux + (size_t)AUX_FIELDS * kNoAllocCells;
constexpr size_t kNoAllocDoubles = kNoAllocTail + 32;
static_assert(kNoAllocCells % 64 == 0, "scratch regions stay 256-byte aligned");
static_assert(sizeof(StepConsts) <= (size_t)SOA_FIELDS * kNoAllocCells * sizeof(double),
              "constants staging fits in the SOA region");
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

// ---- per-process entries (CalcSize, Coagulation): one thread per cell
__global__ void __launch_bounds__(128) calcsize_process_kernel(const __grid_constant__ CalcSizeArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.ncell)
    calcsize_process_cell(c_k, a, c);
}

// In two stages, as the step's pair_kernel and post_kernel: one thread per
// (cell, mode pair) for the coefficients (the FP64 exp/pow/sqrt chains,
// with many warps resident), then one thread per cell for the update.
__global__ void __launch_bounds__(128) coag_pair_process_kernel(const __grid_constant__ CoagProcessArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const CoagTables T = {kCoagBm0ij, kCoagBm3i, kCoagBm0};
  const int p = blockIdx.y;
  const size_t n = (size_t)a.ncell;
  double bij0, bij3, bii0, bjj0;
  coag_process_pair(c_k, T, a, c, p, bij0, bij3, bii0, bjj0);
  a.cc[p * n + c] = bij0;
  a.cc[(3 + p) * n + c] = bij3;
  a.cc[(6 + p) * n + c] = bii0;
  a.cc[(9 + p) * n + c] = bjj0;
}

__global__ void __launch_bounds__(128) coag_process_kernel(const __grid_constant__ CoagProcessArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  const size_t n = (size_t)a.ncell;
  double cc[12];
#pragma unroll
  for (int k = 0; k < 12; ++k)
    cc[k] = a.cc[k * n + c];
  coag_process_update(a, c, cc);
}

// ---- aqueous sulfate chemistry (setsox), one thread per cell
struct SetsoxArgs {
  const double *press, *temp, *lwc, *cldfrc, *cldnum, *xhnm;
  double *qin, *qcw;  // [31][ld]
  double *dso4, *dh2so4;  // [3][ld] or null
  size_t ld;
  long long ncell;
  double dt;
};

__global__ void __launch_bounds__(128) setsox_kernel(const __grid_constant__ SetsoxArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  constexpr int kIn[4] = {0, 1, 2, 3};
  constexpr int kCw[7] = {6, 13, 14, 18, 21, 26, 30};
  double qin[31], qcw[31];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    qin[kIn[k]] = a.qin[(size_t)kIn[k] * a.ld + c];
#pragma unroll
  for (int k = 0; k < 7; ++k)
    qcw[kCw[k]] = a.qcw[(size_t)kCw[k] * a.ld + c];
  double dso4[3], dh2so4[3];
  sox::setsox_cell(a.dt, a.press[c], a.temp[c], a.lwc[c], a.cldfrc[c], a.cldnum[c], a.xhnm[c],
                   qin, qcw, dso4, dh2so4);
#pragma unroll
  for (int k = 1; k < 4; ++k)
    a.qin[(size_t)k * a.ld + c] = qin[k];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    a.qcw[(size_t)sox::so4_cw(m) * a.ld + c] = qcw[sox::so4_cw(m)];
    if (a.dso4)
      a.dso4[(size_t)m * a.ld + c] = dso4[m];
    if (a.dh2so4)
      a.dh2so4[(size_t)m * a.ld + c] = dh2so4[m];
  }
}

// ---- gas-phase chemistry (gas_phase_chemistry), one thread per cell
struct GasChemArgs {
  const double *temp, *photo;
  const double *extfrc, *inv, *het;  // [9][ld], [8][ld], [31][ld]
  double *qq;                        // [31][ld]
  size_t ld;
  long long ncell;
  double dt;
};

// 4 blocks of 128 per SM (128 registers, the solver's spills in L1): 2.0 ms
// on 65,536 x 72 cells against 3.0 ms unconstrained at 247 registers.
__global__ void __launch_bounds__(128, 4) gaschem_kernel(const __grid_constant__ GasChemArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  double ext[gch::kExt], inv[gch::kInv], qq[gch::kTracers];
  // O3 is neither read nor changed
  auto start = [&](int t) { return t == 0 ? 0.0 : a.qq[(size_t)t * a.ld + c]; };
#pragma unroll
  for (int e = 0; e < gch::kExt; ++e)
    ext[e] = __ldg(a.extfrc + (size_t)e * a.ld + c);
#pragma unroll
  for (int i = 0; i < gch::kInv; ++i)
    inv[i] = __ldg(a.inv + (size_t)i * a.ld + c);
  // removal rates are read where used (each Newton iteration): after the
  // first read they come from L1, and the solver's registers stay free
  const double *het_c = a.het + c;
  const size_t ld = a.ld;
  auto het = [het_c, ld](int t) { return __ldg(het_c + (size_t)t * ld); };
  gch::gas_chemistry_from(__ldg(a.temp + c), a.dt, __ldg(a.photo + c), ext, inv, het, start, qq);
#pragma unroll
  for (int k = 1; k < gch::kTracers; ++k)
    a.qq[(size_t)k * a.ld + c] = qq[k];
}

// ---- aerosol activation (ndrop get_activate_frac), one thread per cell
struct ActivateArgs {
  const double *temp, *aer[NPOP], *rho, *w;
  double *out;  // [17][ld]
  size_t ld;
  long long ncell;
};

__global__ void __launch_bounds__(128) activate_kernel(const __grid_constant__ ActivateArgs a) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell)
    return;
  double ai[NPOP], out[17];
#pragma unroll
  for (int p = 0; p < NPOP; ++p)
    ai[p] = __ldg(a.aer[p] + c);
  const double rho = __ldg(a.rho + c);
  act::activate_cell(c_k, ai, rho, rho, __ldg(a.w + c), __ldg(a.temp + c), out);
#pragma unroll
  for (int k = 0; k < 17; ++k)
    a.out[(size_t)k * a.ld + c] = out[k];
}

// ---- aerosol optics (modal_aero_lw_k, modal_aero_sw) in three launches, as
// the step is split: mode sizes per cell (calcsize, RH), water uptake and
// what the bands take of a mode per (cell, mode), then the products per
// (cell, band) summed over the modes in order. Scratch rows (per cell): dry
// diameter [4], RH, ModeOptics [4][4], extinction of geometric optics [4]
// (shortwave; 0: use the fit), visible-band optical depth of each mode [4]
// (shortwave).
//
// With trop (aero_rad_props) the volcanic extinction is put over the modal
// optics at and above the column's tropopause level in the same pass: at the
// level the two are averaged, above it the volcanic values replace the modal
// ones (volcanic_cmip_sw, aero_rad_props.hpp:38-119;
// compute_odap_volcanic_at/above_troplayer_lw :121-208), whose computation
// is then skipped but for the visible band of the column optical depth.
enum { OS_DGN = 0, OS_RH = 4, OS_MODE = 5, OS_GEO = 21, OS_AOD = 25, OS_FIELDS = 29,
       OS_LW_FIELDS = 21 };
struct OpticsArgs {
  const double *in[MAM4B_NIN];
  const double *pdeldry;
  const double *tables;          // packed bands (opt::pack_band)
  double *out;                   // longwave [16][ld]; shortwave [4][14][ld]: tauxar, wa, ga, fa
  double *scr;                   // [OS_FIELDS or OS_LW_FIELDS][ncell]
  double *aodvis;                // shortwave: [ncol] or null
  const int *trop;               // [ncol] or null: tropopause levels
  const int *modal;              // with trop: the cells at or below the tropopause level
  const unsigned *nmodal;        // their number
  const double *zi;              // [col * (nlev + 1) + k]: interface height (with trop)
  const double *ext, *ssa, *af;  // [band][ld] (with trop; ssa, af shortwave)
  size_t ld;
  long long ncell;
  int ncol, nlev;
  double dt;
};

// Level of a cell relative to its column's tropopause: -1 above (the
// volcanic values replace the modal ones), 0 at it, 1 below; 1 without trop.
__device__ __forceinline__ int rel_to_tropopause(const OpticsArgs &a, long long c) {
  if (!a.trop)
    return 1;
  const unsigned col = (unsigned)c / (unsigned)a.nlev;
  const int k = (int)((unsigned)c - col * (unsigned)a.nlev), lev = __ldg(a.trop + col);
  return k < lev ? -1 : k == lev ? 0 : 1;
}
__device__ __forceinline__ double layer_thickness(const OpticsArgs &a, long long c) {
  const size_t i = (size_t)c + (unsigned)c / (unsigned)a.nlev;
  return __ldg(a.zi + i) - __ldg(a.zi + i + 1);
}
// The cell of work item i of the modal stages, -1 for none: every cell, or
// with trop the listed ones when nothing needs the others.
__device__ __forceinline__ long long modal_cell(const OpticsArgs &a, long long i) {
  if (!a.trop || a.aodvis)
    return i < a.ncell ? i : -1;
  return i < (long long)*a.nmodal ? a.modal[i] : -1;
}

__global__ void __launch_bounds__(128) optics_size_kernel(const __grid_constant__ OpticsArgs a) {
  const long long c = modal_cell(a, (long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (c < 0)
    return;
  double ai[NPOP], ac[NPOP], dgn_a[NMODE], pt_i[NPOP], pt_c[NPOP];
#pragma unroll
  for (int p = 0; p < NPOP; ++p) {
    ai[p] = __ldg(a.in[MAM4B_IN_AER_I + p] + c);
    ac[p] = __ldg(a.in[MAM4B_IN_AER_C + p] + c);
  }
  calcsize(c_k, ai, ac, a.dt, dgn_a, pt_i, pt_c);
  const size_t n = (size_t)a.ncell;
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    a.scr[(OS_DGN + m) * n + c] = dgn_a[m];
  a.scr[OS_RH * n + c] = water_uptake_rh(__ldg(a.in[MAM4B_IN_QV] + c), __ldg(a.in[MAM4B_IN_T] + c),
                                         __ldg(a.in[MAM4B_IN_P] + c), __ldg(a.in[MAM4B_IN_CLD] + c));
}

template <int M, bool SW>
__device__ __forceinline__ void optics_mode_work(const OpticsArgs &a, long long c) {
  const size_t n = (size_t)a.ncell;
  double sp[7];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    sp[s] = (s < K::nspec(M)) ? __ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0;
  double dgn_w, qw, wd;
  water_uptake_mode<M>(c_k, sp, a.scr[OS_RH * n + c], a.scr[(OS_DGN + M) * n + c], dgn_w, qw,
                       wd);
  // modal_size_parameters: the log of the surface-mode radius by method 2
  // (longwave) or of the radius itself (shortwave, method 1)
  const double alnsg = log(K::sig(M));
  double lrad;
  if constexpr (SW) {
    const double rad = 0.5 * dgn_w * exp(2.0 * alnsg * alnsg);
    lrad = log(rad);
    a.scr[(OS_GEO + M) * n + c] = lrad <= log(25.e-6) ? 0.0 : 1.5 / (rad * 1.0e3);
  } else {
    lrad = log(0.5 * dgn_w) + 2.0 * alnsg * alnsg;
  }
  const opt::ModeOptics o = opt::mode_optics<M>(sp, lrad, qw, SW);
  double *s = a.scr + (OS_MODE + 4 * M) * n + c;
  s[0] = o.xrad;
  s[n] = o.water;
  s[2 * n] = o.inv_wet;
  s[3 * n] = o.wet1000;
}

// Cells regrouped by humidity, as in mode_kernel.
template <bool SW>
__global__ void __launch_bounds__(256) optics_mode_kernel(const __grid_constant__ OpticsArgs a) {
  const long long c0 = modal_cell(a, (long long)blockIdx.x * blockDim.x + threadIdx.x);
  const long long i = group_cells(
      c0 >= 0, c0 >= 0 && a.scr[OS_RH * (size_t)a.ncell + c0] < K::rh_cryst);
  if (i < 0)
    return;
  const long long c = modal_cell(a, i);
  switch (blockIdx.y) {
  case 0: optics_mode_work<0, SW>(a, c); break;
  case 1: optics_mode_work<1, SW>(a, c); break;
  case 2: optics_mode_work<2, SW>(a, c); break;
  default: optics_mode_work<3, SW>(a, c); break;
  }
}

// What a band reads of mode M of a cell. The next mode's values are loaded
// before the current one's fits, whose arithmetic hides the latency.
struct ModeIn {
  opt::ModeOptics o;
  double geo, sp[7];
};
template <int M, bool SW>
__device__ __forceinline__ ModeIn load_mode(const OpticsArgs &a, long long c) {
  const size_t n = (size_t)a.ncell;
  const double *q = a.scr + (OS_MODE + 4 * M) * n + c;
  ModeIn x;
  x.o = {q[0], q[n], q[2 * n], q[3 * n]};
  x.geo = 0.0;
  if constexpr (SW)
    x.geo = a.scr[(OS_GEO + M) * n + c];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    x.sp[s] = s < K::nspec(M) ? __ldg(a.in[MAM4B_IN_AER_I + K::spec0(M) + (s < K::nspec(M) ? s : 0)] + c) : 0.0;
  return x;
}
// The four modes of a cell in the staged band s: the NQ fits of each mode
// go to put(mode, fit, its ModeIn).
template <int NQ, int NODE, class Put>
__device__ __forceinline__ void band_modes(const OpticsArgs &a, const double *s, long long c,
                                           const Put &put) {
  constexpr bool SW = NQ == 3;
  double fit[NQ];
  const ModeIn m0 = load_mode<0, SW>(a, c);
  const ModeIn m1 = load_mode<1, SW>(a, c);
  opt::mode_fit<0, NQ, NODE>(s, m0.sp, m0.o, fit);
  put(std::integral_constant<int, 0>(), fit, m0);
  const ModeIn m2 = load_mode<2, SW>(a, c);
  opt::mode_fit<1, NQ, NODE>(s, m1.sp, m1.o, fit);
  put(std::integral_constant<int, 1>(), fit, m1);
  const ModeIn m3 = load_mode<3, SW>(a, c);
  opt::mode_fit<2, NQ, NODE>(s, m2.sp, m2.o, fit);
  put(std::integral_constant<int, 2>(), fit, m2);
  opt::mode_fit<3, NQ, NODE>(s, m3.sp, m3.o, fit);
  put(std::integral_constant<int, 3>(), fit, m3);
}
// The block's band into shared memory.
template <int DOUBLES>
__device__ __forceinline__ void stage_band(const OpticsArgs &a, int b, double *s) {
  const double2 *g = reinterpret_cast<const double2 *>(a.tables + (size_t)b * DOUBLES);
  for (int i = threadIdx.x; i < DOUBLES / 2; i += blockDim.x)
    reinterpret_cast<double2 *>(s)[i] = __ldg(g + i);
  __syncthreads();
}
static_assert(opt::kLwBandDoubles % 2 == 0 && opt::kSwBandDoubles % 2 == 0 &&
                  opt::kBandNodes % 2 == 0 && opt::kBandGrids % 2 == 0 &&
                  opt::kGridDoubles % 2 == 0 && opt::kPointsRe % 2 == 0 && opt::kLwNode % 2 == 0 && opt::kSwNode % 2 == 0,
              "16-byte loads of the staged tables");

// The band is the grid's fastest index: the blocks of one group of cells
// run back to back for every band, so each cell's inputs come from DRAM
// once and from L2 for the other bands. Each block stages its band's tables
// once and steps several groups of cells with them: the cells with modal
// optics (listed ones with trop, whose warps are then full), then the cells
// above the tropopause.
constexpr int kBandBlock = 256;
// blocks per band at most: 256, 512 and 1,024 took 0.974, 0.966 and 0.998 ms
// longwave and 1.72, 1.69 and 1.69 shortwave on 16,384 x 72 cells
constexpr unsigned kBandCellBlocks = 512;
template <class Modal, class Above>
__device__ __forceinline__ void band_cells(const OpticsArgs &a, bool all, const Modal &modal,
                                           const Above &above) {
  const long long i0 = (long long)blockIdx.y * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.y * blockDim.x;
  if (!a.trop || all) {
    for (long long c = i0; c < a.ncell; c += stride)
      modal(c);
    return;
  }
  const long long nm = (long long)*a.nmodal;
  for (long long i = i0; i < nm; i += stride)
    modal((long long)__ldg(a.modal + i));
  for (long long c = i0; c < a.ncell; c += stride)
    if (rel_to_tropopause(a, c) < 0)
      above(c);
}

__global__ void __launch_bounds__(kBandBlock, 3) optics_band_kernel(const __grid_constant__ OpticsArgs a) {
  __shared__ __align__(16) double s[opt::kLwBandDoubles];
  const int b = blockIdx.x;
  stage_band<opt::kLwBandDoubles>(a, b, s);
  double *out = a.out + (size_t)b * a.ld;
  auto volcanic = [&](long long c) {
    return layer_thickness(a, c) * __ldg(a.ext + (size_t)b * a.ld + c);
  };
  band_cells(
      a, false,
      [&](long long c) {
        const double mass = __ldg(a.pdeldry + c) * (1.0 / 9.80616);
        double tau = 0.0;
        band_modes<1, opt::kLwNode>(a, s, c, [&](auto, const double (&fit)[1], const ModeIn &x) {
          tau = fma(dmax(0.0, fit[0] * x.o.wet1000), mass, tau);
        });
        if (rel_to_tropopause(a, c) == 0)
          tau = 0.5 * (tau + volcanic(c));
        out[c] = tau;
      },
      [&](long long c) { out[c] = volcanic(c); });
}

// Bound by the instructions of the mixing, the bracket search and the fits
// (about 230 per mode and band) and by shared-memory reads of the brackets'
// corners (32 of 16 bytes per lane, mode and band: 120 cycles per warp at
// least). With the tables as the host gives them (one 8-byte read per
// coefficient and corner, linear search, species volumes and two divisions
// again in every band) 920 instructions per mode and band: the shortwave
// entry of 16,384 x 72 cells took 3.84 ms (this kernel 2.9) and takes 1.67,
// the longwave one 2.78 and 0.93.
__global__ void __launch_bounds__(kBandBlock, 3) optics_sw_band_kernel(const __grid_constant__ OpticsArgs a) {
  __shared__ __align__(16) double s[opt::kSwBandDoubles];
  const int b = blockIdx.x;
  const size_t n = (size_t)a.ncell;
  stage_band<opt::kSwBandDoubles>(a, b, s);
  const bool diag = a.aodvis && b == opt::kSwDiagBand;
  auto store = [&](long long c, const double (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      a.out[((size_t)q * opt::kSwBands + b) * a.ld + c] = v[q];
  };
  auto volcanic = [&](long long c, double (&v)[4]) {
    const double ext = layer_thickness(a, c) * __ldg(a.ext + (size_t)b * a.ld + c);
    const double asym = __ldg(a.af + (size_t)b * a.ld + c);
    v[0] = ext;
    v[1] = ext * __ldg(a.ssa + (size_t)b * a.ld + c);
    v[2] = v[1] * asym;
    v[3] = v[2] * asym;
  };
  band_cells(
      a, diag,
      [&](long long c) {
        const double mass = __ldg(a.pdeldry + c) * (1.0 / 9.80616);
        double sum[4] = {0.0, 0.0, 0.0, 0.0};
        band_modes<3, opt::kSwNode>(a, s, c, [&](auto mode, const double (&fit)[3], const ModeIn &x) {
          constexpr int M = decltype(mode)::value;
          if (opt::no_optics(x.o)) {
            if (diag)
              a.scr[(OS_AOD + M) * n + c] = 0.0;
            return;
          }
          const double pext = (x.geo == 0.0 ? exp(fit[0]) : x.geo) * x.o.wet1000;
          const double pabs = bound(0.0, pext, fit[1] * x.o.wet1000);
          const double palb = 1.0 - pabs / dmax(pext, 1.e-40);
          double o = pext * mass;
          if (diag)
            a.scr[(OS_AOD + M) * n + c] = o;
          sum[0] += o;
          o *= palb;
          sum[1] += o;
          o *= fit[2];
          sum[2] += o;
          sum[3] = fma(o, fit[2], sum[3]);
        });
        const int rel = rel_to_tropopause(a, c);
        if (rel <= 0) {
          double v[4];
          volcanic(c, v);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            sum[q] = rel == 0 ? 0.5 * (sum[q] + v[q]) : v[q];
        }
        store(c, sum);
      },
      [&](long long c) {
        double v[4];
        volcanic(c, v);
        store(c, v);
      });
}

// visible optical depth of each column: its levels' mode optical depths
// summed, one warp per column
__global__ void __launch_bounds__(128) optics_sw_aod_kernel(const __grid_constant__ OpticsArgs a) {
  const int lane = threadIdx.x & 31;
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= a.ncol)
    return;  // the whole warp
  const size_t n = (size_t)a.ncell;
  double s = 0.0;
  for (int k = lane; k < a.nlev; k += 32) {
    const size_t c = (size_t)col * a.nlev + k;
#pragma unroll
    for (int m = 0; m < NMODE; ++m)
      s += a.scr[(OS_AOD + m) * n + c];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0)
    a.aodvis[col] = s;
}

// ---- aero_rad_props: the tropopause of each column
struct RadArgs {
  const double *temp, *pmid;     // step input fields (cell = col * nlev + k)
  const double *pint;            // [col * (nlev + 1) + k]: interface pressure
  int *trop;                     // [ncol]
  int *modal;                    // [ncol * nlev]: the cells at or below the level
  unsigned *nmodal;              // their number (zero at the launch)
  int ncol, nlev;
};

// one warp per column: the lanes compute every layer's lapse-rate
// quantities (the pow-heavy part) into shared memory, then one lane runs
// the scan on them, and the column's cells at or below the level go to the
// list of cells with modal optics
__global__ void __launch_bounds__(128) tropopause_kernel(const __grid_constant__ RadArgs r) {
  extern __shared__ double tsm[];  // [warps][4][nlev]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nlev = r.nlev;
  const int col = blockIdx.x * (blockDim.x >> 5) + warp;
  if (col >= r.ncol)
    return;  // the whole warp: col is the same on every lane
  double *s = tsm + (size_t)warp * 4 * nlev;
  const size_t c0 = (size_t)col * nlev, i0 = (size_t)col * (nlev + 1);
  auto T = [&](int k) { return __ldg(r.temp + c0 + k); };
  auto P = [&](int k) { return __ldg(r.pmid + c0 + k); };
  // p^kappa of every level first (in the last row, whose layer values
  // replace it): a layer needs those of both its levels
  double *pk = s + 3 * nlev;
  for (int k = lane; k < nlev; k += 32)
    pk[k] = rad::p_kappa(P(k));
  __syncwarp();
  for (int k0 = 1; k0 < nlev; k0 += 32) {
    const int k = k0 + lane;
    rad::LapsePair q;
    if (k < nlev)
      q = rad::lapse_pair(T, P, k, pk[k - 1], pk[k]);
    __syncwarp();  // the next 32 layers still read pk[k0 + 31] and above
    if (k < nlev) {
      s[k] = q.pmk;
      s[nlev + k] = q.pm;
      s[2 * nlev + k] = q.dtdz;
      // layer k + 31's pk[k - 1 + 32] is read by the next round: write one
      // below, where this round was the last reader
      pk[k - 1] = q.tm;
    }
    __syncwarp();
  }
  int lev = 0;
  if (lane == 0) {
    auto pair = [&](int k) {
      rad::LapsePair q;
      q.pmk = s[k];
      q.pm = s[nlev + k];
      q.dtdz = s[2 * nlev + k];
      q.tm = pk[k - 1];
      return q;
    };
    auto PI = [&](int k) { return __ldg(r.pint + i0 + k); };
    lev = rad::tropopause_level_at(rad::twmo_from_pairs(pair, nlev), PI, nlev);
    r.trop[col] = lev;
  }
  lev = __shfl_sync(0xffffffffu, lev, 0);
  unsigned base = 0;
  if (lane == 0)
    base = atomicAdd(r.nmodal, (unsigned)(nlev - lev));
  base = __shfl_sync(0xffffffffu, base, 0);
  for (int k = lev + lane; k < nlev; k += 32)
    r.modal[base + (k - lev)] = (int)(c0 + k);
}

// ---- droplet activation and vertical mixing (ndrop dropmixnuc) in three
// launches: the activations per cell, the columns' cloud changes and
// sub-stepped mixing, the CCN per cell.
struct DropmixArgs {
  const double *in[MAM4B_NIN];  // step input fields: T, p, z, cloud fraction, populations
  const double *mix;            // [MAM4B_DROPMIX_NIN][ld]
  const double *pint, *kvh;     // [col * (nlev + 1) + k]
  double *out;                  // [MAM4B_DROPMIX_NOUT][ld]
  double *act;                  // [DA_FIELDS][ncol * nlev]: activation results
  unsigned *flags;
  size_t ld;
  int ncol, nlev, top_lev, vertical_mix;
  double dt;
};
// activation results of a level, computed ahead by dropmix_act_kernel:
// growing cloud (computed flag, fn, fm) and cloud base (flag, fn, fluxn,
// fluxm)
enum { DA_NEW_OK = 0, DA_NEW_FN = 1, DA_NEW_FM = 5, DA_BASE_OK = 9, DA_BASE_FN = 10,
       DA_BASE_FLUXN = 14, DA_BASE_FLUXM = 18, DA_FIELDS = 22 };

constexpr int kDmMaxSub = 100000;  // bound on the mixing sub-steps
constexpr int kDmActBlock = 256;

// The activations of every level (they read only the inputs) ahead of the
// column kernel: growing cloud activates the level's own aerosol, a cloud
// base the aerosol of the level below. Both are wanted in a fraction of the
// cells, so a block collects the activations of its cells in a list and its
// threads take them from there: a thread per cell ran them with 6.6 of 32
// lanes active (0.92 ms on 16,384 x 72 cells).
__global__ void __launch_bounds__(kDmActBlock) dropmix_act_kernel(const __grid_constant__ DropmixArgs a) {
  __shared__ int s_task[2 * kDmActBlock];  // 2 * (cell of the block) + (cloud base)
  __shared__ unsigned s_count;
  const long long n = (long long)a.ncol * a.nlev;
  const long long b0 = (long long)blockIdx.x * blockDim.x;
  auto IN = [&](int f, long long cc) { return __ldg(a.in[f] + cc); };
  if (threadIdx.x == 0)
    s_count = 0;
  __syncthreads();
  {
    const long long c = b0 + threadIdx.x;
    bool grow = false, base = false;
    if (c < n) {
      a.act[(size_t)DA_NEW_OK * n + c] = 0.0;
      a.act[(size_t)DA_BASE_OK * n + c] = 0.0;
      const int k = (int)(c % a.nlev);
      if (k >= a.top_lev) {
        const double cldn = IN(MAM4B_IN_CLD, c);
        grow = cldn - __ldg(a.mix + (size_t)MAM4B_DROPMIX_IN_CLDO * a.ld + c) > 0.01;
        base = k < a.nlev - 1 && cldn > 0.01 && cldn - IN(MAM4B_IN_CLD, c + 1) > 0.01;
      }
    }
    const unsigned mg = __ballot_sync(0xffffffffu, grow), mb = __ballot_sync(0xffffffffu, base);
    const int lane = threadIdx.x & 31;
    unsigned at = 0;
    if (lane == 0)
      at = atomicAdd(&s_count, (unsigned)(__popc(mg) + __popc(mb)));
    at = __shfl_sync(0xffffffffu, at, 0);
    const unsigned below = (1u << lane) - 1u;
    if (grow)
      s_task[at + __popc(mg & below)] = 2 * threadIdx.x;
    if (base)
      s_task[at + __popc(mg) + __popc(mb & below)] = 2 * threadIdx.x + 1;
  }
  __syncthreads();
  const double rair = act::kRAir;
  for (unsigned i = threadIdx.x; i < s_count; i += blockDim.x) {
    const int task = s_task[i];
    const bool base = task & 1;
    const long long c = b0 + (task >> 1), from = base ? c + 1 : c;  // the aerosol's level
    const double temp = IN(MAM4B_IN_T, c), cs = IN(MAM4B_IN_P, c) / (rair * temp);
    const double cs1 = IN(MAM4B_IN_P, from) / (rair * IN(MAM4B_IN_T, from));
    const double wtke = dmax(__ldg(a.mix + (size_t)MAM4B_DROPMIX_IN_WSUB * a.ld + c), 0.1);
    double ai[NPOP], o[17];
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      ai[p] = IN(MAM4B_IN_AER_I + p, from);
    const bool ok = act::activate_cell(c_k, ai, cs1, cs, wtke, temp, o);
    double *r = a.act + c;
    r[(size_t)(base ? DA_BASE_OK : DA_NEW_OK) * n] = ok ? 1.0 : 0.0;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      r[(size_t)((base ? DA_BASE_FN : DA_NEW_FN) + m) * n] = o[m];
      if (base) {
        r[(size_t)(DA_BASE_FLUXN + m) * n] = o[8 + m];
        r[(size_t)(DA_BASE_FLUXM + m) * n] = o[12 + m];
      } else {
        r[(size_t)(DA_NEW_FM + m) * n] = o[4 + m];
      }
    }
  }
}

// Level fields of a column in shared memory (doubles, [field][nlev]).
enum {
  DM_CS = 0, DM_DZ, DM_ZN, DM_ZS, DM_EDDY, DM_CSBOT, DM_CSBOT_CSCEN, DM_WTKE,
  // coefficients of a sub-step (explmix, explmix_act), its length multiplied
  // in: what level k + 1 and k - 1 give to the cloud-borne (WP, WM) and
  // interstitial (RP, RM) amounts, the interstitial gain from the neighbours'
  // cloud-borne amounts where the cloud does not overlap (XP, XM), the loss
  // (C); zero above top_lev
  DM_WP, DM_WM, DM_RP, DM_RM, DM_XP, DM_XM, DM_C,
  DM_FRAC,                         // relative loss of a shrinking cloud (DM_CHANGE < 0)
  DM_GROW,                         // growth of a growing cloud (DM_CHANGE > 0)
  DM_CHANGE,                       // -1 shrinking, 1 growing, 0 neither
  DM_CLEAR,                        // 1: no cloud left, what was cloud-borne is released
  DM_QCLD, DM_NSOURCE,             // droplet number before mixing, its source
  // activation rates, times the sub-step once it is known
  DM_NACT, DM_MACT = DM_NACT + NMODE, DM_FNUM = DM_MACT + NMODE, DM_FM = DM_FNUM + NMODE,
  DM_FIELDS = DM_FM + NMODE
};
// warps per column; each has a row of staging for whole-line loads and stores
constexpr int kDmWarps = 4;

// Populations by warp: the four numbers (and the droplet number, which the
// activation of the numbers feeds) go to one warp, seven masses to each of
// the others.
__device__ __forceinline__ int dm_mass_pop(int i) {
  // mass i (0..20) in population order
  return i + (i >= 7) + (i >= 11) + (i >= 18);
}

// The column: cloud changes, cloud-base activation and the mixing
// coefficients per level in shared memory by all threads, then the sub-steps
// in registers, a lane holding L consecutive levels and taking its
// neighbours' by shuffles. Populations are independent (the droplet number
// alone reads the four aerosol numbers), so there is no barrier in the
// sub-steps. With the populations in shared memory (73 KB a column, nine
// warps per SM), a work item per (level, population) and a barrier per
// sub-step the column kernel took 6.4 ms on 16,384 x 72 cells (now 2.1); with four
// populations at a time the loops outgrow the instruction cache (a warp
// waits 10 cycles per instruction).
template <int L>
__global__ void __launch_bounds__(32 * kDmWarps, L <= 3 ? 4 : L <= 4 ? 3 : 2)
    dropmix_kernel(const __grid_constant__ DropmixArgs a) {
  extern __shared__ double sm[];
  const int col = blockIdx.x, nlev = a.nlev, top = a.top_lev;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // numbers (0) or masses: the numbers' longer loop goes to another SM
  // partition from block to block
  const int role = (warp + blockIdx.x) & (kDmWarps - 1);
  const size_t c0 = (size_t)col * nlev, i0 = (size_t)col * (nlev + 1), ld = a.ld;
  double *stage = sm + (size_t)(DM_FIELDS + warp) * nlev;
  auto S = [&](int f, int k) -> double & { return sm[(size_t)f * nlev + k]; };
  auto IN = [&](int f, int k) { return __ldg(a.in[f] + c0 + k); };
  auto MIX = [&](int f, int k) { return __ldg(a.mix + (size_t)f * ld + c0 + k); };
  const size_t ncell = (size_t)a.ncol * nlev;
  auto ACT = [&](int f, int k) { return __ldg(a.act + (size_t)f * ncell + c0 + k); };
  const double dt = a.dt, dtinv = 1.0 / dt;
  const double gravity = act::kGravity, rair = act::kRAir;

  // per-level quantities (dropmixnuc :1440-1490) and the new cloud
  // (update_from_newcld): shrinking cloud releases, growing cloud activates
  // the level's own aerosol
  for (int k = threadIdx.x; k < nlev; k += blockDim.x) {
    const double cs = IN(MAM4B_IN_P, k) / (rair * IN(MAM4B_IN_T, k));
    const double rpdel = 1.0 / MIX(MAM4B_DROPMIX_IN_PDEL, k);
    S(DM_CS, k) = cs;
    S(DM_DZ, k) = 1.0 / (cs * gravity * rpdel);
    S(DM_ZN, k) = gravity * rpdel;
    S(DM_WTKE, k) = dmax(MIX(MAM4B_DROPMIX_IN_WSUB, k), 0.1);
    // levels above top_lev keep zero, as the reference's work arrays
    double zs = 0.0, eddy = 0.0, csbot = 0.0, csr = 0.0;
    double qcld = MIX(MAM4B_DROPMIX_IN_NCLDWTR, k), nsource = 0.0, frac = 0.0, grow = 0.0,
           change = 0.0, clear = 0.0, fnum[NMODE] = {0, 0, 0, 0}, fm[NMODE] = {0, 0, 0, 0};
    if (k >= top) {
      if (k < nlev - 1) {
        zs = 1.0 / (IN(MAM4B_IN_ZM, k) - IN(MAM4B_IN_ZM, k + 1));
        eddy = bound(0.01, 100.0, __ldg(a.kvh + i0 + k + 1));
        csbot = 2.0 * __ldg(a.pint + i0 + k + 1) /
                (rair * (IN(MAM4B_IN_T, k) + IN(MAM4B_IN_T, k + 1)));
        csr = csbot / cs;
      } else {
        zs = 1.0 / (IN(MAM4B_IN_ZM, k - 1) - IN(MAM4B_IN_ZM, k));
        csbot = IN(MAM4B_IN_P, k) / (rair * IN(MAM4B_IN_T, k));
        csr = 1.0;
      }
      const double cldn = IN(MAM4B_IN_CLD, k), cldo = MIX(MAM4B_DROPMIX_IN_CLDO, k);
      if (cldn < cldo) {
        change = -1.0;
        nsource += qcld * (cldn - cldo) / cldo * dtinv;
        frac = (cldn - cldo) / cldo;
        qcld *= (1.0 + frac);
      }
      if (cldn - cldo > 0.01) {
        change = 1.0;
        grow = cldn - cldo;
        if (ACT(DA_NEW_OK, k) != 0.0) {
#pragma unroll
          for (int m = 0; m < NMODE; ++m) {
            fnum[m] = ACT(DA_NEW_FN + m, k);
            fm[m] = ACT(DA_NEW_FM + m, k);
          }
        }
#pragma unroll
        for (int m = 0; m < NMODE; ++m) {
          const double dact = grow * fnum[m] * IN(MAM4B_IN_AER_I + K::numslot(m), k);
          qcld += dact;
          nsource += dact * dtinv;
        }
      }
      clear = k < nlev - 1 && !(cldn > 0.01) ? 1.0 : 0.0;
    }
    S(DM_ZS, k) = zs;
    S(DM_EDDY, k) = eddy;
    S(DM_CSBOT, k) = csbot;
    S(DM_CSBOT_CSCEN, k) = csr;
    S(DM_QCLD, k) = qcld;
    S(DM_NSOURCE, k) = nsource;
    S(DM_FRAC, k) = frac;
    S(DM_GROW, k) = grow;
    S(DM_CHANGE, k) = change;
    S(DM_CLEAR, k) = clear;
#pragma unroll
    for (int f = DM_WP; f <= DM_C; ++f)
      S(f, k) = 0.0;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      S(DM_NACT + m, k) = 0.0;
      S(DM_MACT + m, k) = 0.0;
      S(DM_FNUM + m, k) = fnum[m];
      S(DM_FM + m, k) = fm[m];
    }
  }
  __syncthreads();

  // amounts of population p (mode m) at level k after the new cloud
  auto new_cloud = [&](int m, int p, int k, double &r, double &w) {
    const double change = S(DM_CHANGE, k);
    if (change < 0.0) {
      const double dact = w * S(DM_FRAC, k);
      w += dact;
      r -= dact;
    } else if (change > 0.0) {
      const double f = p == K::numslot(m) ? S(DM_FNUM + m, k) : S(DM_FM + m, k);
      const double d = S(DM_GROW, k) * f * IN(MAM4B_IN_AER_I + p, k);
      w += d;
      r -= d;
    }
  };

  // cloud-base activation (update_from_cldn_profile): reads the number of
  // the level below after the new cloud, before that level's clearing
  for (int k = top + threadIdx.x; k < nlev - 1; k += blockDim.x) {
    const double cldn = IN(MAM4B_IN_CLD, k), cldn1 = IN(MAM4B_IN_CLD, k + 1);
    if (cldn > 0.01 && cldn - cldn1 > 0.01) {
      S(DM_EDDY, k) = S(DM_WTKE, k) / S(DM_ZS, k);
      const double cs = S(DM_CS, k);
      const bool ok = ACT(DA_BASE_OK, k) != 0.0;
      const double delz_cld = cldn - cldn1;
      double fluxntot = 0.0;
      const double crdz = S(DM_CSBOT_CSCEN, k) / S(DM_DZ, k);
#pragma unroll
      for (int m = 0; m < NMODE; ++m) {
        const double fluxn = ok ? ACT(DA_BASE_FLUXN + m, k) : 0.0;
        const double fluxm = ok ? ACT(DA_BASE_FLUXM + m, k) : 0.0;
        S(DM_NACT + m, k) += fluxn * crdz * delz_cld;
        S(DM_MACT + m, k) += fluxm * crdz * delz_cld;
        double r = IN(MAM4B_IN_AER_I + K::numslot(m), k + 1);
        double w = IN(MAM4B_IN_AER_C + K::numslot(m), k + 1);
        new_cloud(m, K::numslot(m), k + 1, r, w);
        fluxntot += fluxn * delz_cld * r * cs;
      }
      S(DM_NSOURCE, k) += fluxntot / (cs * S(DM_DZ, k));
    }
    if (S(DM_CLEAR, k) != 0.0) {
      S(DM_NSOURCE, k) -= S(DM_QCLD, k) * dtinv;
      S(DM_QCLD, k) = 0.0;
    }
  }
  __syncthreads();

  // mixing set-up (update_from_explmix :1192-1225); the time-step bound is
  // a minimum over levels, the same in any order
  double dtmin = 1.79769313486231570e+308;
  for (int k = top + threadIdx.x; k < nlev; k += blockDim.x) {
    const int kp1 = k + 1 < nlev ? k + 1 : nlev - 1, km1 = k - 1 > top ? k - 1 : top;
    const double cld = IN(MAM4B_IN_CLD, k), cldp = IN(MAM4B_IN_CLD, kp1), cldm = IN(MAM4B_IN_CLD, km1);
    const double ovp = cldp > 1e-10 ? dmin(cld / cldp, 1.0) : 1.0;
    const double ovm = cldm > 1e-10 ? dmin(cld / cldm, 1.0) : 1.0;
    const double ekp = S(DM_ZN, k) * S(DM_EDDY, k) * S(DM_CSBOT, k) * S(DM_ZS, k);
    // top_lev >= 1: level k - 1 exists (above top_lev its terms are zero)
    const double ekm = S(DM_ZN, k) * S(DM_EDDY, k - 1) * S(DM_CSBOT, k - 1) * S(DM_ZS, km1);
    S(DM_RP, k) = ekp;
    S(DM_RM, k) = ekm;
    S(DM_WP, k) = ekp * ovp;
    S(DM_WM, k) = ekm * ovm;
    S(DM_XP, k) = ekp * (1.0 - ovp);
    S(DM_XM, k) = ekm * (1.0 - ovm);
    S(DM_C, k) = ekp + ekm;
    const double tinv = ekp + ekm;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      S(DM_NACT + m, k) = dmin(S(DM_NACT + m, k), ekp);
      S(DM_MACT + m, k) = dmin(S(DM_MACT + m, k), ekp);
    }
    if (tinv > 1e-6)
      dtmin = dmin(dtmin, 1.0 / tinv);
  }
  __shared__ double red[kDmWarps];
  for (int o = 16; o > 0; o >>= 1)
    dtmin = dmin(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, o));
  if (lane == 0)
    red[warp] = dtmin;
  __syncthreads();
  dtmin = red[0];
#pragma unroll
  for (int w = 1; w < kDmWarps; ++w)
    dtmin = dmin(dtmin, red[w]);
  double dtmix = 0.9 * dtmin;
  const double nsub_d = dt / dtmix + 1;
  const int nsubmix = nsub_d < (double)kDmMaxSub ? (int)nsub_d : kDmMaxSub;
  if (!(nsub_d < (double)kDmMaxSub) && threadIdx.x == 0)
    atomicOr(a.flags, MAM4B_FLAG_NONFINITE_OUTPUT);
  dtmix = dt / nsubmix;
  for (int k = top + threadIdx.x; k < nlev; k += blockDim.x) {
#pragma unroll
    for (int f = DM_WP; f <= DM_C; ++f)
      S(f, k) *= dtmix;
#pragma unroll
    for (int f = DM_NACT; f < DM_NACT + 2 * NMODE; ++f)
      S(f, k) *= dtmix;
  }
  __syncthreads();

  // the lane's levels k0 .. k0 + L - 1; the column's lowest level is the
  // last lane's last, levels above top_lev take no part and hold zero
  const int k0 = nlev - 32 * L + lane * L;
  // a level field at the lane's levels (level 0, above top_lev, for those
  // beyond the column)
  auto field = [&](int f, double (&x)[L]) {
#pragma unroll
    for (int i = 0; i < L; ++i)
      x[i] = S(f, max(k0 + i, 0));
  };
  // row of global memory <-> the lane's levels, through the warp's staging
  auto load = [&](const double *g, double (&x)[L]) {
    __syncwarp();
    for (int k = top + lane; k < nlev; k += 32)
      stage[k] = __ldg(g + c0 + k);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < L; ++i)
      x[i] = k0 + i >= top ? stage[k0 + i] : 0.0;
  };
  auto to_stage = [&](const double (&x)[L]) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < L; ++i)
      if (k0 + i >= top)
        stage[k0 + i] = x[i];
    __syncwarp();
  };
  auto store = [&](int f, const double (&x)[L]) {
    to_stage(x);
    double *o = a.out + (size_t)f * ld + c0;
    for (int k = lane; k < nlev; k += 32)
      o[k] = k < top ? 0.0 : stage[k];
  };
  // population p (mode m) before mixing: the inputs ai, the amounts r, w
  // after the new cloud and the release where no cloud is left
  auto begin = [&](int m, int p, double (&ai)[L], double (&r)[L], double (&w)[L]) {
    load(a.in[MAM4B_IN_AER_I + p], ai);
    load(a.in[MAM4B_IN_AER_C + p], w);
#pragma unroll
    for (int i = 0; i < L; ++i) {
      r[i] = ai[i];
      if (k0 + i < top)
        continue;
      new_cloud(m, p, k0 + i, r[i], w[i]);
      if (S(DM_CLEAR, k0 + i) != 0.0) {
        r[i] += w[i];
        w[i] = 0.0;
      }
    }
  };
  // tendencies and the updated cloud-borne population; clear-sky levels give
  // their cloud-borne aerosol back
  auto finish = [&](int p, const double (&ai)[L], double (&r)[L], double (&w)[L]) {
#pragma unroll
    for (int i = 0; i < L; ++i) {
      if (k0 + i >= top && IN(MAM4B_IN_CLD, k0 + i) == 0.0) {
        r[i] += w[i];
        w[i] = 0.0;
      }
      r[i] = (r[i] - ai[i]) * dtinv;
      w[i] = dmax(w[i], 0.0);
    }
    store(MAM4B_DROPMIX_OUT_PTEND + p, r);
    store(MAM4B_DROPMIX_OUT_QQCW + p, w);
  };
  // the levels above the lane's first and below its last; the column's top
  // and lowest level stand in for the missing ones
  auto neighbours = [&](const double (&x)[L], double (&up)[L], double &dn) {
    up[0] = __shfl_up_sync(0xffffffffu, x[L - 1], 1);
    dn = __shfl_down_sync(0xffffffffu, x[0], 1);
    if (lane == 31)
      dn = x[L - 1];
#pragma unroll
    for (int i = 0; i < L; ++i) {
      if (i > 0)
        up[i] = x[i - 1];
      if (k0 + i == top)
        up[i] = x[i];
    }
  };
  struct Coef {
    double wp[L], wm[L], rp[L], rm[L], xp[L], xm[L], c[L];
  };
  auto coefficients = [&](Coef &cf) {
    field(DM_WP, cf.wp);
    field(DM_WM, cf.wm);
    field(DM_RP, cf.rp);
    field(DM_RM, cf.rm);
    field(DM_XP, cf.xp);
    field(DM_XM, cf.xm);
    field(DM_C, cf.c);
  };
  // One sub-step of a population: src receives what the activation of the
  // level below (at the lowest level of the level itself, at the rate low)
  // moves from the interstitial to the cloud-borne amount. rs: the
  // interstitial amounts read; without vertical mixing the interstitial
  // buffers are the initial one and one that stays zero, in turn, as in the
  // reference.
  const bool vmix = a.vertical_mix != 0;
  auto substep = [&](const Coef &cf, const double (&act_)[L], double low, double (&r)[L],
                     double (&w)[L], const double (&rs)[L], double (&src)[L]) {
    double ru[L], wu[L], rd, wd, rn[L], wn[L];
    neighbours(rs, ru, rd);
    neighbours(w, wu, wd);
#pragma unroll
    for (int i = 0; i < L; ++i) {
      const double rb = i < L - 1 ? rs[i < L - 1 ? i + 1 : 0] : rd;
      const double wb = i < L - 1 ? w[i < L - 1 ? i + 1 : 0] : wd;
      src[i] = act_[i] * rb;
      if (i == L - 1 && lane == 31)
        src[i] = dmax(0.0, rs[i] * low + w[i] * low);
      double dw = fma(cf.wp[i], wb, src[i]);
      dw = fma(cf.wm[i], wu[i], dw);
      wn[i] = dmax(w[i] + fma(-cf.c[i], w[i], dw), 0.0);
      double dr = fma(cf.rp[i], rb, -src[i]);
      dr = fma(cf.rm[i], ru[i], dr);
      dr = fma(cf.xp[i], wb, dr);
      dr = fma(cf.xm[i], wu[i], dr);
      rn[i] = dmax(rs[i] + fma(-cf.c[i], rs[i], dr), 0.0);
    }
#pragma unroll
    for (int i = 0; i < L; ++i) {
      w[i] = wn[i];
      if (vmix)
        r[i] = rn[i];
    }
  };
  if (role > 0) {
    Coef cf;
    coefficients(cf);
#pragma unroll 1
    for (int j = 0; j < 7; ++j) {
      const int p = dm_mass_pop(7 * (role - 1) + j), m = dmx::mode_of(p);
      double ai[L], r[L], w[L], mact[L], src[L];
      begin(m, p, ai, r, w);
      field(DM_MACT + m, mact);
      const double low = S(DM_NACT + m, nlev - 1);
      if (vmix) {
#pragma unroll 1
        for (int isub = 0; isub < nsubmix; ++isub)
          substep(cf, mact, low, r, w, r, src);
      } else {
#pragma unroll 1
        for (int isub = 0; isub < nsubmix; ++isub) {
          double rs[L];
#pragma unroll
          for (int i = 0; i < L; ++i)
            rs[i] = isub & 1 ? 0.0 : r[i];
          substep(cf, mact, low, r, w, rs, src);
        }
        if (nsubmix & 1) {
#pragma unroll
          for (int i = 0; i < L; ++i)
            r[i] = 0.0;
        }
      }
      finish(p, ai, r, w);
    }
    return;
  }
  // numbers, and the droplets, which gain what the numbers activate. The
  // coefficients are read again for every population: with them and the five
  // states in registers too few warps would fit on an SM.
  double r[NMODE][L], w[NMODE][L], q[L], ai[L];
#pragma unroll
  for (int m = 0; m < NMODE; ++m)
    begin(m, K::numslot(m), ai, r[m], w[m]);
#pragma unroll
  for (int i = 0; i < L; ++i)
    q[i] = k0 + i >= top ? S(DM_QCLD, k0 + i) : 0.0;
#pragma unroll 1
  for (int isub = 0; isub < nsubmix; ++isub) {
    double srcn[L];
#pragma unroll
    for (int i = 0; i < L; ++i)
      srcn[i] = 0.0;
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
      asm volatile("" ::: "memory");
      Coef cf;
      coefficients(cf);
      double nact[L], src[L], rs[L];
      field(DM_NACT + m, nact);
#pragma unroll
      for (int i = 0; i < L; ++i)
        rs[i] = !vmix && (isub & 1) ? 0.0 : r[m][i];
      // the lowest level's own number counts as the level below it, besides
      // its activation
      if (lane == 31)
        srcn[L - 1] += nact[L - 1] * rs[L - 1];
      substep(cf, nact, nact[L - 1], r[m], w[m], rs, src);
#pragma unroll
      for (int i = 0; i < L; ++i)
        srcn[i] += src[i];
    }
    if (vmix) {
      asm volatile("" ::: "memory");
      double wp[L], wm[L], cl[L], qu[L], qd, qn[L];
      field(DM_WP, wp);
      field(DM_WM, wm);
      field(DM_C, cl);
      neighbours(q, qu, qd);
#pragma unroll
      for (int i = 0; i < L; ++i) {
        const double qb = i < L - 1 ? q[i < L - 1 ? i + 1 : 0] : qd;
        double dq = fma(wp[i], qb, srcn[i]);
        dq = fma(wm[i], qu[i], dq);
        qn[i] = dmax(q[i] + fma(-cl[i], q[i], dq), 0.0);
      }
#pragma unroll
      for (int i = 0; i < L; ++i)
        q[i] = qn[i];
    }
  }
#pragma unroll
  for (int m = 0; m < NMODE; ++m) {
    if (!vmix && (nsubmix & 1)) {
#pragma unroll
      for (int i = 0; i < L; ++i)
        r[m][i] = 0.0;
    }
    load(a.in[MAM4B_IN_AER_I + K::numslot(m)], ai);
    finish(K::numslot(m), ai, r[m], w[m]);
  }
  to_stage(q);
  for (int k = lane; k < nlev; k += 32) {
    double *o = a.out + c0 + k;
    o[(size_t)MAM4B_DROPMIX_OUT_WTKE * ld] = S(DM_WTKE, k);
    const double ncldwtr = MIX(MAM4B_DROPMIX_IN_NCLDWTR, k);
    const bool in = k >= top;
    const double qcld = !in ? ncldwtr : IN(MAM4B_IN_CLD, k) == 0.0 ? 0.0 : stage[k];
    const double nsource = S(DM_NSOURCE, k);
    o[(size_t)MAM4B_DROPMIX_OUT_QCLD * ld] = qcld;
    o[(size_t)MAM4B_DROPMIX_OUT_NDROPMIX * ld] = in ? (qcld - ncldwtr) * dtinv - nsource : 0.0;
    o[(size_t)MAM4B_DROPMIX_OUT_TENDND * ld] = in ? (dmax(qcld, 1.e-6) - ncldwtr) * dtinv : 0.0;
    o[(size_t)MAM4B_DROPMIX_OUT_NDROPCOL * ld] =
        in ? ncldwtr * MIX(MAM4B_DROPMIX_IN_PDEL, k) / gravity : 0.0;
    o[(size_t)MAM4B_DROPMIX_OUT_NSOURCE * ld] = in ? nsource : 0.0;
    // activated fractions: the cloud base's where there is one
    const bool base = in && k < nlev - 1 && IN(MAM4B_IN_CLD, k) > 0.01 &&
                      IN(MAM4B_IN_CLD, k) - IN(MAM4B_IN_CLD, k + 1) > 0.01 &&
                      ACT(DA_BASE_OK, k) != 0.0;
#pragma unroll
    for (int m = 0; m < NMODE; ++m)
      o[(size_t)(MAM4B_DROPMIX_OUT_FACTNUM + m) * ld] =
          base ? ACT(DA_BASE_FN + m, k) : S(DM_FNUM + m, k);
  }
}

// CCN of every cell from the interstitial and the updated cloud-borne
// aerosol (zero above top_lev), one thread per cell.
__global__ void __launch_bounds__(128) dropmix_ccn_kernel(const __grid_constant__ DropmixArgs a) {
  const long long n = (long long)a.ncol * a.nlev;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n)
    return;
  double ccn[dmx::kPsat] = {};
  if ((int)(c % a.nlev) >= a.top_lev) {
    double ai[NPOP], qcb_shift[NMODE][7], qcb_num[NMODE];
#pragma unroll
    for (int p = 0; p < NPOP; ++p)
      ai[p] = __ldg(a.in[MAM4B_IN_AER_I + p] + c);
#pragma unroll
    for (int m = 0; m < NMODE; ++m) {
#pragma unroll
      for (int s = 0; s < 7; ++s)
        qcb_shift[m][s] = 0.0;
#pragma unroll
      for (int l = 0; l < K::nspec(m); ++l) {
        const double q = a.out[(size_t)(MAM4B_DROPMIX_OUT_QQCW + dmx::pop_of(m, l)) * a.ld + c];
        if (l == 0)
          qcb_num[m] = q;
        else
          qcb_shift[m][l] = q;  // species l - 1's mass, read as species l
      }
    }
    const double temp = __ldg(a.in[MAM4B_IN_T] + c);
    dmx::ccn_cell(c_k, ai, qcb_shift, qcb_num, temp,
                  __ldg(a.in[MAM4B_IN_P] + c) / (act::kRAir * temp), ccn);
  }
#pragma unroll
  for (int l = 0; l < dmx::kPsat; ++l)
    a.out[(size_t)(MAM4B_DROPMIX_OUT_CCN + l) * a.ld + c] = ccn[l];
}

}  // namespace mam4b

// =============================================================== C ABI
namespace mam4b {
// Column gather/scatter of mam4b_step_columns: tab[f * ncol + col] points
// at column col of field f (nlev doubles); slab is [nfield][ncol * nlev].
__global__ void __launch_bounds__(128) gather_columns_kernel(const double *const *tab, double *slab,
                                                             int ncol, int nlev) {
  const long long ncell = (long long)ncol * nlev;
  const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= ncell)
    return;
  const int f = blockIdx.y;
  const int col = (int)(cell / nlev), lev = (int)(cell - (long long)col * nlev);
  slab[(size_t)f * ncell + cell] = tab[(size_t)f * ncol + col][lev];
}
// first nadd fields added to their columns, the rest written; null columns skipped
__global__ void __launch_bounds__(128) scatter_columns_kernel(double *const *tab,
                                                              const double *slab, int ncol,
                                                              int nlev, int nadd) {
  const long long ncell = (long long)ncol * nlev;
  const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= ncell)
    return;
  const int f = blockIdx.y;
  const int col = (int)(cell / nlev), lev = (int)(cell - (long long)col * nlev);
  double *p = tab[(size_t)f * ncol + col];
  if (!p)
    return;
  const double v = slab[(size_t)f * ncell + cell];
  p[lev] = (f < nadd) ? p[lev] + v : v;
}
}  // namespace mam4b

using namespace mam4b;

// Host-buffer path: columns are processed in chunks of about kHostChunkCells
// cells on one stream per stage: all host->device copies back to back on
// the copy-in stream, each chunk's kernels on one of kComputeStreams
// streams once its inputs have arrived, each chunk's device->host copy on
// the copy-out stream once its kernels are done. Both copy engines stay
// busy from the first chunk to the last (the copies, not the kernels,
// bound this path); the chunks' kernels overlap, which hides the tail of
// each chunk's SOA solver (its longest loop).
constexpr int kComputeStreams = 4;
constexpr int kHostStreams = 2 + kComputeStreams;  // in, compute..., out
constexpr long long kHostChunkCells = 1LL << 18;
constexpr int kMaxChunks = 64;

struct mam4b_ctx {
  mam4b_config cfg;
  int device;
  unsigned *d_flags;
  cudaStream_t last_stream;
  char err[256];
  std::atomic<unsigned long long> launches;
  // host-path scratch (device slabs), grown on demand
  double *d_in, *d_out, *d_pblh;
  size_t cap_in, cap_out, cap_pblh;
  // pipeline scratch: SOA loop state, hand-off, queued cells, counters
  // (grown on demand)
  double *d_soa;
  double *d_hand;
  int *d_done, *d_order;
  double *d_aux;
  unsigned *d_counters;  // CNT_WORDS per chunk of the host path
  size_t cap_cells;
  int sms;              // SMs of the device (persistent solver grid = sms x blocks per SM)
  mam4b_tuning tune;    // launch shape of the forward pipeline
  bool tune_given;      // the caller's: set, autotuned or in MAM4B_TUNING_FILE
  // graph mode (mam4b_set_graph_mode): the pipeline of the last call,
  // captured once and replayed while the call's arguments stay the same
  bool use_graph;
  cudaStream_t cap_stream;
  cudaGraph_t graph;
  cudaGraphExec_t graph_exec;
  StepArgs graph_args;
  int graph_precision;
  mam4b_tuning graph_tune;
  // adjoint: SOA checkpoints of the persistent threads (allocated on first
  // use) and the cotangent scratch of the pipelined adjoint (grown)
  double *d_ck;
  int adj_grid;
  double *d_ck2, *d_abar, *d_lbar;
  int adj_ck;           // SOA checkpoint interval of the pipelined adjoint (0 = 1)
  int ck2_slots;        // SOA states per solver thread d_ck2 holds
  int *d_npass;         // [cap_adj]: passes of each SOA loop
  double *d_optics_lw;  // longwave optics tables (16 packed bands), set by the host
  double *d_optics_sw;  // shortwave optics tables (14 packed bands), set by the host
  double *d_optics_scr; // optics scratch (optics_scratch), grown
  size_t cap_optics_scr;
  int *d_trop;          // [cap_trop]: tropopause level per column (aero_rad_props)
  size_t cap_trop;
  double *d_diag;       // scratch of the step with process tendencies
  size_t cap_diag;      // its cells
  double *d_dmx;        // dropmixnuc activation results (DA_FIELDS per cell), grown
  double *d_coag_cc;    // coagulation process: 12 coefficients per cell, grown
  size_t cap_coag_cc;
  size_t cap_dmx;
  unsigned *d_bins;     // [2 kPassBins]: loops per pass count, start offsets
  // mam4b_step_columns: device pointer tables of the columns (grown) and
  // their host staging
  void **d_coltab;
  size_t cap_coltab;
  std::vector<void *> h_coltab;
  int adj_soa_grid;
  size_t cap_adj;
  // host path: copy/compute streams and their events (created on first use)
  cudaStream_t hs[kHostStreams];
  cudaEvent_t ev_start, ev_done[kHostStreams];
  cudaEvent_t ev_in[kMaxChunks], ev_comp[kMaxChunks];  // per chunk: inputs in, kernels done
  bool host_streams;
};

namespace {
std::mutex g_init_mu;
bool g_consts_ready[64];

mam4b_status set_err(mam4b_ctx *ctx, mam4b_status st, const char *what, cudaError_t e) {
  if (ctx)
    snprintf(ctx->err, sizeof(ctx->err), "%s: %s", what,
             e == cudaSuccess ? "invalid argument" : cudaGetErrorString(e));
  return st;
}

cudaError_t ensure_consts(int dev) {
  std::lock_guard<std::mutex> lk(g_init_mu);
  if (dev < 0 || dev >= 64)
    return cudaErrorInvalidDevice;
  if (g_consts_ready[dev])
    return cudaSuccess;
  StepConsts *d_tmp = nullptr;
  cudaError_t e = cudaMalloc(&d_tmp, sizeof(StepConsts));
  if (e == cudaSuccess) {
    init_consts_kernel<<<1, 1>>>(d_tmp);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaDeviceSynchronize();
  if (e == cudaSuccess)
    e = cudaMemcpyToSymbol(c_k, d_tmp, sizeof(StepConsts), 0, cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess)
    e = cudaDeviceSynchronize();
  cudaFree(d_tmp);
  if (e == cudaSuccess)
    g_consts_ready[dev] = true;
  return e;
}

bool valid_config(const mam4b_config *c) {
  return c && (c->gaexch_h2so4_uptake_optaa == 1 || c->gaexch_h2so4_uptake_optaa == 2);
}

cudaError_t ensure_solver_scratch(mam4b_ctx *ctx, size_t ncell) {
  cudaError_t e = cudaSuccess;
  if (!ctx->d_counters)
    e = cudaMalloc(&ctx->d_counters, (size_t)CNT_WORDS * kMaxChunks * sizeof(unsigned));
  if (e != cudaSuccess || ctx->cap_cells >= ncell)
    return e;
  cudaFree(ctx->d_soa);
  cudaFree(ctx->d_hand);
  cudaFree(ctx->d_done);
  cudaFree(ctx->d_order);
  cudaFree(ctx->d_aux);
  ctx->d_aux = nullptr;
  ctx->d_soa = nullptr;
  ctx->d_hand = nullptr;
  ctx->d_done = nullptr;
  ctx->d_order = nullptr;
  ctx->cap_cells = 0;
  e = cudaMalloc(&ctx->d_soa, (size_t)SOA_FIELDS * ncell * sizeof(double));
  if (e == cudaSuccess)
    e = cudaMalloc(&ctx->d_hand, (size_t)H_FIELDS * ncell * sizeof(double));
  if (e == cudaSuccess)
    e = cudaMalloc(&ctx->d_done, ncell * sizeof(int));
  if (e == cudaSuccess)
    e = cudaMalloc(&ctx->d_order, ncell * sizeof(int));
  if (e == cudaSuccess)
    e = cudaMalloc(&ctx->d_aux, (size_t)AUX_FIELDS * ncell * sizeof(double));
  if (e == cudaSuccess)
    ctx->cap_cells = ncell;
  return e;
}

// How the solver treats long loops. A batch with fewer cells than about
// 3,500 per SM is bound by its longest loops (up to 1,000 passes of about
// 400 ns with one lane per loop, about 700 ns when the SM is full): those
// run four lanes to a loop, 520 ns a pass alone. Larger batches are bound by
// throughput, where one lane per loop does more work per instruction, and
// only start their longest loops early. FP64 step, 1..1,000 sub-steps per
// cell, four lanes / one lane: 37 k cells 0.78 / 1.34 ms, 295 k cells 2.17 /
// 2.40 ms, 590 k cells 3.70 / 3.60 ms, 2.4 M cells 13.2 / 10.7 ms. Loops
// below 150 expected passes end before the long ones either way. The host
// path asks for each of its chunks, which run several at a time; there the
// copies hide the difference (65,536 x 72 cells, four lanes / one lane in every
// chunk: 52.45 / 52.45 ms uneven, 53.67 / 53.64 uniform).
void set_solver(StepArgs &a, int sms) {
  a.quads = a.ncell < 3500LL * sms;
  a.long_steps = a.quads ? 150.0 : 300.0;
}

void set_step_config(const mam4b_ctx *ctx, StepArgs &a, long long ncell, int nlev, double dt) {
  a.flags = ctx->d_flags;
  a.ncell = ncell;
  a.nlev = nlev;
  a.dt = dt;
  a.do_cond = ctx->cfg.do_cond;
  a.do_rename = ctx->cfg.do_rename;
  a.do_newnuc = ctx->cfg.do_newnuc;
  a.do_coag = ctx->cfg.do_coag;
  a.optaa = ctx->cfg.gaexch_h2so4_uptake_optaa;
  a.nmono = ctx->cfg.n_so4_monolayers_pcage;
  set_solver(a, ctx->sms);
}

// Pipeline scratch of the cells [c0, c0 + a.ncell) of a batch (one host
// chunk; c0 = 0 for a whole batch); chunk selects its counters.
void set_step_scratch(const mam4b_ctx *ctx, StepArgs &a, size_t c0, int chunk) {
  a.soa = ctx->d_soa + (size_t)SOA_FIELDS * c0;
  a.hand = ctx->d_hand + (size_t)H_FIELDS * c0;
  a.done = ctx->d_done + c0;
  a.order = ctx->d_order + c0;
  a.aux = ctx->d_aux + (size_t)AUX_FIELDS * c0;
  a.counters = ctx->d_counters + (size_t)CNT_WORDS * chunk;
}

// Scratch of the step with process tendencies, an allocation of its own that
// only such steps grow. False when there is none to be had: under capture
// (such a step has always been capturable from its first call, and what it
// captures must not depend on a later call's growth) or out of memory.
bool set_diag_scratch(mam4b_ctx *ctx, StepArgs &a, cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (!a.do_cond || cudaStreamIsCapturing(s, &cap) != cudaSuccess ||
      cap != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return false;
  }
  const size_t n = (size_t)a.ncell, fields = SOA_FIELDS + H_FIELDS + AUX_FIELDS;
  if (ctx->cap_diag < n) {
    cudaFree(ctx->d_diag);
    ctx->d_diag = nullptr;
    ctx->cap_diag = 0;
    if (cudaMalloc(&ctx->d_diag, n * (fields * sizeof(double) + 2 * sizeof(int)) +
                                     CNT_WORDS * sizeof(unsigned)) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    ctx->cap_diag = n;
  }
  a.soa = ctx->d_diag;
  a.hand = a.soa + SOA_FIELDS * n;
  a.aux = a.hand + H_FIELDS * n;
  a.done = (int *)(a.aux + AUX_FIELDS * n);
  a.order = a.done + n;
  a.counters = (unsigned *)(a.order + n);
  return true;
}

// ----------------------------------------------------- launch shapes
// The forward pipeline's launch shape (mam4b_tuning): block sizes, register
// caps (compiled variants of the whole-cell kernels) and cells per thread.
// Every shape runs the same arithmetic, so results are bit for bit equal.
bool valid_block(int b, int regs) {
  return (b == 64 || b == 128 || b == 256) && (long long)b * regs <= 65536;
}
bool valid_tuning(const mam4b_tuning &t) {
  return (t.size_regs == 255 || t.size_regs == 128 || t.size_regs == 96) &&
         valid_block(t.size_block, t.size_regs) &&
         valid_block(t.mode_block, 64) && valid_block(t.pair_block, 128) &&
         (t.pre_regs == 255 || t.pre_regs == 168 || t.pre_regs == 128) &&
         valid_block(t.pre_block, t.pre_regs) &&
         (t.post_regs == 255 || t.post_regs == 168 || t.post_regs == 128) &&
         valid_block(t.post_block, t.post_regs) &&
         (t.soa_regs == 64 || t.soa_regs == 96 || t.soa_regs == 128) &&
         (t.soa_block == 128 || t.soa_block == 256) &&
         (long long)t.soa_block * t.soa_regs <= 65536 && t.soa_blocks_per_sm >= 1 &&
         t.soa_blocks_per_sm <= 16 &&
         (t.cells_per_thread == 1 || t.cells_per_thread == 2 || t.cells_per_thread == 4) &&
         (t.inline_scale == 0 || t.inline_scale == 1 || t.inline_scale == 4 ||
          t.inline_scale == 16 || t.inline_scale == 64);
}

unsigned grid_for(long long n, int block, int cpt) {
  const long long per = (long long)block * cpt;
  const long long g = (n + per - 1) / per;
  return (unsigned)(g > 0 ? g : 1);
}

// Stage launchers. Stage order: 0 front (its shape is the tuning's size_*;
// with chemistry chem_size_kernel), 1 mode (with chemistry then
// chem_cell_kernel and chem_subarea_kernel), 2 pair, 3 pre, 4 soa, 5 post.
template <bool LOOP>
void launch_front_t(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s) {
  const int cells = t.size_block / 2;
  const dim3 g(grid_for(a.ncell, cells, t.cells_per_thread), 2);
  const size_t smem = (size_t)XF_FIELDS * cells * sizeof(double);
  if (t.size_regs == 96)
    front_kernel<96, LOOP><<<g, t.size_block, smem, s>>>(a);
  else if (t.size_regs == 128)
    front_kernel<128, LOOP><<<g, t.size_block, smem, s>>>(a);
  else
    front_kernel<255, LOOP><<<g, t.size_block, smem, s>>>(a);
}
void launch_front(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s) {
  if (t.cells_per_thread > 1)
    launch_front_t<true>(t, a, s);
  else
    launch_front_t<false>(t, a, s);
}
void launch_mode(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s, bool mixed) {
  const dim3 g(grid_for(a.ncell, t.mode_block, 1), NMODE);
  if (mixed)
    mode_kernel<true><<<g, t.mode_block, 0, s>>>(a);
  else
    mode_kernel<false><<<g, t.mode_block, 0, s>>>(a);
}
void launch_pair(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s, bool mixed) {
  const dim3 g(grid_for(a.ncell, t.pair_block, 1), 3);
  if (mixed)
    pair_kernel<true><<<g, t.pair_block, 0, s>>>(a);
  else
    pair_kernel<false><<<g, t.pair_block, 0, s>>>(a);
}
// Only the form that finishes cells has code for the register caps to shape;
// the other needs 54 (MIXED 82).
template <bool MIXED, bool FUSE>
void launch_pre_t(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s) {
  const unsigned g = grid_for(a.ncell, t.pre_block, 1);
  if (!FUSE || t.pre_regs == 128)
    pre_kernel<128, MIXED, FUSE><<<g, t.pre_block, 0, s>>>(a);
  else if constexpr (FUSE) {
    if (t.pre_regs == 168)
      pre_kernel<168, MIXED, FUSE><<<g, t.pre_block, 0, s>>>(a);
    else
      pre_kernel<255, MIXED, FUSE><<<g, t.pre_block, 0, s>>>(a);
  }
}
// fuse: cells with short SOA loops finish in pre (a.inline_scale > 0)
void launch_pre(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s, bool mixed = false,
                bool fuse = false) {
  if (mixed)
    fuse ? launch_pre_t<true, true>(t, a, s) : launch_pre_t<true, false>(t, a, s);
  else
    fuse ? launch_pre_t<false, true>(t, a, s) : launch_pre_t<false, false>(t, a, s);
}
template <int SOA>
void launch_soa_t(const mam4b_tuning &t, int sms, const StepArgs &a, cudaStream_t s) {
  const unsigned g = (unsigned)(sms * t.soa_blocks_per_sm);
  if (t.soa_regs == 128)
    soa_kernel<SOA, 128><<<g, t.soa_block, 0, s>>>(a);
  else if (t.soa_regs == 96)
    soa_kernel<SOA, 96><<<g, t.soa_block, 0, s>>>(a);
  else
    soa_kernel<SOA, 64><<<g, t.soa_block, 0, s>>>(a);
}
// the SOA loop of each precision (mam4b_precision)
void launch_soa(const mam4b_tuning &t, int sms, const StepArgs &a, cudaStream_t s,
                int precision) {
  if (precision == MAM4B_MIXED_FAST)
    launch_soa_t<2>(t, sms, a, s);
  else if (precision == MAM4B_MIXED)
    launch_soa_t<1>(t, sms, a, s);
  else
    launch_soa_t<0>(t, sms, a, s);
}
template <bool LOOP>
void launch_post_t(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s) {
  const unsigned g = grid_for(a.ncell, t.post_block, t.cells_per_thread);
  if (t.post_regs == 255)
    post_kernel<255, LOOP><<<g, t.post_block, 0, s>>>(a);
  else if (t.post_regs == 168)
    post_kernel<168, LOOP><<<g, t.post_block, 0, s>>>(a);
  else
    post_kernel<128, LOOP><<<g, t.post_block, 0, s>>>(a);
}
void launch_post(const mam4b_tuning &t, const StepArgs &a, cudaStream_t s) {
  if (t.cells_per_thread > 1)
    launch_post_t<true>(t, a, s);
  else
    launch_post_t<false>(t, a, s);
}

// Clears the counters and queues the pipeline kernels on s in the
// arithmetic of `precision` (mam4b_precision) with launch shape t on a
// device of `sms` SMs. With ch (FP64 only) the cells' chemistry runs after
// the mode stage. With ev (7 events), ev[k] is recorded before stage k and
// ev[6] after the last: the per-stage times of mam4b_autotune.
cudaError_t launch_pipeline_t(const mam4b_tuning &t, int sms, const StepArgs &a_in,
                              cudaStream_t s, int precision, const ChemArgs *ch, cudaEvent_t *ev,
                              std::atomic<unsigned long long> *launches, bool diag = false) {
  StepArgs a = a_in;
  a.mixed = precision != MAM4B_FP64;
  // short SOA loops finish in pre unless the adjoint needs every loop's
  // pass count (npass) or the loop runs in FP32 (MIXED_FAST)
  const bool fuse =
      t.inline_scale > 0 && !a.npass && precision != MAM4B_MIXED_FAST && !diag;
  a.inline_scale = fuse ? (double)t.inline_scale : 0.0;
  cudaError_t e = cudaMemsetAsync(a.counters, 0, CNT_WORDS * sizeof(unsigned), s);
  if (e != cudaSuccess)
    return e;
  if (!a.do_cond) {
    // no SOA loop to pipeline
    const int block = 128;
    const unsigned grid = (unsigned)((a.ncell + block - 1) / block);
    if (ch)
      chem_step_kernel<<<grid, block, 0, s>>>(a, *ch);
    else
      full_kernel<false><<<grid, block, 0, s>>>(a);
    e = cudaGetLastError();
    if (e == cudaSuccess && launches)
      *launches += 1;
    return e;
  }
  const bool mixed = precision != MAM4B_FP64;
  auto mark = [&](int k) {
    if (ev)
      cudaEventRecord(ev[k], s);
  };
  mark(0);
  const dim3 pairs(grid_for(a.ncell, 64, 1), 2);  // blocks of 64 cells, two modes
  const size_t xf = (size_t)XF_FIELDS * 64 * sizeof(double);
  if (ch)
    chem_size_kernel<<<pairs, 128, xf, s>>>(a);
  else if (diag)
    front_kernel<128, false, true><<<pairs, 128, xf, s>>>(a);
  else
    launch_front(t, a, s);
  mark(1);
  launch_mode(t, a, s, mixed);
  if (ch) {
    chem_cell_kernel<<<grid_for(a.ncell, 256, 1), 256, 0, s>>>(a, *ch);
    chem_subarea_kernel<<<pairs, 128, xf, s>>>(a);
  }
  mark(2);
  launch_pair(t, a, s, mixed);
  mark(3);
  launch_pre(t, a, s, mixed, fuse);
  mark(4);
  launch_soa(t, sms, a, s, precision);
  mark(5);
  // the adjoint's forward (npass set) has no post stage: adj_post_kernel
  // recomputes the suffix from the hand-off, and the forward's outputs are
  // not returned
  if (diag)
    post_diag_kernel<<<grid_for(a.ncell, 128, 1), 128, 0, s>>>(a);
  else if (!a.npass)
    launch_post(t, a, s);
  mark(6);
  e = cudaGetLastError();
  if (e == cudaSuccess && launches)
    *launches += ch ? 8 : a.npass ? 5 : 6;
  return e;
}

void drop_graph(mam4b_ctx *ctx) {
  if (ctx->graph_exec)
    cudaGraphExecDestroy(ctx->graph_exec);
  if (ctx->graph)
    cudaGraphDestroy(ctx->graph);
  ctx->graph_exec = nullptr;
  ctx->graph = nullptr;
}

// The context's launch shape for a step. One that the caller did not choose was
// chosen on the FP64 step; the FP32 loop fits 64 registers, so where a thread
// runs a loop the SM holds twice the 128-register shape's blocks (16,384 x 72
// uniform cells: 4.10 ms against 4.65). With four lanes to a loop, in small
// batches, the loops are fewer than the lanes and the wider shape is the
// faster (1,024 columns: 0.70 against 0.88).
mam4b_tuning step_shape(const mam4b_ctx *ctx, const StepArgs &a, int precision) {
  mam4b_tuning t = ctx->tune;
  if (!ctx->tune_given && precision == MAM4B_MIXED_FAST && !a.quads && t.soa_regs == 128) {
    t.soa_regs = 64;
    t.soa_blocks_per_sm *= 2;
  }
  return t;
}

// The forward pipeline with the context's launch shape. With graph mode on
// and `graph` set (mam4b_step's device entry), the pipeline is captured on
// a private stream into a CUDA graph, instantiated once and replayed on s;
// a call with other arguments (pointers, sizes, precision, launch shape)
// recaptures and updates the instantiated graph in place, or
// re-instantiates it when the update is refused.
cudaError_t launch_pipeline(mam4b_ctx *ctx, const StepArgs &a, cudaStream_t s, int precision,
                            const ChemArgs *ch = nullptr, bool graph = false) {
  const mam4b_tuning tune = step_shape(ctx, a, precision);
  if (!graph || !ctx->use_graph || ch || !a.do_cond)
    return launch_pipeline_t(tune, ctx->sms, a, s, precision, ch, nullptr, &ctx->launches);
  const bool same = ctx->graph_exec && memcmp(&ctx->graph_args, &a, sizeof(StepArgs)) == 0 &&
                    ctx->graph_precision == precision &&
                    memcmp(&ctx->graph_tune, &tune, sizeof(mam4b_tuning)) == 0;
  cudaError_t e = cudaSuccess;
  if (!same) {
    if (!ctx->cap_stream)
      e = cudaStreamCreateWithFlags(&ctx->cap_stream, cudaStreamNonBlocking);
    cudaGraph_t g = nullptr;
    if (e == cudaSuccess)
      e = cudaStreamBeginCapture(ctx->cap_stream, cudaStreamCaptureModeRelaxed);
    if (e == cudaSuccess) {
      const cudaError_t el = launch_pipeline_t(tune, ctx->sms, a, ctx->cap_stream, precision,
                                               nullptr, nullptr, nullptr);
      e = cudaStreamEndCapture(ctx->cap_stream, &g);
      if (e == cudaSuccess)
        e = el;
    }
    if (e == cudaSuccess && ctx->graph_exec) {
      cudaGraphExecUpdateResultInfo info;
      if (cudaGraphExecUpdate(ctx->graph_exec, g, &info) != cudaSuccess) {
        (void)cudaGetLastError();  // the refusal is not an error of the step
        cudaGraphExecDestroy(ctx->graph_exec);
        ctx->graph_exec = nullptr;
      }
    }
    if (e == cudaSuccess && !ctx->graph_exec)
      e = cudaGraphInstantiate(&ctx->graph_exec, g, 0);
    if (ctx->graph)
      cudaGraphDestroy(ctx->graph);
    ctx->graph = g;
    if (e != cudaSuccess) {
      drop_graph(ctx);
      return e;
    }
    ctx->graph_args = a;
    ctx->graph_precision = precision;
    ctx->graph_tune = tune;
  }
  e = cudaGraphLaunch(ctx->graph_exec, s);
  if (e == cudaSuccess)
    ctx->launches += 6;
  return e;
}

cudaError_t ensure_host_streams(mam4b_ctx *ctx) {
  if (ctx->host_streams)
    return cudaSuccess;
  // created in order; on failure everything created so far is released
  int ns = 0, ne = 0;
  cudaEvent_t *evs[1 + kHostStreams + 2 * kMaxChunks];
  evs[ne] = &ctx->ev_start;
  cudaError_t e = cudaEventCreateWithFlags(evs[ne], cudaEventDisableTiming);
  if (e == cudaSuccess)
    ++ne;
  for (; ns < kHostStreams && e == cudaSuccess; ++ns) {
    e = cudaStreamCreateWithFlags(&ctx->hs[ns], cudaStreamNonBlocking);
    if (e != cudaSuccess)
      break;
  }
  for (int k = 0; k < kHostStreams && e == cudaSuccess; ++k) {
    evs[ne] = &ctx->ev_done[k];
    e = cudaEventCreateWithFlags(evs[ne], cudaEventDisableTiming);
    if (e == cudaSuccess)
      ++ne;
  }
  for (int i = 0; i < kMaxChunks && e == cudaSuccess; ++i) {
    evs[ne] = &ctx->ev_in[i];
    e = cudaEventCreateWithFlags(evs[ne], cudaEventDisableTiming);
    if (e != cudaSuccess)
      break;
    ++ne;
    evs[ne] = &ctx->ev_comp[i];
    e = cudaEventCreateWithFlags(evs[ne], cudaEventDisableTiming);
    if (e == cudaSuccess)
      ++ne;
  }
  if (e != cudaSuccess) {
    for (int j = 0; j < ns; ++j)
      cudaStreamDestroy(ctx->hs[j]);
    for (int j = 0; j < ne; ++j)
      cudaEventDestroy(*evs[j]);
    return e;
  }
  ctx->host_streams = true;
  return cudaSuccess;
}

// Per-device state of mam4b_step_slab_noalloc, filled once per device by
// noalloc_setup with that device current.
struct NoAllocDevice {
  bool ready;
  double *scratch;  // device address of g_noalloc_scratch on this device
  int sms;          // SMs of the device (the solver's persistent grid)
};
NoAllocDevice g_noalloc[64];

cudaError_t noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lk(g_init_mu);
  if (dev < 0 || dev >= 64)
    return cudaErrorInvalidDevice;
  if (g_noalloc[dev].ready)
    return cudaSuccess;
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess)
    return e;
  if (!g_consts_ready[dev]) {
    // derived constants without a temporary allocation: staged in the
    // scratch array (no step can be using it before set-up ends)
    StepConsts *stage = reinterpret_cast<StepConsts *>(p);
    init_consts_kernel<<<1, 1>>>(stage);
    e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaDeviceSynchronize();
    if (e == cudaSuccess)
      e = cudaMemcpyToSymbol(c_k, stage, sizeof(StepConsts), 0, cudaMemcpyDeviceToDevice);
    if (e == cudaSuccess)
      e = cudaDeviceSynchronize();
    if (e != cudaSuccess)
      return e;
    g_consts_ready[dev] = true;
  }
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess)
    return e;
  g_noalloc[dev].scratch = static_cast<double *>(p);
  g_noalloc[dev].sms = sms;
  g_noalloc[dev].ready = true;
  return cudaSuccess;
}
// ------------------------------------------------------- tuning files
// A tuning file is a flat JSON object with the integer fields of
// mam4b_tuning under their own names and the device name it was chosen on
// ("device": "NVIDIA B200"), e.g. as written by mam4xx_b200/autotune.py.
const char *const kTuningKeys[] = {"size_block", "size_regs", "mode_block", "pair_block",
                                   "pre_block", "pre_regs", "post_block", "post_regs",
                                   "soa_block", "soa_regs", "soa_blocks_per_sm",
                                   "cells_per_thread", "inline_scale"};
int *tuning_field(mam4b_tuning &t, int k) {
  int *f[] = {&t.size_block, &t.size_regs, &t.mode_block, &t.pair_block, &t.pre_block,
              &t.pre_regs, &t.post_block, &t.post_regs, &t.soa_block, &t.soa_regs,
              &t.soa_blocks_per_sm, &t.cells_per_thread, &t.inline_scale};
  return f[k];
}

// Value text after "key": in json, or nullptr.
const char *json_value(const char *json, const char *key) {
  char pat[64];
  snprintf(pat, sizeof(pat), "\"%s\"", key);
  const char *p = strstr(json, pat);
  if (!p)
    return nullptr;
  p += strlen(pat);
  while (*p == ' ' || *p == '\t' || *p == '\n' || *p == '\r')
    ++p;
  if (*p != ':')
    return nullptr;
  ++p;
  while (*p == ' ' || *p == '\t' || *p == '\n' || *p == '\r')
    ++p;
  return p;
}

mam4b_status parse_tuning(const char *json, mam4b_tuning *t, char *device, size_t device_len) {
  mam4b_tuning r;
  mam4b_default_tuning(&r);
  for (int k = 0; k < (int)(sizeof(kTuningKeys) / sizeof(kTuningKeys[0])); ++k) {
    const char *v = json_value(json, kTuningKeys[k]);
    if (!v)
      return MAM4B_ERR_INVALID_ARGUMENT;
    char *end = nullptr;
    const long x = strtol(v, &end, 10);
    if (end == v || x < 0 || x > 4096)
      return MAM4B_ERR_INVALID_ARGUMENT;
    *tuning_field(r, k) = (int)x;
  }
  if (!valid_tuning(r))
    return MAM4B_ERR_INVALID_ARGUMENT;
  if (device && device_len) {
    device[0] = '\0';
    const char *v = json_value(json, "device");
    if (v && *v == '"') {
      const char *q = strchr(v + 1, '"');
      if (q) {
        size_t n = (size_t)(q - v - 1);
        if (n >= device_len)
          n = device_len - 1;
        memcpy(device, v + 1, n);
        device[n] = '\0';
      }
    }
  }
  *t = r;
  return MAM4B_OK;
}

mam4b_status read_tuning_file(const char *path, mam4b_tuning *t, char *device, size_t device_len) {
  FILE *f = fopen(path, "rb");
  if (!f)
    return MAM4B_ERR_INVALID_ARGUMENT;
  char buf[4096];
  const size_t n = fread(buf, 1, sizeof(buf) - 1, f);
  fclose(f);
  buf[n] = '\0';
  return parse_tuning(buf, t, device, device_len);
}

// The tuning a new context starts with: the file named by MAM4B_TUNING_FILE,
// else mam4b_tuning.json next to this library, when it exists, parses and
// was chosen on a device of the current device's name; else the defaults.
// Whether it is the named file's.
bool initial_tuning(int dev, mam4b_tuning *t) {
  mam4b_default_tuning(t);
  char path[1024] = {0};
  const char *env = getenv("MAM4B_TUNING_FILE");
  const bool named = env && *env;
  if (named) {
    snprintf(path, sizeof(path), "%s", env);
  } else {
    Dl_info info;
    if (!dladdr((void *)&initial_tuning, &info) || !info.dli_fname)
      return false;
    snprintf(path, sizeof(path), "%s", info.dli_fname);
    char *slash = strrchr(path, '/');
    if (!slash)
      return false;
    snprintf(slash + 1, sizeof(path) - (size_t)(slash + 1 - path), "mam4b_tuning.json");
  }
  mam4b_tuning r;
  char name[256];
  if (read_tuning_file(path, &r, name, sizeof(name)) != MAM4B_OK)
    return false;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess || strcmp(prop.name, name) != 0)
    return false;
  *t = r;
  return named;
}
}  // namespace

extern "C" {

int mam4b_abi_version(void) { return MAM4B_ABI_VERSION; }

void mam4b_default_tuning(mam4b_tuning *t) {
  if (!t)
    return;
  t->size_block = 128;
  t->size_regs = 128;
  t->mode_block = 128;
  t->pair_block = 128;
  t->pre_block = 128;
  t->pre_regs = 255;
  t->post_block = 128;
  t->post_regs = 128;
  t->soa_block = 128;
  t->soa_regs = 128;
  t->soa_blocks_per_sm = 4;
  t->cells_per_thread = 1;
  t->inline_scale = 0;
}

mam4b_status mam4b_tuning_from_json(const char *path, mam4b_tuning *t, char *device,
                                    size_t device_len) {
  if (!path || !t)
    return MAM4B_ERR_INVALID_ARGUMENT;
  return read_tuning_file(path, t, device, device_len);
}

mam4b_status mam4b_get_tuning(const mam4b_ctx *ctx, mam4b_tuning *t) {
  if (!ctx || !t)
    return MAM4B_ERR_INVALID_ARGUMENT;
  *t = ctx->tune;
  return MAM4B_OK;
}

mam4b_status mam4b_set_tuning(mam4b_ctx *ctx, const mam4b_tuning *t) {
  if (!ctx || !t || !valid_tuning(*t))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_set_tuning", cudaSuccess);
  ctx->tune = *t;
  ctx->tune_given = true;
  return MAM4B_OK;
}

mam4b_status mam4b_set_adjoint_checkpoint(mam4b_ctx *ctx, int interval) {
  if (!ctx || (interval != 1 && interval != 4))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_set_adjoint_checkpoint: interval 1 or 4",
                   cudaSuccess);
  ctx->adj_ck = interval;
  return MAM4B_OK;
}

mam4b_status mam4b_set_graph_mode(mam4b_ctx *ctx, int enable) {
  if (!ctx)
    return MAM4B_ERR_INVALID_ARGUMENT;
  ctx->use_graph = enable != 0;
  if (!ctx->use_graph)
    drop_graph(ctx);
  return MAM4B_OK;
}

void mam4b_default_config(mam4b_config *cfg) {
  if (!cfg)
    return;
  cfg->do_cond = 1;
  cfg->do_rename = 1;
  cfg->do_newnuc = 1;
  cfg->do_coag = 1;
  cfg->gaexch_h2so4_uptake_optaa = 2;
  cfg->newnuc_h2so4_conc_optaa = 2;
  cfg->n_so4_monolayers_pcage = 8;
}

mam4b_status mam4b_create(mam4b_ctx **out, const mam4b_config *cfg) {
  if (!out)
    return MAM4B_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  mam4b_config c;
  if (cfg)
    c = *cfg;
  else
    mam4b_default_config(&c);
  if (!valid_config(&c))
    return MAM4B_ERR_INVALID_ARGUMENT;
  mam4b_ctx *ctx = new (std::nothrow) mam4b_ctx();
  if (!ctx)
    return MAM4B_ERR_INVALID_ARGUMENT;
  ctx->cfg = c;
  ctx->launches = 0;
  cudaError_t e = cudaGetDevice(&ctx->device);
  if (e == cudaSuccess)
    e = ensure_consts(ctx->device);
  if (e == cudaSuccess)
    e = cudaMalloc(&ctx->d_flags, sizeof(unsigned));
  if (e == cudaSuccess)
    e = cudaMemset(ctx->d_flags, 0, sizeof(unsigned));
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, ctx->device);
  if (e != cudaSuccess) {
    if (ctx->d_flags)
      cudaFree(ctx->d_flags);
    delete ctx;
    return MAM4B_ERR_CUDA;
  }
  ctx->tune_given = initial_tuning(ctx->device, &ctx->tune);
  *out = ctx;
  return MAM4B_OK;
}

mam4b_status mam4b_destroy(mam4b_ctx *ctx) {
  if (!ctx)
    return MAM4B_ERR_INVALID_ARGUMENT;
  drop_graph(ctx);
  if (ctx->cap_stream)
    cudaStreamDestroy(ctx->cap_stream);
  cudaFree(ctx->d_coltab);
  cudaFree(ctx->d_flags);
  cudaFree(ctx->d_in);
  cudaFree(ctx->d_out);
  cudaFree(ctx->d_pblh);
  cudaFree(ctx->d_soa);
  cudaFree(ctx->d_hand);
  cudaFree(ctx->d_done);
  cudaFree(ctx->d_order);
  cudaFree(ctx->d_aux);
  cudaFree(ctx->d_counters);
  cudaFree(ctx->d_ck);
  cudaFree(ctx->d_ck2);
  cudaFree(ctx->d_abar);
  cudaFree(ctx->d_lbar);
  cudaFree(ctx->d_npass);
  cudaFree(ctx->d_bins);
  cudaFree(ctx->d_optics_lw);
  cudaFree(ctx->d_optics_scr);
  cudaFree(ctx->d_optics_sw);
  cudaFree(ctx->d_trop);
  cudaFree(ctx->d_diag);
  cudaFree(ctx->d_dmx);
  cudaFree(ctx->d_coag_cc);
  if (ctx->host_streams) {
    for (int k = 0; k < kHostStreams; ++k) {
      cudaStreamDestroy(ctx->hs[k]);
      cudaEventDestroy(ctx->ev_done[k]);
    }
    for (int i = 0; i < kMaxChunks; ++i) {
      cudaEventDestroy(ctx->ev_in[i]);
      cudaEventDestroy(ctx->ev_comp[i]);
    }
    cudaEventDestroy(ctx->ev_start);
  }
  delete ctx;
  return MAM4B_OK;
}

mam4b_status mam4b_step(mam4b_ctx *ctx, const mam4b_state_view *in, const mam4b_tend_view *out,
                        int ncol, int nlev, double dt, int precision, void *stream) {
  if (!ctx || !in || !out || ncol < 0 || nlev <= 0 || !(dt > 0.0) || !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step", cudaSuccess);
  if (precision != MAM4B_FP64 && precision != MAM4B_MIXED && precision != MAM4B_MIXED_FAST)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step: precision", cudaSuccess);
  StepArgs a;
  memset(&a, 0, sizeof(a));
  bool diag = false;
  for (int f = 0; f < MAM4B_NIN; ++f) {
    if (!in->field[f])
      return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step: null input field", cudaSuccess);
    a.in[f] = in->field[f];
  }
  if (!in->pblh)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step: null pblh", cudaSuccess);
  a.pblh = in->pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f) {
    if (!out->field[f])
      return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step: null output field", cudaSuccess);
    a.out[f] = out->field[f];
  }
  for (int f = 0; f < MAM4B_NDIAG; ++f) {
    a.diag[f] = out->diag[f];
    diag = diag || (out->diag[f] != nullptr);
  }
  set_step_config(ctx, a, (long long)ncol * nlev, nlev, dt);
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (a.ncell == 0)
    return MAM4B_OK;
  const int block = 128;
  const long long grid = (a.ncell + block - 1) / block;
  if (a.ncell > 0x7fffffffLL)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step: too many cells", cudaSuccess);
  cudaError_t e;
  if (diag && precision != MAM4B_FP64)
    return set_err(ctx, MAM4B_ERR_NOT_SUPPORTED,
                   "mam4b_step: process diagnostics are FP64 only", cudaSuccess);
  // with process tendencies, in the pipeline's stages where their scratch can
  // be had (1,024 x 72 cells: 0.28 ms against 0.78 ms start to end in one
  // thread per cell, which waits for instructions and spilled registers)
  if (diag && set_diag_scratch(ctx, a, s)) {
    e = launch_pipeline_t(ctx->tune, ctx->sms, a, s, precision, nullptr, nullptr, &ctx->launches,
                          true);
    if (e != cudaSuccess)
      return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step launch", e);
    return MAM4B_OK;
  }
  if (diag) {
    full_kernel<true><<<(unsigned)grid, block, 0, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess)
      return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step launch", e);
    ctx->launches += 1;
    return MAM4B_OK;
  }
  e = ensure_solver_scratch(ctx, (size_t)a.ncell);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step scratch", e);
  set_step_scratch(ctx, a, 0, 0);
  e = launch_pipeline(ctx, a, s, precision, nullptr, true);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step launch", e);
  return MAM4B_OK;
}

mam4b_status mam4b_step_slab(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                             double *out_slab, size_t ld, int ncol, int nlev, double dt,
                             int precision, void *stream) {
  if (!ctx || !in_slab || !pblh || !out_slab || ncol < 0 || nlev <= 0 ||
      ld < (size_t)ncol * (size_t)nlev)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_slab", cudaSuccess);
  mam4b_state_view iv;
  mam4b_tend_view ov;
  memset(&iv, 0, sizeof(iv));
  memset(&ov, 0, sizeof(ov));
  for (int f = 0; f < MAM4B_NIN; ++f)
    iv.field[f] = in_slab + (size_t)f * ld;
  iv.pblh = pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f)
    ov.field[f] = out_slab + (size_t)f * ld;
  return mam4b_step(ctx, &iv, &ov, ncol, nlev, dt, precision, stream);
}

// Autotuner (include/mam4b.h): times every candidate launch shape of each
// pipeline stage on the caller's batch, stage by stage from events
// recorded between the launches (a stage's time does not depend on the
// other stages' shapes), keeps the fastest shape of each stage, then the
// fastest cells-per-thread of the whole-cell kernels, and adopts the result
// when the whole pipeline is faster with it than with the defaults.
mam4b_status mam4b_autotune(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                            double *out_slab, size_t ld, int ncol, int nlev, double dt,
                            int precision, int reps, void *stream, mam4b_tuning *best,
                            float *default_ms, float *best_ms) {
  const char *what = "mam4b_autotune";
  if (!ctx || !in_slab || !pblh || !out_slab || ncol <= 0 || nlev <= 0 || !(dt > 0.0) ||
      ld < (size_t)ncol * (size_t)nlev || reps < 1 || reps > 100 ||
      (long long)ncol * nlev > 0x7fffffffLL ||
      (precision != MAM4B_FP64 && precision != MAM4B_MIXED && precision != MAM4B_MIXED_FAST))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  if (!ctx->cfg.do_cond)
    return set_err(ctx, MAM4B_ERR_NOT_SUPPORTED, "mam4b_autotune: condensation off (one kernel)",
                   cudaSuccess);
  StepArgs a;
  memset(&a, 0, sizeof(a));
  for (int f = 0; f < MAM4B_NIN; ++f)
    a.in[f] = in_slab + (size_t)f * ld;
  a.pblh = pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f)
    a.out[f] = out_slab + (size_t)f * ld;
  set_step_config(ctx, a, (long long)ncol * nlev, nlev, dt);
  cudaError_t e = ensure_solver_scratch(ctx, (size_t)a.ncell);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  set_step_scratch(ctx, a, 0, 0);
  cudaStream_t s = (cudaStream_t)stream;
  cudaEvent_t ev[7];
  int nev = 0;
  for (; nev < 7; ++nev)
    if ((e = cudaEventCreate(&ev[nev])) != cudaSuccess)
      break;
  // per-stage candidates
  const int blocks[3] = {64, 128, 256};
  std::vector<mam4b_tuning> cand[6];
  mam4b_tuning d;
  mam4b_default_tuning(&d);
  for (int b : blocks) {
    for (int r : {255, 128, 96}) {
      mam4b_tuning t = d;
      t.size_block = b;
      t.size_regs = r;
      if (valid_tuning(t))
        cand[0].push_back(t);
    }
    mam4b_tuning t = d;
    t.mode_block = b;
    cand[1].push_back(t);
    t = d;
    t.pair_block = b;
    cand[2].push_back(t);
    t = d;
    t.pre_block = b;
    cand[3].push_back(t);
    for (int r : {255, 168, 128}) {
      t = d;
      t.post_block = b;
      t.post_regs = r;
      if (valid_tuning(t))
        cand[5].push_back(t);
    }
  }
  for (int b : {128, 256})
    for (int r : {64, 96, 128}) {
      const int resident = (int)(65536 / ((long long)b * r));
      for (int bps : {resident, resident / 2}) {
        mam4b_tuning t = d;
        t.soa_block = b;
        t.soa_regs = r;
        t.soa_blocks_per_sm = bps < 1 ? 1 : (bps > 16 ? 16 : bps);
        if (valid_tuning(t))
          cand[4].push_back(t);
      }
    }
  size_t kmax = 0;
  for (auto &c : cand)
    kmax = std::max(kmax, c.size());
  std::vector<float> stage_ms[6];
  for (int k = 0; k < 6; ++k)
    stage_ms[k].assign(cand[k].size(), 1e30f);
  auto combine = [&](size_t i) {
    // stage k of the combined shape from candidate i of stage k
    mam4b_tuning t = d;
    const mam4b_tuning &c0 = cand[0][i % cand[0].size()];
    t.size_block = c0.size_block;
    t.size_regs = c0.size_regs;
    t.mode_block = cand[1][i % cand[1].size()].mode_block;
    t.pair_block = cand[2][i % cand[2].size()].pair_block;
    t.pre_block = cand[3][i % cand[3].size()].pre_block;
    const mam4b_tuning &c4 = cand[4][i % cand[4].size()];
    t.soa_block = c4.soa_block;
    t.soa_regs = c4.soa_regs;
    t.soa_blocks_per_sm = c4.soa_blocks_per_sm;
    const mam4b_tuning &c5 = cand[5][i % cand[5].size()];
    t.post_block = c5.post_block;
    t.post_regs = c5.post_regs;
    return t;
  };
  auto run = [&](const mam4b_tuning &t, float *stages, float *total) -> cudaError_t {
    cudaError_t r = launch_pipeline_t(t, ctx->sms, a, s, precision, nullptr, ev, nullptr);
    if (r == cudaSuccess)
      r = cudaEventSynchronize(ev[6]);
    float ms;
    for (int k = 0; r == cudaSuccess && k < 6; ++k) {
      r = cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
      if (stages)
        stages[k] = ms;
    }
    if (r == cudaSuccess && total)
      r = cudaEventElapsedTime(total, ev[0], ev[6]);
    return r;
  };
  // warm-up
  if (e == cudaSuccess)
    e = run(d, nullptr, nullptr);
  for (size_t i = 0; e == cudaSuccess && i < kmax; ++i) {
    const mam4b_tuning t = combine(i);
    for (int r = 0; e == cudaSuccess && r < reps; ++r) {
      float st[6];
      e = run(t, st, nullptr);
      for (int k = 0; e == cudaSuccess && k < 6; ++k) {
        const size_t j = i % cand[k].size();
        if (i < cand[k].size())
          stage_ms[k][j] = std::min(stage_ms[k][j], st[k]);
      }
    }
  }
  mam4b_tuning b = d;
  if (e == cudaSuccess) {
    size_t arg[6];
    for (int k = 0; k < 6; ++k)
      arg[k] = (size_t)(std::min_element(stage_ms[k].begin(), stage_ms[k].end()) -
                        stage_ms[k].begin());
    b.size_block = cand[0][arg[0]].size_block;
    b.size_regs = cand[0][arg[0]].size_regs;
    b.mode_block = cand[1][arg[1]].mode_block;
    b.pair_block = cand[2][arg[2]].pair_block;
    b.pre_block = cand[3][arg[3]].pre_block;
    b.soa_block = cand[4][arg[4]].soa_block;
    b.soa_regs = cand[4][arg[4]].soa_regs;
    b.soa_blocks_per_sm = cand[4][arg[4]].soa_blocks_per_sm;
    b.post_block = cand[5][arg[5]].post_block;
    b.post_regs = cand[5][arg[5]].post_regs;
  }
  // cells per thread of the whole-cell kernels, then whole-pipeline times
  auto total_of = [&](const mam4b_tuning &t, float &ms) -> cudaError_t {
    ms = 1e30f;
    cudaError_t r = cudaSuccess;
    for (int k = 0; r == cudaSuccess && k < reps; ++k) {
      float x;
      r = run(t, nullptr, &x);
      ms = std::min(ms, x);
    }
    return r;
  };
  float t_best = 1e30f;
  for (int cpt : {1, 2, 4}) {
    mam4b_tuning t = b;
    t.cells_per_thread = cpt;
    float ms = 1e30f;
    if (e == cudaSuccess)
      e = total_of(t, ms);
    if (e == cudaSuccess && ms < t_best) {
      t_best = ms;
      b.cells_per_thread = cpt;
    }
  }
  // short SOA loops finished in pre: changes the work of pre, soa and post
  // together, so it is chosen on the whole step
  for (int sc : {1, 4, 16, 64}) {
    mam4b_tuning t = b;
    t.inline_scale = sc;
    float ms = 1e30f;
    if (e == cudaSuccess)
      e = total_of(t, ms);
    if (e == cudaSuccess && ms < t_best) {
      t_best = ms;
      b.inline_scale = sc;
    }
  }
  float t_def = 1e30f;
  if (e == cudaSuccess)
    e = total_of(d, t_def);
  if (e == cudaSuccess)
    e = total_of(b, t_best);
  for (int k = 0; k < nev; ++k)
    cudaEventDestroy(ev[k]);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  if (!(t_best < t_def)) {
    b = d;
    t_best = t_def;
  }
  ctx->tune = b;
  ctx->tune_given = true;
  if (best)
    *best = b;
  if (default_ms)
    *default_ms = t_def;
  if (best_ms)
    *best_ms = t_best;
  return MAM4B_OK;
}

// The step with gas-phase and aqueous chemistry ahead of amicphys (FP64):
// the forward pipeline with the chemistry in its pre stage; slabs of ld
// doubles per field.
mam4b_status mam4b_step_chem_slab(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                                  const double *chem_in, double *out_slab, double *chem_out,
                                  size_t ld, int ncol, int nlev, double dt, void *stream) {
  const char *what = "mam4b_step_chem_slab";
  if (!ctx || !in_slab || !pblh || !chem_in || !out_slab || !chem_out || ncol < 0 ||
      nlev <= 0 || ld < (size_t)ncol * (size_t)nlev || !(dt > 0.0) || !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  StepArgs a;
  memset(&a, 0, sizeof(a));
  for (int f = 0; f < MAM4B_NIN; ++f)
    a.in[f] = in_slab + (size_t)f * ld;
  a.pblh = pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f)
    a.out[f] = out_slab + (size_t)f * ld;
  set_step_config(ctx, a, (long long)ncol * nlev, nlev, dt);
  ChemArgs ch;
  ch.in = chem_in;
  ch.out = chem_out;
  ch.ld = ld;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (a.ncell == 0)
    return MAM4B_OK;
  if (a.ncell > 0x7fffffffLL)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  cudaError_t e = ensure_solver_scratch(ctx, (size_t)a.ncell);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  set_step_scratch(ctx, a, 0, 0);
  e = launch_pipeline(ctx, a, s, MAM4B_FP64, &ch);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  return MAM4B_OK;
}

static cudaError_t grow(double **p, size_t *cap, size_t need) {
  if (*cap >= need)
    return cudaSuccess;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMalloc(p, need * sizeof(double));
  if (e == cudaSuccess)
    *cap = need;
  return e;
}

mam4b_status mam4b_step_host(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                             double *out_slab, size_t ld, int ncol, int nlev, double dt,
                             int precision, void *stream) {
  if (!ctx || !in_slab || !pblh || !out_slab || ncol < 0 || nlev <= 0 ||
      ld < (size_t)ncol * (size_t)nlev || !(dt > 0.0) || !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_host", cudaSuccess);
  if (precision != MAM4B_FP64 && precision != MAM4B_MIXED && precision != MAM4B_MIXED_FAST)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_host: precision", cudaSuccess);
  const size_t n = (size_t)ncol * (size_t)nlev;
  if (n > 0x7fffffffULL)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_host: too many cells", cudaSuccess);
  cudaStream_t us = (cudaStream_t)stream;
  ctx->last_stream = us;
  if (n == 0)
    return MAM4B_OK;
  cudaError_t e = grow(&ctx->d_in, &ctx->cap_in, (size_t)MAM4B_NIN * n);
  if (e == cudaSuccess)
    e = grow(&ctx->d_out, &ctx->cap_out, (size_t)MAM4B_NOUT * n);
  if (e == cudaSuccess)
    e = grow(&ctx->d_pblh, &ctx->cap_pblh, (size_t)ncol);
  if (e == cudaSuccess)
    e = ensure_solver_scratch(ctx, n);
  if (e == cudaSuccess)
    e = ensure_host_streams(ctx);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step_host scratch", e);
  // chunks of whole columns: the first ones a quarter and a half of the
  // steady size, so that the copy-out engine starts early; at most
  // kMaxChunks (the steady size grows for very large batches)
  int chunk_cols = (int)(kHostChunkCells / nlev);
  if (chunk_cols < 1)
    chunk_cols = 1;
  if ((ncol + chunk_cols - 1) / chunk_cols > kMaxChunks - 2)
    chunk_cols = (ncol + kMaxChunks - 3) / (kMaxChunks - 2);
  int chunk_start[kMaxChunks + 1];
  int nchunk = 0;
  for (int col = 0; col < ncol; ++nchunk) {
    chunk_start[nchunk] = col;
    const int want = nchunk == 0 ? (chunk_cols + 3) / 4 : nchunk == 1 ? (chunk_cols + 1) / 2 : chunk_cols;
    col += want < ncol - col ? want : ncol - col;
  }
  chunk_start[nchunk] = ncol;
  // the internal streams start after the work already queued on us
  e = cudaEventRecord(ctx->ev_start, us);
  for (int k = 0; k < kHostStreams && e == cudaSuccess; ++k)
    e = cudaStreamWaitEvent(ctx->hs[k], ctx->ev_start, 0);
  const size_t dp = n * sizeof(double), hp = ld * sizeof(double);
  cudaStream_t s_in = ctx->hs[0], s_out = ctx->hs[kHostStreams - 1];
  for (int i = 0; i < nchunk && e == cudaSuccess; ++i) {
    cudaStream_t s = ctx->hs[1 + i % kComputeStreams];
    const int col0 = chunk_start[i];
    const int ncc = chunk_start[i + 1] - col0;
    const size_t c0 = (size_t)col0 * nlev, nc = (size_t)ncc * nlev;
    // field f of the chunk: nc doubles at f*ld + c0 on the host, f*n + c0 on the device
    e = cudaMemcpy2DAsync(ctx->d_in + c0, dp, in_slab + c0, hp, nc * sizeof(double), MAM4B_NIN,
                          cudaMemcpyHostToDevice, s_in);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(ctx->d_pblh + col0, pblh + col0, (size_t)ncc * sizeof(double),
                          cudaMemcpyHostToDevice, s_in);
    if (e == cudaSuccess)
      e = cudaEventRecord(ctx->ev_in[i], s_in);
    if (e == cudaSuccess)
      e = cudaStreamWaitEvent(s, ctx->ev_in[i], 0);
    if (e != cudaSuccess)
      break;
    StepArgs a;
    memset(&a, 0, sizeof(a));
    for (int f = 0; f < MAM4B_NIN; ++f)
      a.in[f] = ctx->d_in + (size_t)f * n + c0;
    a.pblh = ctx->d_pblh + col0;
    for (int f = 0; f < MAM4B_NOUT; ++f)
      a.out[f] = ctx->d_out + (size_t)f * n + c0;
    set_step_config(ctx, a, (long long)nc, nlev, dt);
    set_step_scratch(ctx, a, c0, i);
    e = launch_pipeline(ctx, a, s, precision);
    if (e == cudaSuccess)
      e = cudaEventRecord(ctx->ev_comp[i], s);
    if (e == cudaSuccess)
      e = cudaStreamWaitEvent(s_out, ctx->ev_comp[i], 0);
    if (e == cudaSuccess)
      e = cudaMemcpy2DAsync(out_slab + c0, hp, ctx->d_out + c0, dp, nc * sizeof(double),
                            MAM4B_NOUT, cudaMemcpyDeviceToHost, s_out);
  }
  // us waits for every internal stream, then the call returns
  for (int k = 0; k < kHostStreams; ++k) {
    cudaError_t e2 = cudaEventRecord(ctx->ev_done[k], ctx->hs[k]);
    if (e2 == cudaSuccess)
      e2 = cudaStreamWaitEvent(us, ctx->ev_done[k], 0);
    if (e == cudaSuccess)
      e = e2;
  }
  cudaError_t e3 = cudaStreamSynchronize(us);
  if (e == cudaSuccess)
    e = e3;
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step_host", e);
  return MAM4B_OK;
}

// The step on per-column arrays (include/mam4b.h, mam4b_step_columns):
// gather the columns into the context's staging slabs, the pipeline, then
// add the tendencies to (and write the mode outputs into) the caller's
// columns. Two pointer tables go to the device per call, synchronously.
mam4b_status mam4b_step_columns(mam4b_ctx *ctx, const mam4b_column *cols, int ncol, int nlev,
                                double dt, int precision, void *stream) {
  const char *what = "mam4b_step_columns";
  if (!ctx || !cols || ncol < 0 || nlev <= 0 || !(dt > 0.0) || !isfinite(dt) ||
      (long long)ncol * nlev > 0x7fffffffLL ||
      (precision != MAM4B_FP64 && precision != MAM4B_MIXED && precision != MAM4B_MIXED_FAST))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  for (int c = 0; c < ncol; ++c)
    for (int f = 0; f < MAM4B_NIN; ++f)
      if (!cols[c].in[f])
        return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_columns: null input column",
                       cudaSuccess);
  if (ncol == 0)
    return MAM4B_OK;
  const size_t ncell = (size_t)ncol * nlev;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  cudaError_t e = grow(&ctx->d_in, &ctx->cap_in, (size_t)MAM4B_NIN * ncell);
  if (e == cudaSuccess)
    e = grow(&ctx->d_out, &ctx->cap_out, (size_t)MAM4B_NOUT * ncell);
  if (e == cudaSuccess)
    e = grow(&ctx->d_pblh, &ctx->cap_pblh, (size_t)ncol);
  const size_t ntab = (size_t)(MAM4B_NIN + MAM4B_NOUT) * ncol;
  if (e == cudaSuccess && ctx->cap_coltab < ntab) {
    cudaFree(ctx->d_coltab);
    ctx->d_coltab = nullptr;
    ctx->cap_coltab = 0;
    e = cudaMalloc(&ctx->d_coltab, ntab * sizeof(void *));
    if (e == cudaSuccess)
      ctx->cap_coltab = ntab;
  }
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_step_columns scratch", e);
  // tables [input fields][col], then [output fields][col]; pblh per column
  ctx->h_coltab.assign(ntab + (size_t)ncol, nullptr);
  double *pb = reinterpret_cast<double *>(ctx->h_coltab.data() + ntab);
  for (int c = 0; c < ncol; ++c) {
    for (int f = 0; f < MAM4B_NIN; ++f)
      ctx->h_coltab[(size_t)f * ncol + c] = const_cast<double *>(cols[c].in[f]);
    for (int f = 0; f < MAM4B_NUM_PROG; ++f)
      ctx->h_coltab[(size_t)(MAM4B_NIN + f) * ncol + c] = cols[c].tend[f];
    for (int f = 0; f < MAM4B_NOUT - MAM4B_NUM_PROG; ++f)
      ctx->h_coltab[(size_t)(MAM4B_NIN + MAM4B_NUM_PROG + f) * ncol + c] = cols[c].mode_out[f];
    pb[c] = cols[c].pblh;
  }
  static_assert(sizeof(double) == sizeof(void *), "pblh shares the pointer staging");
  e = cudaMemcpyAsync(ctx->d_coltab, ctx->h_coltab.data(), ntab * sizeof(void *),
                      cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ctx->d_pblh, pb, (size_t)ncol * sizeof(double), cudaMemcpyHostToDevice, s);
  // the host staging is reused by the next call: wait for the copies
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(s);
  const int block = 128;
  const unsigned gx = (unsigned)((ncell + block - 1) / block);
  if (e == cudaSuccess) {
    gather_columns_kernel<<<dim3(gx, MAM4B_NIN), block, 0, s>>>(
        reinterpret_cast<const double *const *>(ctx->d_coltab), ctx->d_in, ncol, nlev);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  const mam4b_status st = mam4b_step_slab(ctx, ctx->d_in, ctx->d_pblh, ctx->d_out, ncell, ncol,
                                          nlev, dt, precision, stream);
  if (st != MAM4B_OK)
    return st;
  scatter_columns_kernel<<<dim3(gx, MAM4B_NOUT), block, 0, s>>>(
      reinterpret_cast<double *const *>(ctx->d_coltab) + (size_t)MAM4B_NIN * ncol, ctx->d_out,
      ncol, nlev, MAM4B_NUM_PROG);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

mam4b_status mam4b_synchronize(mam4b_ctx *ctx) {
  if (!ctx)
    return MAM4B_ERR_INVALID_ARGUMENT;
  const cudaError_t e = cudaStreamSynchronize(ctx->last_stream);
  return e == cudaSuccess ? MAM4B_OK : set_err(ctx, MAM4B_ERR_CUDA, "mam4b_synchronize", e);
}

// Allocation-free step for callers that cannot call cudaMalloc (a host
// model whose memory pool owns the GPU's memory, or that forbids the
// device-wide synchronisation of cudaMalloc/cudaFree once it runs). Same
// kernels as mam4b_step, with their scratch in g_noalloc_scratch. Nothing
// here allocates: set-up uses cudaGetSymbolAddress, a kernel, copies into
// the constant bank and occupancy queries; each step clears the counters
// with cudaMemsetAsync and launches the six pipeline kernels (size, mode,
// pair, pre, soa, post), or the one full_kernel when condensation is off.
// All calls share the array, so calls that overlap on the GPU race.
mam4b_status mam4b_step_slab_noalloc(const mam4b_config *cfg, const double *in_slab,
                                     const double *pblh, double *out_slab, size_t ld, int ncol,
                                     int nlev, double dt, uint32_t *flags, void *stream) {
  mam4b_config c;
  if (cfg)
    c = *cfg;
  else
    mam4b_default_config(&c);
  if (!valid_config(&c) || !in_slab || !pblh || !out_slab || ncol < 0 || nlev <= 0 ||
      !(dt > 0.0) || !isfinite(dt) || ld < (size_t)ncol * (size_t)nlev)
    return MAM4B_ERR_INVALID_ARGUMENT;
  const long long ncell = (long long)ncol * nlev;
  if (ncell > (long long)MAM4B_NOALLOC_MAX_CELLS)
    return MAM4B_ERR_TOO_MANY_CELLS;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = noalloc_setup(dev);
  if (e != cudaSuccess)
    return MAM4B_ERR_CUDA;
  if (ncell == 0)
    return MAM4B_OK;
  const NoAllocDevice &nd = g_noalloc[dev];
  StepArgs a;
  memset(&a, 0, sizeof(a));
  for (int f = 0; f < MAM4B_NIN; ++f)
    a.in[f] = in_slab + (size_t)f * ld;
  a.pblh = pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f)
    a.out[f] = out_slab + (size_t)f * ld;
  unsigned *tail = reinterpret_cast<unsigned *>(nd.scratch + kNoAllocTail);
  a.counters = tail;  // CNT_WORDS queue counters, then the spare flag word
  a.flags = flags ? reinterpret_cast<unsigned *>(flags) : tail + CNT_WORDS;
  a.soa = nd.scratch + kNoAllocSoa;
  a.hand = nd.scratch + kNoAllocHand;
  a.done = reinterpret_cast<int *>(nd.scratch + kNoAllocDone);
  a.order = reinterpret_cast<int *>(nd.scratch + kNoAllocOrder);
  a.aux = nd.scratch + kNoAllocAux;
  a.ncell = ncell;
  a.nlev = nlev;
  a.dt = dt;
  a.do_cond = c.do_cond;
  a.do_rename = c.do_rename;
  a.do_newnuc = c.do_newnuc;
  a.do_coag = c.do_coag;
  a.optaa = c.gaexch_h2so4_uptake_optaa;
  a.nmono = c.n_so4_monolayers_pcage;
  set_solver(a, nd.sms);
  cudaStream_t s = (cudaStream_t)stream;
  // the counters (and the spare flag word) must start every step at zero
  e = cudaMemsetAsync(tail, 0, (CNT_WORDS + 1) * sizeof(unsigned), s);
  if (e != cudaSuccess)
    return MAM4B_ERR_CUDA;
  const int block = 128;
  const unsigned grid = (unsigned)((ncell + block - 1) / block);
  if (!a.do_cond) {
    // no SOA loop to pipeline (and no scratch used)
    full_kernel<false><<<grid, block, 0, s>>>(a);
  } else {
    // the default launch shape (mam4b_default_tuning)
    mam4b_tuning t;
    mam4b_default_tuning(&t);
    launch_front(t, a, s);
    launch_mode(t, a, s, false);
    launch_pair(t, a, s, false);
    launch_pre(t, a, s);
    launch_soa(t, nd.sms, a, s, MAM4B_FP64);
    launch_post(t, a, s);
  }
  e = cudaGetLastError();
  return e == cudaSuccess ? MAM4B_OK : MAM4B_ERR_CUDA;
}

// Reverse-mode adjoint (include/mam4b.h). With condensation on: the
// forward pipeline (without its post stage) into the context's output
// scratch, then eight reverse launches (suffix, the counting sort of the
// SOA loops, the loops, front, water uptake, calcsize); otherwise one
// thread per cell (adjoint_kernel).
mam4b_status mam4b_adjoint_slab(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                                const double *out_bar, double *in_bar, size_t ld, int ncol,
                                int nlev, double dt, void *stream) {
  return mam4b_adjoint_slab_ex(ctx, in_slab, pblh, out_bar, in_bar, ld, ncol, nlev, dt,
                               MAM4B_FP64, stream);
}

mam4b_status mam4b_adjoint_slab_ex(mam4b_ctx *ctx, const double *in_slab, const double *pblh,
                                   const double *out_bar, double *in_bar, size_t ld, int ncol,
                                   int nlev, double dt, int precision, void *stream) {
  if (!ctx || !in_slab || !pblh || !out_bar || !in_bar || ncol < 0 || nlev <= 0 ||
      ld < (size_t)ncol * (size_t)nlev || !(dt > 0.0) || !isfinite(dt) ||
      (precision != MAM4B_FP64 && precision != MAM4B_MIXED && precision != MAM4B_MIXED_FAST))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_adjoint_slab", cudaSuccess);
  if (!ctx->cfg.do_cond && !ctx->cfg.do_newnuc)
    return set_err(ctx, MAM4B_ERR_NOT_SUPPORTED,
                   "mam4b_adjoint_slab: needs condensation or nucleation on", cudaSuccess);
  if (precision == MAM4B_MIXED_FAST || (precision == MAM4B_MIXED && !ctx->cfg.do_cond))
    return set_err(ctx, MAM4B_ERR_NOT_SUPPORTED,
                   "mam4b_adjoint_slab: precision not supported (FP64; MIXED with condensation on)",
                   cudaSuccess);
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  const long long ncell = (long long)ncol * nlev;
  if (ncell == 0)
    return MAM4B_OK;
  if (ncell > 0x7fffffffLL)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_adjoint_slab: too many cells", cudaSuccess);
  const adj::AdjCfg cfg = {ctx->cfg.do_cond, ctx->cfg.do_rename, ctx->cfg.do_newnuc,
                           ctx->cfg.do_coag, ctx->cfg.gaexch_h2so4_uptake_optaa,
                           ctx->cfg.n_so4_monolayers_pcage};
  cudaError_t e = cudaSuccess;
  if (!ctx->cfg.do_cond) {
    if (!ctx->d_ck) {
      int dev = 0, sms = 0, per_sm = 0;
      e = cudaGetDevice(&dev);
      if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, adjoint_kernel, 128, 0);
      if (e == cudaSuccess) {
        ctx->adj_grid = sms * (per_sm > 0 ? per_sm : 1);
        e = cudaMalloc(&ctx->d_ck, (size_t)6 * adj::kSoaCkMax * ctx->adj_grid * 128 * sizeof(double));
      }
      if (e != cudaSuccess) {
        ctx->d_ck = nullptr;
        return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_adjoint_slab scratch", e);
      }
    }
    AdjArgs a;
    a.in = in_slab;
    a.pblh = pblh;
    a.ybar = out_bar;
    a.xbar = in_bar;
    a.ld = ld;
    a.ncell = ncell;
    a.nlev = nlev;
    a.dt = dt;
    a.cfg = cfg;
    a.ck = ctx->d_ck;
    adjoint_kernel<<<ctx->adj_grid, 128, 0, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess)
      return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_adjoint_slab launch", e);
    ctx->launches += 1;
    return MAM4B_OK;
  }
  // pipelined adjoint
  const size_t n = (size_t)ncell;
  e = grow(&ctx->d_out, &ctx->cap_out, (size_t)MAM4B_NOUT * n);
  if (e == cudaSuccess)
    e = ensure_solver_scratch(ctx, n);
  if (e == cudaSuccess && ctx->cap_adj < n) {
    cudaFree(ctx->d_abar);
    cudaFree(ctx->d_lbar);
    cudaFree(ctx->d_npass);
    ctx->d_abar = ctx->d_lbar = nullptr;
    ctx->d_npass = nullptr;
    ctx->cap_adj = 0;
    e = cudaMalloc(&ctx->d_abar, (size_t)AB_FIELDS * n * sizeof(double));
    if (e == cudaSuccess)
      e = cudaMalloc(&ctx->d_lbar, (size_t)LB_FIELDS * n * sizeof(double));
    if (e == cudaSuccess)
      e = cudaMalloc(&ctx->d_npass, n * sizeof(int));
    if (e == cudaSuccess && !ctx->d_bins)
      e = cudaMalloc(&ctx->d_bins, 2 * kPassBins * sizeof(unsigned));
    if (e == cudaSuccess)
      ctx->cap_adj = n;
  }
  const int ck_interval = ctx->adj_ck > 1 ? ctx->adj_ck : 1;
  if (e == cudaSuccess && ctx->d_ck2 && ctx->ck2_slots < adj_soa_slots(ck_interval)) {
    cudaFree(ctx->d_ck2);
    ctx->d_ck2 = nullptr;
    ctx->ck2_slots = 0;
  }
  if (e == cudaSuccess && !ctx->d_ck2) {
    int dev = 0, sms = 0, per_sm = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
      e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, adj_soa_kernel<1, false>,
                                                        kSoaBlock, 0);
    if (e == cudaSuccess) {
      ctx->adj_soa_grid = sms * (per_sm > 0 ? per_sm : 1);
      const int slots = adj_soa_slots(ck_interval);
      e = cudaMalloc(&ctx->d_ck2, (size_t)6 * slots * ctx->adj_soa_grid * kSoaBlock * sizeof(double));
      if (e != cudaSuccess)
        ctx->d_ck2 = nullptr;
      else
        ctx->ck2_slots = slots;
    }
  }
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_adjoint_slab scratch", e);
  AdjPipeArgs p;
  memset(&p, 0, sizeof(p));
  for (int f = 0; f < MAM4B_NIN; ++f)
    p.s.in[f] = in_slab + (size_t)f * ld;
  p.s.pblh = pblh;
  for (int f = 0; f < MAM4B_NOUT; ++f)
    p.s.out[f] = ctx->d_out + (size_t)f * n;
  set_step_config(ctx, p.s, ncell, nlev, dt);
  set_step_scratch(ctx, p.s, 0, 0);
  p.ybar = out_bar;
  p.xbar = in_bar;
  p.ld = ld;
  p.abar = ctx->d_abar;
  p.lbar = ctx->d_lbar;
  p.ck = ctx->d_ck2;
  p.bins = ctx->d_bins;
  p.cfg = cfg;
  p.s.npass = ctx->d_npass;
  e = launch_pipeline(ctx, p.s, s, precision);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(ctx->d_bins, 0, kPassBins * sizeof(unsigned), s);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_adjoint_slab forward", e);
  const int block = 128;
  const unsigned grid = (unsigned)((ncell + block - 1) / block);
  const unsigned sort_grid = (unsigned)std::min<long long>((ncell + 255) / 256, 4 * 148);
  adj_post_kernel<<<grid, block, 0, s>>>(p);
  adj_hist_kernel<<<sort_grid, 256, 0, s>>>(p);
  adj_scan_kernel<<<1, 1024, 0, s>>>(p);
  adj_sort_kernel<<<sort_grid, 256, 0, s>>>(p);
  const bool fast = precision == MAM4B_MIXED;
  if (ck_interval == 4 && fast)
    adj_soa_kernel<4, true><<<ctx->adj_soa_grid, kSoaBlock, 0, s>>>(p);
  else if (ck_interval == 4)
    adj_soa_kernel<4, false><<<ctx->adj_soa_grid, kSoaBlock, 0, s>>>(p);
  else if (fast)
    adj_soa_kernel<1, true><<<ctx->adj_soa_grid, kSoaBlock, 0, s>>>(p);
  else
    adj_soa_kernel<1, false><<<ctx->adj_soa_grid, kSoaBlock, 0, s>>>(p);
  adj_pre_kernel<<<grid, block, 0, s>>>(p);
  adj_mode_kernel<<<dim3(grid, NMODE), block, 0, s>>>(p);
  adj_fin_kernel<<<grid, block, 0, s>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_adjoint_slab launch", e);
  ctx->launches += 8;
  return MAM4B_OK;
}

// The step on mam4::TracersView-layout arrays (state_q tracer order,
// utils.hpp:205-259): a field table into the caller's rows, then the step.
mam4b_status mam4b_step_tracers(mam4b_ctx *ctx, const double *q, const double *qqcw,
                                size_t tracer_stride, const double *temperature,
                                const double *pressure, const double *height,
                                const double *cloud_fraction, const double *pblh,
                                double *ptend_q, double *ptend_qqcw, double *mode_out,
                                size_t mode_stride, int ncol, int nlev, double dt,
                                int precision, void *stream) {
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !q || !qqcw || !temperature || !pressure || !height || !cloud_fraction || !pblh ||
      !ptend_q || !ptend_qqcw || !mode_out || ncol < 0 || nlev <= 0 || tracer_stride < n ||
      mode_stride < n)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_step_tracers", cudaSuccess);
  constexpr int kQv = 0, kH2so4 = 11, kSoag = 14, kAero = 15;
  mam4b_state_view iv;
  mam4b_tend_view ov;
  memset(&iv, 0, sizeof(iv));
  memset(&ov, 0, sizeof(ov));
  iv.field[MAM4B_IN_T] = temperature;
  iv.field[MAM4B_IN_P] = pressure;
  iv.field[MAM4B_IN_ZM] = height;
  iv.field[MAM4B_IN_QV] = q + (size_t)kQv * tracer_stride;
  iv.field[MAM4B_IN_CLD] = cloud_fraction;
  iv.field[MAM4B_IN_H2SO4] = q + (size_t)kH2so4 * tracer_stride;
  iv.field[MAM4B_IN_SOAG] = q + (size_t)kSoag * tracer_stride;
  ov.field[MAM4B_OUT_TEND + 0] = ptend_q + (size_t)kH2so4 * tracer_stride;
  ov.field[MAM4B_OUT_TEND + 1] = ptend_q + (size_t)kSoag * tracer_stride;
  for (int p = 0; p < MAM4B_NUM_POPS; ++p) {
    iv.field[MAM4B_IN_AER_I + p] = q + (size_t)(kAero + p) * tracer_stride;
    iv.field[MAM4B_IN_AER_C + p] = qqcw + (size_t)(kAero + p) * tracer_stride;
    ov.field[MAM4B_OUT_TEND + 2 + p] = ptend_q + (size_t)(kAero + p) * tracer_stride;
    ov.field[MAM4B_OUT_TEND + 27 + p] = ptend_qqcw + (size_t)(kAero + p) * tracer_stride;
  }
  for (int k = 0; k < 16; ++k)
    ov.field[MAM4B_OUT_DGN_A + k] = mode_out + (size_t)k * mode_stride;
  iv.pblh = pblh;
  return mam4b_step(ctx, &iv, &ov, ncol, nlev, dt, precision, stream);
}

// Copies a set of packed bands into the context (*dev).
static mam4b_status set_optics_tables(mam4b_ctx *ctx, const char *what, double **dev,
                                      const double *specref, const double *water,
                                      const double *refr, const double *refi,
                                      const double *const *tabs, int ntab, int node, int bands) {
  const size_t per = (size_t)opt::band_doubles(node), bytes = per * bands * sizeof(double);
  double *h = (double *)malloc(bytes);
  if (!h)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  for (int b = 0; b < bands; ++b)
    opt::pack_band(specref, MAM4B_OPTICS_NTYPES, water, refr, refi, tabs, ntab, node, bands, b,
                   h + per * b);
  cudaError_t e = cudaSuccess;
  if (!*dev)
    e = cudaMalloc(dev, bytes);
  if (e == cudaSuccess)
    e = cudaMemcpy(*dev, h, bytes, cudaMemcpyHostToDevice);
  free(h);
  return e == cudaSuccess ? MAM4B_OK : set_err(ctx, MAM4B_ERR_CUDA, what, e);
}

// longwave optics tables: the reference's per-type species refractive
// indices mapped to modes by species type (set_device_specrefindex,
// modal_aero_opt.hpp:142-190), water, grids and absorption tables
mam4b_status mam4b_optics_lw_set_tables(mam4b_ctx *ctx, const mam4b_optics_lw_tables *t) {
  const char *what = "mam4b_optics_lw_set_tables";
  if (!ctx || !t || !t->specrefindex || !t->water_refindex || !t->refrtab || !t->refitab ||
      !t->absp)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  const double *tabs[1] = {t->absp};
  return set_optics_tables(ctx, what, &ctx->d_optics_lw, t->specrefindex, t->water_refindex,
                           t->refrtab, t->refitab, tabs, 1, opt::kLwNode, opt::kLwBands);
}

// shortwave optics tables (layouts of mam4b_optics_sw_tables)
mam4b_status mam4b_optics_sw_set_tables(mam4b_ctx *ctx, const mam4b_optics_sw_tables *t) {
  const char *what = "mam4b_optics_sw_set_tables";
  if (!ctx || !t || !t->specrefindex || !t->water_refindex || !t->refrtab || !t->refitab ||
      !t->extp || !t->absp || !t->asmp)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  const double *tabs[3] = {t->extp, t->absp, t->asmp};
  return set_optics_tables(ctx, what, &ctx->d_optics_sw, t->specrefindex, t->water_refindex,
                           t->refrtab, t->refitab, tabs, 3, opt::kSwNode, opt::kSwBands);
}

// The arguments that both optics entries share; volc with the volcanic
// fields for the radiation-facing entries (its trop set), else null.
static mam4b_status run_optics(mam4b_ctx *ctx, const char *what, bool sw, const double *in_slab,
                               size_t ld, const double *pdeldry, double *out, double *aodvis,
                               int ncol, int nlev, double dt, const OpticsArgs *volc,
                               cudaStream_t s) {
  OpticsArgs a;
  memset(&a, 0, sizeof(a));
  if (volc)
    a = *volc;
  const size_t n = (size_t)ncol * nlev;
  for (int f = 0; f < MAM4B_NIN; ++f)
    a.in[f] = in_slab + (size_t)f * ld;
  a.pdeldry = pdeldry;
  a.tables = sw ? ctx->d_optics_sw : ctx->d_optics_lw;
  a.out = out;
  a.aodvis = aodvis;
  a.ld = ld;
  a.ncell = (long long)n;
  a.ncol = ncol;
  a.nlev = nlev;
  a.dt = dt;
  a.scr = ctx->d_optics_scr;
  const unsigned grid = (unsigned)((n + 127) / 128), grid2 = (unsigned)((n + 255) / 256);
  const unsigned cells = std::min((unsigned)((n + kBandBlock - 1) / kBandBlock), kBandCellBlocks);
  optics_size_kernel<<<grid, 128, 0, s>>>(a);
  int launches = 3;
  if (sw) {
    optics_mode_kernel<true><<<dim3(grid2, NMODE), 256, 0, s>>>(a);
    optics_sw_band_kernel<<<dim3(opt::kSwBands, cells), kBandBlock, 0, s>>>(a);
    if (aodvis) {
      optics_sw_aod_kernel<<<(unsigned)((ncol + 3) / 4), 128, 0, s>>>(a);
      ++launches;
    }
  } else {
    optics_mode_kernel<false><<<dim3(grid2, NMODE), 256, 0, s>>>(a);
    optics_band_kernel<<<dim3(opt::kLwBands, cells), kBandBlock, 0, s>>>(a);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += launches;
  return MAM4B_OK;
}

// Doubles of an optics entry's per-cell values. The number and the list of the
// cells with modal optics (n + 1 ints) follow them in the same allocation, so
// that the radiation-facing entries can be captured after any entry of the size.
static size_t optics_scratch(bool sw, size_t n) {
  return (size_t)(sw ? OS_FIELDS : OS_LW_FIELDS) * n;
}
static unsigned *modal_list(const mam4b_ctx *ctx, bool sw, size_t n) {
  return reinterpret_cast<unsigned *>(ctx->d_optics_scr + optics_scratch(sw, n));
}

// Argument checks and scratch of an optics entry; *empty: nothing to do.
static mam4b_status begin_optics(mam4b_ctx *ctx, const char *what, bool sw, const double *in_slab,
                                 size_t ld, const double *pdeldry, const double *out, int ncol,
                                 int nlev, double dt, cudaStream_t s, bool *empty) {
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !in_slab || !pdeldry || !out || ncol < 0 || nlev <= 0 || ld < n || !(dt > 0.0) ||
      !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  if (!(sw ? ctx->d_optics_sw : ctx->d_optics_lw))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT,
                   sw ? "mam4b_optics_sw: tables not set" : "mam4b_optics_lw: tables not set",
                   cudaSuccess);
  ctx->last_stream = s;
  *empty = n == 0;
  if (*empty)
    return MAM4B_OK;
  const cudaError_t e =
      grow(&ctx->d_optics_scr, &ctx->cap_optics_scr, optics_scratch(sw, n) + (n + 2) / 2);
  return e == cudaSuccess ? MAM4B_OK : set_err(ctx, MAM4B_ERR_CUDA, what, e);
}

// modal_aero_opt::modal_aero_sw (modal_aero_opt.hpp:536-878), batched
mam4b_status mam4b_optics_sw(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                             const double *pdeldry, double *out, double *aodvis, int ncol,
                             int nlev, double dt, void *stream) {
  const char *what = "mam4b_optics_sw";
  cudaStream_t s = (cudaStream_t)stream;
  bool empty;
  const mam4b_status st =
      begin_optics(ctx, what, true, in_slab, ld, pdeldry, out, ncol, nlev, dt, s, &empty);
  if (st != MAM4B_OK || empty)
    return st;
  return run_optics(ctx, what, true, in_slab, ld, pdeldry, out, aodvis, ncol, nlev, dt, nullptr, s);
}

// modal_aero_opt::modal_aero_lw_k (modal_aero_opt.hpp:879-989), batched
mam4b_status mam4b_optics_lw(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                             const double *pdeldry, double *tauxar, int ncol, int nlev,
                             double dt, void *stream) {
  const char *what = "mam4b_optics_lw";
  cudaStream_t s = (cudaStream_t)stream;
  bool empty;
  const mam4b_status st =
      begin_optics(ctx, what, false, in_slab, ld, pdeldry, tauxar, ncol, nlev, dt, s, &empty);
  if (st != MAM4B_OK || empty)
    return st;
  return run_optics(ctx, what, false, in_slab, ld, pdeldry, tauxar, nullptr, ncol, nlev, dt,
                    nullptr, s);
}

// Tropopause levels of the columns into *trop_level (the caller's array, or
// the context's, which it is then set to) and the list of cells at or below
// them (modal_list).
static mam4b_status rad_props_tropopause(mam4b_ctx *ctx, const char *what, bool sw,
                                         const double *in_slab, size_t ld, const double *pint,
                                         int ncol, int nlev, int **trop_level, cudaStream_t s) {
  RadArgs r;
  memset(&r, 0, sizeof(r));
  r.temp = in_slab + (size_t)MAM4B_IN_T * ld;
  r.pmid = in_slab + (size_t)MAM4B_IN_P * ld;
  r.pint = pint;
  r.ncol = ncol;
  r.nlev = nlev;
  if (!*trop_level) {
    if (ctx->cap_trop < (size_t)ncol) {
      cudaFree(ctx->d_trop);
      ctx->d_trop = nullptr;
      ctx->cap_trop = 0;
      const cudaError_t e = cudaMalloc(&ctx->d_trop, (size_t)ncol * sizeof(int));
      if (e != cudaSuccess)
        return set_err(ctx, MAM4B_ERR_CUDA, what, e);
      ctx->cap_trop = (size_t)ncol;
    }
    *trop_level = ctx->d_trop;
  }
  r.trop = *trop_level;
  const size_t n = (size_t)ncol * nlev;
  if (n > 0x7fffffffu)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  r.nmodal = modal_list(ctx, sw, n);
  r.modal = reinterpret_cast<int *>(r.nmodal + 1);
  const int block = 128, per_block = block / 32;
  const size_t smem = (size_t)per_block * 4 * nlev * sizeof(double);
  if (smem > 48 * 1024)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  const cudaError_t e0 = cudaMemsetAsync(r.nmodal, 0, sizeof(unsigned), s);
  if (e0 != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e0);
  tropopause_kernel<<<(unsigned)((ncol + per_block - 1) / per_block), block, smem, s>>>(r);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

// aero_rad_props_sw (aero_rad_props.hpp:250-338), batched
mam4b_status mam4b_aero_rad_props_sw(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                                     const double *pdeldry, const double *pint, const double *zi,
                                     const double *ext_sw, const double *ssa_sw,
                                     const double *af_sw, double *out, double *aodvis,
                                     int *trop_level, int ncol, int nlev, double dt,
                                     void *stream) {
  const char *what = "mam4b_aero_rad_props_sw";
  if (!ctx || !pint || !zi || !ext_sw || !ssa_sw || !af_sw || nlev < 2)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  cudaStream_t s = (cudaStream_t)stream;
  bool empty;
  mam4b_status st = begin_optics(ctx, "mam4b_optics_sw", true, in_slab, ld, pdeldry, out, ncol,
                                 nlev, dt, s, &empty);
  if (st != MAM4B_OK || empty)
    return st;
  st = rad_props_tropopause(ctx, what, true, in_slab, ld, pint, ncol, nlev, &trop_level, s);
  if (st != MAM4B_OK)
    return st;
  OpticsArgs v;
  memset(&v, 0, sizeof(v));
  v.trop = trop_level;
  v.nmodal = modal_list(ctx, true, (size_t)ncol * nlev);
  v.modal = reinterpret_cast<const int *>(v.nmodal + 1);
  v.zi = zi;
  v.ext = ext_sw;
  v.ssa = ssa_sw;
  v.af = af_sw;
  return run_optics(ctx, what, true, in_slab, ld, pdeldry, out, aodvis, ncol, nlev, dt, &v, s);
}

// aero_rad_props_lw (aero_rad_props.hpp:339-410), batched
mam4b_status mam4b_aero_rad_props_lw(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                                     const double *pdeldry, const double *pint, const double *zi,
                                     const double *ext_lw, double *odap, int *trop_level,
                                     int ncol, int nlev, double dt, void *stream) {
  const char *what = "mam4b_aero_rad_props_lw";
  if (!ctx || !pint || !zi || !ext_lw || nlev < 2)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  cudaStream_t s = (cudaStream_t)stream;
  bool empty;
  mam4b_status st = begin_optics(ctx, "mam4b_optics_lw", false, in_slab, ld, pdeldry, odap, ncol,
                                 nlev, dt, s, &empty);
  if (st != MAM4B_OK || empty)
    return st;
  st = rad_props_tropopause(ctx, what, false, in_slab, ld, pint, ncol, nlev, &trop_level, s);
  if (st != MAM4B_OK)
    return st;
  OpticsArgs v;
  memset(&v, 0, sizeof(v));
  v.trop = trop_level;
  v.nmodal = modal_list(ctx, false, (size_t)ncol * nlev);
  v.modal = reinterpret_cast<const int *>(v.nmodal + 1);
  v.zi = zi;
  v.ext = ext_lw;
  return run_optics(ctx, what, false, in_slab, ld, pdeldry, odap, nullptr, ncol, nlev, dt, &v, s);
}

// ndrop::dropmixnuc (ndrop.hpp:1393-1714), one block per column
mam4b_status mam4b_dropmixnuc(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                              const double *mix_in, const double *pint, const double *kvh,
                              double *out, int ncol, int nlev, int top_lev, int vertical_mix,
                              double dt, void *stream) {
  const char *what = "mam4b_dropmixnuc";
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !in_slab || !mix_in || !pint || !kvh || !out || ncol < 0 || nlev < 2 || ld < n ||
      top_lev < 1 || top_lev > nlev - 2 || !(dt > 0.0) || !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  // a lane of the column kernel holds at most kDmMaxLevels / 32 levels
  constexpr int kDmMaxLevels = 201;
  if (nlev > kDmMaxLevels)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_dropmixnuc: too many levels",
                   cudaSuccess);
  const size_t smem = (size_t)nlev * (DM_FIELDS + kDmWarps) * sizeof(double);
  DropmixArgs a;
  memset(&a, 0, sizeof(a));
  for (int f = 0; f < MAM4B_NIN; ++f)
    a.in[f] = in_slab + (size_t)f * ld;
  a.mix = mix_in;
  a.pint = pint;
  a.kvh = kvh;
  a.out = out;
  a.flags = ctx->d_flags;
  a.ld = ld;
  a.ncol = ncol;
  a.nlev = nlev;
  a.top_lev = top_lev;
  a.vertical_mix = vertical_mix ? 1 : 0;
  a.dt = dt;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (n == 0)
    return MAM4B_OK;
  cudaError_t e = grow(&ctx->d_dmx, &ctx->cap_dmx, (size_t)DA_FIELDS * n);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_dropmixnuc scratch", e);
  a.act = ctx->d_dmx;
  const unsigned cells = (unsigned)((n + 127) / 128);
  auto columns = [&](auto levels) {
    constexpr int L = decltype(levels)::value;
    const cudaError_t ea = cudaFuncSetAttribute(
        dropmix_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ea == cudaSuccess)
      dropmix_kernel<L><<<(unsigned)ncol, 32 * kDmWarps, smem, s>>>(a);
    return ea;
  };
  dropmix_act_kernel<<<(unsigned)((n + kDmActBlock - 1) / kDmActBlock), kDmActBlock, 0, s>>>(a);
  // levels per lane
  switch ((nlev - top_lev + 31) / 32) {
  case 1: e = columns(std::integral_constant<int, 1>()); break;
  case 2: e = columns(std::integral_constant<int, 2>()); break;
  case 3: e = columns(std::integral_constant<int, 3>()); break;
  case 4: e = columns(std::integral_constant<int, 4>()); break;
  case 5: e = columns(std::integral_constant<int, 5>()); break;
  case 6: e = columns(std::integral_constant<int, 6>()); break;
  default: e = columns(std::integral_constant<int, 7>()); break;
  }
  dropmix_ccn_kernel<<<cells, 128, 0, s>>>(a);
  if (e == cudaSuccess)
    e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 3;
  return MAM4B_OK;
}

// ndrop get_activate_frac (ndrop.hpp:699-765), batched
mam4b_status mam4b_activate(mam4b_ctx *ctx, const double *in_slab, size_t ld,
                            const double *air_density, const double *updraft, double *out,
                            int ncol, int nlev, void *stream) {
  const char *what = "mam4b_activate";
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !in_slab || !air_density || !updraft || !out || ncol < 0 || nlev <= 0 || ld < n)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  ActivateArgs a;
  a.temp = in_slab + (size_t)MAM4B_IN_T * ld;
  for (int p = 0; p < NPOP; ++p)
    a.aer[p] = in_slab + (size_t)(MAM4B_IN_AER_I + p) * ld;
  a.rho = air_density;
  a.w = updraft;
  a.out = out;
  a.ld = ld;
  a.ncell = (long long)n;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (n == 0)
    return MAM4B_OK;
  const int block = 128;
  activate_kernel<<<(unsigned)((n + block - 1) / block), block, 0, s>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

// mo_setsox::setsox_single_level (mo_setsox.hpp:944-1254), batched
mam4b_status mam4b_setsox(mam4b_ctx *ctx, const double *pressure, const double *temperature,
                          const double *lwc, const double *cloud_fraction,
                          const double *cloud_number, const double *air_density, double *qin,
                          double *qcw, size_t ld, double *dqdt_aqso4, double *dqdt_aqh2so4,
                          int ncol, int nlev, double dt, void *stream) {
  const char *what = "mam4b_setsox";
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !pressure || !temperature || !lwc || !cloud_fraction || !cloud_number ||
      !air_density || !qin || !qcw || ncol < 0 || nlev <= 0 || ld < n || !(dt > 0.0) ||
      !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  SetsoxArgs a;
  a.press = pressure;
  a.temp = temperature;
  a.lwc = lwc;
  a.cldfrc = cloud_fraction;
  a.cldnum = cloud_number;
  a.xhnm = air_density;
  a.qin = qin;
  a.qcw = qcw;
  a.dso4 = dqdt_aqso4;
  a.dh2so4 = dqdt_aqh2so4;
  a.ld = ld;
  a.ncell = (long long)n;
  a.dt = dt;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (n == 0)
    return MAM4B_OK;
  const int block = 128;
  setsox_kernel<<<(unsigned)((n + block - 1) / block), block, 0, s>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

// gas_phase_chemistry (gas_phase_chemistry.hpp:40-117), batched
mam4b_status mam4b_gas_chemistry(mam4b_ctx *ctx, const double *temperature,
                                 const double *photo_rates, const double *extfrc,
                                 const double *invariants, const double *het_rates, double *qq,
                                 size_t ld, int ncol, int nlev, double dt, void *stream) {
  const char *what = "mam4b_gas_chemistry";
  const size_t n = (size_t)(ncol > 0 ? ncol : 0) * (size_t)(nlev > 0 ? nlev : 0);
  if (!ctx || !temperature || !photo_rates || !extfrc || !invariants || !het_rates || !qq ||
      ncol < 0 || nlev <= 0 || ld < n || !(dt > 0.0) || !isfinite(dt))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  GasChemArgs a;
  a.temp = temperature;
  a.photo = photo_rates;
  a.extfrc = extfrc;
  a.inv = invariants;
  a.het = het_rates;
  a.qq = qq;
  a.ld = ld;
  a.ncell = (long long)n;
  a.dt = dt;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (n == 0)
    return MAM4B_OK;
  const int block = 128;
  gaschem_kernel<<<(unsigned)((n + block - 1) / block), block, 0, s>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

static bool copy_prog_fields(const mam4b_prog_fields *f, ProgFields &o) {
  if (!f)
    return false;
  for (int m = 0; m < NMODE; ++m) {
    o.n_i[m] = f->n_mode_i[m];
    o.n_c[m] = f->n_mode_c[m];
    for (int x = 0; x < NAER; ++x) {
      o.q_i[m][x] = f->q_aero_i[m][x];
      o.q_c[m][x] = f->q_aero_c[m][x];
    }
  }
  return true;
}

// CalcSize::compute_tendencies (calcsize.hpp:963-1220), batched
mam4b_status mam4b_calcsize_process(mam4b_ctx *ctx, const mam4b_calcsize_config *cfg,
                                    const mam4b_prog_fields *progs,
                                    const mam4b_prog_fields *tends,
                                    double *const dgncur_i[MAM4B_NUM_MODES],
                                    double *const dgncur_c[MAM4B_NUM_MODES], int ncol,
                                    int nlev, double dt, void *stream) {
  const char *what = "mam4b_calcsize_process";
  if (!ctx || ncol < 0 || nlev <= 0 || !(dt > 0.0) || !isfinite(dt) || !dgncur_i || !dgncur_c)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  CalcSizeArgs a;
  memset(&a, 0, sizeof(a));
  if (!copy_prog_fields(progs, a.progs) || !copy_prog_fields(tends, a.tends))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  a.do_aitacc_transfer = cfg ? (cfg->do_aitacc_transfer != 0) : 1;
  a.do_adjust = cfg ? (cfg->do_adjust != 0) : 1;
  // every field the process reads or writes must be given
  for (int m = 0; m < NMODE; ++m) {
    if (!dgncur_i[m] || !dgncur_c[m] || !a.progs.n_i[m] || !a.progs.n_c[m])
      return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_calcsize_process: null field",
                     cudaSuccess);
    a.dgn_i[m] = dgncur_i[m];
    a.dgn_c[m] = dgncur_c[m];
    const bool tn = a.do_adjust && !(a.do_aitacc_transfer && m <= 1);
    const bool tx = a.do_aitacc_transfer && m <= 1;
    if ((tn || tx) && (!a.tends.n_i[m] || !a.tends.n_c[m]))
      return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_calcsize_process: null tendency",
                     cudaSuccess);
    for (int s = 0; s < K::nspec(m); ++s) {
      if (!a.progs.q_i[m][s] || !a.progs.q_c[m][s])
        return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_calcsize_process: null field",
                       cudaSuccess);
    }
  }
  if (a.do_aitacc_transfer) {
    const int acc_s[4] = {0, 2, 5, 6}, ait_s[4] = {0, 1, 2, 3};
    for (int k = 0; k < 4; ++k)
      if (!a.tends.q_i[0][acc_s[k]] || !a.tends.q_c[0][acc_s[k]] || !a.tends.q_i[1][ait_s[k]] ||
          !a.tends.q_c[1][ait_s[k]])
        return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT,
                       "mam4b_calcsize_process: null tendency", cudaSuccess);
  }
  a.ncell = (long long)ncol * nlev;
  a.dt = dt;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (a.ncell == 0)
    return MAM4B_OK;
  const int block = 128;
  calcsize_process_kernel<<<(unsigned)((a.ncell + block - 1) / block), block, 0, s>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 1;
  return MAM4B_OK;
}

// Coagulation::compute_tendencies (coagulation.hpp:1198-1209), batched
mam4b_status mam4b_coagulation_process(mam4b_ctx *ctx, const double *temperature,
                                       const double *pressure,
                                       const double *const wet_density[MAM4B_NUM_MODES],
                                       const double *const wet_diameter_i[MAM4B_NUM_MODES],
                                       const mam4b_prog_fields *progs,
                                       const mam4b_prog_fields *tends, int ncol, int nlev,
                                       double dt, void *stream) {
  const char *what = "mam4b_coagulation_process";
  if (!ctx || ncol < 0 || nlev <= 0 || !(dt > 0.0) || !isfinite(dt) || !temperature ||
      !pressure || !wet_density || !wet_diameter_i)
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  CoagProcessArgs a;
  memset(&a, 0, sizeof(a));
  if (!copy_prog_fields(progs, a.progs) || !copy_prog_fields(tends, a.tends))
    return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, what, cudaSuccess);
  a.temp = temperature;
  a.pmid = pressure;
  for (int m = 0; m < NMODE; ++m) {
    if (!wet_density[m] || !wet_diameter_i[m] || !a.progs.n_i[m] || !a.tends.n_i[m])
      return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT, "mam4b_coagulation_process: null field",
                     cudaSuccess);
    a.wet_density[m] = wet_density[m];
    a.dgn_awet[m] = wet_diameter_i[m];
    for (int x = 0; x < NAER; ++x)
      if (!a.progs.q_i[m][x] || !a.tends.q_i[m][x])
        return set_err(ctx, MAM4B_ERR_INVALID_ARGUMENT,
                       "mam4b_coagulation_process: null field", cudaSuccess);
  }
  a.ncell = (long long)ncol * nlev;
  a.dt = dt;
  cudaStream_t s = (cudaStream_t)stream;
  ctx->last_stream = s;
  if (a.ncell == 0)
    return MAM4B_OK;
  cudaError_t e = grow(&ctx->d_coag_cc, &ctx->cap_coag_cc, (size_t)12 * a.ncell);
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  a.cc = ctx->d_coag_cc;
  const int block = 128;
  const unsigned grid = (unsigned)((a.ncell + block - 1) / block);
  coag_pair_process_kernel<<<dim3(grid, 3), block, 0, s>>>(a);
  coag_process_kernel<<<grid, block, 0, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, what, e);
  ctx->launches += 2;
  return MAM4B_OK;
}

mam4b_status mam4b_last_status(mam4b_ctx *ctx, uint32_t *flags) {
  if (!ctx || !flags)
    return MAM4B_ERR_INVALID_ARGUMENT;
  cudaError_t e = cudaStreamSynchronize(ctx->last_stream);
  unsigned h = 0;
  if (e == cudaSuccess)
    e = cudaMemcpy(&h, ctx->d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess)
    e = cudaMemset(ctx->d_flags, 0, sizeof(unsigned));
  if (e != cudaSuccess)
    return set_err(ctx, MAM4B_ERR_CUDA, "mam4b_last_status", e);
  *flags = h;
  return (h & MAM4B_FLAGS_ERROR_MASK) ? MAM4B_ERR_DEVICE_FLAGS : MAM4B_OK;
}

void mam4b_last_error(mam4b_ctx *ctx, char *buf, size_t len) {
  if (!buf || len == 0)
    return;
  const char *m = ctx ? ctx->err : "null context";
  snprintf(buf, len, "%s", m);
}

uint64_t mam4b_launch_count(mam4b_ctx *ctx) { return ctx ? (uint64_t)ctx->launches : 0; }

}  // extern "C"
