// physics.cuh -- device-side physics of the ECHO-QGP step: equation of
// state, reconstruction, fluxes, sources, primitive<->conserved maps.
//
// Every routine restates a reference Fortran routine (file:line given on
// each) with the same operation order and parenthesisation, so that a build
// with -fmad=false reproduces the CPU restatement bit for bit (IEEE division
// and square root are correctly rounded on both sides).  The `KIND`
// template parameter selects the equation set at compile time:
//   KIND_HD      ideal hydro, nv = 5
//   KIND_VISC    Israel-Stewart viscous hydro, nv = 12
//   KIND_MHD     ideal MHD, nv = 8
//   KIND_MHDGLM  ideal MHD with GLM divergence cleaning, nv = 9
//   KIND_RES     resistive MHD (E a primitive) with GLM, nv = 12
#pragma once

#include <cstdint>
#include <math.h>

#include "../../include/echo_gpu.h"

namespace echo {

enum { KIND_HD = 0, KIND_VISC = 1, KIND_MHD = 2, KIND_MHDGLM = 3, KIND_RES = 4 };

template <int KIND>
struct Traits;
template <>
struct Traits<KIND_HD> {
  static constexpr int NV = 5, KG = -1;
  static constexpr bool MHD = false, VISC = false, GLM = false, RES = false;
};
template <>
struct Traits<KIND_VISC> {
  static constexpr int NV = 12, KG = -1;
  static constexpr bool MHD = false, VISC = true, GLM = false, RES = false;
};
template <>
struct Traits<KIND_MHD> {
  static constexpr int NV = 8, KG = -1;
  static constexpr bool MHD = true, VISC = false, GLM = false, RES = false;
};
template <>
struct Traits<KIND_MHDGLM> {
  static constexpr int NV = 9, KG = 8;
  static constexpr bool MHD = true, VISC = false, GLM = true, RES = false;
};
// resistive runs (MHD = 2): B, E, psi (system.f90:92-105, 113-116)
template <>
struct Traits<KIND_RES> {
  static constexpr int NV = 12, KG = 11;
  static constexpr bool MHD = true, VISC = false, GLM = true, RES = true;
};

// variable indices (common.f90:63), 0-based
enum { KRH = 0, KVX = 1, KVY = 2, KVZ = 3, KPR = 4, KPIBU = 5, KPIXY = 6, KPIXZ = 7,
       KPIYZ = 8, KPIXX = 9, KPIYY = 10, KPIZZ = 11 };
enum { KBX = 5, KBY = 6, KBZ = 7, KGLM = 8 };  // KGLM: ideal MHD; Traits<K>::KG in general
enum { KEX = 8, KEY = 9, KEZ = 10 };              // resistive E^i
// derivative indices (common.f90:70-71), 0-based
enum { DTX = 0, DTY, DTZ, DXX, DXY, DXZ, DYX, DYY, DYZ, DZX, DZY, DZZ, DTT, DXT, DYT, DZT, NDER = 16 };

// One interval of the EoS table, rows i and i + 1: everything a lookup in it
// reads, in one 64-byte line (the columns are 2048 entries apart).  e(p) from
// the first half, p(e) from te, tp and the third quarter, c_s^2 the last.
struct __align__(16) EosRec {
  double tp, te;     // p, e of row i
  double sl_ep, tp1; // de/dp; p of row i + 1
  double sl_pe, te1; // dp/de = (dp/dT) / (de/dT); e of row i + 1
  double tc, sl_ce;  // c_s^2 of row i; d(c_s^2)/de
};
// A bucket of the bracket search (tab_bracket): the lower bound h of the
// bracket of its values and the table value h stands for
struct __align__(16) EosBucket {
  double node;
  int h, pad;
};

// Parameters and per-step metric, passed by value to every kernel.
struct DevPhys {
  int eqstate, coordinates, recal, obtained_zz, init_type, bulkvis;
  int nt;
  const double* __restrict__ tT;
  const double* __restrict__ te;
  const double* __restrict__ tp;
  const double* __restrict__ tc;
  // bracket accelerators for te and tp (see tab_bracket); null = plain search
  const int* __restrict__ bke;
  const int* __restrict__ bkp;
  long long bke0, bkp0;
  int nbke, nbkp;
  // product build: the intervals of the table as records and the buckets of
  // their bracket search (null: search the columns and interpolate with
  // divisions, as the reference does); the table's first and last e and p
  const struct EosRec* __restrict__ rec;
  const struct EosBucket* __restrict__ qe;
  const struct EosBucket* __restrict__ qp;
  double emin, emax, pmin, pmax;
  double maxspeed, eta_over_s, tau_pi_coeff, enezero, przero, glm_alpha;
  double sigma_el, sigma_chiral;  // resistive runs: conductivities (code units)
};

// metric (system_metric_*, system.f90:132-160), derived from t on device.
// g_11 = g_22 = 1 in both coordinate systems of the reference (Minkowski
// and Bjorken), so they are compile-time ones: x * 1.0 is exactly x, and
// the multiplications the reference writes with them drop out.
struct Metric {
  static constexpr double g1 = 1.0, g2 = 1.0;
  double g3, gp, gm, g0, t, t3, ig3;
};

__device__ __forceinline__ Metric make_metric(int coordinates, double t, double t3) {
  Metric m;
  m.g0 = -1.;
  m.t = t;
  m.t3 = t3;
  if (coordinates == ECHO_BJORKEN) {
    m.g3 = t * t;
    m.gp = t;
    m.gm = 1. / m.gp;
  } else {
    m.g3 = 1.;
    m.gp = 1.;
    m.gm = 1.;
  }
  m.ig3 = 1. / m.g3;
  return m;
}

// x / g3 and x / gp as the reference writes them; the product build
// multiplies by the reciprocals, computed once per thread
__device__ __forceinline__ double over_g3(const Metric& M, double x) {
#ifdef ECHO_EXACT
  return x / M.g3;
#else
  return x * M.ig3;
#endif
}
__device__ __forceinline__ double over_gp(const Metric& M, double x) {
#ifdef ECHO_EXACT
  return x / M.gp;
#else
  return x * M.gm;
#endif
}

#ifndef ECHO_EXACT
// ---------------------------------------------------------------------------
// Reciprocal, reciprocal square root, square root and quotient of the product
// build: the hardware's approximation (PTX rcp.approx.ftz.f64,
// rsqrt.approx.ftz.f64, relative errors of about 2^-23) and one third-order
// Householder correction each (Householder, The Numerical Treatment of a Single
// Nonlinear Equation, 1970, ch. 4: x (1 + e + e^2) for 1/a with e = 1 - a x,
// y (1 + e/2 + 3 e^2 / 8) for 1/sqrt(a) with e = 1 - a y^2), without the
// special-case branches of the division and of sqrt().
//
// Errors over normal operands and results: reciprocal, square root and quotient
// within 0.51 ulp, rsqrt within 1.01 (the rounding of a y enters e).
//
// *_h3 return the division's and sqrt's own results at 0, infinity and NaN: a
// con2prim that starts at v^2 = 1 or from no pressure meets 1 - v^2 = 0 and an
// infinite or zero enthalpy.  There the correction is NaN (of 0 times infinity)
// and the approximation the result.  Subnormal operands and results count as 0;
// the square roots take operands below 1e-290 as 0.
//
// *_n, where operands and results are normal or a NaN is as good as the
// division's result: the WENO weights' denominators, the speeds of a face state
// (v^2 < 1), table spacings, the Newton steps of newton3 (which leave NaN to
// BRENTM).  With the test for NaN in the speeds and in newton3 too a step of
// 97 x 97 x 81 RMHD took 965 us, 954 without it there.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool is_nan(double r) { return (unsigned)__double2hiint(r) << 1 > 0xffe00000u; }
__device__ __forceinline__ double rcp_approx(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  return x;
}
__device__ __forceinline__ double rsqrt_approx(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return y;
}
__device__ __forceinline__ double rcp_step(double a, double x) {
  const double e = fma(-a, x, 1.);
  return fma(x, fma(e, e, e), x);
}
__device__ __forceinline__ double rsqrt_step(double a, double y) {
  const double e = fma(-a * y, y, 1.);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double rcp_n(double a) { return rcp_step(a, rcp_approx(a)); }
__device__ __forceinline__ double rcp_h3(double a) {
  const double x = rcp_approx(a), r = rcp_step(a, x);
  return is_nan(r) ? x : r;
}
__device__ __forceinline__ double rsqrt_n(double a) { return rsqrt_step(a, rsqrt_approx(a)); }
__device__ __forceinline__ double rsqrt_h3(double a) {
  const double y = rsqrt_approx(a), r = rsqrt_step(a, y);
  return is_nan(r) ? y : r;
}
__device__ __forceinline__ double sqrt_n(double a) {
  const double y = rsqrt_n(a), r = a * y;
  return fabs(a) < 1e-290 ? 0. : fma(fma(-r, r, a), 0.5 * y, r);
}
__device__ __forceinline__ double sqrt_h3(double a) { return __double2hiint(a) == 0x7ff00000 ? a : sqrt_n(a); }
// b / a, the quotient of rcp_n corrected by its residual
__device__ __forceinline__ double div_n(double b, double a) {
  const double x = rcp_n(a), q = b * x;
  return fma(fma(-q, a, b), x, q);
}
#endif

// ---------------------------------------------------------------------------
// equation of state (eos.f90)
// ---------------------------------------------------------------------------

// the bracket search of eos.f90:430-442; returns indxh (1-based)
__device__ __forceinline__ int tab_search(const double* __restrict__ arr, int n, double val) {
  int lo = 1, hi = n, mid = (lo + hi) / 2;
  while (lo + 1 != hi) {
    if (val > __ldg(arr + mid - 1)) {
      lo = mid;
    } else {
      hi = mid;
    }
    mid = (lo + hi) / 2;
  }
  return hi;
}

// The bracket of the search above in O(1): the index of a positive double's
// bit pattern >> BK_SHIFT is monotonic in its value (128 buckets per binade);
// bk[b] holds, for bucket b, a lower bound of the bracket of every value in
// the bucket, built on the host from the table itself.  A short forward scan
// then lands on exactly the index the binary search returns:
// max(2, smallest i with arr(i) >= val) for arr(1) <= val <= arr(n).
#define BK_SHIFT 45
__device__ __forceinline__ int tab_bracket(const double* __restrict__ arr, const int* __restrict__ bk,
                                           long long k0, int nb, int n, double val) {
  if (bk == nullptr) return tab_search(arr, n, val);
  long long key = (__double_as_longlong(val) >> BK_SHIFT) - k0;
  key = key < 0 ? 0 : (key >= nb ? nb - 1 : key);
  int h = __ldg(bk + key);
  while (h < n && __ldg(arr + h - 1) < val) h++;
  return h;
}
#ifdef ECHO_EXACT
struct EosAt {
  int h;
};
#else
// Product build: the interval of a lookup.  The bracket is tab_search's (the
// smallest row h >= 2 with arr(h) >= val), found with two dependent loads --
// the bucket, then the record, which holds the values that confirm it -- where
// bucket, scan and columns took four: the lookups of the fluxes and of the
// con2prim Newton loops are latency.  Kept across the steps of a Newton
// iteration: an interval that still holds the value is not looked up again.
struct EosAt {
  double p0, e0, sl;  // row i; slope of the looked-up direction
  double hi;          // upper end of the interval in the looked-up variable
  int h;              // bracket (rows h - 1, h; 1-based), 0 = none yet
};
__device__ __forceinline__ int eos_bucket(const EosBucket* __restrict__ q, long long k0, int nb, int n, double val) {
  long long key = (__double_as_longlong(val) >> BK_SHIFT) - k0;
  key = key < 0 ? 0 : (key >= nb ? nb - 1 : key);
  const double2 b = __ldg((const double2*)(q + key));
  const int h = __double2loint(b.y);
  return h < n && b.x < val ? h + 1 : h;
}
// interval of the p column that holds pr (pmin <= pr <= pmax)
__device__ __forceinline__ void eos_at_p(const DevPhys& P, double pr, EosAt& a) {
  int h = eos_bucket(P.qp, P.bkp0, P.nbkp, P.nt, pr);
  const double2* r = (const double2*)(P.rec + (h - 2));
  double2 x = __ldg(r), y = __ldg(r + 1);
  while (h < P.nt && y.y < pr) {
    h++;
    r += 4;
    x = __ldg(r);
    y = __ldg(r + 1);
  }
  a.p0 = x.x;
  a.e0 = x.y;
  a.sl = y.x;
  a.hi = y.y;
  a.h = h;
}
// interval of the e column that holds en (emin <= en <= emax)
__device__ __forceinline__ void eos_at_e(const DevPhys& P, double en, EosAt& a) {
  int h = eos_bucket(P.qe, P.bke0, P.nbke, P.nt, en);
  const double2* r = (const double2*)(P.rec + (h - 2));
  double2 x = __ldg(r), y = __ldg(r + 2);
  while (h < P.nt && y.y < en) {
    h++;
    r += 4;
    x = __ldg(r);
    y = __ldg(r + 2);
  }
  a.p0 = x.x;
  a.e0 = x.y;
  a.sl = y.x;
  a.hi = y.y;
  a.h = h;
}
// whether the interval of an earlier lookup is the one of val (its lower end lo)
__device__ __forceinline__ bool eos_holds(const EosAt& a, double lo, double val) {
  return a.h > 0 && (val > lo || (a.h == 2 && val == lo)) && val <= a.hi;
}
#endif
#define SEARCH_E(P, val) tab_bracket((P).te, (P).bke, (P).bke0, (P).nbke, (P).nt, (val))
#define SEARCH_P(P, val) tab_bracket((P).tp, (P).bkp, (P).bkp0, (P).nbkp, (P).nt, (val))

// eos_energy: get_energy (eos.f90:468-523) / eos_energy_ana (eos.f90:1104-1185)
__device__ __forceinline__ int eos_energy(const DevPhys& P, double rh, double* en, double pr) {
  if (P.eqstate == ECHO_EOS_TABLE) {
#ifndef ECHO_EXACT
    if (P.rec) {
      if (pr < P.pmin) return 125;
      if (pr > P.pmax) return 126;
      EosAt a;
      eos_at_p(P, pr, a);
      *en = a.e0 + (pr - a.p0) * a.sl;
      return 0;
    }
#endif
    if (pr < __ldg(P.tp)) return 125;
    if (pr > __ldg(P.tp + P.nt - 1)) return 126;
    int h = SEARCH_P(P, pr);
    double p2 = __ldg(P.tp + h - 1), p1 = __ldg(P.tp + h - 2);
    double e2 = __ldg(P.te + h - 1), e1 = __ldg(P.te + h - 2);
    *en = e1 + (e2 - e1) * (pr - p1) / (p2 - p1);
    return 0;
  }
  if (pr <= P.przero) {
    *en = P.enezero * pr / P.przero;
    return 0;
  }
  if (P.eqstate == ECHO_EOS_CONFORMAL)
    *en = 3. * pr;
  else
    *en = rh + pr / (4.0 / 3.0 - 1.);
  return 0;
}

#ifndef ECHO_EXACT
// p(e) of a table with records; a holds the interval of the last call (h = 0: none)
__device__ __forceinline__ int eos_pressure_at(const DevPhys& P, double en, double* pr, double* dprdrh,
                                               double* dprden, EosAt& a) {
  if (!eos_holds(a, a.e0, en)) {
    if (en < P.emin) return 123;
    if (en > P.emax) return 124;
    eos_at_e(P, en, a);
  }
  *pr = a.p0 + (en - a.e0) * a.sl;
  *dprdrh = 0;
  *dprden = a.sl;
  return 0;
}
#endif

// eos_pressure: get_pressure (eos.f90:399-464) / eos_pressure_ana (eos.f90:886-922)
__device__ __forceinline__ int eos_pressure(const DevPhys& P, double rh, double en, double* pr,
                                            double* dprdrh, double* dprden) {
  if (P.eqstate == ECHO_EOS_TABLE) {
#ifndef ECHO_EXACT
    if (P.rec) {
      EosAt a;
      a.h = 0;
      return eos_pressure_at(P, en, pr, dprdrh, dprden, a);
    }
#endif
    if (en < __ldg(P.te)) return 123;
    if (en > __ldg(P.te + P.nt - 1)) return 124;
    int h = SEARCH_E(P, en);
    double p2 = __ldg(P.tp + h - 1), p1 = __ldg(P.tp + h - 2);
    double e2 = __ldg(P.te + h - 1), e1 = __ldg(P.te + h - 2);
    double t2 = __ldg(P.tT + h - 1), t1 = __ldg(P.tT + h - 2);
    *pr = p1 + (p2 - p1) * (en - e1) / (e2 - e1);
    double dpt = (p2 - p1) / (t2 - t1);
    double det = (e2 - e1) / (t2 - t1);
    *dprdrh = 0;
    *dprden = dpt / det;
    return 0;
  }
  if (P.eqstate == ECHO_EOS_CONFORMAL) {
    double a = 3.0;
    *pr = en / a;
    *dprdrh = 0.;
    *dprden = 1. / 3.;
  } else {
    double gam = 4.0 / 3.0;
    *pr = (gam - 1.) * (en - rh);
    *dprdrh = -gam + 1.;
    *dprden = gam - 1.;
  }
  return 0;
}

#ifndef ECHO_EXACT
// Product build, the face states of system_flux: e(p), and the interval for
// eos_sound_at.  a.h = 0 when the EoS is not a table with records (then
// eos_energy / eos_sound are used).
__device__ __forceinline__ int eos_energy_h(const DevPhys& P, double rh, double* en, double pr, EosAt& a) {
  if (P.eqstate == ECHO_EOS_TABLE && P.rec) {
    if (pr < P.pmin) return 125;
    if (pr > P.pmax) return 126;
    eos_at_p(P, pr, a);
    *en = a.e0 + (pr - a.p0) * a.sl;
    return 0;
  }
  a.h = 0;
  return eos_energy(P, rh, en, pr);
}
// c_s^2(e) for the e just interpolated: e lies in the same interval of the e
// column (e(p) is monotonic; at a node both neighbouring intervals give the
// node value), so get_sound's search is skipped
__device__ __forceinline__ double eos_sound_at(const DevPhys& P, const EosAt& a, double en) {
  const double2 c = __ldg((const double2*)(P.rec + (a.h - 2)) + 3);
  return c.x + (en - a.e0) * c.y;
}
#endif

// eos_sound: get_sound (eos.f90:590-641) / eos_sound_ana (eos.f90:926-952)
__device__ __forceinline__ int eos_sound(const DevPhys& P, double rh, double en, double pr, double* cs2) {
  if (P.eqstate == ECHO_EOS_TABLE) {
#ifndef ECHO_EXACT
    if (P.rec) {
      if (en < P.emin) return 131;
      if (en > P.emax) return 132;
      EosAt a;
      eos_at_e(P, en, a);
      *cs2 = eos_sound_at(P, a, en);
      return 0;
    }
#endif
    if (en < __ldg(P.te)) return 131;
    if (en > __ldg(P.te + P.nt - 1)) return 132;
    int h = SEARCH_E(P, en);
    double s2 = __ldg(P.tc + h - 1), s1 = __ldg(P.tc + h - 2);
    double e2 = __ldg(P.te + h - 1), e1 = __ldg(P.te + h - 2);
    *cs2 = s1 + (s2 - s1) * (en - e1) / (e2 - e1);
    return 0;
  }
  double dprden, dprdrh;
  if (P.eqstate == ECHO_EOS_CONFORMAL) {
    dprden = 1. / 3.;
    dprdrh = 0.;
  } else {
    double gam = 4.0 / 3.0;
    dprden = gam - 1.;
    dprdrh = -gam + 1.;
  }
  double c;
  if (en + pr == 0)
    c = dprden;
  else
    c = dprden + (rh / (en + pr)) * dprdrh;
  *cs2 = c > 0.0 ? c : 0.0;
  return 0;
}

// eos_pressure inside a Newton loop: a is the interval of the last call
// (a.h = 0 before the first)
__device__ __forceinline__ int eos_pressure_it(const DevPhys& P, double rh, double en, double* pr, double* dprdrh,
                                               double* dprden, EosAt& a) {
#ifndef ECHO_EXACT
  if (P.eqstate == ECHO_EOS_TABLE && P.rec) return eos_pressure_at(P, en, pr, dprdrh, dprden, a);
#endif
  return eos_pressure(P, rh, en, pr, dprdrh, dprden);
}

// get_derived_data: get_derived_data_tab (eos.f90:645-701) / _ana (eos.f90:956-968)
__device__ __forceinline__ int get_derived_data(const DevPhys& P, double rh, double pr, double* en,
                                                double* temp, double* s) {
  if (P.eqstate == ECHO_EOS_TABLE) {
#ifndef ECHO_EXACT
    if (P.rec) {
      if (pr < P.pmin) return 135;
      if (pr > P.pmax) return 136;
      EosAt a;
      eos_at_p(P, pr, a);
      const double e1 = a.e0, e2 = __ldg(&P.rec[a.h - 2].te1);
      const double t1 = __ldg(P.tT + a.h - 2), t2 = __ldg(P.tT + a.h - 1);
      const double fac = (pr - a.p0) / (a.hi - a.p0);
      *temp = t1 + (t2 - t1) * fac;
      *en = e1 + (e2 - e1) * fac;
      *s = (*en + pr) / *temp;
      return 0;
    }
#endif
    if (pr < __ldg(P.tp)) return 135;
    if (pr > __ldg(P.tp + P.nt - 1)) return 136;
    int h = SEARCH_P(P, pr);
    double p2 = __ldg(P.tp + h - 1), p1 = __ldg(P.tp + h - 2);
    double e2 = __ldg(P.te + h - 1), e1 = __ldg(P.te + h - 2);
    double t2 = __ldg(P.tT + h - 1), t1 = __ldg(P.tT + h - 2);
    double fac = (pr - p1) / (p2 - p1);
    *temp = t1 + (t2 - t1) * fac;
    *en = e1 + (e2 - e1) * fac;
    *s = (*en + pr) / *temp;
    return 0;
  }
  int err = eos_energy(P, rh, en, pr);
  *temp = 0.148909 * pow(*en, 0.25);
  if (*temp == 0)
    *s = 0.;
  else
    *s = (*en + pr) / *temp;
  return err;
}

// ---------------------------------------------------------------------------
// reconstruction (holib.f90)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double fsign1(double d) { return copysign(1.0, d); }

__device__ __forceinline__ double mm2(double d1, double d2) {  // holib.f90:440-452
  double s1 = fsign1(d1), s2 = fsign1(d2);
  double a1 = fabs(d1), a2 = fabs(d2);
  return .5 * (s1 + s2) * (a1 < a2 ? a1 : a2);
}
__device__ __forceinline__ double fmin3(double a, double b, double c) {
  double r = a;
  if (b < r) r = b;
  if (c < r) r = c;
  return r;
}
__device__ __forceinline__ double fmax3(double a, double b, double c) {
  double r = a;
  if (b > r) r = b;
  if (c > r) r = c;
  return r;
}
__device__ __forceinline__ double mm4(double d1, double d2, double d3, double d4) {  // :472-486
  double s1 = fsign1(d1), s2 = fsign1(d2), s3 = fsign1(d3), s4 = fsign1(d4);
  double m = fabs(d1);
  if (fabs(d2) < m) m = fabs(d2);
  if (fabs(d3) < m) m = fabs(d3);
  if (fabs(d4) < m) m = fabs(d4);
  return .125 * (s1 + s2) * fabs((s1 + s3) * (s1 + s4)) * m;
}
__device__ __forceinline__ double ceno3(double d0, double d1, double d2) {  // :490-510
  const double alpha = 0.7;
  double r = 0.;
  int s = (int)fsign1(d0) + (int)fsign1(d1) + (int)fsign1(d2);
  if (abs(s) == 3) {
    double w0 = fabs(d0), w1 = alpha * fabs(d1), w2 = fabs(d2);
    double wm = w0;
    r = d0;
    if (w1 < wm) {
      wm = w1;
      r = d1;
    }
    if (w2 < wm) {
      wm = w2;
      r = d2;
    }
  }
  return r;
}
__device__ __forceinline__ double mp5(double f, double f1, double f2, double f3, double f4, double f5) {
  double r = f;  // holib.f90:514-536
  double ful = f3 + 2 * (f3 - f2);
  double fmp = f3 + mm2(f4 - f3, ful - f3);
  if ((f - f3) * (f - fmp) > 0.) {
    double dm = f1 - 2 * f2 + f3;
    double d0 = f2 - 2 * f3 + f4;
    double dp = f3 - 2 * f4 + f5;
    double fmd = .5 * (f3 + f4) - .5 * mm4(4 * d0 - dp, 4 * dp - d0, d0, dp);
    double flc = f3 + .5 * (f3 - f2) + (4. / 3.) * mm4(4 * d0 - dm, 4 * dm - d0, d0, dm);
    double lo1 = fmin3(f3, f4, fmd), lo2 = fmin3(f3, ful, flc);
    double hi1 = fmax3(f3, f4, fmd), hi2 = fmax3(f3, ful, flc);
    double fmin = lo1 > lo2 ? lo1 : lo2;
    double fmax = hi1 < hi2 ? hi1 : hi2;
    r = f + mm2(fmin - f, fmax - f);
  }
  return r;
}

// WENO5 one side: f1..f5 in the reference's naming (holib.f90:198-212)
#ifndef ECHO_EXACT
// Product build: the scheme in differences of neighbouring values.  With d_i
// the first and D_i the second differences of a side's stencil f1..f5:
//  - 4 (beta_k / 12 + eps) is 4 d^2 + 4 d D + 16/3 D^2 + 4 eps with the d
//    beside f3 and the sub-stencil's D (4 d^2 - 4 d D for the third);
//  - the sub-stencil values are f3 + d / 2 + 3/8 D1, f3 + d / 2 + 3/8 D2 and
//    f3 + d / 2 + 1/2 D2 - 1/8 D3, so a state is f3 + d / 2 plus a weighted
//    mean of second differences;
//  - the common denominator of the weights is multiplied through,
//    sum_k d_k x_k / q_k^2 / sum_k d_k / q_k^2 = sum_k d_k x_k Q_j Q_l /
//    sum_k d_k Q_j Q_l with Q = q^2 (q >= 4e-6, so the products cannot
//    underflow), and the two states share one reciprocal: n1/m1 and n2/m2 =
//    (n1 m2, n2 m1) / (m1 m2), where m1, m2 >= 1e-21 and stay far below 1e150
//    for the values a run holds.
// 50 FP64 instructions for both states of a cell (written in values, 101 for
// the two states of a face), with less rounding: the cancellations of nearly
// equal values are the exact differences.
__device__ __forceinline__ double weno5_q(double D, double d4, double A) {  // d4 = 4 d, A = 4 d^2 + 4 eps
  return fma(D, fma(16. / 3., D, d4), A);
}
// 8/3 of the numerator beyond f3 + d / 2, and the denominator, of a side from
// its second differences and w1 = Q2 Q3, w2 = Q1 Q3, w3 = Q1 Q2; g = w2 D2,
// H = 20/3 D2
__device__ __forceinline__ void weno5_nm(double D1, double D3, double g, double H, double w1, double w2, double w3,
                                         double& n, double& m) {
  n = fma(w3, fma(-5. / 3., D3, H), fma(10., g, w1 * D1));
  m = fma(5., w3, fma(10., w2, w1));
}
// Both face states of one cell from its five-point stencil f1..f5 =
// v(c-2..c+2): plus = the state at c+1/2 (the left state of the face above,
// holib.f90:198-212 on f1..f5), minus = the state at c-1/2 (the right state of
// the face below, the same formula on f5..f1).  The two orientations share
// their three smoothness indicators.
__device__ __forceinline__ void weno5_cell(double f1, double f2, double f3, double f4, double f5, double& plus,
                                           double& minus) {
  const double d0 = f2 - f1, d1 = f3 - f2, d2 = f4 - f3, d3 = f5 - f4;
  const double Da = d1 - d0, Db = d2 - d1, Dc = d3 - d2;
  const double e1 = 4. * d1, e2 = -4. * d2;
  const double A1 = fma(e1, d1, 4.e-6), A2 = fma(-e2, d2, 4.e-6);
  const double qa = weno5_q(Da, e1, A1), qb = weno5_q(Db, e1, A1), qc = weno5_q(Dc, e2, A2);
  const double Qa = qa * qa, Qb = qb * qb, Qc = qc * qc;
  const double wbc = Qb * Qc, wac = Qa * Qc, wab = Qa * Qb;
  const double g = wac * Db, H = (20. / 3.) * Db;
  double np, mp, nm, mm;
  weno5_nm(Da, Dc, g, H, wbc, wac, wab, np, mp);
  weno5_nm(Dc, Da, g, H, wab, wac, wbc, nm, mm);  // reversed: the first differences change sign
  const double inv = 0.375 * rcp_n(mp * mm);
  plus = f3 + fma(np * mm, inv, 0.5 * d1);  // one rounding at the size of f3
  minus = f3 + fma(nm * mp, inv, -0.5 * d2);
}
// weno5_cell of the two neighbouring cells f[2] and f[3]: they share three first
// and two second differences and a smoothness term (42.5 FP64 instructions a
// cell)
__device__ __forceinline__ void weno5_pair(const double f[6], double plus[2], double minus[2]) {
  double d[5], D[5], e[4], A[4];
#pragma unroll
  for (int i = 0; i < 5; i++) d[i] = f[i + 1] - f[i];
#pragma unroll
  for (int i = 1; i < 5; i++) D[i] = d[i] - d[i - 1];
#pragma unroll
  for (int i = 1; i < 4; i++) {
    e[i] = 4. * d[i];
    A[i] = fma(e[i], d[i], 4.e-6);
  }
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const double Da = D[c + 1], Db = D[c + 2], Dc = D[c + 3];
    const double qa = weno5_q(Da, e[c + 1], A[c + 1]), qb = weno5_q(Db, e[c + 1], A[c + 1]);
    const double qc = weno5_q(Dc, -e[c + 2], A[c + 2]);
    const double Qa = qa * qa, Qb = qb * qb, Qc = qc * qc;
    const double wbc = Qb * Qc, wac = Qa * Qc, wab = Qa * Qb;
    const double g = wac * Db, H = (20. / 3.) * Db;
    double np, mp, nm, mm;
    weno5_nm(Da, Dc, g, H, wbc, wac, wab, np, mp);
    weno5_nm(Dc, Da, g, H, wab, wac, wbc, nm, mm);
    const double inv = 0.375 * rcp_n(mp * mm);
    plus[c] = f[c + 2] + fma(np * mm, inv, 0.5 * d[c + 1]);
    minus[c] = f[c + 2] + fma(nm * mp, inv, -0.5 * d[c + 2]);
  }
}
// Left and right state of the face between s[2] and s[3]
__device__ __forceinline__ void weno5_face(const double s[6], double& gl, double& gr) {
  const double d0 = s[1] - s[0], d1 = s[2] - s[1], d2 = s[3] - s[2], d3 = s[4] - s[3], d4 = s[5] - s[4];
  const double D1 = d1 - d0, D2 = d2 - d1, D3 = d3 - d2, D4 = d4 - d3;
  const double e1 = 4. * d1, e2 = 4. * d2, e3 = 4. * d3;
  const double A1 = fma(e1, d1, 4.e-6), A2 = fma(e2, d2, 4.e-6), A3 = fma(e3, d3, 4.e-6);
  double q1 = weno5_q(D1, e1, A1), q2 = weno5_q(D2, e1, A1), q3 = weno5_q(D3, -e2, A2);
  double Q1 = q1 * q1, Q2 = q2 * q2, Q3 = q3 * q3, w = Q1 * Q3, nl, ml, nr, mr;
  weno5_nm(D1, D3, w * D2, (20. / 3.) * D2, Q2 * Q3, w, Q1 * Q2, nl, ml);
  q1 = weno5_q(D4, -e3, A3);
  q2 = weno5_q(D3, -e3, A3);
  q3 = weno5_q(D2, e2, A2);
  Q1 = q1 * q1;
  Q2 = q2 * q2;
  Q3 = q3 * q3;
  w = Q1 * Q3;
  weno5_nm(D4, D2, w * D3, (20. / 3.) * D3, Q2 * Q3, w, Q1 * Q2, nr, mr);
  const double inv = 0.375 * rcp_n(ml * mr);
  gl = s[2] + fma(nl * mr, inv, 0.5 * d1);
  gr = s[3] + fma(nr * ml, inv, -0.5 * d3);
}
#else
__device__ __forceinline__ double weno5_side(double f1, double f2, double f3, double f4, double f5) {
  const double d1 = 1 / 16., d2 = 10 / 16., d3 = 5 / 16., eps = 1.e-6;
  const double c11 = 3 / 8., c21 = -10 / 8., c31 = 15 / 8.;
  const double c12 = -1 / 8., c22 = 6 / 8., c32 = 3 / 8.;
  const double c13 = 3 / 8., c23 = 6 / 8., c33 = -1 / 8.;
  double t1, t2, b1, b2, b3, q, a1, a2, a3;
  t1 = f3 - 2 * f2 + f1;
  t2 = 3. * f3 - 4. * f2 + f1;
  b1 = 13. * (t1 * t1) + 3. * (t2 * t2);
  t1 = f4 - 2 * f3 + f2;
  t2 = f4 - f2;
  b2 = 13. * (t1 * t1) + 3. * (t2 * t2);
  t1 = f5 - 2 * f4 + f3;
  t2 = f5 - 4. * f4 + 3. * f3;
  b3 = 13. * (t1 * t1) + 3. * (t2 * t2);
  q = b1 / 12. + eps;
  a1 = d1 / (q * q);
  q = b2 / 12. + eps;
  a2 = d2 / (q * q);
  q = b3 / 12. + eps;
  a3 = d3 / (q * q);
  double p1 = c11 * f1 + c21 * f2 + c31 * f3;
  double p2 = c12 * f2 + c22 * f3 + c32 * f4;
  double p3 = c13 * f3 + c23 * f4 + c33 * f5;
  return (a1 * p1 + a2 * p2 + a3 * p3) / (a1 + a2 + a3);
}
#endif

__device__ __forceinline__ double weno3_side(double f1, double f2, double f3) {  // :149-158
  const double d1 = 1 / 3., d2 = 2 / 3., eps = 1.e-6;
  const double c11 = -1 / 2., c21 = 3 / 2., c12 = 1 / 2., c22 = 1 / 2.;
  double b1 = (f2 - f1) * (f2 - f1);
  double b2 = (f3 - f2) * (f3 - f2);
  double a1 = d1 / ((b1 + eps) * (b1 + eps));
  double a2 = d2 / ((b2 + eps) * (b2 + eps));
  double p1 = c11 * f1 + c21 * f2;
  double p2 = c12 * f2 + c22 * f3;
  return (a1 * p1 + a2 * p2) / (a1 + a2);
}

__device__ __forceinline__ double ceno3_side(double f1, double f2, double f3, double f4, double f5) {
  const double c11 = 3 / 8., c21 = -10 / 8., c31 = 15 / 8.;  // holib.f90:98-109
  const double c12 = -1 / 8., c22 = 6 / 8., c32 = 3 / 8.;
  const double c13 = 3 / 8., c23 = 6 / 8., c33 = -1 / 8.;
  double p = f3 + .5 * mm2(f3 - f2, f4 - f3);
  double d0 = c11 * f1 + c21 * f2 + c31 * f3 - p;
  double d1 = c12 * f2 + c22 * f3 + c32 * f4 - p;
  double d2 = c13 * f3 + c23 * f4 + c33 * f5 - p;
  return p + ceno3(d0, d1, d2);
}

__device__ __forceinline__ double ppm4_side(double f1, double f2, double f3, double f4) {  // :250-255
  return f2 + .5 * (f3 - f2) - .125 * (mm2(f4 - f3, f3 - f2) - mm2(f3 - f2, f2 - f1));
}

// Left and right states at face i+1/2 from the 6-point stencil
// s[0..5] = f(i-2..i+3) (work_rec, work.f90:420-525).
__device__ __forceinline__ void recon_any(int recal, const double s[6], double& gl, double& gr) {
  switch (recal) {
    case ECHO_REC_TVD2: {  // holib.f90:47-77, rewritten per face
      gl = s[2] + .5 * mm2(s[2] - s[1], s[3] - s[2]);
      gr = s[3] - .5 * mm2(s[3] - s[2], s[4] - s[3]);
      break;
    }
    case ECHO_REC_CENO3:
      gl = ceno3_side(s[0], s[1], s[2], s[3], s[4]);
      gr = ceno3_side(s[5], s[4], s[3], s[2], s[1]);
      break;
    case ECHO_REC_WENO3:
      gl = weno3_side(s[1], s[2], s[3]);
      gr = weno3_side(s[4], s[3], s[2]);
      break;
    case ECHO_REC_WENO5:
#ifdef ECHO_EXACT
      gl = weno5_side(s[0], s[1], s[2], s[3], s[4]);
      gr = weno5_side(s[5], s[4], s[3], s[2], s[1]);
#else
      weno5_face(s, gl, gr);
#endif
      break;
    case ECHO_REC_PPM4:
      gl = ppm4_side(s[1], s[2], s[3], s[4]);
      gr = ppm4_side(s[4], s[3], s[2], s[1]);
      break;
    case ECHO_REC_MPE3: {  // holib.f90:272-294
      const double d1 = -1 / 8., d2 = 6 / 8., d3 = 3 / 8.;
      double l = d1 * s[1] + d2 * s[2] + d3 * s[3];
      double r = d1 * s[4] + d2 * s[3] + d3 * s[2];
      gl = mp5(l, s[0], s[1], s[2], s[3], s[4]);
      gr = mp5(r, s[5], s[4], s[3], s[2], s[1]);
      break;
    }
    default: {  // MPE5, holib.f90:298-320
      const double d1 = 3 / 128., d2 = -20 / 128., d3 = 90 / 128., d4 = 60 / 128., d5 = -5 / 128.;
      double l = d1 * s[0] + d2 * s[1] + d3 * s[2] + d4 * s[3] + d5 * s[4];
      double r = d1 * s[5] + d2 * s[4] + d3 * s[3] + d4 * s[2] + d5 * s[1];
      gl = mp5(l, s[0], s[1], s[2], s[3], s[4]);
      gr = mp5(r, s[5], s[4], s[3], s[2], s[1]);
      break;
    }
  }
}

// The reconstruction fixed at compile time (REC = ECHO_REC_*) or chosen at
// run time (REC = REC_RUNTIME).  The face kernels reconstruct every
// variable with an unrolled loop; a run-time switch inside it puts all seven
// schemes into the kernel once per variable, so the common scheme gets a
// kernel of its own.
enum { REC_RUNTIME = -1 };
template <int REC>
__device__ __forceinline__ void recon_face(int recal, const double s[6], double& gl, double& gr) {
  recon_any(REC >= 0 ? REC : recal, s, gl, gr);
}

// Both face states of the cell f[2] from its five-point stencil: plus as
// recon_any's left state of the face above it, minus as its right state of
// the face below (the same expressions, so the parity build's bits).
template <int REC>
__device__ __forceinline__ void recon_cell(int recal, const double f[5], double& plus, double& minus) {
  switch (REC >= 0 ? REC : recal) {
    case ECHO_REC_TVD2: {
      const double h = .5 * mm2(f[2] - f[1], f[3] - f[2]);
      plus = f[2] + h;
      minus = f[2] - h;
      break;
    }
    case ECHO_REC_CENO3:
      plus = ceno3_side(f[0], f[1], f[2], f[3], f[4]);
      minus = ceno3_side(f[4], f[3], f[2], f[1], f[0]);
      break;
    case ECHO_REC_WENO3:
      plus = weno3_side(f[1], f[2], f[3]);
      minus = weno3_side(f[3], f[2], f[1]);
      break;
    case ECHO_REC_WENO5:
#ifdef ECHO_EXACT
      plus = weno5_side(f[0], f[1], f[2], f[3], f[4]);
      minus = weno5_side(f[4], f[3], f[2], f[1], f[0]);
#else
      weno5_cell(f[0], f[1], f[2], f[3], f[4], plus, minus);
#endif
      break;
    case ECHO_REC_PPM4:
      plus = ppm4_side(f[1], f[2], f[3], f[4]);
      minus = ppm4_side(f[3], f[2], f[1], f[0]);
      break;
    case ECHO_REC_MPE3: {
      const double d1 = -1 / 8., d2 = 6 / 8., d3 = 3 / 8.;
      double l = d1 * f[1] + d2 * f[2] + d3 * f[3];
      double r = d1 * f[3] + d2 * f[2] + d3 * f[1];
      plus = mp5(l, f[0], f[1], f[2], f[3], f[4]);
      minus = mp5(r, f[4], f[3], f[2], f[1], f[0]);
      break;
    }
    default: {  // MPE5
      const double d1 = 3 / 128., d2 = -20 / 128., d3 = 90 / 128., d4 = 60 / 128., d5 = -5 / 128.;
      double l = d1 * f[0] + d2 * f[1] + d3 * f[2] + d4 * f[3] + d5 * f[4];
      double r = d1 * f[4] + d2 * f[3] + d3 * f[2] + d4 * f[1] + d5 * f[0];
      plus = mp5(l, f[0], f[1], f[2], f[3], f[4]);
      minus = mp5(r, f[4], f[3], f[2], f[1], f[0]);
      break;
    }
  }
}

// recon_cell of the N neighbouring cells f[2], f[3], ... from f[0..N+3]
template <int REC, int N>
__device__ __forceinline__ void recon_cells(int recal, const double* f, double* plus, double* minus) {
#ifndef ECHO_EXACT
  if (REC == ECHO_REC_WENO5 && N == 2) {
    weno5_pair(f, plus, minus);
    return;
  }
#endif
#pragma unroll
  for (int i = 0; i < N; i++) recon_cell<REC>(recal, f + i, plus[i], minus[i]);
}

// ---------------------------------------------------------------------------
// viscous helpers (viscous.f90)
// ---------------------------------------------------------------------------
struct Pit {
  double tt, tx, ty, tz, zz;
};

// get_derived_pi (viscous.f90:244-255)
__device__ __forceinline__ void derived_pi(const Metric& M, const double* p, Pit& o) {
  double g1 = M.g1, g2 = M.g2, g3 = M.g3;
  o.tx = p[KPIXX] * p[KVX] * g1 + p[KPIXY] * p[KVY] * g2 + p[KPIXZ] * p[KVZ] * g3;
  o.ty = p[KPIXY] * p[KVX] * g1 + p[KPIYY] * p[KVY] * g2 + p[KPIYZ] * p[KVZ] * g3;
  o.tz = p[KPIXZ] * p[KVX] * g1 + p[KPIYZ] * p[KVY] * g2 + p[KPIZZ] * p[KVZ] * g3;
  o.tt = o.tx * p[KVX] * g1 + o.ty * p[KVY] * g2 + o.tz * p[KVZ] * g3;
  o.zz = p[KPIZZ];
}

// get_derived_pi_zz (viscous.f90:259-279)
__device__ __forceinline__ void derived_pi_zz(const Metric& M, const double* p, Pit& o) {
  double g1 = M.g1, g2 = M.g2, g3 = M.g3;
  double vx = p[KVX], vy = p[KVY], vz = p[KVZ];
  double pixy = p[KPIXY], pixx = p[KPIXX], piyy = p[KPIYY], piyz = p[KPIYZ], pixz = p[KPIXZ];
  if (vz == 0.) {
    // v^eta = 0 (every cell of a boost-invariant run): the terms below with
    // a factor vz are exact zeros and 1 - vz^2 g3 is exactly 1, so these are
    // the same sums in the same order, with the same bits
    o.tt = vx * g1 * pixy * vy * g2 + vx * vx * g1 * g1 * pixx + vy * g1 * g1 * pixy * vx + vy * vy * g1 * piyy * g2;
    o.tx = pixx * vx * g1 + pixy * vy * g2;
    o.ty = pixy * vx * g1 + piyy * vy * g2;
    o.tz = pixz * vx * g1 + piyz * vy * g2;
    o.zz = 1. / g3 *
           (vx * g1 * pixy * vy * g2 - pixx * g1 - piyy * g2 + vx * vx * g1 * g1 * pixx + vy * g1 * g1 * pixy * vx +
            vy * vy * g1 * piyy * g2);
    return;
  }
  o.tt = 1. / (1. - vz * vz * g3) *
         (vx * g1 * pixy * vy * g2 + vx * vx * g1 * g1 * pixx + vy * g1 * piyz * vz * g3 +
          2. * vx * g1 * pixz * vz * g3 + vy * g1 * g1 * pixy * vx + vy * vy * g1 * piyy * g2 +
          vz * g3 * piyz * vy * g2 - pixx * g1 * vz * vz * g3 - piyy * g2 * vz * vz * g3);
  o.tx = pixx * vx * g1 + pixy * vy * g2 + pixz * vz * g3;
  o.ty = pixy * vx * g1 + piyy * vy * g2 + piyz * vz * g3;
  o.tz = 1. / (1. - vz * vz * g3) *
         (pixz * vx * g1 + pixz * vx * g1 * vz * vz * g3 + piyz * vy * g2 +
          vz * vx * g1 * pixy * vy * g2 - vz * pixx * g1 - vz * piyy * g2 +
          vz * vx * vx * g1 * g1 * pixx + vy * g1 * piyz * vz * vz * g3 +
          vz * vy * g1 * g1 * pixy * vx + vz * vy * vy * g1 * piyy * g2);
  o.zz = 1. / (g3 * (1. - vz * vz * g3)) *
         (vx * g1 * pixy * vy * g2 - pixx * g1 - piyy * g2 + vx * vx * g1 * g1 * pixx +
          vy * g1 * piyz * vz * g3 + 2. * vx * g1 * pixz * vz * g3 + vy * g1 * g1 * pixy * vx +
          vy * vy * g1 * piyy * g2 + vz * g3 * piyz * vy * g2);
}

__device__ __forceinline__ void derived_pi_any(const DevPhys& P, const Metric& M, double* p, Pit& o) {
  if (P.obtained_zz) {
    derived_pi_zz(M, p, o);
    p[KPIZZ] = o.zz;
  } else {
    derived_pi(M, p, o);
  }
}

// get_viscous_parameters (viscous.f90:172-199)
__device__ __forceinline__ int viscous_parameters(const DevPhys& P, double dens, double press,
                                                  double* eta, double* zeta, double* tau_pi,
                                                  double* tau_pi_big) {
  double en = 0, temp = 0, s = 0, cs2 = 0;
  (void)get_derived_data(P, dens, press, &en, &temp, &s);
  int err = eos_sound(P, dens, en, press, &cs2);
  const double hbar = 0.197326;
  *eta = hbar * P.eta_over_s * s;
  if (P.init_type == 2) *eta = P.eta_over_s;
  if (P.bulkvis)
    *zeta = 2. * *eta * (1. / 3. - cs2);
  else
    *zeta = 0.;
  if (temp == 0 || s == 0)
    *tau_pi = 0.;
  else
    *tau_pi = P.tau_pi_coeff * *eta / (temp * s);
  if (P.init_type == 5) *tau_pi = 5. * *eta / (temp * s);
  *tau_pi_big = *tau_pi;
  return err;
}

// ---------------------------------------------------------------------------
// electromagnetic helpers (system.f90:1846-1897)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void e_ideal(const Metric& M, double vx, double vy, double vz, double bx,
                                        double by, double bz, double E[3]) {
  double gp = M.gp;
  E[0] = -gp * (vy * bz - vz * by);
  E[1] = -gp * (vz * bx - vx * bz);
  E[2] = -gp * (vx * by - vy * bx);
}
__device__ __forceinline__ void exb(const Metric& M, const double E[3], double bx, double by, double bz,
                                    double o[3]) {
  double e0 = E[0], e1 = E[1], e2 = over_g3(M, E[2]), gp = M.gp;
  o[0] = gp * (e1 * bz - e2 * by);
  o[1] = gp * (e2 * bx - e0 * bz);
  o[2] = gp * (e0 * by - e1 * bx);
}
// covariant E_i of a cell: the resistive primitive E^i lowered
// (system.f90:203-205; the reference's system_flux omits g_33 for E_3,
// system.f90:1365, which only Minkowski coordinates forgive), or -v x B
template <int KIND>
__device__ __forceinline__ void e_field(const Metric& M, const double* v, double E[3]) {
  if (Traits<KIND>::RES) {
    E[0] = v[KEX];
    E[1] = v[KEY];
    E[2] = v[KEZ] * M.g3;
  } else {
    e_ideal(M, v[KVX], v[KVY], v[KVZ], v[KBX], v[KBY], v[KBZ], E);
  }
}

// ---------------------------------------------------------------------------
// system_prim2cons (system.f90:164-263)
// ---------------------------------------------------------------------------
template <int KIND>
__device__ __forceinline__ int prim2cons(const DevPhys& P, const Metric& M, double* v, double* u) {
  typedef Traits<KIND> T;
  double g1 = M.g1, g2 = M.g2, g3 = M.g3, gp = M.gp;
  double rh = v[KRH], vx = v[KVX], vy = v[KVY], vz = v[KVZ], pr = v[KPR];
  double en = 0;
  int err = eos_energy(P, rh, &en, pr);
  if (err) return err;
  double v2 = g1 * vx * vx + g2 * vy * vy + g3 * vz * vz;
  double glf = 1. / sqrt(1. - v2);
  double w = en + pr;
  double ww = w * (glf * glf);
  u[KRH] = rh * glf;
  if (T::VISC) {
    w = w + v[KPIBU];
    ww = w * (glf * glf);
    Pit pi;
    derived_pi_any(P, M, v, pi);
    u[KVX] = (ww * vx + pi.tx);
    u[KVY] = (ww * vy + pi.ty);
    u[KVZ] = (ww * vz + pi.tz) * g3;
    u[KPR] = ww - pr - v[KPIBU] - pi.tt * M.g0;
    u[KPIBU] = v[KPIBU] * u[KRH];
    u[KPIZZ] = v[KPIZZ] * u[KRH];
    u[KPIXZ] = v[KPIXZ] * u[KRH];
    u[KPIXY] = v[KPIXY] * u[KRH];
    u[KPIYZ] = v[KPIYZ] * u[KRH];
    u[KPIXX] = v[KPIXX] * u[KRH];
    u[KPIYY] = v[KPIYY] * u[KRH];
  } else if (T::MHD) {
    double E[3], EXB[3];
    e_field<KIND>(M, v, E);
    double E2 = E[0] * E[0] + E[1] * E[1] + (E[2] * E[2]) / g3;
    exb(M, E, v[KBX], v[KBY], v[KBZ], EXB);
    double bx = v[KBX], by = v[KBY], bz = v[KBZ];
    double B2 = bx * bx + by * by + (bz * bz) * g3;
    double EEM = 0.5 * (E2 + B2);
    u[KVX] = ww * vx + EXB[0];
    u[KVY] = ww * vy + EXB[1];
    u[KVZ] = ww * vz * g3 + EXB[2];
    u[KPR] = ww - pr + EEM;
    u[KBX] = v[KBX];
    u[KBY] = v[KBY];
    u[KBZ] = v[KBZ];
    if (T::RES) {
      u[KEX] = v[KEX];
      u[KEY] = v[KEY];
      u[KEZ] = v[KEZ];
    }
    if (T::GLM) u[T::KG] = v[T::KG] / gp;
  } else {
    u[KVX] = ww * vx;
    u[KVY] = ww * vy;
    u[KVZ] = ww * vz * g3;
    u[KPR] = ww - pr;
  }
#pragma unroll
  for (int k = 0; k < T::NV; k++) u[k] = u[k] * gp;
  return 0;
}

// ---------------------------------------------------------------------------
// system_flux (system.f90:1316-1583); DIR 1..3
// ---------------------------------------------------------------------------
template <int KIND, int DIR>
__device__ __forceinline__ int system_flux(const DevPhys& P, const Metric& M, double* v, double* u,
                                           double* f, double& vfp, double& vfm) {
  typedef Traits<KIND> T;
  const int NV = T::NV;
  double g1 = M.g1, g2 = M.g2, g3 = M.g3, gp = M.gp, gm = M.gm;
  double rh = v[KRH], vx = v[KVX], vy = v[KVY], vz = v[KVZ], pr = v[KPR];
  double en = 0;
#ifdef ECHO_EXACT
  int err = eos_energy(P, rh, &en, pr);
#else
  EosAt at;
  int err = eos_energy_h(P, rh, &en, pr, at);
#endif
  if (err) return err;
  double v2 = g1 * vx * vx + g2 * vy * vy + g3 * vz * vz;
  if (v2 > 1) return 333;
#ifdef ECHO_EXACT
  double glf = 1. / sqrt(1. - v2);
#else
  double glf = rsqrt(1. - v2);
#endif
  double w, E[3] = {0, 0, 0}, EXB[3] = {0, 0, 0}, E2 = 0, B2 = 0, EEM = 0;
  Pit pi = {0, 0, 0, 0, 0};
  if (!T::VISC) {
    w = en + pr;
    if (T::MHD) {
      e_field<KIND>(M, v, E);
      E2 = E[0] * E[0] + E[1] * E[1] + over_g3(M, E[2] * E[2]);
      exb(M, E, v[KBX], v[KBY], v[KBZ], EXB);
      B2 = v[KBX] * v[KBX] + v[KBY] * v[KBY] + (v[KBZ] * v[KBZ]) * g3;
      EEM = 0.5 * (E2 + B2);
    }
  } else {
    w = en + pr + v[KPIBU];
  }
  double ww = w * (glf * glf);
  u[KRH] = rh * glf;
  if (T::VISC) {
    derived_pi_any(P, M, v, pi);
#pragma unroll
    for (int k = KPIBU; k < NV; k++) u[k] = v[k] * u[KRH];
    u[KVX] = ww * vx + pi.tx;
    u[KVY] = ww * vy + pi.ty;
    u[KVZ] = (ww * vz + pi.tz) * g3;
    u[KPR] = ww - pr - v[KPIBU] - pi.tt * M.g0;
  } else if (T::MHD) {
    u[KVX] = ww * vx + EXB[0];
    u[KVY] = ww * vy + EXB[1];
    u[KVZ] = ww * vz * g3 + EXB[2];
    u[KPR] = ww - pr + EEM;
    u[KBX] = v[KBX];
    u[KBY] = v[KBY];
    u[KBZ] = v[KBZ];
    if (T::RES) {
      u[KEX] = v[KEX];
      u[KEY] = v[KEY];
      u[KEZ] = v[KEZ];
    }
    if (T::GLM) u[T::KG] = over_gp(M, v[T::KG]);
  } else {
    u[KVX] = ww * vx;
    u[KVY] = ww * vy;
    u[KVZ] = ww * vz * g3;
    u[KPR] = ww - pr;
  }
  double wwdir, vdir, gcov_dir;
  if (DIR == 1) {
    wwdir = ww * vx;
    vdir = vx;
    gcov_dir = g1;
    f[KRH] = rh * glf * vx;
    if (T::VISC) {
      f[KVX] = wwdir * vx * g1 + pr + v[KPIBU] + v[KPIXX] * g1;
      f[KVY] = wwdir * vy * g2 + v[KPIXY] * g2;
      f[KVZ] = wwdir * vz * g3 + v[KPIXZ] * g3;
      f[KPR] = wwdir + pi.tx;
#pragma unroll
      for (int k = 5; k < NV; k++) f[k] = u[k] * vx;
    } else if (T::MHD) {
      f[KVX] = wwdir * vx - E[0] * E[0] - v[KBX] * v[KBX] + pr + EEM;
      f[KVY] = wwdir * vy - E[0] * E[1] - v[KBX] * v[KBY];
      f[KVZ] = wwdir * vz * g3 - E[0] * E[2] - v[KBX] * v[KBZ] * g3;
      f[KPR] = wwdir + EXB[0];
      f[KBX] = 0.;
      f[KBY] = -E[2] * gm;
      f[KBZ] = +E[1] * gm;
      if (T::RES) {  // E fluxes (system.f90:1450-1452)
        f[KEX] = 0.;
        f[KEY] = +v[KBZ] * g3 * gm;
        f[KEZ] = -v[KBY] * g2 * gm;
      }
      if (T::GLM) {
        f[KBX] = v[T::KG];
        f[T::KG] = over_gp(M, v[KBX]);
      }
    } else {
      f[KVX] = wwdir * vx * g1 + pr;
      f[KVY] = wwdir * vy * g2;
      f[KVZ] = wwdir * vz * g3;
      f[KPR] = wwdir;
    }
  } else if (DIR == 2) {
    wwdir = ww * vy;
    vdir = vy;
    gcov_dir = g2;
    f[KRH] = rh * glf * vy;
    if (T::VISC) {
      f[KVX] = wwdir * vx * g1 + v[KPIXY] * g1;
      f[KVY] = wwdir * vy * g2 + pr + v[KPIBU] + v[KPIYY] * g2;
      f[KVZ] = wwdir * vz * g3 + v[KPIYZ] * g3;
      f[KPR] = wwdir + pi.ty;
#pragma unroll
      for (int k = 5; k < NV; k++) f[k] = u[k] * vy;
    } else if (T::MHD) {
      f[KVX] = wwdir * vx - E[1] * E[0] - v[KBY] * v[KBX];
      f[KVY] = wwdir * vy - E[1] * E[1] - v[KBY] * v[KBY] + pr + EEM;
      f[KVZ] = wwdir * vz * g3 - E[1] * E[2] - v[KBY] * v[KBZ] * g3;
      f[KPR] = wwdir + EXB[1];
      f[KBX] = E[2] * gm;
      f[KBY] = 0.;
      f[KBZ] = -E[0] * gm;
      if (T::RES) {  // system.f90:1491-1493
        f[KEX] = -v[KBZ] * g3 * gm;
        f[KEY] = 0.;
        f[KEZ] = +v[KBX] * g1 * gm;
      }
      if (T::GLM) {
        f[KBY] = v[T::KG];
        f[T::KG] = over_gp(M, v[KBY]);
      }
    } else {
      f[KVX] = wwdir * vx * g1;
      f[KVY] = wwdir * vy * g2 + pr;
      f[KVZ] = wwdir * vz * g3;
      f[KPR] = wwdir;
    }
  } else {
    wwdir = ww * vz;
    vdir = vz;
    gcov_dir = g3;
    f[KRH] = rh * glf * vz;
    if (T::VISC) {
      f[KVX] = wwdir * vx * g1 + v[KPIXZ] * g1;
      f[KVY] = wwdir * vy * g2 + v[KPIYZ] * g2;
      f[KVZ] = wwdir * vz * g3 + pr + v[KPIBU] + v[KPIZZ] * g3;
      f[KPR] = wwdir + pi.tz;
#pragma unroll
      for (int k = 5; k < NV; k++) f[k] = u[k] * vz;
    } else if (T::MHD) {
      f[KVX] = wwdir * vx - over_g3(M, E[2]) * E[0] - v[KBZ] * v[KBX];
      f[KVY] = wwdir * vy - over_g3(M, E[2]) * E[1] - v[KBZ] * v[KBY];
      f[KVZ] = wwdir * vz * g3 - over_g3(M, E[2] * E[2]) - (v[KBZ] * v[KBZ]) * g3 + pr + EEM;
      f[KPR] = wwdir + over_g3(M, EXB[2]);
      f[KBX] = -E[1] * gm;
      f[KBY] = E[0] * gm;
      f[KBZ] = 0.;
      if (T::RES) {  // system.f90:1532-1534
        f[KEX] = +v[KBY] * g2 * gm;
        f[KEY] = -v[KBX] * g1 * gm;
        f[KEZ] = 0.;
      }
      if (T::GLM) {
        f[KBZ] = over_g3(M, v[T::KG]);
        f[T::KG] = over_gp(M, v[KBZ]);
      }
    } else {
      f[KVX] = wwdir * vx * g1;
      f[KVY] = wwdir * vy * g2;
      f[KVZ] = wwdir * vz * g3 + pr;
      f[KPR] = wwdir;
    }
  }
#pragma unroll
  for (int k = 0; k < NV; k++) u[k] = u[k] * gp;
#pragma unroll
  for (int k = 0; k < NV; k++) f[k] = f[k] * gp;
  double ca2;
  if (T::MHD) {
    double bb2 = B2 - E2;
    ca2 = bb2 / (bb2 + (en + pr));
  } else {
    ca2 = 0.;
  }
  double cs2 = 0;
#ifdef ECHO_EXACT
  err = eos_sound(P, rh, en, pr, &cs2);
#else
  if (at.h)
    cs2 = eos_sound_at(P, at, en);
  else
    err = eos_sound(P, rh, en, pr, &cs2);
#endif
  if (err) return err;
  double a2 = cs2 + ca2 - cs2 * ca2;
  double den = 1. / (1. - v2 * a2);
  double vf1 = den * (1. - a2) * vdir;
  // g_11 = g_22 = 1 in both metrics, so only the eta direction divides
  double hdir = DIR == 3 ? over_g3(M, 1. - v2 * a2) : (1. - v2 * a2);
  (void)gcov_dir;
  double vf2 = den * sqrt(a2 * (1. - v2) * (hdir - (1. - a2) * (vdir * vdir)));
  vfp = vf1 + vf2;
  vfm = vf1 - vf2;
  if (T::RES) {
    // resistive: the light cone bounds the Riemann fan of the E, B waves (the
    // reference keeps the ideal fast speed here, system.f90:1557-1580)
    vfp = 1. / sqrt(DIR == 3 ? g3 : 1.);
    vfm = -vfp;
  }
  return 0;
}

}  // namespace echo
