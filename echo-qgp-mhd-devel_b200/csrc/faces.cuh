// faces.cuh -- the flux sweeps of a stage, cell-centred tiles.
//
// A block owns a tile of C = 2^LC consecutive cells (ghost cells included) and
// the faces between them.  Phase 1: every thread reconstructs both face states
// of its CPT neighbouring cells, one variable after another (recon_cells), into
// shared memory.  Phase 2: the flux of a face takes the upper state of the cell
// below and the lower state of the cell above.
//
// What bounds it: L1 and FP64 together (x / y / eta sweep of 97 x 97 x 81 ideal RMHD:
// L1 70 / 61 / 55 % of its peak, FP64 pipe 44 / 47 / 44 %, issue 42 / 45 / 43 %), in
// phases that the 21 to 23 warps of an SM overlap in part.
// One thread per face with all its variables in registers (the arrangement
// before) evaluated the smoothness indicators of a cell twice, unrolled every
// variable into one body and spilled about 600 bytes a thread at the 72
// registers its occupancy needed.  Here a cell's indicators serve both its
// faces, two neighbouring cells of a thread share loads (6 for 10) and
// differences, the reconstruction is a loop over the variables and the flux
// reads its operands from shared memory where it uses them.
//
// Tiles.  Along x the cells 0..nx+1 of all pencils (padded to an even number)
// are numbered through and tile t covers C of them from t (C - 2) on.  Along y
// and eta a tile is W = 2^lw neighbouring pencils (consecutive in memory) by
// C / W cells, one row more than it has faces; W = 16 keeps every load at whole
// 128-byte lines.
//
// Measured, x / y / eta us a launch, one thread per face before and this: ideal
// RMHD 97 x 97 x 81 111 / 108 / 114 and 76 / 70 / 73; resistive 193 x 193 x 129
// 742 / 733 / 844 and 451 / 500 / 530.  With the loads, the reconstruction or
// the flux left out in turn the RMHD x sweep took 62, 69 and 72 us: no one of
// them bounds it.
#pragma once

// Variables of phase 1 unrolled together.  Measured, 1 / 2 / 3, us for the passes
// of whole steps: ideal RMHD 97 x 97 x 81 4796 / 4771 / 4761, resistive
// 193 x 193 x 129 19453 / 19466 / 19517, hydro MPE5 75 x 67 x 49 1002 / 1012 / 1026,
// viscous 61 x 57 x 41 877 / 887 / 900.
#ifndef ECHO_SWEEP_UNROLL
#define ECHO_SWEEP_UNROLL 2
#endif

namespace echo {

struct SweepArgs {
  FaceArgs A[3];          // x, y, eta
  unsigned first[4];      // block range of each direction
  int lw;                 // log2 of the pencils of a y or eta tile
  // with last set, the block that finishes last runs the stage's scalar logic:
  // one launch fewer on the chain of every stage
  int last;
  ScalarArgs S;
};

// 64 KB of shared memory a block at most: 2 x (NV + 4) x 256 doubles
template <int KIND>
__host__ __device__ constexpr int tile_rows_of_states() {
  return Traits<KIND>::NV + (Traits<KIND>::VISC ? 4 : 0);
}
template <int KIND>
__host__ __device__ constexpr size_t tile_smem(int lc) {
  return sizeof(double) * 2 * (size_t)tile_rows_of_states<KIND>() * ((size_t)1 << lc);
}

// tiles of a sweep of grid g (cells, faces and the padded cells of x pencils, at
// most twice the cells, are counted below 2^32: the arrays of the smallest run,
// 1-D hydro, have 265 bytes a cell)
__host__ __device__ inline unsigned tiles_of(const Grid& g, int dir, int lc, int lw) {
  const unsigned C = 1u << lc;
  if (dir == 0) {
    const unsigned e = (((unsigned)g.nx + 3u) & ~1u) * (unsigned)g.ny * (unsigned)g.nz;
    return (e + C - 3) / (C - 2);
  }
  const unsigned n = (unsigned)(dir == 1 ? g.ny : g.nz), cols = (unsigned)g.nx * (unsigned)(dir == 1 ? g.nz : g.ny);
  const unsigned rows = (C >> lw) - 1;
  return ((cols + (1u << lw) - 1) >> lw) * ((n + 1 + rows - 1) / rows);
}

// index of the face above cell c (0..n) of a pencil: its transverse position
// (ta, tb), first cell base and stride
template <int DIR>
__host__ __device__ __forceinline__ unsigned face_index(const Grid& g, unsigned c, unsigned ta, unsigned tb,
                                                        unsigned base, unsigned stride) {
  const unsigned nx = (unsigned)g.nx, ny = (unsigned)g.ny;
  return DIR == 0 ? (tb * ny + ta) * (nx + 1) + c : DIR == 1 ? (tb * (ny + 1) + c) * nx + ta : c * stride + base;
}

// Whether the sweeps of grid g need 64-bit byte offsets.  2^29 cells and more
// fit the device in ideal hydro alone (265, 305 and 345 bytes a cell in 1-D, 2-D
// and 3-D; the next set, 1-D RMHD, has 385).  Not always: the stencil's offsets
// as 64-bit pairs cost the sweeps 0.5 to 1 % (75 x 67 x 49 hydro MPE5 1010 us
// for 5 steps with 32 bits, 1021 with 64).
inline bool wide_grid(const Grid& g) {
  const size_t lim = (size_t)1 << 29;
  return g.ncell > lim || (g.nx > 1 && faces_of<0>(g) > lim) || (g.ny > 1 && faces_of<1>(g) > lim) ||
         (g.nz > 1 && faces_of<2>(g) > lim);
}

#ifndef ECHO_EXACT
// What the flux of one side of a face needs beside the primitives w[k * ld].
struct FaceSide {
  double ww, D, em;  // w gamma^2, rho gamma, electromagnetic energy
  double i1, vB;     // ideal MHD: 1 / gamma^2 and v.B, with ww = w gamma^2 + B^2 and em = b^2 / 2
};

// Energy density, enthalpy and the signal speeds of one side (system_flux).
template <int KIND, int DIR>
__device__ __forceinline__ int side_speeds(const DevPhys& P, const Metric& M, const double* w, int ld, FaceSide& s,
                                           double& vfp, double& vfm) {
  typedef Traits<KIND> T;
  const double rh = w[KRH * ld], pr = w[KPR * ld];
  const double vx = w[KVX * ld], vy = w[KVY * ld], vz = w[KVZ * ld];
  double en = 0.;
  EosAt at;
  int err = eos_energy_h(P, rh, &en, pr, at);
  if (err) return err;
  const double v2 = vx * vx + vy * vy + M.g3 * (vz * vz);
  if (v2 > 1) return 333;
  const double i1 = 1. - v2, glf = rsqrt_n(i1), h = en + pr;
  s.ww = (T::VISC ? h + w[KPIBU * ld] : h) * (glf * glf);
  s.D = rh * glf;
  s.em = 0.;
  double b = 0.;  // B^2 - E^2
  if (T::MHD) {
    const double bx = w[KBX * ld], by = w[KBY * ld], bz = w[KBZ * ld];
    const double B2 = bx * bx + by * by + M.g3 * (bz * bz);
    if (T::RES) {
      const double ex = w[KEX * ld], ey = w[KEY * ld], ez = w[KEZ * ld];
      s.em = 0.5 * (ex * ex + ey * ey + M.g3 * (ez * ez) + B2);
    } else {
      s.vB = vx * bx + vy * by + M.g3 * (vz * bz);
      s.i1 = i1;
      b = fma(s.vB, s.vB, B2 * i1);
      s.em = 0.5 * b;
      s.ww += B2;
    }
  }
  if (T::RES) {
    // the light cone bounds the Riemann fan of the E, B waves
    vfp = DIR == 3 ? sqrt_h3(M.ig3) : 1.;
    vfm = -vfp;
    return 0;
  }
  double cs2 = 0.;
  if (at.h)
    cs2 = eos_sound_at(P, at, en);
  else
    err = eos_sound(P, rh, en, pr, &cs2);
  if (err) return err;
  const double vd = DIR == 1 ? vx : DIR == 2 ? vy : vz;
  // in the reference's order, each operation rounded as there or within an ulp:
  // where fluid and field are at rest the flux is (a+ f_l + a- f_r) / (a+ + a-)
  // of equal terms, and the last bits of the speeds are its noise
  double a2 = cs2;
  if (T::MHD) {
    const double ca2 = div_n(b, b + h);
    a2 = cs2 + ca2 - cs2 * ca2;
  }
  const double x = 1. - v2 * a2, den = div_n(1., x), hd = DIR == 3 ? over_g3(M, x) : x;
  const double vf1 = den * (1. - a2) * vd;
  const double vf2 = den * sqrt_n(a2 * i1 * (hd - (1. - a2) * (vd * vd)));
  vfp = vf1 + vf2;
  vfm = vf1 - vf2;
  return 0;
}

// F += c (f + lam u) of one side for every variable but the momentum normal to
// the face, f and u those of system_flux without their sqrt(-g) (in c): c = g
// a+ / (a+ + a-), lam = a- on the left, c = g a- / (a+ + a-), lam = -a+ on the
// right.  fn, un: the normal momentum's flux and value (hll_flux).
template <int KIND, int DIR>
__device__ __forceinline__ void side_flux(const DevPhys& P, const Metric& M, const double* w, int ld,
                                          const FaceSide& s, double c, double lam, double* F, double& fn, double& un) {
  typedef Traits<KIND> T;
  constexpr int d = DIR - 1, ia = DIR % 3, ib = (DIR + 1) % 3;
  const double v[3] = {w[KVX * ld], w[KVY * ld], w[KVZ * ld]};
  const double pr = w[KPR * ld], g3 = M.g3, gd = DIR == 3 ? g3 : 1.;
  const double a = v[d] + lam, ca = c * a;
  F[KRH] = fma(ca, s.D, F[KRH]);
  if (T::MHD && !T::RES) {
    // Ideal MHD with b the field in the fluid frame: S_i = W v_i - (v.B) B_i,
    // W = w gamma^2 + B^2; T^d_i = S_i v^d - B^d (B_i / gamma^2 + (v.B) v_i) +
    // delta p_t, p_t = p + b^2 / 2; U = W - p_t; and v^d B^a - v^a B^d.  The
    // same tensor as with E = -v x B, in half the operations.
    const double B[3] = {w[KBX * ld], w[KBY * ld], w[KBZ * ld]};
    const double cB = -c * B[d], pt = pr + s.em;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double S = fma(s.ww, v[i], -s.vB * B[i]), m = fma(s.i1, B[i], s.vB * v[i]);
      if (i == d) {
        un = gd * S;
        fn = fma(gd, S * v[d] - B[d] * m, pt);
        F[KPR] = fma(c, fma(lam, s.ww - pt, S), F[KPR]);
      } else {
        const double x = fma(ca, S, cB * m);
        F[KVX + i] = i == 2 ? fma(g3, x, F[KVX + i]) : F[KVX + i] + x;
      }
    }
    F[KBX + ia] = fma(ca, B[ia], fma(cB, v[ia], F[KBX + ia]));
    F[KBX + ib] = fma(ca, B[ib], fma(cB, v[ib], F[KBX + ib]));
    if (T::GLM) {
      const double psi = w[T::KG * ld];
      F[KBX + d] = fma(c, fma(lam, B[d], DIR == 3 ? over_g3(M, psi) : psi), F[KBX + d]);
      F[T::KG] = fma(c, over_gp(M, fma(lam, psi, B[d])), F[T::KG]);
    } else {
      F[KBX + d] = fma(c, lam * B[d], F[KBX + d]);
    }
    return;
  }
  const double cwa = ca * s.ww, wd = s.ww * v[d];
  // beyond the w gamma^2 v_i terms: value and flux of the momenta, energy
  double u[3] = {0., 0., 0.}, f[3] = {0., 0., 0.}, pt = pr, fe = -lam * pr;
  if (T::VISC) {
    double p[T::NV];
#pragma unroll
    for (int k = KVX; k < T::NV; k++) p[k] = w[k * ld];
    Pit pi;
    derived_pi_any(P, M, p, pi);  // with obtained_zz also p[KPIZZ]
    u[0] = pi.tx;
    u[1] = pi.ty;
    u[2] = pi.tz * g3;
    f[0] = DIR == 1 ? p[KPIXX] : DIR == 2 ? p[KPIXY] : p[KPIXZ];
    f[1] = DIR == 1 ? p[KPIXY] : DIR == 2 ? p[KPIYY] : p[KPIYZ];
    f[2] = g3 * (DIR == 1 ? p[KPIXZ] : DIR == 2 ? p[KPIYZ] : p[KPIZZ]);
    pt += p[KPIBU];
    fe = fma(lam, pi.tt - pt, DIR == 1 ? pi.tx : DIR == 2 ? pi.ty : pi.tz);
    const double cda = ca * s.D;
#pragma unroll
    for (int k = KPIBU; k < T::NV; k++) F[k] = fma(cda, p[k], F[k]);
  }
  if (T::RES) {
    const double B[3] = {w[KBX * ld], w[KBY * ld], w[KBZ * ld]};
    const double E[3] = {w[KEX * ld], w[KEY * ld], w[KEZ * ld] * g3};
    exb(M, E, B[0], B[1], B[2], u);
    const double Ed = w[(KEX + d) * ld], Bd = B[d];
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = -Ed * E[i] - Bd * B[i] * (i == 2 ? g3 : 1.);
    pt += s.em;
    fe = fma(lam, s.em - pr, DIR == 3 ? over_g3(M, u[d]) : u[d]);
    // Faraday's and Ampere's laws (system.f90:1450-1452, 1491-1493,
    // 1532-1534): f_a = -E_b / sqrt(-g), f_b = E_a / sqrt(-g) for B and
    // B_b / sqrt(-g), -B_a / sqrt(-g) for E, (d, a, b) cyclic
    F[KBX + ia] = fma(c, fma(lam, B[ia], -E[ib] * M.gm), F[KBX + ia]);
    F[KBX + ib] = fma(c, fma(lam, B[ib], E[ia] * M.gm), F[KBX + ib]);
    const double psi = w[T::KG * ld];
    F[KBX + d] = fma(c, fma(lam, Bd, DIR == 3 ? over_g3(M, psi) : psi), F[KBX + d]);
    F[T::KG] = fma(c, over_gp(M, fma(lam, psi, Bd)), F[T::KG]);
    const double ga = ia == 2 ? g3 : 1., gb = ib == 2 ? g3 : 1.;
    F[KEX + ia] = fma(c, fma(lam, w[(KEX + ia) * ld], B[ib] * gb * M.gm), F[KEX + ia]);
    F[KEX + ib] = fma(c, fma(lam, w[(KEX + ib) * ld], -B[ia] * ga * M.gm), F[KEX + ib]);
    F[KEX + d] = fma(c, lam * Ed, F[KEX + d]);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    if (i == d) continue;
    const double vi = i == 2 ? v[i] * g3 : v[i];
    F[KVX + i] = T::VISC || T::RES ? fma(cwa, vi, fma(c, fma(lam, u[i], f[i]), F[KVX + i])) : fma(cwa, vi, F[KVX + i]);
  }
  un = fma(gd, wd, u[d]);
  fn = fma(gd * wd, v[d], f[d]) + pt;
  F[KPR] += fma(c, fe, cwa);
}

// The HLL flux of a face (times sqrt(-g)) from both sides' states and signal
// speeds ap, am (work.f90:195-229).  The momentum normal to the face holds the
// pressure, large and nearly equal on the two sides, and its rounding is the
// noise of the velocities: it is combined once, from both sides' whole terms.
template <int KIND, int DIR>
__device__ __forceinline__ void hll_flux(const DevPhys& P, const Metric& M, const double* wl, const double* wr, int ld,
                                         const FaceSide& L, const FaceSide& R, double ap, double am, double* F) {
  double a1 = 1.;
  if (!(ap == 0. && am == 0.)) {
    a1 = div_n(1., ap + am);
  }
#pragma unroll
  for (int k = 0; k < Traits<KIND>::NV; k++) F[k] = 0.;
  const double ga = M.gp * a1;
  double fl, ul, fr, ur;
  side_flux<KIND, DIR>(P, M, wl, ld, L, ga * ap, am, F, fl, ul);
  side_flux<KIND, DIR>(P, M, wr, ld, R, ga * am, -ap, F, fr, ur);
  F[KVX + DIR - 1] = fma(ga * ap, fma(am, ul, fl), ga * am * fma(-ap, ur, fr));
}
#endif

// the m values from cell c - 2 on of one variable with boundary codes of its
// own (differing between variables, or extrapolation): out of line
struct Stencil6 {
  double f[6];
};
static __device__ __noinline__ Stencil6 stencil_general(const double* __restrict__ a, size_t base, long long stride,
                                                        int n, int c, int m, int code_l, int code_r) {
  Stencil6 r;
#pragma unroll 1
  for (int q = 0; q < m; q++) r.f[q] = ghost_val(a, base, stride, n, c - 2 + q, code_l, code_r);
  return r;
}

// the fix-ups of a face's states (evolve.f90:334-369) with w0 = the cell left
// of the face (pencil index i, which may be a ghost): p <= 0 takes its p,
// v^2 >= 1 its velocity, scaled to maxspeed if that is superluminal too
template <int KIND>
static __device__ __noinline__ void fix_states(const FaceArgs& A, const Metric& M, size_t base, long long stride,
                                               int n, int i, double* wl, double* wr, int ld) {
  double w0[5];
  for (int k = KVX; k <= KPR; k++)
    w0[k] = ghost_val(A.v + (size_t)k * A.g.ncell, base, stride, n, i, A.bc.c[k][0], A.bc.c[k][1]);
  for (int side = 0; side < 2; side++) {
    double* w = side == 0 ? wr : wl;
    if (w[KPR * ld] <= 0) w[KPR * ld] = w0[KPR];
    double v2 = 0;
    v2 = v2 + w[KVX * ld] * w[KVX * ld] * M.g1;
    v2 = v2 + w[KVY * ld] * w[KVY * ld] * M.g2;
    v2 = v2 + w[KVZ * ld] * w[KVZ * ld] * M.g3;
    if (v2 >= 1.) {
      for (int k = KVX; k <= KVZ; k++) w[k * ld] = w0[k];
      v2 = 0;
      v2 = v2 + w[KVX * ld] * w[KVX * ld] * M.g1;
      v2 = v2 + w[KVY * ld] * w[KVY * ld] * M.g2;
      v2 = v2 + w[KVZ * ld] * w[KVZ * ld] * M.g3;
      if (v2 >= 1) {
        for (int k = KVX; k <= KVZ; k++) {
          w0[k] = w0[k] * A.P.maxspeed / (sqrt(v2));
          w[k * ld] = w0[k];
        }
      }
    }
  }
}

// The flux of the face above cell c of a pencil (base, stride) from its states
// wl, wr (variable k at k * C; changed in place by the fix-ups and the GLM
// upwinding): writes A.F (and A.WD), the signal speed into amax.
template <int KIND, int DIR, int C, bool WIDE>
__device__ __forceinline__ void face_one(const FaceArgs& A, const Metric& M, unsigned base, unsigned stride, int n,
                                         int c, int ta, int tb, double* wl, double* wr, double& amax) {
  typedef Traits<KIND> T;
  constexpr int NV = T::NV;
  const Grid& g = A.g;
  amax = 0.;
  const size_t nfaces = faces_of<DIR>(g);
  const unsigned fid = face_index<DIR>(g, (unsigned)c, (unsigned)ta, (unsigned)tb, base, stride);
  if (T::VISC) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      A.WD[(size_t)q * nfaces + fid] = wl[(NV + q) * C];
      A.WD[(size_t)(4 + q) * nfaces + fid] = wr[(NV + q) * C];
    }
  }
  const double ch = A.sc->glm_ch_old;
  double F[NV];
  int err;
#ifdef ECHO_EXACT
  double ql[NV], qr[NV], w0[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) {
    ql[k] = T::VISC && k == KPIZZ && A.P.obtained_zz ? 0. : wl[k * C];
    qr[k] = T::VISC && k == KPIZZ && A.P.obtained_zz ? 0. : wr[k * C];
    w0[k] = 0.;
  }
#pragma unroll 1
  for (int k = KVX; k <= KPR; k++)
    w0[k] = ghost_val(A.v + (size_t)k * g.ncell, base, stride, n, c, A.bc.c[k][0], A.bc.c[k][1]);
  err = face_tail<KIND, DIR>(A.P, M, ch, ql, qr, w0, F, amax);
#else
  {
    const double lv = wl[KVX * C] * wl[KVX * C] + wl[KVY * C] * wl[KVY * C] + M.g3 * (wl[KVZ * C] * wl[KVZ * C]);
    const double rv = wr[KVX * C] * wr[KVX * C] + wr[KVY * C] * wr[KVY * C] + M.g3 * (wr[KVZ * C] * wr[KVZ * C]);
    if (wl[KPR * C] <= 0 || wr[KPR * C] <= 0 || lv >= 1. || rv >= 1.)
      fix_states<KIND>(A, M, base, stride, n, c, wl, wr, C);
  }
  if (T::GLM) {
    // work_glm[xyz]: psi and the normal B of the face (the second's
    // correction has the factor psi_r - psi_l, which is zero by then)
    const int kb = KBX + DIR;
    const double bl = wl[kb * C], br = wr[kb * C];
    const double psi = 0.5 * ((wl[T::KG * C] + wr[T::KG * C]) - (br - bl) * ch), bn = 0.5 * (bl + br);
    wl[T::KG * C] = psi;
    wr[T::KG * C] = psi;
    wl[kb * C] = bn;
    wr[kb * C] = bn;
  }
  FaceSide L, R;
  double vflp, vflm, vfrp, vfrm;
  err = side_speeds<KIND, DIR + 1>(A.P, M, wl, C, L, vflp, vflm);
  if (!err) err = side_speeds<KIND, DIR + 1>(A.P, M, wr, C, R, vfrp, vfrm);
  if (!err) {
    double ap = 0., am = 0.;
    if (vflp > ap) ap = vflp;
    if (vfrp > ap) ap = vfrp;
    if (-vflm > am) am = -vflm;
    if (-vfrm > am) am = -vfrm;
    amax = ap > am ? ap : am;
    hll_flux<KIND, DIR + 1>(A.P, M, wl, wr, C, L, R, ap, am, F);
  }
#endif
  if (err) {
    amax = 0.;
    const size_t cell = base + (size_t)((c >= 1 ? c : 1) - 1) * stride;
    atomicMin(&A.sc->err_key, ((unsigned long long)cell << 20) | (unsigned long long)err);
#pragma unroll
    for (int k = 0; k < NV; k++) F[k] = 0.0;
  }
#pragma unroll
  for (int k = 0; k < NV; k++) *(double*)((char*)(A.F + (size_t)k * nfaces) + off8<WIDE>(fid)) = F[k];
  if (!err) {
    // GLM speed of the reference: the last face of the last pencil (work.f90:217,310,401)
    const int na = DIR == 0 ? g.ny : g.nx, nb = DIR == 2 ? g.ny : g.nz;
    if (c == n && ta == na - 1 && tb == nb - 1) A.sc->aflux[DIR] = amax;
  }
}

// The checks of a face alone (face_one without its flux): the EoS range and
// superluminal errors of both states, left first, and the signal speed, which
// is the light cone's.  Resistive runs, first IMEX-SSP stage: the flux of U1
// has weight 0 in every later combination, its errors and the speed of the
// cleaning wave are all that stage leaves behind.
template <int KIND, int DIR, int C>
__device__ __forceinline__ void face_check(const FaceArgs& A, const Metric& M, unsigned base, unsigned stride, int n,
                                           int c, int ta, int tb, double* wl, double* wr, double& amax) {
  const Grid& g = A.g;
  auto speed2 = [&](const double* w) {
    return w[KVX * C] * w[KVX * C] + w[KVY * C] * w[KVY * C] + M.g3 * (w[KVZ * C] * w[KVZ * C]);
  };
  if (wl[KPR * C] <= 0 || wr[KPR * C] <= 0 || speed2(wl) >= 1. || speed2(wr) >= 1.)
    fix_states<KIND>(A, M, base, stride, n, c, wl, wr, C);
  auto bad = [&](const double* w) {
    if (A.P.eqstate == ECHO_EOS_TABLE) {  // eos_energy
      if (w[KPR * C] < __ldg(A.P.tp)) return 125;
      if (w[KPR * C] > __ldg(A.P.tp + A.P.nt - 1)) return 126;
    }
    return speed2(w) > 1. ? 333 : 0;
  };
  int err = bad(wl);
  if (!err) err = bad(wr);
  amax = 0.;
  if (err) {
    const size_t cell = base + (size_t)((c >= 1 ? c : 1) - 1) * stride;
    atomicMin(&A.sc->err_key, ((unsigned long long)cell << 20) | (unsigned long long)err);
    return;
  }
  amax = 1. / sqrt(DIR == 2 ? M.g3 : 1.);
  const int na = DIR == 0 ? g.ny : g.nx, nb = DIR == 2 ? g.ny : g.nz;
  if (c == n && ta == na - 1 && tb == nb - 1) A.sc->aflux[DIR] = amax;
}

// One tile of the sweep along DIR; returns the largest signal speed of this
// thread's faces.  Called by every thread of the block: NG groups of C / CPT
// threads, the groups sharing the variables of phase 1.  sm:
// tile_smem<KIND>(LC) bytes.  CHECK: velocity and pressure, face_check.  WIDE:
// wide_grid.
template <int KIND, int DIR, int REC, int LC, int CPT, int NG, bool CHECK, bool WIDE>
__device__ __forceinline__ double face_tile(const FaceArgs& A, unsigned tile, int lw, double* sm) {
  typedef Traits<KIND> T;
  constexpr int NV = T::NV, C = 1 << LC, NT = C / CPT, NS = CPT + 4, UNROLL = ECHO_SWEEP_UNROLL;
  const Grid& g = A.g;
  const int t = NG > 1 ? (int)threadIdx.x & (NT - 1) : (int)threadIdx.x;
  const int grp = NG > 1 ? (int)threadIdx.x / NT : 0;
  const int n = DIR == 0 ? g.nx : DIR == 1 ? g.ny : g.nz;
  const int W = DIR == 0 ? 1 : 1 << lw;
  // cell j of thread t is slot j NT + t (the shared accesses of a warp are
  // consecutive)
  double* plus = sm;                                       // upper face state of a cell
  double* minus = sm + tile_rows_of_states<KIND>() * C;    // its lower face state
  const double mt = A.sc->t, mt3 = A.sc->t3;

  // this thread's first cell: pencil index c (0 and n + 1 are the ghosts next
  // to the grid), first cell and stride of its pencil, transverse position
  int c, ta, tb;
  unsigned base;
  bool ok;
  const unsigned stride = DIR == 0 ? 1u : DIR == 1 ? (unsigned)g.nx : (unsigned)g.nx * (unsigned)g.ny;
  if (DIR == 0) {
    const unsigned e = tile * (unsigned)(C - 2) + (unsigned)(t * CPT);
    const unsigned pen = fast_div(e, g.dnx2);
    c = (int)(e - pen * (((unsigned)g.nx + 3u) & ~1u));
    tb = (int)fast_div(pen, g.dny);
    ta = (int)(pen - (unsigned)tb * (unsigned)g.ny);
    ok = tb < g.nz;
    base = pen * (unsigned)g.nx;
  } else {
    const unsigned cols = (unsigned)g.nx * (unsigned)(DIR == 1 ? g.nz : g.ny);
    const unsigned nct = (cols + (unsigned)W - 1) >> lw;
    const unsigned rt = tile / nct, ct = tile - rt * nct;
    const unsigned p = (ct << lw) + (unsigned)(t & (W - 1));
    tb = (int)fast_div(p, g.dnx);
    ta = (int)(p - (unsigned)tb * (unsigned)g.nx);
    c = (int)(rt * (unsigned)((C >> lw) - 1)) + (t >> lw) * CPT;
    ok = p < cols;
    base = DIR == 1 ? (unsigned)tb * (unsigned)(g.ny * g.nx) + (unsigned)ta : p;
  }
  ok = ok && c <= n + 1;

  if (ok) {
    // byte offsets of the stencil from cell c - 2 on, with the ghost fill of
    // evolve_bc[xyz]; the last cell's own upper neighbour is not read
    const int last = c + CPT - 1 <= n + 1 ? NS - 1 : NS - 2;
    Off<WIDE> off[NS];
    int neg = 0;
    if (c >= 3 && c + CPT + 1 <= n) {
#pragma unroll
      for (int q = 0; q < NS; q++) off[q] = off8<WIDE>(base + (unsigned)(c - 3 + q) * stride);
    } else {
#pragma unroll
      for (int q = 0; q < NS; q++) {
        int qq;
        double sg;
        map_ghost(c - 2 + (q < last ? q : last), n, A.bc.c[0][0], A.bc.c[0][1], qq, sg);
        off[q] = off8<WIDE>(base + (unsigned)(qq - 1) * stride);
        if (sg < 0.) neg |= 1 << q;
      }
    }
    auto load = [&](int k, double* f) {
      const char* vk = (const char*)(A.v + (size_t)k * g.ncell);
      if (A.bc_uniform) {
#pragma unroll
        for (int q = 0; q < NS; q++) f[q] = __ldg((const double*)(vk + off[q]));
        if (A.bc_signed) {
#pragma unroll
          for (int q = 0; q < NS; q++) f[q] = (neg >> q) & 1 ? -f[q] : f[q];
        }
      } else {
        const Stencil6 s = stencil_general((const double*)vk, base, stride, n, c, last + 1, A.bc.c[k][0], A.bc.c[k][1]);
#pragma unroll
        for (int q = 0; q < NS; q++) f[q] = q <= last ? s.f[q] : s.f[q - 1];
      }
    };
    auto put = [&](int k, const double* f) {
      double pl[CPT], mi[CPT];
      recon_cells<REC, CPT>(A.P.recal, f, pl, mi);
#pragma unroll
      for (int j = 0; j < CPT; j++) {
        plus[k * C + j * NT + t] = pl[j];
        minus[k * C + j * NT + t] = mi[j];
      }
    };
    // pi^{eta eta} of a face state follows from the others (derived_pi_zz)
    const int nr = CHECK ? KPR + 1 : T::VISC && A.P.obtained_zz ? NV - 1 : NV;
    int k = CHECK ? KVX + grp : grp;
#pragma unroll UNROLL
    for (; k < nr; k += NG) {
      double f[NS];
      load(k, f);
      put(k, f);
    }
    // u^mu for the viscous derivatives (work_rec(n,1,4,1)), by the group
    // whose turn it is
    if (T::VISC && k == nr) {
      const double g3 = A.coordinates == ECHO_BJORKEN ? mt * mt : 1.;
      double vx[NS], vy[NS], vz[NS], gg[NS];
      load(KVX, vx);
      load(KVY, vy);
      load(KVZ, vz);
#pragma unroll
      for (int q = 0; q < NS; q++) {
#ifdef ECHO_EXACT
        gg[q] = 1. / sqrt(1. - vx[q] * vx[q] - vy[q] * vy[q] - g3 * (vz[q] * vz[q]));
#else
        gg[q] = rsqrt_h3(1. - vx[q] * vx[q] - vy[q] * vy[q] - g3 * (vz[q] * vz[q]));
#endif
        vx[q] = gg[q] * vx[q];
        vy[q] = gg[q] * vy[q];
        vz[q] = gg[q] * vz[q];
      }
      put(NV + 0, gg);
      put(NV + 1, vx);
      put(NV + 2, vy);
      put(NV + 3, vz);
    }
  }
  __syncthreads();

  // the faces above this thread's cells
  double amax = 0.;
  const Metric M = make_metric(A.coordinates, mt, mt3);
#pragma unroll 1
  for (int j = 0; j < CPT; j++) {
    // the cell above is this thread's next one or the first of the thread W
    // further on; the last pair of an x tile is the first of the next
    const bool own = CPT > 1 && j < CPT - 1;
    const int cf = c + j;
    if (!(grp == 0 && ok && cf <= n && (own ? DIR > 0 || t < NT - 1 : t + W < NT - (DIR == 0 && CPT == 1 ? 1 : 0)))) continue;
    double* wl = plus + j * NT + t;
    double* wr = minus + (own ? (j + 1) * NT + t : t + W);
    double am;
    if (CHECK)
      face_check<KIND, DIR, C>(A, M, base, stride, n, cf, ta, tb, wl, wr, am);
    else
      face_one<KIND, DIR, C, WIDE>(A, M, base, stride, n, cf, ta, tb, wl, wr, am);
    amax = am > amax ? am : amax;
  }
  return amax;
}

// Cells of a thread in the large tiles (256 cells): two share loads and
// differences, but a thread then holds 4 NV doubles of shared memory, which
// for the twelve variables of the viscous and resistive sets leaves 12 to 16
// warps an SM; and the limiters of MPE5, the scheme of ideal hydro runs that
// do not choose, gain nothing from it.  Measured, x / y / eta us a launch:
// ideal RMHD 97 x 97 x 81 78 / 79 / 84 with one cell, 76 / 70 / 73 with two;
// resistive 193 x 193 x 129 453 / 496 / 518 with one, 508 / 518 / 547 with
// two; ideal hydro MPE5 75 x 67 x 49 33 / 27 / 32 with one, 35 / 28 / 36 with two.
template <int KIND>
__host__ __device__ constexpr int sweep_cpt(int lc) {
  return lc == 8 && (KIND == KIND_MHD || KIND == KIND_MHDGLM) ? 2 : 1;
}
// threads of a block; the small tiles' (32 cells) are eight groups
template <int KIND>
__host__ __device__ constexpr int sweep_threads(int lc) {
  return 256 / sweep_cpt<KIND>(lc);
}
// Blocks of an SM, the register bound.  Measured with one fewer / this / one more,
// us for the passes of whole steps: ideal RMHD 97 x 97 x 81 4824 / 4771 / 4929,
// hydro MPE5 75 x 67 x 49 1067 / 1012 / 1020, viscous 61 x 57 x 41 980 / 887 / 934,
// resistive 193 x 193 x 129 21279 / 19466 / 22144; small tiles (hydro 101 x 101)
// 2359 / 2030 / 2055.
#ifndef ECHO_SWEEP_MINB
#define ECHO_SWEEP_MINB 6
#endif
#ifndef ECHO_SWEEP_MINB_HD
#define ECHO_SWEEP_MINB_HD 4
#endif
#ifndef ECHO_SWEEP_MINB_VISC
#define ECHO_SWEEP_MINB_VISC 3
#endif
#ifndef ECHO_SWEEP_MINB_RES
#define ECHO_SWEEP_MINB_RES 4
#endif
#ifndef ECHO_SWEEP_MINB_SMALL
#define ECHO_SWEEP_MINB_SMALL 3
#endif
template <int KIND>
constexpr int sweep_minb(int lc) {
  return lc != 8             ? ECHO_SWEEP_MINB_SMALL
         : KIND == KIND_HD   ? ECHO_SWEEP_MINB_HD
         : KIND == KIND_VISC ? ECHO_SWEEP_MINB_VISC
         : KIND == KIND_RES  ? ECHO_SWEEP_MINB_RES
                             : ECHO_SWEEP_MINB;
}

// The sweeps of a stage in one launch: the blocks of the directions one after
// another, so that the partial last wave of one overlaps the next.  They are
// independent: each writes its own face fluxes and signal-speed slots.
template <int KIND, int REC, int LC, bool CHECK = false, bool WIDE = false>
__global__ void __launch_bounds__(sweep_threads<KIND>(LC), sweep_minb<KIND>(LC)) sweep_kernel(const __grid_constant__ SweepArgs S) {
  extern __shared__ double sm[];
  constexpr int CPT = sweep_cpt<KIND>(LC), NG = (sweep_threads<KIND>(LC) * CPT) >> LC;
  __shared__ double red[sweep_threads<KIND>(LC) / 32];
  const unsigned b = blockIdx.x;
  double amax;
  int dir;
  if (b < S.first[1]) {
    dir = 0;
    amax = face_tile<KIND, 0, REC, LC, CPT, NG, CHECK, WIDE>(S.A[0], b, S.lw, sm);
  } else if (b < S.first[2]) {
    dir = 1;
    amax = face_tile<KIND, 1, REC, LC, CPT, NG, CHECK, WIDE>(S.A[1], b - S.first[1], S.lw, sm);
  } else {
    dir = 2;
    amax = face_tile<KIND, 2, REC, LC, CPT, NG, CHECK, WIDE>(S.A[2], b - S.first[2], S.lw, sm);
  }
  DevScalars* sc = S.A[0].sc;
  block_max_atomic(amax, &sc->amax_bits[dir], red);
  // thread 0 has the block's maximum and, past the barrier above, every
  // thread's aflux behind it
  if (S.last && threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&sc->done, 1u) == gridDim.x - 1) {
      __threadfence();
      stage_scalars_last(S.S);
    }
  }
}

}  // namespace echo
