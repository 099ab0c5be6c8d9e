// faces.cuh -- the flux sweeps of a stage, cell-centred tiles.
//
// A block owns a tile of C = 2^lc consecutive cells (ghost cells included) and
// the faces between them.  Phase 1: every thread reconstructs both face states
// of its cell, one variable after another (recon_cell), into shared memory.
// Phase 2: one thread per face takes the upper state of the cell below and the
// lower state of the cell above and computes the HLL flux.
//
// What bounds it: FP64 issue.  One thread per face with all its variables in
// registers (the arrangement before) evaluated the smoothness indicators of a
// cell twice, unrolled every variable into one body and spilled about 600 bytes
// a thread at the 72 registers its occupancy needed.  Here a cell's indicators
// serve both its faces, the reconstruction is a rolled loop over the variables
// (one variable's operands live, the next one's loads in flight) and the flux
// reads its operands from shared memory where it uses them.
//
// Tiles.  Along x the cells 0..nx+1 of all pencils are numbered through and
// tile t covers C of them from t (C - 1) on, so that C - 1 faces (2 % of them
// between two pencils) come from C cells.  Along y and eta a tile is W = 2^lw
// neighbouring pencils (consecutive in memory) by C / W cells, one row more
// than it has faces; W = 16 keeps every load at whole 128-byte lines.
//
// Measured (97 x 97 x 81 ideal RMHD, B200): x / y / eta sweep 111 / 108 / 114 us
// with one thread per face, 80 / 82 / 86 us here, 39 to 44 million warp
// instructions instead of 60 to 64 (half of them FP64 in both); resistive
// 193 x 193 x 129: 742 / 733 / 844 us before, 476 / 527 / 549 us here.
#pragma once

#ifndef ECHO_SWEEP_UNROLL
#define ECHO_SWEEP_UNROLL 3
#endif

namespace echo {

struct SweepArgs {
  FaceArgs A[3];          // x, y, eta
  unsigned first[4];      // block range of each direction
  int lw;                 // log2 of the pencils of a tile (y, eta)
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

// tiles of a sweep of grid g (face and cell counts are below 2^32: the arrays
// of a larger grid would not fit the device)
__host__ __device__ inline unsigned tiles_of(const Grid& g, int dir, int lc, int lw) {
  const unsigned C = 1u << lc;
  if (dir == 0) {
    const unsigned e = (unsigned)(g.nx + 2) * (unsigned)g.ny * (unsigned)g.nz - 1;  // pairs of neighbours
    return (e + C - 2) / (C - 1);
  }
  const unsigned n = (unsigned)(dir == 1 ? g.ny : g.nz), cols = (unsigned)g.nx * (unsigned)(dir == 1 ? g.nz : g.ny);
  const unsigned rows = (C >> lw) - 1;
  return ((cols + (1u << lw) - 1) >> lw) * ((n + 1 + rows - 1) / rows);
}

#ifndef ECHO_EXACT
// What the flux of one side of a face needs beside the primitives w[k * ld].
struct FaceSide {
  double ww, D, em;  // w gamma^2, rho gamma, electromagnetic energy
};

// Energy density, enthalpy and the signal speeds of one side (system_flux).
// With w = e + p, b = B^2 - E^2 and a^2 = (c_s^2 w + b) / (w + b), the fast
// speeds' 1 / (1 - v^2 a^2) and 1 / (w + b) are one reciprocal.
template <int KIND, int DIR>
__device__ __forceinline__ int side_speeds(const DevPhys& P, const Metric& M, const double* w, int ld, FaceSide& s,
                                           double& vfp, double& vfm) {
  typedef Traits<KIND> T;
  const double rh = w[KRH * ld], pr = w[KPR * ld];
  const double vx = w[KVX * ld], vy = w[KVY * ld], vz = w[KVZ * ld];
  double en = 0.;
  int hb = 0;
  int err = eos_energy_h(P, rh, &en, pr, &hb);
  if (err) return err;
  const double v2 = vx * vx + vy * vy + M.g3 * (vz * vz);
  if (v2 > 1) return 333;
  const double i1 = 1. - v2, glf = rsqrt_h3(i1), h = en + pr;
  s.ww = (T::VISC ? h + w[KPIBU * ld] : h) * (glf * glf);
  s.D = rh * glf;
  s.em = 0.;
  double b = 0.;
  if (T::MHD) {
    const double bx = w[KBX * ld], by = w[KBY * ld], bz = w[KBZ * ld];
    double E[3];
    if (T::RES) {
      E[0] = w[KEX * ld];
      E[1] = w[KEY * ld];
      E[2] = w[KEZ * ld] * M.g3;
    } else {
      e_ideal(M, vx, vy, vz, bx, by, bz, E);
    }
    const double E2 = E[0] * E[0] + E[1] * E[1] + M.ig3 * (E[2] * E[2]);
    const double B2 = bx * bx + by * by + M.g3 * (bz * bz);
    s.em = 0.5 * (E2 + B2);
    b = B2 - E2;
  }
  if (T::RES) {
    // the light cone bounds the Riemann fan of the E, B waves
    vfp = DIR == 3 ? sqrt_h3(M.ig3) : 1.;
    vfm = -vfp;
    return 0;
  }
  double cs2 = 0.;
  if (hb)
    cs2 = eos_sound_at(P, hb, en);
  else
    err = eos_sound(P, rh, en, pr, &cs2);
  if (err) return err;
  const double vd = DIR == 1 ? vx : DIR == 2 ? vy : vz;
  // a^2 = N / q, 1 - a^2 = O / q, 1 - v^2 a^2 = Dn / q
  const double q = T::MHD ? h + b : 1., N = T::MHD ? fma(cs2, h, b) : cs2, O = T::MHD ? h - cs2 * h : 1. - cs2;
  const double Dn = fma(-v2, N, q), r = rcp_h3(Dn);
  const double hd = DIR == 3 ? M.ig3 * Dn : Dn;
  const double vf1 = O * vd * r;
  const double vf2 = r * sqrt_h3(N * i1 * fma(-O, vd * vd, hd));
  vfp = vf1 + vf2;
  vfm = vf1 - vf2;
  return 0;
}

// F += c (f + lam u) of one side, f and u those of system_flux without their
// sqrt(-g) (in c): c = a+ / (a+ + a-), lam = a- on the left,
// c = a- / (a+ + a-), lam = -a+ on the right.
template <int KIND, int DIR>
__device__ __forceinline__ void side_flux(const DevPhys& P, const Metric& M, const double* w, int ld,
                                          const FaceSide& s, double c, double lam, double* F) {
  typedef Traits<KIND> T;
  const double v[3] = {w[KVX * ld], w[KVY * ld], w[KVZ * ld]};
  const double pr = w[KPR * ld], g3 = M.g3;
  const double a = v[DIR - 1] + lam;
  F[KRH] = fma(c * s.D, a, F[KRH]);
  const double cwa = c * s.ww * a;
  F[KVX] = fma(cwa, v[0], F[KVX]);
  F[KVY] = fma(cwa, v[1], F[KVY]);
  F[KVZ] = fma(cwa, v[2] * g3, F[KVZ]);
  double pt = pr, fe = -lam * pr;  // f + lam u beyond the w gamma^2 terms: normal stress, energy
  if (T::VISC) {
    double p[T::NV];
#pragma unroll
    for (int k = KVX; k < T::NV; k++) p[k] = w[k * ld];
    Pit pi;
    derived_pi_any(P, M, p, pi);  // with obtained_zz also p[KPIZZ]
    const double pd[3] = {DIR == 1 ? p[KPIXX] : DIR == 2 ? p[KPIXY] : p[KPIXZ],
                          DIR == 1 ? p[KPIXY] : DIR == 2 ? p[KPIYY] : p[KPIYZ],
                          DIR == 1 ? p[KPIXZ] : DIR == 2 ? p[KPIYZ] : p[KPIZZ]};
    F[KVX] = fma(c, fma(lam, pi.tx, pd[0]), F[KVX]);
    F[KVY] = fma(c, fma(lam, pi.ty, pd[1]), F[KVY]);
    F[KVZ] = fma(c * g3, fma(lam, pi.tz, pd[2]), F[KVZ]);
    pt += p[KPIBU];
    fe = fma(lam, pi.tt - pt, DIR == 1 ? pi.tx : DIR == 2 ? pi.ty : pi.tz);
    const double cda = c * s.D * a;
#pragma unroll
    for (int k = KPIBU; k < T::NV; k++) F[k] = fma(cda, p[k], F[k]);
  }
  if (T::MHD) {
    const double B[3] = {w[KBX * ld], w[KBY * ld], w[KBZ * ld]};
    double E[3], X[3];
    if (T::RES) {
      E[0] = w[KEX * ld];
      E[1] = w[KEY * ld];
      E[2] = w[KEZ * ld] * g3;
    } else {
      e_ideal(M, v[0], v[1], v[2], B[0], B[1], B[2], E);
    }
    exb(M, E, B[0], B[1], B[2], X);
    pt += s.em;
    fe = lam * (s.em - pr);
    const double Ed = DIR == 3 ? over_g3(M, E[2]) : E[DIR - 1], Bd = B[DIR - 1];
    F[KVX] = fma(c, lam * X[0] - Ed * E[0] - Bd * B[0], F[KVX]);
    F[KVY] = fma(c, lam * X[1] - Ed * E[1] - Bd * B[1], F[KVY]);
    F[KVZ] = fma(c, lam * X[2] - Ed * E[2] - Bd * (B[2] * g3), F[KVZ]);
    fe += DIR == 3 ? over_g3(M, X[2]) : X[DIR - 1];
    // Faraday's law: f_a = -E_b / sqrt(-g), f_b = E_a / sqrt(-g), (d, a, b) cyclic
    const int ia = DIR % 3, ib = (DIR + 1) % 3;
    F[KBX + ia] = fma(c, fma(lam, B[ia], -E[ib] * M.gm), F[KBX + ia]);
    F[KBX + ib] = fma(c, fma(lam, B[ib], E[ia] * M.gm), F[KBX + ib]);
    if (T::GLM) {
      const double psi = w[T::KG * ld];
      F[KBX + DIR - 1] = fma(c, fma(lam, Bd, DIR == 3 ? over_g3(M, psi) : psi), F[KBX + DIR - 1]);
      F[T::KG] = fma(c, over_gp(M, fma(lam, psi, Bd)), F[T::KG]);
    } else {
      F[KBX + DIR - 1] = fma(c, lam * Bd, F[KBX + DIR - 1]);
    }
    if (T::RES) {  // Ampere's law (system.f90:1450-1452, 1491-1493, 1532-1534)
      const double ga = ia == 2 ? g3 : 1., gb = ib == 2 ? g3 : 1.;
      F[KEX + ia] = fma(c, fma(lam, w[(KEX + ia) * ld], B[ib] * gb * M.gm), F[KEX + ia]);
      F[KEX + ib] = fma(c, fma(lam, w[(KEX + ib) * ld], -B[ia] * ga * M.gm), F[KEX + ib]);
      F[KEX + DIR - 1] = fma(c, lam * w[(KEX + DIR - 1) * ld], F[KEX + DIR - 1]);
    }
  }
  F[KVX + DIR - 1] = fma(c, pt, F[KVX + DIR - 1]);
  F[KPR] += fma(c, fe, cwa);
}
#endif

// the five-point stencil of one variable with boundary codes of its own
// (differing between variables, or extrapolation): out of line
struct Stencil5 {
  double f[5];
};
static __device__ __noinline__ Stencil5 stencil_general(const double* __restrict__ a, size_t base, long long stride,
                                                        int n, int c, int code_l, int code_r) {
  Stencil5 r;
#pragma unroll 1
  for (int q = 0; q < 5; q++) r.f[q] = ghost_val(a, base, stride, n, c - 2 + q, code_l, code_r);
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

// One tile of the sweep along DIR; returns the largest signal speed of this
// thread's faces.  Called by every thread of the block; blockDim.x is a
// multiple of the tile's cells: the further groups of threads share the
// variables of phase 1.  sm: tile_smem<KIND>(lc) bytes.
template <int KIND, int DIR, int REC, int LC, int NG>
__device__ __forceinline__ double face_tile(const FaceArgs& A, unsigned tile, int lw, double* sm) {
  typedef Traits<KIND> T;
  constexpr int NV = T::NV, C = 1 << LC, UNROLL = ECHO_SWEEP_UNROLL;
  const Grid& g = A.g;
  const int slot = threadIdx.x & (C - 1), grp = threadIdx.x >> LC;
  const int n = DIR == 0 ? g.nx : DIR == 1 ? g.ny : g.nz;
  const int W = DIR == 0 ? 1 : 1 << lw;
  double* plus = sm;                                       // upper face state of a cell
  double* minus = sm + tile_rows_of_states<KIND>() * C;    // its lower face state
  const Metric M = make_metric(A.coordinates, A.sc->t, A.sc->t3);

  // this thread's cell: pencil index c (0 and n + 1 are the ghosts next to the
  // grid), first cell and stride of its pencil, transverse position.  Cell and
  // face indices are below 2^29 (their doubles' byte offsets below 2^32): the
  // arrays of a larger grid do not fit the device.
  int c, ta, tb;
  unsigned base;
  bool ok;
  const unsigned stride = DIR == 0 ? 1u : DIR == 1 ? (unsigned)g.nx : (unsigned)g.nx * (unsigned)g.ny;
  if (DIR == 0) {
    const unsigned e = tile * (unsigned)(C - 1) + (unsigned)slot;
    const unsigned pen = fast_div(e, g.dnx2);
    c = (int)(e - pen * (unsigned)(g.nx + 2));
    tb = (int)fast_div(pen, g.dny);
    ta = (int)(pen - (unsigned)tb * (unsigned)g.ny);
    ok = tb < g.nz;
    base = pen * (unsigned)g.nx;
  } else {
    const unsigned cols = (unsigned)g.nx * (unsigned)(DIR == 1 ? g.nz : g.ny);
    const unsigned nct = (cols + (unsigned)W - 1) >> lw;
    const unsigned rt = tile / nct, ct = tile - rt * nct;
    const unsigned p = (ct << lw) + (unsigned)(slot & (W - 1));
    tb = (int)fast_div(p, g.dnx);
    ta = (int)(p - (unsigned)tb * (unsigned)g.nx);
    c = (int)(rt * (unsigned)((C >> lw) - 1)) + (slot >> lw);
    ok = p < cols && c <= n + 1;
    base = DIR == 1 ? (unsigned)tb * (unsigned)(g.ny * g.nx) + (unsigned)ta : p;
  }

  if (ok) {
    // byte offsets of the stencil c-2..c+2, with the ghost fill of evolve_bc[xyz]
    unsigned off[5];
    int neg = 0;
    if (c >= 3 && c <= n - 2) {
#pragma unroll
      for (int q = 0; q < 5; q++) off[q] = 8u * (base + (unsigned)(c - 3 + q) * stride);
    } else {
#pragma unroll
      for (int q = 0; q < 5; q++) {
        int qq;
        double sg;
        map_ghost(c - 2 + q, n, A.bc.c[0][0], A.bc.c[0][1], qq, sg);
        off[q] = 8u * (base + (unsigned)(qq - 1) * stride);
        if (sg < 0.) neg |= 1 << q;
      }
    }
    auto load = [&](int k, double* f) {
      const char* vk = (const char*)(A.v + (size_t)k * g.ncell);
      if (A.bc_uniform) {
#pragma unroll
        for (int q = 0; q < 5; q++) f[q] = __ldg((const double*)(vk + off[q]));
        if (A.bc_signed) {
#pragma unroll
          for (int q = 0; q < 5; q++) f[q] = (neg >> q) & 1 ? -f[q] : f[q];
        }
      } else {
        const Stencil5 s = stencil_general((const double*)vk, base, stride, n, c, A.bc.c[k][0], A.bc.c[k][1]);
#pragma unroll
        for (int q = 0; q < 5; q++) f[q] = s.f[q];
      }
    };
    // pi^{eta eta} of a face state follows from the others (derived_pi_zz)
    const int nr = T::VISC && A.P.obtained_zz ? NV - 1 : NV;
    int k = NG > 1 ? grp : 0;
#pragma unroll UNROLL
    for (; k < nr; k += NG) {
      double f[5], pl, mi;
      load(k, f);
      recon_cell<REC>(A.P.recal, f, pl, mi);
      plus[k * C + slot] = pl;
      minus[k * C + slot] = mi;
    }
    // u^mu for the viscous derivatives (work_rec(n,1,4,1)), by the group
    // whose turn it is
    if (T::VISC && k == nr) {
      double vx[5], vy[5], vz[5], gg[5];
      load(KVX, vx);
      load(KVY, vy);
      load(KVZ, vz);
#pragma unroll
      for (int q = 0; q < 5; q++) {
#ifdef ECHO_EXACT
        gg[q] = 1. / sqrt(1. - vx[q] * vx[q] - vy[q] * vy[q] - M.g3 * (vz[q] * vz[q]));
#else
        gg[q] = rsqrt_h3(1. - vx[q] * vx[q] - vy[q] * vy[q] - M.g3 * (vz[q] * vz[q]));
#endif
        vx[q] = gg[q] * vx[q];
        vy[q] = gg[q] * vy[q];
        vz[q] = gg[q] * vz[q];
      }
      recon_cell<REC>(A.P.recal, gg, plus[(NV + 0) * C + slot], minus[(NV + 0) * C + slot]);
      recon_cell<REC>(A.P.recal, vx, plus[(NV + 1) * C + slot], minus[(NV + 1) * C + slot]);
      recon_cell<REC>(A.P.recal, vy, plus[(NV + 2) * C + slot], minus[(NV + 2) * C + slot]);
      recon_cell<REC>(A.P.recal, vz, plus[(NV + 3) * C + slot], minus[(NV + 3) * C + slot]);
    }
  }
  __syncthreads();

  // the face between cell c and the next one of its pencil
  double amax = 0.;
  if (grp == 0 && ok && slot < C - W && c <= n) {
    const size_t nfaces = faces_of<DIR>(g);
    const unsigned fid = DIR == 0   ? ((unsigned)tb * (unsigned)g.ny + (unsigned)ta) * (unsigned)(g.nx + 1) + (unsigned)c
                         : DIR == 1 ? ((unsigned)tb * (unsigned)(g.ny + 1) + (unsigned)c) * (unsigned)g.nx + (unsigned)ta
                                    : (unsigned)c * stride + base;
    double* wl = plus + slot;
    double* wr = minus + slot + W;
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
      const double a1 = M.gp * (ap == 0. && am == 0. ? 1. : rcp_h3(ap + am));
#pragma unroll
      for (int k = 0; k < NV; k++) F[k] = 0.;
      side_flux<KIND, DIR + 1>(A.P, M, wl, C, L, a1 * ap, am, F);
      side_flux<KIND, DIR + 1>(A.P, M, wr, C, R, a1 * am, -ap, F);
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
    for (int k = 0; k < NV; k++) *(double*)((char*)(A.F + (size_t)k * nfaces) + 8u * fid) = F[k];
    if (!err) {
      // GLM speed of the reference: the last face of the last pencil (work.f90:217,310,401)
      const int na = DIR == 0 ? g.ny : g.nx, nb = DIR == 2 ? g.ny : g.nz;
      if (c == n && ta == na - 1 && tb == nb - 1) A.sc->aflux[DIR] = amax;
    }
  }
  return amax;
}

// threads of a sweep block
#define ECHO_SWEEP_NT 256
#ifndef ECHO_SWEEP_MINB
#define ECHO_SWEEP_MINB 4
#endif
#ifndef ECHO_SWEEP_MINB_VISC
#define ECHO_SWEEP_MINB_VISC 3
#endif
#ifndef ECHO_SWEEP_MINB_RES
#define ECHO_SWEEP_MINB_RES 4
#endif
#define ECHO_SWEEP_BOUNDS(KIND)                                                          \
  __launch_bounds__(ECHO_SWEEP_NT, (KIND) == KIND_VISC  ? ECHO_SWEEP_MINB_VISC       \
                                   : (KIND) == KIND_RES ? ECHO_SWEEP_MINB_RES : ECHO_SWEEP_MINB)

// The sweeps of a stage in one launch: the blocks of the directions one after
// another, so that the partial last wave of one overlaps the next.  They are
// independent: each writes its own face fluxes and signal-speed slots.
template <int KIND, int REC, int LC>
__global__ void ECHO_SWEEP_BOUNDS(KIND) sweep_kernel(const __grid_constant__ SweepArgs S) {
  extern __shared__ double sm[];
  __shared__ double red[ECHO_SWEEP_NT / 32];
  const unsigned b = blockIdx.x;
  double amax;
  int dir;
  if (b < S.first[1]) {
    dir = 0;
    amax = face_tile<KIND, 0, REC, LC, (ECHO_SWEEP_NT >> LC)>(S.A[0], b, S.lw, sm);
  } else if (b < S.first[2]) {
    dir = 1;
    amax = face_tile<KIND, 1, REC, LC, (ECHO_SWEEP_NT >> LC)>(S.A[1], b - S.first[1], S.lw, sm);
  } else {
    dir = 2;
    amax = face_tile<KIND, 2, REC, LC, (ECHO_SWEEP_NT >> LC)>(S.A[2], b - S.first[2], S.lw, sm);
  }
  block_max_atomic(amax, &S.A[0].sc->amax_bits[dir], red);
}

}  // namespace echo
