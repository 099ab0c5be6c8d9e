// unit_tests.cu -- kernel-level entry points for parity tests
// (echo_gpu_test_recon, echo_gpu_test_c2p in include/echo_gpu.h).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/echo_gpu.h"
#include "ctx.cuh"

#define CK(x)                                                                               \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess) {                                                                \
      fprintf(stderr, "echo_gpu: CUDA error %s at %s:%d\n", cudaGetErrorString(e_), __FILE__, \
              __LINE__);                                                                    \
      return ECHO_ERR_CUDA;                                                                 \
    }                                                                                       \
  } while (0)

bool echo_make_buckets(const double* arr, int n, std::vector<int>& bk, long long& k0);
int echo_kind_of(const EchoParams* p);
int echo_nv_of(int kind);

// ---------------------------------------------------------------------------
// kernel-level entry points for parity tests
// ---------------------------------------------------------------------------
namespace echo {
__global__ void recon_test_kernel(int recal, int m, int n, const double* f, double* gl, double* gr) {
  size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (size_t)m * (n + 1)) return;
  int row = (int)(id / (n + 1)), i = (int)(id % (n + 1));
  const double* fr = f + (size_t)row * (n + 8) + 4;  // fr[j] = f(j)
  double s[6];
  for (int q = 0; q < 6; q++) s[q] = fr[i - 2 + q];
  double l, r;
  recon_any(recal, s, l, r);
  gl[id] = l;
  gr[id] = r;
}

template <int KIND>
__global__ void c2p_test_kernel(DevPhys P, Metric M, int algo, double tol, int ncells, const double* u, double* v,
                                int* err, int* iters) {
  typedef Traits<KIND> T;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  double uu[T::NV], vv[T::NV];
  for (int k = 0; k < T::NV; k++) {
    uu[k] = u[(size_t)c * T::NV + k];
    vv[k] = v[(size_t)c * T::NV + k];
  }
  int it = 0;
  int e = cons2prim<KIND, true>(P, M, algo, tol, uu, vv, &it);
  for (int k = 0; k < T::NV; k++) v[(size_t)c * T::NV + k] = vv[k];
  if (err) err[c] = e;
  if (iters) iters[c] = it;
}
}  // namespace echo

template <int KIND>
static void launch_c2p_test(DevPhys P, Metric M, int algo, double tol, int ncells, const double* u, double* v,
                            int* err, int* iters) {
  c2p_test_kernel<KIND><<<(ncells + 127) / 128, 128>>>(P, M, algo, tol, ncells, u, v, err, iters);
}

static __global__ void fastdiv_test_kernel(const unsigned* d, int nd, const unsigned* n, int nn, unsigned* q) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nd * nn) return;
  const int i = (int)(t / nn), j = (int)(t % nn);
  q[t] = echo::fast_div(n[j], echo::make_fastdiv(d[i]));
}

extern "C" int echo_gpu_test_fastdiv(const unsigned* d, int nd, const unsigned* n, int nn, unsigned* q) {
  (void)cudaGetLastError();
  if (nd <= 0 || nn <= 0 || !d || !n || !q) return ECHO_ERR_ARG;
  for (int i = 0; i < nd; i++)
    if (d[i] == 0) return ECHO_ERR_ARG;
  const size_t nq = (size_t)nd * nn;
  unsigned *dd, *dn, *dq;
  CK(cudaMalloc(&dd, nd * sizeof(unsigned)));
  CK(cudaMalloc(&dn, nn * sizeof(unsigned)));
  CK(cudaMalloc(&dq, nq * sizeof(unsigned)));
  CK(cudaMemcpy(dd, d, nd * sizeof(unsigned), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(dn, n, nn * sizeof(unsigned), cudaMemcpyHostToDevice));
  fastdiv_test_kernel<<<(unsigned)((nq + 127) / 128), 128>>>(dd, nd, dn, nn, dq);
  CK(cudaGetLastError());
  CK(cudaMemcpy(q, dq, nq * sizeof(unsigned), cudaMemcpyDeviceToHost));
  cudaFree(dd);
  cudaFree(dn);
  cudaFree(dq);
  return ECHO_OK;
}

// product build: the reciprocals of physics.cuh; parity build: CUDA's operators
static __global__ void recip_test_kernel(int op, int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
#ifdef ECHO_EXACT
  out[i] = op == 1 || op == 5 ? 1. / sqrt(a[i]) : op == 2 || op == 6 ? sqrt(a[i]) : op == 3 ? b[i] / a[i] : 1. / a[i];
#else
  out[i] = op == 0   ? echo::rcp_h3(a[i])
           : op == 1 ? echo::rsqrt_h3(a[i])
           : op == 2 ? echo::sqrt_h3(a[i])
           : op == 3 ? echo::div_n(b[i], a[i])
           : op == 4 ? echo::rcp_n(a[i])
           : op == 5 ? echo::rsqrt_n(a[i])
                     : echo::sqrt_n(a[i]);
#endif
}

extern "C" int echo_gpu_test_recip(int op, int n, const double* a, const double* b, double* out) {
  (void)cudaGetLastError();
  if (op < 0 || op > 6 || n <= 0 || !a || !b || !out) return ECHO_ERR_ARG;
  const size_t nb = (size_t)n * sizeof(double);
  double *da, *db, *dc;
  CK(cudaMalloc(&da, nb));
  CK(cudaMalloc(&db, nb));
  CK(cudaMalloc(&dc, nb));
  CK(cudaMemcpy(da, a, nb, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(db, b, nb, cudaMemcpyHostToDevice));
  recip_test_kernel<<<(n + 127) / 128, 128>>>(op, n, da, db, dc);
  CK(cudaGetLastError());
  CK(cudaMemcpy(out, dc, nb, cudaMemcpyDeviceToHost));
  cudaFree(da);
  cudaFree(db);
  cudaFree(dc);
  return ECHO_OK;
}

extern "C" int echo_gpu_test_offsets(int nx, int ny, int nz, unsigned long long* off) {
  if (nx < 1 || ny < 1 || nz < 1 || !off) return ECHO_ERR_ARG;
  echo::Grid g;
  memset(&g, 0, sizeof(g));
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.ncell = (size_t)nx * ny * nz;
  const unsigned x = (unsigned)nx, y = (unsigned)ny, z = (unsigned)nz;
  const unsigned i[4] = {(unsigned)(g.ncell - 1), echo::face_index<0>(g, x, y - 1, z - 1, (z * y - 1) * x, 1),
                         echo::face_index<1>(g, y, x - 1, z - 1, (z - 1) * x * y + x - 1, x),
                         echo::face_index<2>(g, z, x - 1, y - 1, x * y - 1, x * y)};
  const bool wide = echo::wide_grid(g);
  for (int q = 0; q < 4; q++) off[q] = wide ? echo::off8<true>(i[q]) : echo::off8<false>(i[q]);
  off[4] = echo::off8<true>(i[0]);  // the updates' (always 64-bit)
  return ECHO_OK;
}

extern "C" int echo_gpu_test_recon(int recal, int m, int n, const double* f, double* gl, double* gr) {
  (void)cudaGetLastError();  // a failed launch of an earlier call must not be reported here
  if (m <= 0 || n <= 0 || !f || !gl || !gr) return ECHO_ERR_ARG;
  size_t nf = (size_t)m * (n + 8), nfc = (size_t)m * (n + 1);
  double *df, *dl, *dr;
  CK(cudaMalloc(&df, nf * sizeof(double)));
  CK(cudaMalloc(&dl, nfc * sizeof(double)));
  CK(cudaMalloc(&dr, nfc * sizeof(double)));
  CK(cudaMemcpy(df, f, nf * sizeof(double), cudaMemcpyHostToDevice));
  recon_test_kernel<<<(unsigned)((nfc + 127) / 128), 128>>>(recal, m, n, df, dl, dr);
  CK(cudaGetLastError());
  CK(cudaMemcpy(gl, dl, nfc * sizeof(double), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(gr, dr, nfc * sizeof(double), cudaMemcpyDeviceToHost));
  cudaFree(df);
  cudaFree(dl);
  cudaFree(dr);
  return ECHO_OK;
}

extern "C" int echo_gpu_test_c2p(const EchoParams* p, const double* eos_table, int n_eos, int ncells, double g3,
                                 double gp, const double* u, double* v, int* err, int* iters) {
  if (!p || ncells <= 0 || !u || !v) return ECHO_ERR_ARG;
  if (p->mhd > 1) return ECHO_ERR_UNSUPPORTED;  // the resistive inversion is tested through the step
  (void)cudaGetLastError();
  int kind = echo_kind_of(p), nv = echo_nv_of(kind);
  size_t nb = (size_t)ncells * nv * sizeof(double);
  double *du, *dv, *dtab = nullptr;
  int *derr, *dit;
  CK(cudaMalloc(&du, nb));
  CK(cudaMalloc(&dv, nb));
  CK(cudaMalloc(&derr, ncells * sizeof(int)));
  CK(cudaMalloc(&dit, ncells * sizeof(int)));
  CK(cudaMemcpy(du, u, nb, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(dv, v, nb, cudaMemcpyHostToDevice));
  DevPhys P;
  memset(&P, 0, sizeof(P));
  int* dbk = nullptr;
  if (eos_table && n_eos > 0) {
    std::vector<double> cols((size_t)4 * n_eos);
    for (int i = 0; i < n_eos; i++)
      for (int q = 0; q < 4; q++) cols[(size_t)q * n_eos + i] = eos_table[4 * i + q];
    CK(cudaMalloc(&dtab, sizeof(double) * 4 * n_eos));
    CK(cudaMemcpy(dtab, cols.data(), sizeof(double) * 4 * n_eos, cudaMemcpyHostToDevice));
    P.nt = n_eos;
    P.tT = dtab;
    P.te = dtab + n_eos;
    P.tp = dtab + 2 * n_eos;
    P.tc = dtab + 3 * n_eos;
    std::vector<int> be, bp;
    long long ke0 = 0, kp0 = 0;
    if (echo_make_buckets(cols.data() + n_eos, n_eos, be, ke0) && echo_make_buckets(cols.data() + 2 * n_eos, n_eos, bp, kp0)) {
      CK(cudaMalloc(&dbk, sizeof(int) * (be.size() + bp.size())));
      CK(cudaMemcpy(dbk, be.data(), sizeof(int) * be.size(), cudaMemcpyHostToDevice));
      CK(cudaMemcpy(dbk + be.size(), bp.data(), sizeof(int) * bp.size(), cudaMemcpyHostToDevice));
      P.bke = dbk;
      P.bkp = dbk + be.size();
      P.bke0 = ke0;
      P.bkp0 = kp0;
      P.nbke = (int)be.size();
      P.nbkp = (int)bp.size();
    }
  }
  P.eqstate = p->eqstate;
  P.coordinates = p->coordinates;
  P.recal = p->recal;
  P.obtained_zz = p->obtained_zz;
  P.init_type = p->init_type;
  P.bulkvis = p->bulkvis;
  P.maxspeed = p->maxspeed;
  P.eta_over_s = p->eta_over_s;
  P.tau_pi_coeff = p->tau_pi_coeff;
  P.enezero = p->enezero;
  P.przero = p->przero;
  P.glm_alpha = p->glm_alpha;
  Metric M;
  M.g0 = -1.;
  M.g3 = g3;
  M.gp = gp;
  M.gm = 1. / gp;
  M.ig3 = 1. / g3;
  M.t = gp;
  M.t3 = pow(gp, 3.);
  switch (kind) {
    case KIND_HD: launch_c2p_test<KIND_HD>(P, M, p->algo_solver, p->c2p_tol, ncells, du, dv, derr, dit); break;
    case KIND_VISC: launch_c2p_test<KIND_VISC>(P, M, p->algo_solver, p->c2p_tol, ncells, du, dv, derr, dit); break;
    case KIND_MHD: launch_c2p_test<KIND_MHD>(P, M, p->algo_solver, p->c2p_tol, ncells, du, dv, derr, dit); break;
    default: launch_c2p_test<KIND_MHDGLM>(P, M, p->algo_solver, p->c2p_tol, ncells, du, dv, derr, dit); break;
  }
  CK(cudaGetLastError());
  CK(cudaMemcpy(v, dv, nb, cudaMemcpyDeviceToHost));
  if (err) CK(cudaMemcpy(err, derr, ncells * sizeof(int), cudaMemcpyDeviceToHost));
  if (iters) CK(cudaMemcpy(iters, dit, ncells * sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(du);
  cudaFree(dv);
  cudaFree(derr);
  cudaFree(dit);
  cudaFree(dtab);
  cudaFree(dbk);
  return ECHO_OK;
}

// ---------------------------------------------------------------------------
// con2prim of independent ideal-RMHD cells with the learned seed (weights !=
// NULL) or with Newton from the guess in v (weights == NULL): the seed's
// gain, cell by cell, at the same residual.
// ---------------------------------------------------------------------------
namespace echo {
template <int KIND>
__global__ void c2p_seed_kernel(DevPhys P, Metric M, MlpDev net, int use_seed, double tol, int ncells,
                                const double* u, double* v, int* err, int* iters, int* seed_failed) {
  typedef Traits<KIND> T;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  bool active = c < ncells;
  double uu[T::NV], vv[T::NV];
  for (int k = 0; k < T::NV; k++) {
    uu[k] = active ? u[(size_t)c * T::NV + k] : 1.0;
    vv[k] = active ? v[(size_t)c * T::NV + k] : 0.0;
  }
  float seed[2] = {0.f, 0.f};
  if (use_seed) {
    mlp_seed<KIND>(net, M, active, uu, seed);
  }
  if (!active) return;
  int it = 0, sf = 0;
  int e = cons2prim<KIND>(P, M, use_seed ? ECHO_C2P_MLP : ECHO_C2P_NEWTON, tol, uu, vv, &it,
                          use_seed ? seed : nullptr, &sf);
  for (int k = 0; k < T::NV; k++) v[(size_t)c * T::NV + k] = vv[k];
  err[c] = e;
  iters[c] = it;
  seed_failed[c] = sf;
}
}  // namespace echo

bool echo_mlp_pack(const float* W, const float* norm, std::vector<unsigned>& frag, std::vector<float>& par);

extern "C" int echo_gpu_test_c2p_seeded(const EchoParams* p, const double* eos_table, int n_eos, int ncells,
                                        double g3, double gp, const float* weights, const float* norm,
                                        const double* u, double* v, int* err, int* iters, int* seed_failed) {
  if (!p || !p->mhd || p->viscosity || ncells <= 0 || !u || !v || !err || !iters || !seed_failed)
    return ECHO_ERR_ARG;
  if (p->mhd > 1) return ECHO_ERR_UNSUPPORTED;
  (void)cudaGetLastError();
  int kind = echo_kind_of(p), nv = echo_nv_of(kind);
  size_t nb = (size_t)ncells * nv * sizeof(double);
  double *du, *dv, *dtab = nullptr;
  int *derr, *dit, *dsf;
  unsigned* dfrag = nullptr;
  float* dpar = nullptr;
  CK(cudaMalloc(&du, nb));
  CK(cudaMalloc(&dv, nb));
  CK(cudaMalloc(&derr, ncells * sizeof(int)));
  CK(cudaMalloc(&dit, ncells * sizeof(int)));
  CK(cudaMalloc(&dsf, ncells * sizeof(int)));
  CK(cudaMemcpy(du, u, nb, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(dv, v, nb, cudaMemcpyHostToDevice));
  DevPhys P;
  memset(&P, 0, sizeof(P));
  std::vector<double> cols((size_t)4 * n_eos);
  for (int i = 0; i < n_eos; i++)
    for (int q = 0; q < 4; q++) cols[(size_t)q * n_eos + i] = eos_table[4 * i + q];
  CK(cudaMalloc(&dtab, sizeof(double) * 4 * n_eos));
  CK(cudaMemcpy(dtab, cols.data(), sizeof(double) * 4 * n_eos, cudaMemcpyHostToDevice));
  P.nt = n_eos;
  P.tT = dtab;
  P.te = dtab + n_eos;
  P.tp = dtab + 2 * n_eos;
  P.tc = dtab + 3 * n_eos;
  P.eqstate = p->eqstate;
  P.coordinates = p->coordinates;
  P.enezero = p->enezero;
  P.przero = p->przero;
  MlpDev net{nullptr, nullptr};
  if (weights) {
    std::vector<unsigned> frag;
    std::vector<float> par;
    echo_mlp_pack(weights, norm, frag, par);
    CK(cudaMalloc(&dfrag, sizeof(unsigned) * frag.size()));
    CK(cudaMalloc(&dpar, sizeof(float) * par.size()));
    CK(cudaMemcpy(dfrag, frag.data(), sizeof(unsigned) * frag.size(), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(dpar, par.data(), sizeof(float) * par.size(), cudaMemcpyHostToDevice));
    net.frag = dfrag;
    net.par = dpar;
  }
  Metric M;
  M.g0 = -1.;
  M.g3 = g3;
  M.gp = gp;
  M.gm = 1. / gp;
  M.ig3 = 1. / g3;
  M.t = gp;
  M.t3 = pow(gp, 3.);
  unsigned blocks = (unsigned)((ncells + 127) / 128);
  if (kind == KIND_MHDGLM)
    c2p_seed_kernel<KIND_MHDGLM><<<blocks, 128>>>(P, M, net, weights != nullptr, p->c2p_tol, ncells, du, dv, derr,
                                                  dit, dsf);
  else
    c2p_seed_kernel<KIND_MHD><<<blocks, 128>>>(P, M, net, weights != nullptr, p->c2p_tol, ncells, du, dv, derr, dit,
                                               dsf);
  CK(cudaGetLastError());
  CK(cudaMemcpy(v, dv, nb, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(err, derr, ncells * sizeof(int), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(iters, dit, ncells * sizeof(int), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(seed_failed, dsf, ncells * sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(du);
  cudaFree(dv);
  cudaFree(derr);
  cudaFree(dit);
  cudaFree(dsf);
  cudaFree(dtab);
  cudaFree(dfrag);
  cudaFree(dpar);
  return ECHO_OK;
}

// ---------------------------------------------------------------------------
// FP64 peak of this GPU: the roofline the step kernels' FP64 work is
// measured against.  Every thread runs 8 independent multiply-add chains
// (x = x * a + b, a fixed point at 1, so no value leaves the normal range)
// for `iters` rounds; one round is 8 DFMA = 16 FLOP per thread.
// ---------------------------------------------------------------------------
namespace echo {
__global__ void __launch_bounds__(256) fp64_peak_kernel(int iters, double a, double b, double* out) {
  double x0 = 1.0 + threadIdx.x * 1e-9, x1 = x0 + 1e-9, x2 = x0 + 2e-9, x3 = x0 + 3e-9;
  double x4 = x0 + 4e-9, x5 = x0 + 5e-9, x6 = x0 + 6e-9, x7 = x0 + 7e-9;
#pragma unroll 4
  for (int i = 0; i < iters; i++) {
    x0 = fma(x0, a, b);
    x1 = fma(x1, a, b);
    x2 = fma(x2, a, b);
    x3 = fma(x3, a, b);
    x4 = fma(x4, a, b);
    x5 = fma(x5, a, b);
    x6 = fma(x6, a, b);
    x7 = fma(x7, a, b);
  }
  double s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == 12345.0) out[0] = s;  // never true: keeps the chains live
}
}  // namespace echo

extern "C" int echo_gpu_fp64_peak(double* gflops, double* ms) {
  if (!gflops) return ECHO_ERR_ARG;
  int dev = 0, nsm = 0, per_sm = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, echo::fp64_peak_kernel, 256, 0));
  if (per_sm < 1) per_sm = 1;
  const int iters = 1 << 11;
  const unsigned blocks = (unsigned)(nsm * per_sm);
  double* d_out = nullptr;
  CK(cudaMalloc(&d_out, sizeof(double)));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  echo::fp64_peak_kernel<<<blocks, 256>>>(iters, 0.999999, 1e-6, d_out);  // warm-up
  float best = 1e30f;
  for (int r = 0; r < 5; r++) {
    CK(cudaEventRecord(e0));
    echo::fp64_peak_kernel<<<blocks, 256>>>(iters, 0.999999, 1e-6, d_out);
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    float t = 0.f;
    CK(cudaEventElapsedTime(&t, e0, e1));
    if (t < best) best = t;
  }
  CK(cudaGetLastError());
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d_out);
  double flop = 16.0 * (double)iters * (double)blocks * 256.0;
  *gflops = flop / (best * 1e-3) / 1e9;
  if (ms) *ms = best;
  return ECHO_OK;
}
