// rel_kernels.cu -- relativistic species (src/ALPS_fns_rel.f90).
//
// Setup per run (launch_rel_prepare): the (Gamma, pparbar) grid spanning the
// f0 table, a thin-plate-spline interpolation of log f0 onto it (dense
// saddle-point system, LU with partial pivoting as dgesv does), the subluminal-cone
// mask (f0_rel = -1 outside), normalisation, and the one-sided derivatives at
// the cone edge (derivative_f0_rel, :36-289; polyharmonic_spline, :293-426),
// then the ee term (int_ee_rel, :1097-1215).
// Per k (launch_rel_bessel): the Bessel products of int_T_rel (:1256-1369) at
// every (Gamma, pparbar) node, whose arguments do not depend on omega, and the
// coefficients of CBESSJ's power series.
// Per omega batch (launch_rel_orders): REL_RB blocks per (omega, species, n):
// the resonance test over the whole (pperp, ppar) grid (determine_resonances,
// src/ALPS_fns.f90:680-702), then either the regular-grid trapezoid sum with
// the Lorentz factor in resU (src/ALPS_fns.f90:799-864, 1560-1596) or the
// Gamma-row integrals with their principal-value windows and the Landau term
// (integrate_res_rel :460-913, landau_integrate_rel :1005-1092).
#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include <cusolverDn.h>

#include "alps_internal.cuh"
#include "device_math.cuh"

namespace {

__device__ __host__ inline double cube(double x) { return x * x * x; }

// ---------------------------------------------------------------------------
// thin-plate spline
// ---------------------------------------------------------------------------
__device__ inline double tps_phi(double r) {
  if (r >= 1.0) return r * r * log(r);
  if (r == 0.0) return 0.0;
  return r * log(pow(r, r));
}

// column-major (n+3)^2 system of polyharmonic_spline, the smoothing added
// on the diagonal of the kernel block
__global__ void k_tps_matrix(const double* __restrict__ gc, const double* __restrict__ pc, int n, double smoothing,
                             double* A) {
  long m = n + 3;
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * m) return;
  int i = (int)(t % m), j = (int)(t / m);
  double v = 0.0;
  if (i < n && j < n) {
    double dg = gc[i] - gc[j], dp = pc[i] - pc[j];
    v = tps_phi(sqrt(dg * dg + dp * dp));
    if (i == j) v = v + smoothing;
  } else if (i < n && j >= n) {
    v = (j == n) ? 1.0 : (j == n + 1 ? gc[i] : pc[i]);
  } else if (j < n && i >= n) {
    v = (i == n) ? 1.0 : (i == n + 1 ? gc[j] : pc[j]);
  }
  A[t] = v;
}

// Dense LU with partial pivoting, column by column (the dgetrf/dgetrs pair of
// dgesv).  Column-major m x m.  Step k: k_lu_pivot (one block) picks the
// first row of largest |A(i,k)|, swaps the whole rows and scales column k;
// k_lu_update applies the rank-1 update to columns k+1..m-1.
__global__ void k_lu_pivot(double* A, int m, int k, int* piv, int* status) {
  __shared__ double sv[1024];
  __shared__ int si[1024];
  __shared__ int sp;
  if (*status) return;
  double mx = -1.0;
  int p = m;
  for (int i = k + threadIdx.x; i < m; i += blockDim.x) {
    double v = fabs(A[(size_t)i + (size_t)m * k]);
    if (v > mx) {
      mx = v;
      p = i;
    }
  }
  sv[threadIdx.x] = mx;
  si[threadIdx.x] = p;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      double v2 = sv[threadIdx.x + s];
      int i2 = si[threadIdx.x + s];
      if (v2 > sv[threadIdx.x] || (v2 == sv[threadIdx.x] && i2 < si[threadIdx.x])) {
        sv[threadIdx.x] = v2;
        si[threadIdx.x] = i2;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    int q = si[0];
    if (q >= m) q = k;  // column of NaNs: keep the diagonal
    sp = q;
    piv[k] = q;
    if (A[(size_t)q + (size_t)m * k] == 0.0) *status = 1;
  }
  __syncthreads();
  const int q = sp;
  if (q != k)
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
      double t = A[(size_t)k + (size_t)m * j];
      A[(size_t)k + (size_t)m * j] = A[(size_t)q + (size_t)m * j];
      A[(size_t)q + (size_t)m * j] = t;
    }
  __syncthreads();
  const double dk = A[(size_t)k + (size_t)m * k];
  if (dk != 0.0)
    for (int i = k + 1 + threadIdx.x; i < m; i += blockDim.x)
      A[(size_t)i + (size_t)m * k] = __ddiv_rn(A[(size_t)i + (size_t)m * k], dk);
}

__global__ void k_lu_update(double* A, int m, int k, const int* status) {
  if (*status) return;
  const int j = k + 1 + blockIdx.x;
  if (j >= m) return;
  const double f = A[(size_t)k + (size_t)m * j];
  if (f == 0.0) return;
  double* colj = A + (size_t)m * j;
  const double* colk = A + (size_t)m * k;
  for (int i = k + 1 + threadIdx.x; i < m; i += blockDim.x) colj[i] = __dsub_rn(colj[i], __dmul_rn(colk[i], f));
}

// row interchanges, then the unit-lower and upper triangular solves
__global__ void k_lu_solve(const double* A, int m, const int* piv, double* w, const int* status) {
  if (*status) return;
  if (threadIdx.x == 0)
    for (int k = 0; k < m; ++k) {
      double t = w[k];
      w[k] = w[piv[k]];
      w[piv[k]] = t;
    }
  __syncthreads();
  for (int j = 0; j < m; ++j) {
    const double wj = w[j];
    for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x)
      w[i] = __dsub_rn(w[i], __dmul_rn(A[(size_t)i + (size_t)m * j], wj));
    __syncthreads();
  }
  for (int j = m - 1; j >= 0; --j) {
    if (threadIdx.x == 0) w[j] = __ddiv_rn(w[j], A[(size_t)j + (size_t)m * j]);
    __syncthreads();
    const double wj = w[j];
    for (int i = threadIdx.x; i < j; i += blockDim.x)
      w[i] = __dsub_rn(w[i], __dmul_rn(A[(size_t)i + (size_t)m * j], wj));
    __syncthreads();
  }
}

// f0_rel = exp(spline) on the fine grid, -1 outside the subluminal cone
__global__ void k_tps_eval(const double* __restrict__ w, const double* __restrict__ gc, const double* __restrict__ pc,
                           int n, const double* __restrict__ grel, const double* __restrict__ prel, int ng, int np,
                           double* f0rel) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (ng + 1) * (np + 1)) return;
  int ig = t / (np + 1), ip = t % (np + 1);
  double g = grel[ig], pb = prel[ip], f = 0.0;
  for (int k = 0; k < n; ++k) {
    double dg = g - gc[k], dp = pb - pc[k];
    double r = sqrt(dg * dg + dp * dp);
    if (r >= 1.0) f = f + w[k] * r * r * log(r);
    else if (r != 0.0) f = f + w[k] * r * log(pow(r, r));
  }
  f = f + w[n] + w[n + 1] * g + w[n + 2] * pb;
  f = exp(f);
  // outside the subluminal cone, decided as the reference rounds it (no FMA)
  if (__dsub_rn(__dmul_rn(g, g), 1.0) < __dmul_rn(pb, pb)) f = -1.0;
  f0rel[t] = f;
}

// integral of f0_rel over the cone (one block, fixed reduction order)
__global__ void k_rel_norm(double* f0rel, const double* __restrict__ grel, int ng, int np, double scale) {
  __shared__ double red[256];
  double acc = 0.0;
  int tot = (ng + 1) * (np + 1);
  for (int t = threadIdx.x; t < tot; t += blockDim.x) {
    double f = f0rel[t];
    if (f > -1.0) acc += grel[t / (np + 1)] * f * scale;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  double integ = red[0];
  __syncthreads();
  for (int t = threadIdx.x; t < tot; t += blockDim.x)
    if (f0rel[t] != -1.0) f0rel[t] = f0rel[t] / integ;
}

__global__ void k_rel_deriv(const double* __restrict__ f, const double* __restrict__ grel,
                            const double* __restrict__ prel, int ng, int np, double* d1, double* d2) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (ng + 1) * (np + 1)) return;
  int ig = t / (np + 1), ip = t % (np + 1);
  d1[t] = 0.0;
  d2[t] = 0.0;
  if (ig < 1 || ig > ng - 1 || ip < 1 || ip > np - 1) return;
  int L = np + 1;
  auto F = [&](int a, int b) { return f[a * L + b]; };
  if ((F(ig - 1, ip) > 0.0) && (F(ig + 1, ip) > 0.0)) d1[t] = (F(ig + 1, ip) - F(ig - 1, ip)) / (grel[ig + 1] - grel[ig - 1]);
  if ((F(ig, ip + 1) > 0.0) && (F(ig, ip - 1) > 0.0)) d2[t] = (F(ig, ip + 1) - F(ig, ip - 1)) / (prel[ip + 1] - prel[ip - 1]);
  if (F(ig, ip) >= 0.0) {
    if ((F(ig, ip + 1) <= 0.0) && (F(ig, ip - 1) > 0.0)) d2[t] = (F(ig, ip) - F(ig, ip - 1)) / (prel[ip] - prel[ip - 1]);
    if ((F(ig, ip + 1) > 0.0) && (F(ig, ip - 1) <= 0.0)) d2[t] = (F(ig, ip + 1) - F(ig, ip)) / (prel[ip + 1] - prel[ip]);
  }
}

__device__ inline void cone_limits(const double* fr, int np, int& lower, int& upper) {
  bool fl = false, fu = false;
  lower = 1;
  upper = np - 1;
  for (int ip = 1; ip <= np - 1; ++ip) {
    if (!fl && fr[ip - 1] <= -1.0 && fr[ip] > -1.0) { lower = ip; fl = true; }
    if (!fu && fr[ip] > -1.0 && fr[ip + 1] <= -1.0) { upper = ip; fu = true; }
  }
}

// int_ee_rel: one block
__global__ void k_rel_ee(const double* __restrict__ f0rel, const double* __restrict__ dfr2,
                         const double* __restrict__ prel, int ng, int np, double scale, double* out) {
  __shared__ double red[256];
  double acc = 0.0;
  int L = np + 1;
  for (int ig = 1 + threadIdx.x; ig <= ng - 1; ig += blockDim.x) {
    int lo, up;
    cone_limits(f0rel + (size_t)ig * L, np, lo, up);
    auto t = [&](int ip) { return prel[ip] * dfr2[(size_t)ig * L + ip]; };
    double wi = (ig == ng - 1) ? 1.0 : 2.0;   // Gamma weight; pparbar weights 1 at ends, 2 inside
    double row = t(lo) + t(up);
    for (int ip = lo + 1; ip <= up - 1; ++ip) row += 2.0 * t(ip);
    acc += wi * row;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0] * scale;
}

// J_n(z(ig, ip)), z = (k_perp m/(vA q)) sqrt(Gamma^2 - 1 - pparbar^2)
__global__ void k_rel_jtab(const double* __restrict__ grel, const double* __restrict__ prel, int ng, int np, int nrows,
                           double zfac, double* jrel) {
  long tot = (long)(ng + 1) * (np + 1);
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= tot * nrows) return;
  int n = (int)(t / tot);
  long pt = t % tot;
  int ig = (int)(pt / (np + 1)), ip = (int)(pt % (np + 1));
  double g = grel[ig], pb = prel[ip];
  double pperpbar = sqrt(g * g - 1.0 - pb * pb);
  double z = zfac * pperpbar;
  jrel[t] = (z == z) ? alps_bessj(n, z) : z;
}

// The Bessel products of int_T_rel at every node, planes fam[(n*3 + F)] of
// (ng+1)(np+1): F = 0: J_n^2, 1: J_n'^2 pperpbar^2, 2: J_n J_n' pperpbar, from
// the planes J_0 .. J_nmax+1.  They are the same for orders n and -n.
__global__ void k_rel_families(const double* __restrict__ jrel, const double* __restrict__ grel,
                               const double* __restrict__ prel, int ng, int np, int nmax, double* fam) {
  const long tot = (long)(ng + 1) * (np + 1);
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= tot * (nmax + 1)) return;
  const int n = (int)(t / tot);
  const long pt = t % tot;
  const double g = grel[pt / (np + 1)], pb = prel[pt % (np + 1)];
  const double pp = sqrt(g * g - 1.0 - pb * pb);
  const double b = jrel[n * tot + pt];
  const double bp = n == 0 ? -jrel[tot + pt] : 0.5 * (jrel[(n - 1) * tot + pt] - jrel[(n + 1) * tot + pt]);
  fam[(n * 3L + 0) * tot + pt] = b * b;
  fam[(n * 3L + 1) * tot + pt] = bp * bp * pp * pp;
  fam[(n * 3L + 2) * tot + pt] = b * bp * pp;
}

// gamma on the (pperp, ppar) grid, g2/gamma, and gamma in FP32 (the resonance
// test's estimate)
__global__ void k_rel_gamma(const double* __restrict__ pperp, const double* __restrict__ ppar,
                            const double* __restrict__ g2, int N, int M, double vA, double ms, double* gam,
                            double* g2g, float* gf) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)(N + 1) * (M + 1)) return;
  const double p1 = pperp[t / (M + 1)], p2 = ppar[t % (M + 1)];
  const double g = sqrt((p1 * p1 + p2 * p2) * (vA * vA) / (ms * ms) + 1.0);
  gam[t] = g;
  g2g[t] = g2[t] / g;
  gf[t] = (float)g;
}

// first and last pparbar index inside the cone of each Gamma row
// (integrate_resU_rel, src/ALPS_fns_rel.f90:603-617)
__global__ void k_rel_cone(const double* __restrict__ f0rel, int ng, int np, int2* cone) {
  int ig = blockIdx.x * blockDim.x + threadIdx.x;
  if (ig > ng) return;
  int lo, up;
  cone_limits(f0rel + (size_t)ig * (np + 1), np, lo, up);
  cone[ig] = make_int2(lo, up);
}

// right-hand side of the spline system: log f at the samples, three zeros
__global__ void k_tps_rhs(const double* __restrict__ f, int n, double* w) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) w[k] = log(f[k]);
  else if (k < n + 3) w[k] = 0.0;
}

// spline (log f) on the tensor grid pperp[i] x ppar[j], [i*(npar+1) + j]
// (the evaluation loop of polyharmonic_spline, interpolation.f90:610-630)
__global__ void k_tps_eval_grid(const double* __restrict__ w, const double* __restrict__ gc,
                                const double* __restrict__ pc, int n, const double* __restrict__ pperp,
                                const double* __restrict__ ppar, int nperp, int npar, double* g) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (nperp + 1) * (npar + 1)) return;
  const int i = t / (npar + 1), j = t % (npar + 1);
  const double x = pperp[i], y = ppar[j];
  double f = 0.0;
  for (int k = 0; k < n; ++k) {
    double dg = x - gc[k], dp = y - pc[k];
    double r = sqrt(dg * dg + dp * dp);
    if (r >= 1.0) f = f + w[k] * r * r * log(r);
    else if (r != 0.0) f = f + w[k] * r * log(pow(r, r));
  }
  g[t] = f + w[n] + w[n + 1] * x + w[n + 2] * y;
}

// f = mult exp(g - shift), shift = log(2 pi dpperp dppar sum_ij exp(g) pperp_i)
// when normalising (normalize, interpolation.f90:520-552); one block, fixed
// reduction order
__global__ void k_interp_finish(const double* __restrict__ g, const double* __restrict__ pperp, int nperp, int npar,
                                double dpp, double dpl, int normalize, double mult, double* f) {
  __shared__ double red[256];
  const int tot = (nperp + 1) * (npar + 1);
  double shift = 0.0;
  if (normalize) {
    double acc = 0.0;
    for (int t = threadIdx.x; t < tot; t += blockDim.x) acc += exp(g[t]) * pperp[t / (npar + 1)];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
      __syncthreads();
    }
    shift = log(red[0] * dpp * dpl * 2.0 * ALPS_PI);
  }
  for (int t = threadIdx.x; t < tot; t += blockDim.x) f[t] = mult * exp(g[t] - shift);
}

}  // namespace

// ---------------------------------------------------------------------------
// Large spline systems: cuSOLVER's blocked LU with partial pivoting (getrf,
// getrs: the dgesv pair), loaded on first use.  The column-by-column LU above
// restates dgesv's arithmetic for the sizes the oracle can check; from
// TPS_BLOCKED_M unknowns on (a 128 x 256 input grid has 33 156) its one pass
// per column would take minutes, and the blocked factorisation runs at the
// FP64 GEMM rate instead.
// ---------------------------------------------------------------------------
#define TPS_BLOCKED_M 4096

struct CusolverApi {
  bool tried = false, ok = false;
  cusolverStatus_t (*create)(cusolverDnHandle_t*) = nullptr;
  cusolverStatus_t (*destroy)(cusolverDnHandle_t) = nullptr;
  cusolverStatus_t (*set_stream)(cusolverDnHandle_t, cudaStream_t) = nullptr;
  cusolverStatus_t (*getrf_ws)(cusolverDnHandle_t, int, int, double*, int, int*) = nullptr;
  cusolverStatus_t (*getrf)(cusolverDnHandle_t, int, int, double*, int, double*, int*, int*) = nullptr;
  cusolverStatus_t (*getrs)(cusolverDnHandle_t, cublasOperation_t, int, int, const double*, int, const int*,
                            double*, int, int*) = nullptr;
};
std::mutex g_cusolver_mu;
CusolverApi g_cusolver;

const CusolverApi* cusolver_api() {
  std::lock_guard<std::mutex> lk(g_cusolver_mu);
  if (g_cusolver.tried) return g_cusolver.ok ? &g_cusolver : nullptr;
  g_cusolver.tried = true;
  const char* names[] = {"libcusolver.so.12", "libcusolver.so", "/usr/local/cuda/lib64/libcusolver.so.12",
                         "/usr/local/cuda/lib64/libcusolver.so"};
  void* h = nullptr;
  for (const char* nm : names)
    if ((h = dlopen(nm, RTLD_NOW | RTLD_LOCAL))) break;
  if (!h) return nullptr;
  CusolverApi& a = g_cusolver;
  a.create = reinterpret_cast<decltype(a.create)>(dlsym(h, "cusolverDnCreate"));
  a.destroy = reinterpret_cast<decltype(a.destroy)>(dlsym(h, "cusolverDnDestroy"));
  a.set_stream = reinterpret_cast<decltype(a.set_stream)>(dlsym(h, "cusolverDnSetStream"));
  a.getrf_ws = reinterpret_cast<decltype(a.getrf_ws)>(dlsym(h, "cusolverDnDgetrf_bufferSize"));
  a.getrf = reinterpret_cast<decltype(a.getrf)>(dlsym(h, "cusolverDnDgetrf"));
  a.getrs = reinterpret_cast<decltype(a.getrs)>(dlsym(h, "cusolverDnDgetrs"));
  a.ok = a.create && a.destroy && a.set_stream && a.getrf_ws && a.getrf && a.getrs;
  return a.ok ? &a : nullptr;
}

// LU with partial pivoting and the solve of A w = w (column-major m x m, d_A
// overwritten) through cuSOLVER; ALPS_E_SINGULAR for an exactly singular
// pivot, ALPS_E_UNSUPPORTED when the library cannot be loaded
int tps_lu_blocked(double* d_A, int m, double* d_w, cudaStream_t st) {
  const CusolverApi* api = cusolver_api();
  if (!api) return ALPS_E_UNSUPPORTED;
  cusolverDnHandle_t h = nullptr;
  if (api->create(&h) != CUSOLVER_STATUS_SUCCESS) return ALPS_E_CUDA;
  int status = ALPS_OK, lwork = 0, info = 0;
  double* d_work = nullptr;
  int *d_piv = nullptr, *d_info = nullptr;
  if (api->set_stream(h, st) != CUSOLVER_STATUS_SUCCESS || api->getrf_ws(h, m, m, d_A, m, &lwork) !=
                                                               CUSOLVER_STATUS_SUCCESS)
    status = ALPS_E_CUDA;
  if (!status && (cudaMalloc(&d_work, (size_t)std::max(lwork, 1) * sizeof(double)) != cudaSuccess ||
                  cudaMalloc(&d_piv, (size_t)m * sizeof(int)) != cudaSuccess ||
                  cudaMalloc(&d_info, sizeof(int)) != cudaSuccess))
    status = ALPS_E_OOM;
  if (!status && api->getrf(h, m, m, d_A, m, d_work, d_piv, d_info) != CUSOLVER_STATUS_SUCCESS) status = ALPS_E_CUDA;
  if (!status) {
    if (cudaMemcpyAsync(&info, d_info, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      status = ALPS_E_CUDA;
    else if (info != 0)
      status = ALPS_E_SINGULAR;
  }
  if (!status && api->getrs(h, CUBLAS_OP_N, m, 1, d_A, m, d_piv, d_w, m, d_info) != CUSOLVER_STATUS_SUCCESS)
    status = ALPS_E_CUDA;
  if (!status && cudaStreamSynchronize(st) != cudaSuccess) status = ALPS_E_CUDA;
  cudaFree(d_work);
  cudaFree(d_piv);
  cudaFree(d_info);
  api->destroy(h);
  return status;
}

// Weights of the thin-plate spline through n samples (gc, pc) with the
// right-hand side already in d_w (n + 3 entries): the dense system of
// polyharmonic_spline solved by LU with partial pivoting (dgesv).
int tps_solve_device(const double* d_gc, const double* d_pc, int n, double smoothing, double* d_w, cudaStream_t st) {
  const int m = n + 3;
  double* d_A = nullptr;
  int *d_piv = nullptr, *d_info = nullptr;
  int status = ALPS_OK;
  if (cudaMalloc(&d_A, (size_t)m * m * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_piv, m * sizeof(int)) != cudaSuccess || cudaMalloc(&d_info, sizeof(int)) != cudaSuccess) {
    status = ALPS_E_OOM;
  }
  if (!status && cudaMemsetAsync(d_info, 0, sizeof(int), st) != cudaSuccess) status = ALPS_E_CUDA;
  if (!status) {
    long mm = (long)m * m;
    k_tps_matrix<<<(unsigned)((mm + 255) / 256), 256, 0, st>>>(d_gc, d_pc, n, smoothing, d_A);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
  }
  if (!status && m >= TPS_BLOCKED_M) {
    status = tps_lu_blocked(d_A, m, d_w, st);
    cudaFree(d_A);
    cudaFree(d_piv);
    cudaFree(d_info);
    return status;
  }
  for (int k = 0; k < m && !status; ++k) {
    k_lu_pivot<<<1, 1024, 0, st>>>(d_A, m, k, d_piv, d_info);
    if (k + 1 < m) k_lu_update<<<m - k - 1, 256, 0, st>>>(d_A, m, k, d_info);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
  }
  if (!status) {
    k_lu_solve<<<1, 1024, 0, st>>>(d_A, m, d_piv, d_w, d_info);
    int info = 0;
    cudaMemcpyAsync(&info, d_info, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) status = ALPS_E_CUDA;
    else if (info != 0) status = ALPS_E_SINGULAR;
  }
  cudaFree(d_A);
  cudaFree(d_piv);
  cudaFree(d_info);
  return status;
}

// ===========================================================================
int launch_rel_prepare(alps_ctx* c, int is) {
  SpeciesHost& S = c->spec[is];
  const double vA = c->sys.vA, ms = S.sp.ms;
  const int N = c->sys.nperp, M = c->sys.npar, ng = c->sys.ngamma, np = c->sys.npparbar;
  cudaStream_t st = c->stream;
  // grid spanning the table (derivative_f0_rel :120-171), on the host
  double pmin = 999999.0, pmax = -999999.0, gmin = 999999.0, gmax = -1.0;
  int n = (N + 1) * (M + 1);
  std::vector<double> gc(n), pc(n), grid(n);
  for (int i = 0; i <= N; ++i)
    for (int j = 0; j <= M; ++j) {
      double p1 = S.pperp[i], p2 = S.ppar[j];
      double g = std::sqrt((p1 * p1 + p2 * p2) * (vA * vA) / (ms * ms) + 1.0);
      gmax = std::max(gmax, g);
      gmin = std::min(gmin, g);
      pmin = std::min(pmin, p2);
      pmax = std::max(pmax, p2);
      int k = i * (M + 1) + j;
      gc[k] = std::sqrt(1.0 + (p1 * p1 + p2 * p2) * vA * vA / (ms * ms));
      pc[k] = p2 * vA / ms;
      grid[k] = std::log(S.f0[k]);
    }
  pmin = pmin * vA / ms;
  pmax = pmax * vA / ms;
  double pn = S.pperp[N];
  double gmax_use = std::sqrt(1.0 + pn * pn * (vA * vA) / (ms * ms));
  S.grel.resize(ng + 1);
  S.prel.resize(np + 1);
  for (int ig = 0; ig <= ng; ++ig) S.grel[ig] = gmin + ((gmax_use - gmin) * ig) / (1.0 * ng);
  for (int ip = 0; ip <= np; ++ip) S.prel[ip] = pmin + ((pmax - pmin) * ip) / (1.0 * np);
  size_t nf = (size_t)(ng + 1) * (np + 1);
  if (!S.d_grel) ALPS_CUDA_TRY(cudaMalloc(&S.d_grel, (ng + 1) * sizeof(double)));
  if (!S.d_prel) ALPS_CUDA_TRY(cudaMalloc(&S.d_prel, (np + 1) * sizeof(double)));
  if (!S.d_f0rel) ALPS_CUDA_TRY(cudaMalloc(&S.d_f0rel, nf * sizeof(double)));
  if (!S.d_dfr1) ALPS_CUDA_TRY(cudaMalloc(&S.d_dfr1, nf * sizeof(double)));
  if (!S.d_dfr2) ALPS_CUDA_TRY(cudaMalloc(&S.d_dfr2, nf * sizeof(double)));
  if (!S.d_cone) ALPS_CUDA_TRY(cudaMalloc(&S.d_cone, (ng + 1) * sizeof(int2)));
  if (!S.d_relgam) ALPS_CUDA_TRY(cudaMalloc(&S.d_relgam, (size_t)(N + 1) * (M + 1) * 20));
  {
    const size_t nn = (size_t)(N + 1) * (M + 1);
    k_rel_gamma<<<(unsigned)((nn + 127) / 128), 128, 0, st>>>(S.d_pperp, S.d_ppar, S.d_g2, N, M, vA, ms, S.d_relgam,
                                                               S.d_relgam + nn,
                                                               reinterpret_cast<float*>(S.d_relgam + 2 * nn));
    ALPS_CUDA_TRY(cudaGetLastError());
  }
  ALPS_CUDA_TRY(cudaMemcpyAsync(S.d_grel, S.grel.data(), (ng + 1) * sizeof(double), cudaMemcpyHostToDevice, st));
  ALPS_CUDA_TRY(cudaMemcpyAsync(S.d_prel, S.prel.data(), (np + 1) * sizeof(double), cudaMemcpyHostToDevice, st));
  // dense thin-plate-spline system (the reference sets its smoothing to 0
  // for the relativistic remap, src/ALPS_fns_rel.f90:149-151)
  int m = n + 3;
  double *d_gc = nullptr, *d_pc = nullptr, *d_w = nullptr;
  ALPS_CUDA_TRY(cudaMalloc(&d_gc, n * sizeof(double)));
  ALPS_CUDA_TRY(cudaMalloc(&d_pc, n * sizeof(double)));
  ALPS_CUDA_TRY(cudaMalloc(&d_w, m * sizeof(double)));
  std::vector<double> w(m, 0.0);
  for (int k = 0; k < n; ++k) w[k] = grid[k];
  ALPS_CUDA_TRY(cudaMemcpyAsync(d_gc, gc.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
  ALPS_CUDA_TRY(cudaMemcpyAsync(d_pc, pc.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
  ALPS_CUDA_TRY(cudaMemcpyAsync(d_w, w.data(), m * sizeof(double), cudaMemcpyHostToDevice, st));
  int status = tps_solve_device(d_gc, d_pc, n, 0.0, d_w, st);
  if (!status) {
    k_tps_eval<<<(unsigned)((nf + 127) / 128), 128, 0, st>>>(d_w, d_gc, d_pc, n, S.d_grel, S.d_prel, ng, np,
                                                              S.d_f0rel);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
  }
  if (!status) {
    double dgamma = S.grel[2] - S.grel[1], dpb = S.prel[2] - S.prel[1];
    k_rel_norm<<<1, 256, 0, st>>>(S.d_f0rel, S.d_grel, ng, np, 2.0 * ALPS_PI * dgamma * dpb * cube(ms / vA));
    k_rel_deriv<<<(unsigned)((nf + 127) / 128), 128, 0, st>>>(S.d_f0rel, S.d_grel, S.d_prel, ng, np, S.d_dfr1,
                                                                S.d_dfr2);
    k_rel_cone<<<(ng + 1 + 127) / 128, 128, 0, st>>>(S.d_f0rel, ng, np, S.d_cone);
    double* d_ee = nullptr;
    cudaMalloc(&d_ee, sizeof(double));
    double scale = 2.0 * ALPS_PI * S.sp.qs / (ms) * dgamma * dpb * 0.25 * cube(ms / vA);
    k_rel_ee<<<1, 256, 0, st>>>(S.d_f0rel, S.d_dfr2, S.d_prel, ng, np, scale, d_ee);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
    double ee = 0.0;
    cudaMemcpyAsync(&ee, d_ee, sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    cudaFree(d_ee);
    S.int_ee_rel = ee;
  }
  cudaFree(d_gc);
  cudaFree(d_pc);
  cudaFree(d_w);
  return status;
}

// ===========================================================================
// The interpolation tool (interpolation/interpolation.f90): thin-plate
// spline of log f through scattered samples, on a fine tensor grid,
// optionally normalised.
extern "C" int alps_interpolate(const double* pperp_c, const double* ppar_c, const double* f_c, int n,
                                const alps_interp_params* p, double* pperp_out, double* ppar_out, double* f_out) {
  if (!pperp_c || !ppar_c || !f_c || !p || n < 1 || p->nperp < 2 || p->npar < 2) return ALPS_E_INVALID;
  for (int k = 0; k < n; ++k)
    if (!(f_c[k] > 0.0)) return ALPS_E_INVALID;  // log f
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return ALPS_E_NO_DEVICE;
  const int nperp = p->nperp, npar = p->npar, m = n + 3;
  const size_t nf = (size_t)(nperp + 1) * (npar + 1);
  // the fine grid, as the reference forms it
  std::vector<double> pp(nperp + 1), pl(npar + 1);
  for (int i = 0; i <= nperp; ++i) pp[i] = p->pperp_min + (p->pperp_max - p->pperp_min) * i / (1.0 * nperp);
  for (int j = 0; j <= npar; ++j) pl[j] = p->ppar_min + (p->ppar_max - p->ppar_min) * j / (1.0 * npar);
  cudaStream_t st = nullptr;
  ALPS_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  double *d_gc = nullptr, *d_pc = nullptr, *d_f = nullptr, *d_w = nullptr, *d_pp = nullptr, *d_pl = nullptr;
  double *d_g = nullptr, *d_out = nullptr;
  int status = ALPS_OK;
  if (cudaMalloc(&d_gc, n * sizeof(double)) != cudaSuccess || cudaMalloc(&d_pc, n * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_f, n * sizeof(double)) != cudaSuccess || cudaMalloc(&d_w, m * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_pp, (nperp + 1) * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_pl, (npar + 1) * sizeof(double)) != cudaSuccess || cudaMalloc(&d_g, nf * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&d_out, nf * sizeof(double)) != cudaSuccess)
    status = ALPS_E_OOM;
  if (!status) {
    cudaMemcpyAsync(d_gc, pperp_c, n * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_pc, ppar_c, n * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_f, f_c, n * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_pp, pp.data(), (nperp + 1) * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_pl, pl.data(), (npar + 1) * sizeof(double), cudaMemcpyHostToDevice, st);
    k_tps_rhs<<<(m + 127) / 128, 128, 0, st>>>(d_f, n, d_w);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
  }
  if (!status) status = tps_solve_device(d_gc, d_pc, n, p->smoothing, d_w, st);
  if (!status) {
    k_tps_eval_grid<<<(unsigned)((nf + 127) / 128), 128, 0, st>>>(d_w, d_gc, d_pc, n, d_pp, d_pl, nperp, npar, d_g);
    // dpperp = pperp(2,1) - pperp(1,1), dppar = ppar(1,2) - ppar(1,1)
    k_interp_finish<<<1, 256, 0, st>>>(d_g, d_pp, nperp, npar, pp[2] - pp[1], pl[2] - pl[1], p->do_normalize,
                                       p->mult_f, d_out);
    if (cudaGetLastError() != cudaSuccess) status = ALPS_E_CUDA;
  }
  if (!status && f_out && cudaMemcpyAsync(f_out, d_out, nf * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    status = ALPS_E_CUDA;
  if (!status && cudaStreamSynchronize(st) != cudaSuccess) status = ALPS_E_CUDA;
  if (!status)
    for (int i = 0; i <= nperp; ++i)
      for (int j = 0; j <= npar; ++j) {
        if (pperp_out) pperp_out[(size_t)i * (npar + 1) + j] = pp[i];
        if (ppar_out) ppar_out[(size_t)i * (npar + 1) + j] = pl[j];
      }
  cudaFree(d_gc);
  cudaFree(d_pc);
  cudaFree(d_f);
  cudaFree(d_w);
  cudaFree(d_pp);
  cudaFree(d_pl);
  cudaFree(d_g);
  cudaFree(d_out);
  cudaStreamDestroy(st);
  return status;
}

// ===========================================================================
// omega batch
// ===========================================================================
namespace {

struct RelArgs {
  SysDev sys;
  SpecDev sp[ALPS_MAX_SPECIES];
  int relcap;
};

// fit_function for the Gamma rows, fit types 4 and 5 (src/ALPS_analyt.f90:244-258)
__device__ inline double2 eval_fit_rel(const SpecDev& S, int ig, double2 p) {
  double2 ff = cmk(0.0, 0.0);
  const double g = S.grel[ig];
  const int nf = S.nf;
  for (int f = 0; f < nf; ++f) {
    const double* P = S.fit + (size_t)ig * 5 * nf + f;
    const double pc = S.perp_corr[f];
    if (S.fit_type[f] == 4) {
      ff = cadd(ff, cmk(P[0] * exp(-pc * g), 0.0));
    } else {
      double2 d = csub(p, cmk(P[2 * nf], 0.0));
      double2 d2 = cmul(d, d);
      ff = cadd(ff, cscale(cexp_d(cscale(d2, -P[nf])), P[0] * exp(-pc * g)));
    }
  }
  return ff;
}

// the reference's Lanczos Gamma (src/ALPS_fns_rel.f90:1738-1791)
__device__ inline double gamma_lanczos(double xx) {
  const double cof[6] = {76.18009173, -86.50532033, 24.01409822, -1.231739516, 0.120858003e-2, -0.536382e-5};
  double x = xx - 1.0;
  double tmp = x + 5.5;
  tmp = (x + 0.5) * log(tmp) - tmp;
  double ser = 1.0;
  for (int j = 0; j < 6; ++j) {
    x = x + 1.0;
    ser = ser + cof[j] / x;
  }
  return exp(tmp + log(2.50662827465 * ser));
}

// coefficients of CBESSJ's power series (src/ALPS_fns_rel.f90:1502-1553):
// coef[nu*21 + k] = 1 / (k! Gamma(nu + k + 1)), nu = 0 .. nmax + 1
__global__ void k_rel_coef(int nmax, double* coef) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (nmax + 2) * 21) return;
  const int nu = t / 21, k = t % 21;
  double fk = 1.0;
  for (int q = 2; q <= k; ++q) fk = fk * (1.0 * q);
  coef[t] = 1.0 / (fk * gamma_lanczos(1.0 * (nu + k + 1)));
}

// CBESSJ over (z/2)^nu: sum_k coef[k] q^k, q = -z^2/4
__device__ inline double2 cbessj_series(const double* coef, double2 q) {
  double2 s = cmk(coef[20], 0.0);
  for (int k = 19; k >= 0; --k) s = cmk(fma(s.x, q.x, fma(-s.y, q.y, coef[k])), fma(s.x, q.y, s.y * q.x));
  return s;
}

// x^n, n >= 0
__device__ inline double2 cpowi_d(double2 x, int n) {
  double2 pw = cmk(1.0, 0.0);
  for (unsigned u = (unsigned)n; u; u >>= 1) {
    if (u & 1) pw = cmul(pw, x);
    x = cmul(x, x);
  }
  return pw;
}

// The three Bessel products of int_T_res_rel (src/ALPS_fns_rel.f90:1374-1495)
// at complex momentum p: J^2, J'^2 pperpbar^2, J J' pperpbar of order n >= 0.
__device__ inline void res_products(const SpecDev& S, double zfac, int n, double g, double2 p, double2 F[3]) {
  const double2 pp = csqrt_d(csub(cmk(g * g - 1.0, 0.0), cmul(p, p)));
  const double2 z = cscale(pp, zfac), hz = cscale(z, 0.5);
  const double2 q = cscale(cmul(cneg(z), z), 0.25);
  double2 J, Jp;
  if (n == 0) {
    J = cbessj_series(S.relcoef, q);
    Jp = cneg(cmul(hz, cbessj_series(S.relcoef + 21, q)));
  } else {
    const double2 lo = cpowi_d(hz, n - 1), mid = cmul(lo, hz), up = cmul(mid, hz);
    J = cmul(mid, cbessj_series(S.relcoef + n * 21, q));
    Jp = cscale(csub(cmul(lo, cbessj_series(S.relcoef + (n - 1) * 21, q)),
                     cmul(up, cbessj_series(S.relcoef + (n + 1) * 21, q))),
                0.5);
  }
  const double2 b = cmul(Jp, pp);
  F[0] = cmul(J, J);
  F[1] = cmul(b, b);
  F[2] = cmul(J, b);
}

__device__ inline double fr_at(const SpecDev& S, int ig, int ip) {
  if (ip < 0 || ip > S.np || ig < 0 || ig > S.ng) return -1.0;
  return S.f0rel[(size_t)ig * (S.np + 1) + ip];
}

// funct_g_rel's node for a momentum (src/ALPS_fns_rel.f90:918-960): the last
// node k in 0..np-1 with pb[k] <= pp (-2 outside the grid) ...
__device__ inline int rel_piece(const SpecDev& S, double pp) {
  const int np = S.np;
  const double* pb = S.prel;
  if (!(pp >= pb[0] && pp < pb[np])) return -2;
  int k = (int)floor((pp - pb[0]) * ((double)np / (pb[np] - pb[0])));
  k = max(0, min(np - 1, k));
  while (k > 0 && pb[k] > pp) --k;
  while (k < np - 1 && pb[k + 1] <= pp) ++k;
  return k;
}
// ... moved inwards at the subluminal cone's edge and off the grid's ends
__device__ inline int rel_node(const SpecDev& S, int ig, int close, bool at_end) {
  const int np = S.np;
  if (fr_at(S, ig, close + 1) <= -1.0) close = close - 1;
  if (fr_at(S, ig, close - 1) <= -1.0) close = close + 1;
  if (at_end) close = np - 2;
  if (close >= (np - 1)) close = np - 2;
  if (close <= 1) close = 2;
  return close;
}

// one Gamma row's integration limits and resonance (integrate_resU_rel,
// src/ALPS_fns_rel.f90:516-660)
struct RelRow {
  double dR, dI;   // the pole
  double sm;       // spacing of the principal-value samples
  int i0, lo, up, i1;  // trapezoid over i0..lo and up..i1
  int ipres;
  int pv;          // the row has a principal-value window
};

__device__ RelRow rel_row(const SpecDev& S, const SysDev& sy, double2 om, int m, int ig, bool& err) {
  RelRow r;
  const double ms = S.ms, qs = S.qs, vA = sy.vA, kpar = sy.kpar;
  const int M_I = sy.M_I, np = S.np;
  const double* pb = S.prel;
  const double dpb = pb[2] - pb[1];
  const double g = S.grel[ig];
  // the resonance and its window decided as the reference rounds them (no FMA)
  const double x = __ddiv_rn(__dmul_rn(__dsub_rn(__dmul_rn(g, om.x), __ddiv_rn(__dmul_rn(1.0 * m, qs), ms)), vA), kpar);
  int ipres = 0;
  bool found = false;
  if (__dmul_rn(x, x) <= __dsub_rn(__dmul_rn(g, g), 1.0)) {
    // the ip in 1..np-2 with pb[ip] <= x < pb[ip+1]
    if (np - 2 >= 1 && pb[1] <= x && x < pb[np - 1]) {
      int k = 1 + (int)floor((x - pb[1]) / dpb);
      k = max(1, min(np - 2, k));
      while (k > 1 && pb[k] > x) --k;
      while (k < np - 2 && pb[k + 1] <= x) ++k;
      ipres = k;
      found = true;
    }
  }
  for (int ip = 0; ip <= M_I; ++ip) {
    if ((x >= __dsub_rn(pb[0], __dmul_rn(dpb, (double)ip))) && (x < __dsub_rn(pb[0], __dmul_rn(dpb, (double)(ip - 1))))) {
      ipres = -ip;
      found = true;
    }
    if ((x >= __dadd_rn(pb[np - 1], __dmul_rn(dpb, (double)ip))) &&
        (x < __dadd_rn(pb[np - 1], __dmul_rn(dpb, (double)(ip + 1))))) {
      ipres = np - 1 + ip;
      found = true;
    }
  }
  const int2 cn = S.cone[ig];
  const int lowerC = cn.x, upperC = cn.y;
  r.i0 = lowerC;
  if (found) {
    r.i1 = upperC;
    r.lo = ipres - M_I;
    r.up = ipres + M_I + 1;
    if ((ipres >= 0) && (ipres <= np))
      if (fabs(x - pb[ipres]) > (0.5 * dpb)) r.up = r.up + 1;
    if ((r.lo < lowerC) && (r.up > upperC)) {
      err = true;
      r.i0 = 1;  // nothing is summed
      r.lo = 0;
      r.up = 1;
      r.i1 = 0;
      found = false;
    } else if (r.lo <= lowerC) {
      r.i0 = 1;
      r.lo = 0;
      r.up = lowerC;
    } else if (r.up >= upperC) {
      r.lo = upperC;
      r.up = np;
      r.i1 = np - 1;
    }
  } else {
    r.lo = upperC;
    r.i1 = np - 1;
    r.up = np;
  }
  const double gx = ((om.x * g) * vA) / kpar;
  r.dI = ((om.y * g) * vA) / kpar;
  r.dR = gx - (1.0 * m) * (qs / ms) * vA / kpar;
  r.ipres = ipres;
  r.pv = (found && r.lo >= r.i0 && r.up <= r.i1) ? 1 : 0;
  r.sm = r.pv ? (r.dR - pb[ipres - M_I]) / (1.0 * sy.M_P) : 0.0;
  return r;
}

// A principal-value piece: the samples whose interpolant is that of node a
// (close), their weights' sum A and first moment B about the node
struct RelPiece {
  double2 A, B;
  int a;
};

#define REL_WARPS (REL_THREADS / 32)
#define REL_CHUNK 128  // samples a warp sums between two looks at the pieces' ends

#define REL_PRE_WORDS (3 * (REL_CHUNK + 1) + 1)  // even: the pieces after them are 16-byte aligned

// pieces of a row held at a time: both sides of the window and the tiny rest,
// for windows of more than REL_WIDE nodes to a side REL_PART of the former (the
// pieces' node weights add up, so a row may take them part by part)
#define REL_WIDE 128
#define REL_PART 256
__host__ __device__ inline int rel_max_pieces(int M_I) { return 2 * ((M_I < REL_WIDE ? M_I : REL_WIDE) + 4) + 8; }
// shared memory per warp in doubles: prefix sums of a chunk of samples, pieces
__host__ __device__ inline size_t rel_warp_words(int M_I) {
  return REL_PRE_WORDS + (size_t)rel_max_pieces(M_I) * (sizeof(RelPiece) / sizeof(double));
}

// sum of the 32 lanes before this one
__device__ inline double lanes_before(double v, int lane) {
  double s = v;
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  return s - v;
}

// Samples p_k, k = 0 .. K, of the principal-value sums, with the weights
// w_k / (dx - i dI), dx = p_k - dR, cut at given k's: for the lane's cut kc
// (first k beyond its piece) returns the sums over k < kc of w r dx, w r and
// w r dx^2, r = 1/(dx^2 + dI^2).  tiny: the rest beyond the symmetric window.
struct RelSums {
  double s1, s2, s3;
};
struct RelSamples {
  double dR, cap, sm, corr;
  int K;
  bool tiny;
  __device__ double at(int k) const {
    if (!tiny) return k == 0 ? dR : (k == K ? dR + cap : __dadd_rn(dR, __dmul_rn(sm, (double)k)));
    return k == 0 ? dR + cap : __dadd_rn(__dadd_rn(dR, cap), __dmul_rn(__dmul_rn(corr, sm), (double)k));
  }
};
__device__ RelSums rel_cut_sums(const RelSamples& q, double dI2, bool from0, int kc, double* pre, int lane) {
  RelSums out = {0.0, 0.0, 0.0}, carry = {0.0, 0.0, 0.0};
  for (unsigned k0 = 0; k0 <= (unsigned)q.K; k0 += REL_CHUNK) {
    const int n = (int)min((unsigned)REL_CHUNK, (unsigned)q.K + 1u - k0), per = (n + 31) / 32;
    const int b = min(n, lane * per), e = min(n, b + per);
    RelSums loc = {0.0, 0.0, 0.0};
    for (int j = b; j < e; ++j) {
      const int k = (int)k0 + j;
      pre[3 * j] = loc.s1;
      pre[3 * j + 1] = loc.s2;
      pre[3 * j + 2] = loc.s3;
      if (k == 0 && !from0) continue;
      const double dx = q.at(k) - q.dR;
      double r = rcp_fast(fma(dx, dx, dI2));
      r *= (k == 0 || k == q.K) ? 1.0 : 2.0;
      const double t = dx * r;
      loc.s1 += t;
      loc.s2 += r;
      loc.s3 = fma(dx, t, loc.s3);
    }
    const RelSums bef = {carry.s1 + lanes_before(loc.s1, lane), carry.s2 + lanes_before(loc.s2, lane),
                         carry.s3 + lanes_before(loc.s3, lane)};
    for (int j = b; j < e; ++j) {
      pre[3 * j] += bef.s1;
      pre[3 * j + 1] += bef.s2;
      pre[3 * j + 2] += bef.s3;
    }
    carry.s1 = __shfl_sync(0xffffffffu, bef.s1 + loc.s1, 31);
    carry.s2 = __shfl_sync(0xffffffffu, bef.s2 + loc.s2, 31);
    carry.s3 = __shfl_sync(0xffffffffu, bef.s3 + loc.s3, 31);
    __syncwarp();
    const int at = kc - (int)k0;
    if (at >= 0 && at < n) out = {pre[3 * at], pre[3 * at + 1], pre[3 * at + 2]};
    __syncwarp();
  }
  if (kc > q.K) out = carry;
  return out;
}

// The pieces of one row's principal-value sum (principal_integral_rel,
// src/ALPS_fns_rel.f90:724-913), by a warp.  A sample's interpolant is that
// of one node and linear in p, so each piece needs only the sums of its
// samples' weights and of their first moments; the samples are summed once,
// as prefix sums, for both sides of the window, and each lane cuts them at
// the ends of its piece.  Returns the number of pieces left in rec.  WIDE: those
// of one part; more: there are further parts.
template <bool WIDE>
__device__ int rel_pieces(const SpecDev& S, const SysDev& sy, const RelRow& r, int ig, int part, double* pre,
                          RelPiece* rec, int lane, bool& more) {
  const double* pb = S.prel;
  const int np = S.np, M_P = sy.M_P;
  const double dpb = pb[2] - pb[1];
  const double dR = r.dR, dI = r.dI, dI2 = dI * dI;
  const double cap = dR - pb[r.ipres - sy.M_I], sm = r.sm;
  const bool sym = fabs(dI) > sy.Tlim;
  const int cap_rec = rel_max_pieces(sy.M_I);
  int nrec = 0;
  RelSamples q = {dR, cap, sm, 1.0, M_P, false};
  more = false;
  if (sym) {
    const int jc = rel_piece(S, dR);  // the pole's own interval (the window lies inside the grid)
    const int nu = max(0, rel_piece(S, dR + cap) - jc) + 1, nd = max(0, jc - rel_piece(S, 2.0 * dR - (dR + cap))) + 1;
    const int first = WIDE ? part * REL_PART : 0, last = min(nu + nd, WIDE ? first + REL_PART : cap_rec);
    for (int t0 = first; t0 < last; t0 += 32) {
      const int t = t0 + lane;
      const bool has = t < last, down = t >= nu;
      const int i = down ? t - nu : t, j = down ? jc - i : jc + i;
      // first sample beyond the piece: up p_k >= pb[j+1], down 2 dR - p_k < pb[j]
      int kc = M_P + 1;
      if (has && i + 1 < (down ? nd : nu)) {
        const double edge = down ? pb[j] : pb[j + 1];
        auto beyond = [&](int k) { return down ? 2.0 * dR - q.at(k) < edge : q.at(k) >= edge; };
        int k = (int)ceil((down ? dR - edge : edge - dR) / sm);
        k = max(0, min(M_P + 1, k));
        while (k > 0 && beyond(k - 1)) --k;
        while (k <= M_P && !beyond(k)) ++k;
        kc = k;
      }
      const RelSums end = rel_cut_sums(q, dI2, true, kc, pre, lane);
      // less the sums of the piece before (the lane before; a later round of
      // 32 pieces starts from its own cut)
      RelSums beg;
      beg.s1 = __shfl_up_sync(0xffffffffu, end.s1, 1);
      beg.s2 = __shfl_up_sync(0xffffffffu, end.s2, 1);
      beg.s3 = __shfl_up_sync(0xffffffffu, end.s3, 1);
      if (i == 0) beg = {0.0, 0.0, 0.0};
      if (t0 > 0 && __any_sync(0xffffffffu, has && lane == 0 && i > 0)) {
        // the cut at this lane's piece's beginning
        int kb = 0;
        if (lane == 0) {
          const double edge = down ? pb[j + 1] : pb[j];
          auto beyond = [&](int k) { return down ? 2.0 * dR - q.at(k) < edge : q.at(k) >= edge; };
          int k = (int)ceil((down ? dR - edge : edge - dR) / sm);
          k = max(0, min(M_P + 1, k));
          while (k > 0 && beyond(k - 1)) --k;
          while (k <= M_P && !beyond(k)) ++k;
          kb = k;
        }
        const RelSums b0 = rel_cut_sums(q, dI2, true, kb, pre, lane);
        if (lane == 0) beg = b0;
      }
      if (has) {
        const double s1 = end.s1 - beg.s1, s2 = (end.s2 - beg.s2) * dI, s3 = end.s3 - beg.s3;
        const int a = rel_node(S, ig, j, false);
        const double del = dR - pb[a];
        RelPiece pc;
        pc.a = a;
        // up: w/(dx - i dI) = w r (dx + i dI); down: -w/(dx + i dI) at -dx
        pc.A = down ? cmk(-s1, s2) : cmk(s1, s2);
        pc.B = cmk(fma(del, pc.A.x, s3), fma(del, pc.A.y, down ? -dI * s1 : dI * s1));
        rec[t - first] = pc;
      }
    }
    nrec = last - first;
    if (WIDE && last < nu + nd) {
      more = true;
      __syncwarp();
      return nrec;
    }
  } else {
    // g' sum_k w_k dx^2/(dx^2 + dI^2), and +- i pi G(p_res)/smdelta
    const RelSums s = rel_cut_sums(q, dI2, false, M_P + 1, pre, lane);
    if (lane < 3) {
      const double p = lane == 0 ? dR + dpb : (lane == 1 ? dR - dpb : dR);
      const int a = rel_node(S, ig, rel_piece(S, p), p == pb[np]);
      RelPiece pc;
      pc.a = a;
      const double c = s.s3 / dpb;
      if (lane < 2) pc.A = cmk(lane == 0 ? c : -c, 0.0);
      else pc.A = cmk(0.0, dI > 0.0 ? 2.0 * ALPS_PI / sm : (dI < 0.0 ? -2.0 * ALPS_PI / sm : 0.0));
      pc.B = cscale(pc.A, p - pb[a]);
      rec[lane] = pc;
    }
    nrec = 3;
  }
  // the tiny rest between dR + capDelta and the upper limit
  const int ntiny = rest_samples((pb[r.up] - dR - cap) / sm);
  if (ntiny > 0) {
    q.corr = ((pb[r.up] - dR - cap) / (1.0 * ntiny)) / sm;
    q.K = ntiny;
    q.tiny = true;
    const int jc = rel_piece(S, q.at(0)), nu = min(4, max(0, rel_piece(S, q.at(ntiny)) - jc) + 1);
    int kc = ntiny + 1;
    if (lane + 1 < nu) {
      const double edge = pb[jc + lane + 1];
      int k = (int)ceil((edge - q.at(0)) / (q.corr * sm));
      k = max(0, min(ntiny + 1, k));
      while (k > 0 && q.at(k - 1) >= edge) --k;
      while (k <= ntiny && q.at(k) < edge) ++k;
      kc = k;
    }
    const RelSums end = rel_cut_sums(q, dI2, true, kc, pre, lane);
    RelSums beg;
    beg.s1 = __shfl_up_sync(0xffffffffu, end.s1, 1);
    beg.s2 = __shfl_up_sync(0xffffffffu, end.s2, 1);
    beg.s3 = __shfl_up_sync(0xffffffffu, end.s3, 1);
    if (lane == 0) beg = {0.0, 0.0, 0.0};
    if (lane < nu && nrec + lane < cap_rec) {
      const double s1 = (end.s1 - beg.s1) * q.corr, s2 = (end.s2 - beg.s2) * q.corr * dI, s3 = (end.s3 - beg.s3) * q.corr;
      const int j = jc + lane, a = rel_node(S, ig, j, q.at(ntiny) == pb[np] && lane == nu - 1);
      const double del = dR - pb[a];
      RelPiece pc;
      pc.a = a;
      pc.A = cmk(s1, s2);
      pc.B = cmk(fma(del, s1, s3), fma(del, s2, dI * s1));
      rec[nrec + lane] = pc;
    }
    nrec = min(nrec + nu, cap_rec);
  }
  __syncwarp();
  return nrec;
}

// sum of 12 doubles per thread over the block's threads, in warp order; the
// total on thread q < 12
__device__ double block_sum12(double v[12], double* sh /* [REL_WARPS][12] */) {
#pragma unroll
  for (int q = 0; q < 12; ++q)
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 12; ++q)
    if (lane == q) sh[warp * 12 + q] = v[q];
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 12)
    for (int k = 0; k < REL_WARPS; ++k) t += sh[k * 12 + threadIdx.x];
  return t;
}

// determine_resonances, relativistic branch (src/ALPS_fns.f90:680-702): is
// there a node (i, j) with ppar_j <= p_res(gamma_ij) < ppar_j+1?  An FP32
// estimate (error below eps) settles all nodes but those near an interval's
// ends, where the reference's own rounding decides.
__device__ bool rel_resonant(const SpecDev& S, const SysDev& sy, double2 om, int m) {
  const double ms = S.ms, qs = S.qs, vA = sy.vA, kpar = sy.kpar;
  const int N = S.N, M = S.M;
  const float a1 = (float)(ms * om.x / kpar), a2 = (float)((1.0 * m) * qs / kpar);
  const float dp = (float)(S.ppar[2] - S.ppar[1]);
  const float pmax = fmaxf(fabsf((float)S.ppar[0]), fabsf((float)S.ppar[M]));
  const int tcols = min(M, (int)blockDim.x), rows = max(1, (int)blockDim.x / tcols);
  const int c0 = (int)threadIdx.x % tcols, r0 = (int)threadIdx.x / tcols;
  bool res = false;
  if (r0 < rows)
    for (int j = c0; j < M && !res; j += tcols) {
      const float pj = (float)S.ppar[j];
      for (int i = r0; i <= N; i += rows) {
        const float ga = S.relgf[(size_t)i * (M + 1) + j] * a1;
        const float d = (ga - a2) - pj;
        const float eps = 1.0e-6f * (fabsf(ga) + fabsf(a2) + pmax);
        if (d < -eps || d > dp + eps) continue;
        if (d > eps && d < dp - eps) {
          res = true;
          break;
        }
        const double p1 = S.pperp[i], p2 = S.ppar[j];
        const double gamma = __dsqrt_rn(__dadd_rn(
            __ddiv_rn(__dmul_rn(__dadd_rn(__dmul_rn(p1, p1), __dmul_rn(p2, p2)), __dmul_rn(vA, vA)), __dmul_rn(ms, ms)),
            1.0));
        const double pr = __ddiv_rn(__dsub_rn(__dmul_rn(__dmul_rn(gamma, ms), om.x), __dmul_rn(1.0 * m, qs)), kpar);
        if ((S.ppar[j] <= pr) && (S.ppar[j + 1] > pr)) {
          res = true;
          break;
        }
      }
    }
  return __syncthreads_or(res) != 0;
}

// REL_RB blocks per (omega, species, signed order): each takes every
// REL_RB-th Gamma row, or every REL_RB-th row of the regular grid, and writes
// its partial sums to its own slot; k_finalize adds the slots in order.
//
// Bound by the FP64 pipe (two lanes a clock and SM), so the work is laid out
// to spend few operations per node.  The T-tensor's Bessel products come from
// tables (k_rel_families; both signs of an order share them), its constant
// factors, Kc and the derivative's omega are applied once, and a node costs
// one real reciprocal and 30 operations where six complex divisions took 330.
// A principal-value sample costs 10 (see rel_pieces) where two interpolants
// of six entries over three nodes took 1500, and the window then is a few
// more nodes with complex weights.  Rows' decisions are taken a row per lane,
// and so are the Landau rows, by one warp beside the others.
// 8 frequencies, 41 signed orders, 100x200 (Gamma, pparbar): 5340 us before,
// 304 us so.  WIDE: windows of more than REL_WIDE nodes to a side (a loop over
// the parts costs the others 7 us of those).
template <bool WIDE>
__global__ void __launch_bounds__(REL_THREADS) k_rel_orders(RelArgs a, const double2* __restrict__ om, int n_om,
                                                            double2* __restrict__ out, int* flags) {
  extern __shared__ __align__(16) double rel_smem[];
  __shared__ double sh[REL_WARPS * 12];
  __shared__ RelRow rows[32];
  const int w = blockIdx.x, s = blockIdx.z;
  const int rb = blockIdx.y % REL_RB, ord = blockIdx.y / REL_RB;
  const int n = ord >> 1, sg = ord & 1;
  const SpecDev& S = a.sp[s];
  if (w >= n_om || !S.relat || n > S.nmax || n >= a.relcap || (n == 0 && sg == 1)) return;
  const SysDev& sy = a.sys;
  const int m = sg ? -n : n;
  const double2 o = om[w];
  const double ms = S.ms, qs = S.qs, vA = sy.vA, kpar = sy.kpar, kperp = sy.kperp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool kn = sy.kperp_norm != 0;
  const double kf = kn ? 1.0 : kperp, kf2 = kn ? 1.0 : kperp * kperp;
  double2 acc[6];  // sums of the entries xx yy zz xy xz yz without their constant factors
#pragma unroll
  for (int e = 0; e < 6; ++e) acc[e] = cmk(0.0, 0.0);
  double2* dst = out + (((((size_t)w * sy.nspec + s) * a.relcap + n) * 2 + sg) * REL_RB + rb) * 6;
  double v[12];
  auto pack = [&](const double2* x) {
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      v[2 * e] = x[e].x;
      v[2 * e + 1] = x[e].y;
    }
  };
  if (!rel_resonant(S, sy, o, m)) {
    // integrate with the Lorentz factor in resU (src/ALPS_fns.f90:799-864,
    // 1560-1596), rows 1..N-1 (a warp each) and columns 1..M-1
    const int N = S.N, M = S.M, L = M + 1;
    const double z = kn ? kperp / qs : 1.0 / qs;
    const double mox = ms * o.x, moy = ms * o.y, mq = (1.0 * m) * qs, kom = kpar / ms;
    const size_t fs = (size_t)(S.nmax + 1) * (N - 1);
    for (int i = 1 + rb + REL_RB * warp; i <= N - 1; i += REL_RB * REL_WARPS) {
      double2 s0 = cmk(0.0, 0.0), s1 = s0, s2 = s0;
      for (int j = 1 + lane; j <= M - 1; j += 32) {
        const size_t k = (size_t)i * L + j;
        const double p2 = S.ppar[j], ga = S.relgam[k];
        const double wj = (j == 1 || j == M - 1) ? 1.0 : 2.0;
        // num = omega g1 + kpar/(gamma m) g2, den = gamma m omega - kpar p - m q
        const double2 num = cmk(fma(o.x, S.g1[k], kom * S.relg2g[k]), o.y * S.g1[k]);
        const double dx = fma(ga, mox, -fma(kpar, p2, mq)), dy = ga * moy;
        const double r = wj * rcp_fast(fma(dx, dx, dy * dy));
        const double2 t = cmul(num, cmk(dx * r, -dy * r));
        const double2 tp = cscale(t, p2);
        s0 = cadd(s0, t);
        s1 = cadd(s1, tp);
        s2 = cmk(fma(tp.x, p2, s2.x), fma(tp.y, p2, s2.y));
      }
      // the row's Bessel products with its p_perp weight
      const double* R = S.Rw + (size_t)n * (N - 1) + (i - 1);
      const double f0 = R[0], f1 = R[fs], f2 = R[2 * fs];
      auto add = [&](int e, double f, double2 x) { acc[e] = cmk(fma(f, x.x, acc[e].x), fma(f, x.y, acc[e].y)); };
      add(0, f0, s0);
      add(1, f1, s0);
      add(2, f0, s2);
      add(3, f2, s0);
      add(4, f0, s1);
      add(5, f2, s1);
    }
    pack(acc);
    const double t = block_sum12(v, sh);
    if (threadIdx.x < 12) {
      const int e = threadIdx.x >> 1;
      const double pf[6] = {1.0 * (m * m) / (z * z), kf2, kf2, kf * (1.0 * m) / z, kf * (1.0 * m) / z, kf2};
      const double x = t * (qs * pf[e] * (2.0 * ALPS_PI * S.dpperp * S.dppar_abs * 0.25));
      // i for xy, -i for yz
      const int c = threadIdx.x & 1;
      double* d = reinterpret_cast<double*>(dst);
      if (e == 3) d[threadIdx.x ^ 1] = c ? -x : x;
      else if (e == 5) d[threadIdx.x ^ 1] = c ? x : -x;
      else d[threadIdx.x] = x;
    }
    return;
  }
  // integrate_res_rel + landau_integrate_rel over the Gamma rows
  const int np = S.np, ng = S.ng;
  const double* pb = S.prel;
  const double dpb = pb[2] - pb[1], dg = S.grel[2] - S.grel[1], kva = kpar / vA;
  const size_t plane = (size_t)(ng + 1) * (np + 1);
  const double* fam = S.relfam + (size_t)n * 3 * plane;
  const double lw = (o.y > 0.0) ? 0.0 : ((o.y < 0.0) ? 2.0 : 1.0);
  double* wsm = rel_smem + warp * rel_warp_words(sy.M_I);
  RelPiece* rec = reinterpret_cast<RelPiece*>(wsm + REL_PRE_WORDS);
  double2 lacc[6];
#pragma unroll
  for (int e = 0; e < 6; ++e) lacc[e] = cmk(0.0, 0.0);
  bool err = false;
  // adds node ip of row ig with complex weight R: A R F_e, A = omega df/dGamma
  // + (kpar/vA) df/dpparbar
  auto node = [&](int ig, int ip, double2 R) {
    const size_t k = (size_t)ig * (np + 1) + ip;
    const double d1 = S.dfr1[k];
    const double2 t = cmul(cmk(fma(o.x, d1, kva * S.dfr2[k]), o.y * d1), R);
    const double p = pb[ip], f0 = fam[k], f1 = fam[plane + k], f2 = fam[2 * plane + k], f0p = f0 * p;
    auto add = [&](int e, double f) { acc[e] = cmk(fma(f, t.x, acc[e].x), fma(f, t.y, acc[e].y)); };
    add(0, f0);
    add(1, f1);
    add(2, f0p * p);
    add(3, f2);
    add(4, f0p);
    add(5, f2 * p);
  };
  const int nrow = (ng - 1 - rb + REL_RB - 1) / REL_RB;  // rows 1 + rb + REL_RB r of this block
  // the last warp takes the Landau rows where there are any
  const int rwarps = lw != 0.0 ? REL_WARPS - 1 : REL_WARPS;
  for (int r0 = 0; r0 < nrow; r0 += 32) {
    const int nr = min(32, nrow - r0);
    __syncthreads();
    if (warp == 0 && lane < nr) rows[lane] = rel_row(S, sy, o, m, 1 + rb + REL_RB * (r0 + lane), err);
    __syncthreads();
    if (warp < rwarps) {
      for (int q = warp; q < nr; q += rwarps) {
        const int ig = 1 + rb + REL_RB * (r0 + q);
        const RelRow r = rows[q];
        const double wr = (ig <= ng - 2) ? 2.0 : 1.0, dI2 = r.dI * r.dI;
        // trapezoid over the nodes away from the pole; a range's two ends
        // weigh 1 (once if they coincide), the others 2
        for (int h = 0; h < 2; ++h) {
          const int b = h ? r.up : r.i0, e = h ? r.i1 : r.lo;
          for (int ip = b + lane; ip <= e; ip += 32) {
            const double dx = pb[ip] - r.dR;
            double x = wr * dpb * rcp_fast(fma(dx, dx, dI2));
            if (ip != b && ip != e) x *= 2.0;
            node(ig, ip, cmk(dx * x, r.dI * x));
          }
        }
        bool more = r.pv;
        for (int part = 0; more; ++part) {
          const int nrec = rel_pieces<WIDE>(S, sy, r, ig, part, wsm, rec, lane, more);
          more = WIDE && more;
          int a0 = np, a1 = 0;
          for (int t = lane; t < nrec; t += 32) {
            a0 = min(a0, rec[t].a);
            a1 = max(a1, rec[t].a);
          }
          a0 = __reduce_min_sync(0xffffffffu, a0);
          a1 = __reduce_max_sync(0xffffffffu, a1);
          // G = h(a) + (h(a+1) - h(a-1)) (p - pb[a]) / (2 dpb)
          const double hs = 0.5 / dpb, sc = wr * r.sm;
          for (int ip = a0 - 1 + lane; ip <= a1 + 1; ip += 32) {
            double2 W = cmk(0.0, 0.0);
            bool used = false;
            for (int t = 0; t < nrec; ++t) {
              const int d = ip - rec[t].a;
              if (d < -1 || d > 1) continue;
              used = true;
              if (d == 0) W = cadd(W, rec[t].A);
              else W = cadd(W, cscale(rec[t].B, d * hs));
            }
            if (used) node(ig, ip, cscale(W, sc));
          }
          __syncwarp();
        }
      }
    } else if (lane < nr) {
      // landau_integrate_rel (src/ALPS_fns_rel.f90:1005-1092), a row per lane
      const int ig = 1 + rb + REL_RB * (r0 + lane);
      const double g = S.grel[ig];
      double2 pr = cscale(cscale(o, g), vA);
      pr = cmk(pr.x / kpar - (1.0 * m) * qs * vA / (kpar * ms), pr.y / kpar);
      // inside the subluminal cone, decided as the reference rounds it (no FMA)
      if (__dmul_rn(pr.x, pr.x) <= __dsub_rn(__dmul_rn(g, g), 1.0)) {
        const double h = (ig == ng - 1) ? 0.5 : 1.0;
        const double2 dfg = ig == 1 ? cscale(csub(eval_fit_rel(S, ig + 1, pr), eval_fit_rel(S, ig, pr)), 1.0 / dg)
                                    : cscale(csub(eval_fit_rel(S, ig + 1, pr), eval_fit_rel(S, ig - 1, pr)), 0.5 / dg);
        const double2 dfp = cscale(csub(eval_fit_rel(S, ig, cadd(pr, cmk(dpb, 0.0))),
                                        eval_fit_rel(S, ig, csub(pr, cmk(dpb, 0.0)))),
                                   0.5 / dpb);
        const double2 coef = cscale(cadd(cmul(o, dfg), cscale(dfp, kva)), -h);
        double2 F[3];
        res_products(S, kperp * ms / (vA * qs), n, g, pr, F);
        const double2 c0 = cmul(coef, F[0]), c2 = cmul(coef, F[2]), c0p = cmul(c0, pr);
        lacc[0] = cadd(lacc[0], c0);
        lacc[1] = cadd(lacc[1], cmul(coef, F[1]));
        lacc[2] = cadd(lacc[2], cmul(c0p, pr));
        lacc[3] = cadd(lacc[3], c2);
        lacc[4] = cadd(lacc[4], c0p);
        lacc[5] = cadd(lacc[5], cmul(c2, pr));
      }
    }
  }
  if (err) atomicOr(flags, 2);
  pack(acc);
  const double tr = block_sum12(v, sh);
  double tl = 0.0;
  if (lw != 0.0) {
    pack(lacc);
    tl = block_sum12(v, sh);
  }
  if (warp == 0) {
    // Kc = -2 pi (ms/vA)^3 q vA / (kpar m); the Landau sums carry i f lw
    const double zbar = kn ? kperp * ms / (vA * qs) : ms / (vA * qs);
    const double qv = qs * vA / (kpar * ms);
    const double Kc = -2.0 * ALPS_PI * cube(ms / vA) * qv;
    const double f = dg * ALPS_PI * 2.0 * ALPS_PI * qv * cube(ms / vA) * lw;
    const double to = __shfl_xor_sync(0xffffffffu, tl, 1);  // the other component
    if (lane < 12) {
      const int e = lane >> 1, c = lane & 1;
      const double pf[6] = {1.0 * (m * m) / (zbar * zbar), kf2, kf2, (1.0 * m) * kf / zbar, (1.0 * m) * kf / zbar, kf2};
      // i l: (-y, x)
      const double x = pf[e] * fma(tr, Kc * dg * 0.25, (c ? to : -to) * f);
      double* d = reinterpret_cast<double*>(dst);
      if (e == 3) d[lane ^ 1] = c ? -x : x;
      else if (e == 5) d[lane ^ 1] = c ? x : -x;
      else d[lane] = x;
    }
  }
}

}  // namespace

int launch_rel_bessel(alps_ctx* c, int is, double kperp) {
  SpeciesHost& S = c->spec[is];
  const int ng = c->sys.ngamma, np = c->sys.npparbar, nmax = S.nmax, nrows = nmax + 2;
  const size_t plane = (size_t)(ng + 1) * (np + 1), nj = plane * nrows, nfam = plane * 3 * (nmax + 1);
  // J_0 .. J_nmax+1, then the Bessel products, then the series coefficients
  const size_t need = nj + nfam + (size_t)nrows * 21;
  if (need > S.jrel_cap || !S.d_jrel) {
    if (S.d_jrel) cudaFree(S.d_jrel);
    S.d_jrel = nullptr;
    ALPS_CUDA_TRY(cudaMalloc(&S.d_jrel, need * sizeof(double)));
    S.jrel_cap = need;
  }
  S.d_relfam = S.d_jrel + nj;
  S.d_relcoef = S.d_relfam + nfam;
  double zfac = kperp * S.sp.ms / (c->sys.vA * S.sp.qs);
  k_rel_jtab<<<(unsigned)((nj + 127) / 128), 128, 0, c->stream>>>(S.d_grel, S.d_prel, ng, np, nrows, zfac, S.d_jrel);
  k_rel_families<<<(unsigned)((plane * (nmax + 1) + 127) / 128), 128, 0, c->stream>>>(S.d_jrel, S.d_grel, S.d_prel, ng,
                                                                                     np, nmax, S.d_relfam);
  k_rel_coef<<<(nrows * 21 + 127) / 128, 128, 0, c->stream>>>(nmax, S.d_relcoef);
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}

int launch_rel_orders(const SysDev& sys, const SpecDev* sp, int relcap, int n, const double2* d_om, double2* d_out,
                      int* d_flags, cudaStream_t st) {
  RelArgs a;
  a.sys = sys;
  bool any = false;
  for (int s = 0; s < sys.nspec; ++s) {
    a.sp[s] = sp[s];
    any = any || sp[s].relat;
  }
  a.relcap = relcap;
  if (!any || n <= 0) return ALPS_OK;
  const size_t smem = REL_WARPS * rel_warp_words(sys.M_I) * sizeof(double);
  auto kernel = sys.M_I > REL_WIDE ? k_rel_orders<true> : k_rel_orders<false>;
  if (smem > 40 * 1024)
    ALPS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<dim3(n, 2 * relcap * REL_RB, sys.nspec), REL_THREADS, smem, st>>>(a, d_om, n, d_out, d_flags);
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}
