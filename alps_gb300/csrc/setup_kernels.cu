// setup_kernels.cu -- per-run and per-wavevector device preprocessing.
//
//   k_derivatives     derivative_f0 (src/ALPS_fns.f90:103-115), plus the
//                     second RHS vector pperp*df/dppar - ppar*df/dpperp of resU
//   k_int_ee          int_ee (src/ALPS_fns.f90:1457-1555)
//   k_lm_fit          determine_param_fit + LM_nonlinear_fit
//                     (src/ALPS_analyt.f90:365-728, 1183-1636)
//   k_nmax            determine_nmax (src/ALPS_fns.f90:3971-4075)
//   k_bessel_table    determine_bessel_array (src/ALPS_fns.f90:4214-4255)
//   k_bessel_rows     weighted Bessel-product rows of the p_perp contraction
//   k_dgemm           FP64 tiled GEMM for the contraction
//   k_fold_reduced    reduced vectors V[n][j][12] of the omega pass
#include <cooperative_groups.h>

#include <cmath>
#include <cstring>
#include <cstdio>

#include "alps_internal.cuh"
#include "tc_gemm.cuh"
#include "device_math.cuh"

namespace {

__global__ void k_derivatives(const double* __restrict__ f0, const double* __restrict__ pperp,
                              const double* __restrict__ ppar, int N, int M, double* g1, double* g2,
                              double* G) {
  int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int i = blockIdx.y + 1;
  if (i > N - 1 || j > M - 1) return;
  int L = M + 1;
  double df1 = __ddiv_rn(__dsub_rn(f0[(i + 1) * L + j], f0[(i - 1) * L + j]),
                         __dsub_rn(pperp[i + 1], pperp[i - 1]));
  double df2 = __ddiv_rn(__dsub_rn(f0[i * L + j + 1], f0[i * L + j - 1]),
                         __dsub_rn(ppar[j + 1], ppar[j - 1]));
  double gg2 = __dsub_rn(__dmul_rn(pperp[i], df2), __dmul_rn(ppar[j], df1));
  g1[i * L + j] = df1;
  g2[i * L + j] = gg2;
  // contraction RHS, row-major [(i-1)][g*(M-1) + (j-1)]
  size_t row = (size_t)(i - 1) * 2 * (M - 1);
  G[row + (j - 1)] = df1;
  G[row + (M - 1) + (j - 1)] = gg2;
}

// ee term; weights w_perp(i) * w_par(j) of the reference's trapezoid.  Bound by
// the FP64 pipe of the SMs that take part: a cluster of eight blocks, rows over
// the warps, the blocks' sums through distributed shared memory (192x384 grid:
// 116 us in one block, 15 us so).
#define EE_BLOCKS 8
__global__ void __cluster_dims__(EE_BLOCKS, 1, 1) __launch_bounds__(256)
    k_int_ee(const double* __restrict__ g2, const double* __restrict__ ppar, int N, int M, double scale, double* out) {
  __shared__ double red[8];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, L = M + 1;
  double acc = 0.0;
  for (int i = 1 + (int)cl.block_rank() * 8 + warp; i <= N - 1; i += EE_BLOCKS * 8) {
    const double* row = g2 + (size_t)i * L;
    double r = 0.0;
    for (int j = 1 + lane; j <= M - 1; j += 32) {
      const double x = ppar[j] * row[j];
      r += (j == 1 || j == M - 1) ? x : x + x;
    }
    acc += (i <= N - 2) ? r + r : r;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[warp] = acc;
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x == 0) {
    double t = 0.0;
    for (unsigned b = 0; b < EE_BLOCKS; ++b) {
      const double* p = cl.map_shared_rank(red, b);
      for (int w = 0; w < 8; ++w) t += p[w];
    }
    *out = t * scale;
  }
  cl.sync();  // the other blocks' sums stay until they are read
}

// ---------------------------------------------------------------------------
// Levenberg-Marquardt fit of the analytic continuation.  One block walks the
// iperp rows of one species in order (each row starts from the previous
// result, src/ALPS_analyt.f90:518); within a row the threads share the
// points, the warps the entries of J^T J, and one warp solves.  Bound by the
// FP64 pipe of one SM (16 clocks an instruction of any warp): the table's
// logarithms come from the whole chip (k_fit_logs), one warp prepares what all
// need of the parameters, and four warps share what each repeats; one
// Maxwellian in log space takes its normal equations from seven sums of the
// residual pass, and its three unknowns in registers.  193 rows of 385 points,
// one Maxwellian: 3690 us before, 2840 us so (28 thousand clocks a row).
// ---------------------------------------------------------------------------
struct FitArgs {
  int N, M, nf, log_fit;
  int fit_type[ALPS_MAX_FITS];
  double pc[ALPS_MAX_FITS];
  double ms, vA;
  int maxsteps;
  double lambda0, lambdafac, eps;
  // relativistic species: rows of the (Gamma, pparbar) grid
  int rel, ng, np;
  const double* flog;   // log f0 [(N+1)*(M+1)], log fits of a non-relativistic species
  const double* f0rel;  // [(ng+1)*(np+1)]
  const double* grel;   // [ng+1]
  const double* prel;   // [np+1]
};

__device__ int fit_nparams(const FitArgs& a, int t) {
  return (t == 1 || t == 3 || t == 5) ? 3 : (t == 2 ? 5 : (t == 6 ? 4 : 1));
}

// fit_function (src/ALPS_analyt.f90:185-266) at real ppar
__device__ double fit_value_real(const FitArgs& a, const double* params, double pperp, double ppar) {
  double ff = 0.0;
  int par_ind = 0;
  for (int ifit = 1; ifit <= a.nf; ++ifit) {
    int t = a.fit_type[ifit - 1];
    double pc = a.pc[ifit - 1];
    const double* p = params + (ifit + par_ind) - 1;
    double d = ppar - p[2];
    if (t == 1) {
      ff = ff + (p[0] * exp(-pc * (pperp * pperp))) * exp(-p[1] * (d * d));
      par_ind += 2;
    } else if (t == 2) {
      double kp = 1.0 + p[1] * (d * d) + pc * p[4] * (pperp * pperp);
      ff = ff + p[0] * exp(p[3] * log(kp));
      par_ind += 4;
    } else if (t == 3) {
      double sq = sqrt(1.0 + ((pperp * pperp) + d * d) * a.vA * a.vA / (a.ms * a.ms));
      ff = ff + p[0] * exp(-p[1] * sq);
      par_ind += 2;
    } else if (t == 4) {
      ff = ff + p[0] * exp(-pc * pperp);
    } else if (t == 5) {
      ff = ff + p[0] * exp(-pc * pperp) * exp(-p[1] * (d * d));
      par_ind += 2;
    } else if (t == 6) {
      double q = p[3] * pc * (pperp * pperp) + p[1] * (d * d);
      ff = ff + p[0] * exp(0.5 * (q - exp(q)));
      par_ind += 3;
    }
  }
  return ff;
}

// determine_JT (src/ALPS_analyt.f90:1183-1389) for one ppar node
__device__ void fit_jacobian(const FitArgs& a, const double* params, int iperp, double pperp, double ppar,
                             double* J /* nJT */) {
  int par_ind = 0, JT_ind = 0;
  for (int ifit = 1; ifit <= a.nf; ++ifit) {
    int t = a.fit_type[ifit - 1];
    double pc = a.pc[ifit - 1];
    const double* p = params + (ifit + par_ind) - 1;
    double* Jp = J + (ifit + JT_ind) - 1;
    double d = ppar - p[2];
    if (t == 1) {
      double e = exp(-p[1] * (d * d) - pc * (pperp * pperp));
      Jp[0] = e;
      Jp[1] = -((d * d)) * p[0] * e;
      Jp[2] = 2.0 * p[1] * d * p[0] * e;
      par_ind += 2;
      JT_ind += 2;
    } else if (t == 2) {
      double kp = 1.0 + p[1] * (d * d) + pc * p[4] * (pperp * pperp);
      double kpm = pow(kp, p[3] - 1.0);
      Jp[0] = pow(kp, p[3]);
      Jp[1] = p[0] * p[3] * kpm * (d * d);
      Jp[2] = p[0] * p[3] * kpm * 2.0 * p[1] * (p[2] - ppar);
      Jp[3] = log(kp) * p[0] * pow(kp, p[3]);
      if (iperp == 0) {
        JT_ind += 3;
      } else {
        Jp[4] = p[0] * p[3] * kpm * pc * (pperp * pperp);
        JT_ind += 4;
      }
      par_ind += 4;
    } else if (t == 3) {
      double sq = sqrt(1.0 + ((pperp * pperp) + d * d) * a.vA * a.vA / (a.ms * a.ms));
      Jp[0] = exp(-p[1] * sq);
      Jp[1] = -p[0] * exp(-p[1] * sq) * sq;
      Jp[2] = p[0] * exp(-p[1] * sq) * (p[1] / sq) * d * a.vA * a.vA / (a.ms * a.ms);
      par_ind += 2;
      JT_ind += 2;
    } else if (t == 4) {
      Jp[0] = exp(-pc * pperp);
    } else if (t == 5) {
      double e = exp(-p[1] * (d * d)) * exp(-pc * pperp);
      Jp[0] = e;
      Jp[1] = -p[0] * e * (d * d);
      Jp[2] = 2.0 * p[0] * d * p[1] * e;
      par_ind += 2;
      JT_ind += 2;
    } else if (t == 6) {
      double q = p[3] * pc * (pperp * pperp) + p[1] * (d * d);
      double e = exp(0.5 * (q - exp(q)));
      Jp[0] = e;
      Jp[1] = p[0] * e * 0.5 * (d * d) * (1.0 - exp(q));
      Jp[2] = p[0] * e * p[1] * (p[2] - ppar) * (1.0 - exp(q));
      if (iperp == 0) {
        JT_ind += 2;
      } else {
        Jp[3] = p[0] * e * 0.5 * pc * (pperp * pperp) * (1.0 - exp(q));
        JT_ind += 3;
      }
      par_ind += 3;
    }
  }
}

#define FIT_MAXP (5 * ALPS_MAX_FITS)

// One species' fit: fit[(i*5+ip)*nf + ifit] holds the seeds at row 0 on
// entry and the fitted rows on exit.  Rows are the iperp rows of the f0
// table, or for a relativistic species the Gamma rows of f0_rel restricted to
// the subluminal cone (src/ALPS_analyt.f90:546-607).
//
// Bound by the FP64 pipe of one SM (two lanes a clock) and by the chain of
// its iterations: the rows follow one another, so a fit cannot take more than
// one.  Hence few FP64 operations per point and iteration:
//   * the logarithms of a row's table are taken once, for the next row while
//     one warp solves;
//   * an accepted step's residuals are the next iteration's (the reference
//     forms them twice);
//   * one Maxwellian in log space (the usual fit) needs no exponential: its
//     log is linear in (log p0, p1) and its Jacobian over the value is
//     (1/p0, -d^2, 2 p1 d).  Where the value itself would leave the normal
//     numbers the exponentials decide as the reference's do.
// Sums over points are trees (32 lanes), more exact than the reference's
// running sums; the step solves (J^T J + lambda diag) delta = J^T r by the
// same partial-pivot elimination without forming the inverse.
// On a 192x384 grid, two species: 35.7 ms as one warp with the sums in
// series, 2.84 ms so.
#define FIT_THREADS 128
struct FitShared {
  double a[FIT_MAXP * (FIT_MAXP + 1)];  // normal matrix, right-hand side in the last column
  double params[FIT_MAXP], delta[FIT_MAXP];
  double red[FIT_THREADS / 32];
  double logp, ip0, lp;  // one Maxwellian in log space: log p0 and 1/p0 of the parameters, log amplitude on the row
  double acc[2][FIT_THREADS / 32][8];  // one Maxwellian: the pass's sums per warp, two passes in turn
  int lower, upper, singular, plain;
};
// doubles of point storage per point: two rows of table values, residual,
// value, Jacobian
__host__ __device__ inline int fit_point_words(int n_params) { return 4 + n_params; }

__device__ __forceinline__ double fit_block_sum(double v, FitShared& sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = sh.red[0];
  for (int k = 1; k < FIT_THREADS / 32; ++k) t += sh.red[k];
  __syncthreads();
  return t;
}

__device__ void lm_fit_body(const FitArgs& a, const double* __restrict__ f0, const double* __restrict__ pperp,
                            const double* __restrict__ ppar, double* fit, double* pts, int* status,
                            FitShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nf = a.nf, N = a.rel ? a.ng : a.N;
  const int maxpts = a.rel ? a.np : a.M, P = maxpts + 1;
  int n_params = 0;
  for (int f = 0; f < nf; ++f) n_params += fit_nparams(a, a.fit_type[f]);
  if (!a.rel && (1 + a.M) < n_params) {
    if (tid == 0) *status = ALPS_E_FIT_POINTS;
    return;
  }
  double *resid = pts + 2 * (size_t)P, *fval = pts + 3 * (size_t)P, *JT = pts + 4 * (size_t)P;
  const bool maxw = nf == 1 && a.fit_type[0] == 1 && a.log_fit && !a.rel;
  // the seeds
  {
    int par_ind = 0;
    for (int ifit = 1; ifit <= nf; ++ifit) {
      const int np = fit_nparams(a, a.fit_type[ifit - 1]);
      if (tid < np) sh.params[ifit + par_ind + tid - 1] = fit[tid * nf + ifit - 1];
      par_ind += np - 1;
    }
  }
  // the table values of a row (log f0 in log space) to buffer row & 1
  auto load_row = [&](int row, int off, int npts, int t0, int nt) {
    double* g = pts + (size_t)(row & 1) * P;
    for (int j = t0; j <= npts; j += nt) {
      if (a.flog) {
        g[j] = a.flog[(size_t)row * (a.M + 1) + j];
      } else {
        const double v = a.rel ? a.f0rel[(size_t)row * (a.np + 1) + off + j] : f0[row * (a.M + 1) + j];
        g[j] = a.log_fit ? log(v) : v;
      }
    }
  };
  if (!a.rel) load_row(0, 0, a.M, tid, FIT_THREADS);
  __syncthreads();
  for (int iperp = 0; iperp <= N; ++iperp) {
    if (iperp != 0)
      for (int t = tid; t < 5 * nf; t += FIT_THREADS) fit[(iperp * 5) * nf + t] = fit[((iperp - 1) * 5) * nf + t];
    int nJT = n_params;
    unsigned mask = 0xffffffffu;  // parameters that are fitted
    {
      int par_ind = 0;
      for (int ifit = 1; ifit <= nf; ++ifit) {
        const int t = a.fit_type[ifit - 1];
        if (t == 2 && iperp == 0) { nJT -= 1; mask &= ~(1u << (ifit + par_ind + 4 - 1)); }
        if (t == 6 && iperp == 0) { nJT -= 1; mask &= ~(1u << (ifit + par_ind + 3 - 1)); }
        par_ind += fit_nparams(a, t) - 1;
      }
    }
    // points of this row: coordinates and fitted values
    int npts = a.M, off = 0;
    double xperp;
    if (a.rel) {
      const double* fr = a.f0rel + (size_t)iperp * (a.np + 1);
      if (tid == 0) sh.lower = sh.upper = a.np;
      __syncthreads();
      // the cone's ends: the first rise above -1 and the first fall below it
      for (int ip = 1 + tid; ip <= a.np - 1; ip += FIT_THREADS) {
        if (fr[ip - 1] <= -1.0 && fr[ip] > -1.0) atomicMin(&sh.lower, ip);
        if (fr[ip] > -1.0 && fr[ip + 1] <= -1.0) atomicMin(&sh.upper, ip);
      }
      __syncthreads();
      const int lower = sh.lower < a.np ? sh.lower : 1, upper = sh.upper < a.np ? sh.upper : a.np - 1;
      __syncthreads();
      xperp = a.grel[iperp];
      if ((upper - lower) <= 2) {
        if (tid == 0) {
          int pi2 = 0;
          for (int ifit = 1; ifit <= nf; ++ifit) {
            sh.params[ifit + pi2 - 1] = fr[(upper + lower) / 2] / exp(-a.pc[ifit - 1] * a.grel[iperp]);
            if (a.fit_type[ifit - 1] == 5) {
              sh.params[ifit + pi2] = 1.0e-12;
              sh.params[ifit + pi2 + 1] = 0.0;
              pi2 += 2;
            }
          }
        }
        npts = -1;
      } else {
        npts = upper - lower;
        off = lower;
        load_row(iperp, off, npts, tid, FIT_THREADS);
      }
      __syncthreads();
    } else {
      xperp = pperp[iperp];
    }
    const double* g = pts + (size_t)(iperp & 1) * P;
    const double* xp = a.rel ? a.prel + off : ppar;
    bool ahead = a.rel || iperp == N;  // the next row's table values are there (or are not wanted)
    if (npts >= 0) {
      // What every thread needs of the current parameters, by warp 0 (the
      // logarithm on one lane, the reciprocal on another; each warp that
      // repeated them took its share of the SM's FP64 pipe).  Unmoved
      // parameters keep both.
      auto settle = [&](bool moved) {
        if (maxw) {
          const double p0 = sh.params[0], p1 = sh.params[1], p2 = sh.params[2];
          if (moved) {
            if (lane == 0) sh.logp = log(p0);
            if (lane == 1) sh.ip0 = 1.0 / p0;
            __syncwarp();
          }
          if (lane == 0) {
            const double lp = sh.logp - a.pc[0] * (xperp * xperp);
            const double d0 = xp[0] - p2, d1 = xp[npts] - p2, dm = fmax(d0 * d0, d1 * d1);
            sh.plain = p0 > 0.0 && p1 >= 0.0 && fabs(lp) < 600.0 && lp - p1 * dm > -690.0;
            sh.lp = lp;
          }
        } else if (lane == 0) {
          sh.plain = 0;
        }
      };
      // residuals (and values) at the current, settled parameters; returns
      // their sum of squares.  maxw without exponentials, where the value is a
      // normal number on the whole row.
      int buf = 0;
      auto residuals = [&](bool& plain) {
        double s = 0.0;
        plain = sh.plain != 0;
        if (plain) {
          // sums of r^2, r, r d, r d^2 and d, d^2, d^3, d^4, d = x - p2: all
          // that J^T J and J^T r need (columns 1/p0, -d^2, 2 p1 d)
          const double lp = sh.lp, p1 = sh.params[1], p2 = sh.params[2];
          double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          for (int j = tid; j <= npts; j += FIT_THREADS) {
            const double d = xp[j] - p2, d2 = d * d, r = (g[j] - lp) + p1 * d2;
            v[0] = fma(r, r, v[0]);
            v[1] += r;
            v[2] = fma(r, d, v[2]);
            v[3] = fma(r, d2, v[3]);
            v[4] += d;
            v[5] += d2;
            v[6] = fma(d2, d, v[6]);
            v[7] = fma(d2, d2, v[7]);
          }
          // eight sums over the lanes by halving
#pragma unroll
          for (int h = 4; h >= 1; h >>= 1) {
            const int off = 4 * h;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i < h) {
                const double keep = (lane & off) ? v[i + h] : v[i], give = (lane & off) ? v[i] : v[i + h];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
              }
          }
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
          buf ^= 1;
          if ((lane & 3) == 0) sh.acc[buf][warp][((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = v[0];
          __syncthreads();
          for (int w = 0; w < FIT_THREADS / 32; ++w) s += sh.acc[buf][w][0];
          return s;
        } else {
          for (int j = tid; j <= npts; j += FIT_THREADS) {
            const double fv = fit_value_real(a, sh.params, xperp, xp[j]);
            const double r = a.log_fit ? g[j] - log(fv) : g[j] - fv;
            fval[j] = fv;
            resid[j] = r;
            s = fma(r, r, s);
          }
        }
        return fit_block_sum(s, sh);
      };
      double lambda_fit = a.lambda0;
      int counter = 0;
      bool converged = false, plain;
      if (warp == 0) settle(iperp == 0);
      __syncthreads();
      double LSQ = residuals(plain);
      while (!converged) {
        counter++;
        const int ld = nJT + 1;
        if (!plain) {
          for (int j = tid; j <= npts; j += FIT_THREADS) {
            double J[FIT_MAXP];
            fit_jacobian(a, sh.params, iperp, xperp, xp[j], J);
            const double iv = a.log_fit ? 1.0 / fval[j] : 1.0;
            for (int k = 0; k < nJT; ++k) JT[(size_t)k * P + j] = J[k] * iv;
          }
          __syncthreads();
          // J^T J (upper triangle) and J^T r: a warp per entry
          const int nq = nJT * (nJT + 1) / 2 + nJT;
          for (int t = warp; t < nq; t += FIT_THREADS / 32) {
            int k, l;
            if (t < nJT) {
              k = t;
              l = nJT;
            } else {
              int u = t - nJT;
              for (k = 0; u >= nJT - k; ++k) u -= nJT - k;
              l = k + u;
            }
            const double *x = JT + (size_t)k * P, *y = l == nJT ? resid : JT + (size_t)l * P;
            double acc = 0.0;
            for (int j = lane; j <= npts; j += 32) acc = fma(x[j], y[j], acc);
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) {
              if (l == k) acc = acc + lambda_fit * acc;
              sh.a[k * ld + l] = acc;
              if (l < nJT) sh.a[l * ld + k] = acc;
            }
          }
          __syncthreads();
        }
        if (warp == 0) {
          // elimination with partial pivoting on the augmented matrix
          bool singular = false;
          if (plain) {
            // three unknowns, in registers on every lane
            double t[8];
#pragma unroll
            for (int q = 1; q < 8; ++q) {
              t[q] = 0.0;
              for (int w = 0; w < FIT_THREADS / 32; ++w) t[q] += sh.acc[buf][w][q];
            }
            const double i0 = sh.ip0, tp = 2.0 * sh.params[1];
            double m[3][4] = {{(double)(npts + 1) * (i0 * i0), -i0 * t[5], i0 * (tp * t[4]), i0 * t[1]},
                              {-i0 * t[5], t[7], -tp * t[6], -t[3]},
                              {i0 * (tp * t[4]), -tp * t[6], tp * (tp * t[5]), tp * t[2]}};
            double x[3], rp[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) m[k][k] = m[k][k] + lambda_fit * m[k][k];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
              for (int i = k + 1; i < 3; ++i)
                if (fabs(m[i][k]) > fabs(m[k][k])) {
#pragma unroll
                  for (int c = 0; c < 4; ++c) {
                    const double u = m[k][c];
                    m[k][c] = m[i][c];
                    m[i][c] = u;
                  }
                }
              if (m[k][k] == 0.0) singular = true;
              rp[k] = 1.0 / m[k][k];
#pragma unroll
              for (int i = k + 1; i < 3; ++i) {
                const double f = m[i][k] * rp[k];
#pragma unroll
                for (int c = k + 1; c < 4; ++c) m[i][c] -= f * m[k][c];
              }
            }
            x[2] = m[2][3] * rp[2];
            x[1] = (m[1][3] - m[1][2] * x[2]) * rp[1];
            x[0] = ((m[0][3] - m[0][1] * x[1]) - m[0][2] * x[2]) * rp[0];
            if (lane == 0 && !singular) {
              sh.delta[0] = x[0];
              sh.delta[1] = x[1];
              sh.delta[2] = x[2];
            }
            __syncwarp();
          }
          for (int k = 0; k < (plain ? 0 : nJT); ++k) {
            int p = k;
            double mx = fabs(sh.a[k * ld + k]);
            for (int i = k + 1; i < nJT; ++i)
              if (fabs(sh.a[i * ld + k]) > mx) { mx = fabs(sh.a[i * ld + k]); p = i; }
            if (sh.a[p * ld + k] == 0.0) { singular = true; break; }
            __syncwarp();
            if (p != k && lane >= k && lane <= nJT) {
              const double tmp = sh.a[k * ld + lane];
              sh.a[k * ld + lane] = sh.a[p * ld + lane];
              sh.a[p * ld + lane] = tmp;
            }
            __syncwarp();
            const int i = k + 1 + lane;
            double f = 0.0;
            if (i < nJT) f = sh.a[i * ld + k] / sh.a[k * ld + k];
            __syncwarp();
            if (i < nJT) sh.a[i * ld + k] = f;
            __syncwarp();
            const int m = nJT - k;  // columns k + 1 .. nJT
            for (int t = lane; t < (nJT - k - 1) * m; t += 32) {
              const int r = k + 1 + t / m, c = k + 1 + t % m;
              sh.a[r * ld + c] -= sh.a[r * ld + k] * sh.a[k * ld + c];
            }
            __syncwarp();
          }
          if (!singular && !plain)
            for (int i = nJT - 1; i >= 0; --i) {
              const double x = sh.a[i * ld + nJT] / sh.a[i * ld + i];
              __syncwarp();
              if (lane < i) sh.a[lane * ld + nJT] -= sh.a[lane * ld + i] * x;
              if (lane == 0) sh.delta[i] = x;
              __syncwarp();
            }
          if (lane == 0) {
            sh.singular = singular;
            if (!singular)
              for (int k = 0, l = 0; k < n_params; ++k)
                if ((mask >> k) & 1u) sh.params[k] = sh.params[k] + sh.delta[l++];
          }
          __syncwarp();
          if (!singular) settle(true);
        } else if (!ahead) {
          load_row(iperp + 1, 0, a.M, tid - 32, FIT_THREADS - 32);
        }
        ahead = true;
        __syncthreads();
        if (sh.singular) {
          if (tid == 0) *status = ALPS_E_SINGULAR;
          return;
        }
        const double LSQnew = residuals(plain);
        const double diff = fabs(LSQnew - LSQ);
        if (LSQnew > LSQ) {
          if (warp == 0) {
            if (lane == 0)
              for (int k = 0, l = 0; k < n_params; ++k)
                if ((mask >> k) & 1u) sh.params[k] = sh.params[k] - sh.delta[l++];
            __syncwarp();
            settle(true);
          }
          __syncthreads();
          lambda_fit = lambda_fit * a.lambdafac;
        } else {
          lambda_fit = lambda_fit / a.lambdafac;
        }
        if (diff < a.eps) converged = true;
        if (counter == a.maxsteps) converged = true;
        // the residuals at the parameters the next iteration starts from
        if (!converged) LSQ = (LSQnew > LSQ) ? residuals(plain) : LSQnew;
      }
    }
    if (!ahead) load_row(iperp + 1, 0, a.M, tid, FIT_THREADS);
    {
      int par_ind = 0;
      for (int ifit = 1; ifit <= nf; ++ifit) {
        const int np = fit_nparams(a, a.fit_type[ifit - 1]);
        if (tid < np) fit[(iperp * 5 + tid) * nf + ifit - 1] = sh.params[ifit + par_ind + tid - 1];
        par_ind += np - 1;
      }
    }
    __syncthreads();
  }
}

// the fit's point storage: shared memory where it fits, else the global
// scratch (maxpts + 1) fit_point_words(FIT_MAXP) of the species
__device__ __forceinline__ double* fit_points(const FitArgs& a, double* scratch, double* smem, int smem_words) {
  int n_params = 0;
  for (int f = 0; f < a.nf; ++f) n_params += fit_nparams(a, a.fit_type[f]);
  const int P = (a.rel ? a.np : a.M) + 1;
  return (long)P * fit_point_words(n_params) <= smem_words ? smem : scratch;
}

__global__ void __launch_bounds__(FIT_THREADS) k_lm_fit(FitArgs a, const double* __restrict__ f0,
                                                        const double* __restrict__ pperp,
                                                        const double* __restrict__ ppar, double* fit, double* scratch,
                                                        int* status, int smem_words) {
  extern __shared__ double fit_smem[];
  __shared__ FitShared sh;
  if (blockIdx.x != 0) return;
  lm_fit_body(a, f0, pperp, ppar, fit, fit_points(a, scratch, fit_smem, smem_words), status, sh);
}

// Dynamic shared memory (in doubles) that a fit wants, at most FIT_SMEM_WORDS;
// a larger one uses its global scratch
#define FIT_SMEM_WORDS 12288
inline int fit_smem_words(const FitArgs& a) {
  static const int np[7] = {1, 3, 5, 3, 1, 3, 4};  // parameters by fit type
  int n_params = 0;
  for (int f = 0; f < a.nf; ++f) n_params += np[a.fit_type[f] >= 1 && a.fit_type[f] <= 6 ? a.fit_type[f] : 0];
  const long w = (long)((a.rel ? a.np : a.M) + 1) * fit_point_words(n_params);
  return w <= FIT_SMEM_WORDS ? (int)w : 0;
}

}  // namespace

// the fit of one (context, species) in a batched launch
struct FitJob {
  FitArgs a;
  const double *f0, *pperp, *ppar;
  double *fit, *scratch;
  int* status;
};

namespace {

// every job of the batch, one block each: fits of different plasmas are
// independent; within a fit the reference's warm start orders the rows
__global__ void __launch_bounds__(FIT_THREADS) k_lm_fit_many(const FitJob* __restrict__ jobs, int n, int smem_words) {
  extern __shared__ double fit_smem[];
  __shared__ FitShared sh;
  __shared__ FitJob J;
  const int j = blockIdx.x;
  if (j >= n) return;
  if (threadIdx.x == 0) J = jobs[j];
  __syncthreads();
  lm_fit_body(J.a, J.f0, J.pperp, J.ppar, J.fit, fit_points(J.a, J.scratch, fit_smem, smem_words), J.status, sh);
}

// log f0 of a whole table, over the chip
__global__ void k_fit_logs(const double* __restrict__ f0, size_t n, double* flog) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) flog[t] = log(f0[t]);
}

// both fit kernels may take FIT_SMEM_WORDS doubles
int fit_smem_optin() {
  const int bytes = FIT_SMEM_WORDS * (int)sizeof(double);
  ALPS_CUDA_TRY(cudaFuncSetAttribute(k_lm_fit, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  ALPS_CUDA_TRY(cudaFuncSetAttribute(k_lm_fit_many, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return ALPS_OK;
}

// determine_nmax for one species: the smallest n >= 1 with
// max_i |J_n(z_i)| <= Bessel_zero, z_i = k_perp pperp_i / q, or n = limit.
// The maximum exceeds the cutoff exactly when some node's |J_n| does.  The
// orders go in chunks of NMAX_CHUNK, one thread each:
//   * orders whose n lies above the grid's last z (z < 0.95 n): J_n rises on
//     (0, n), so the last node decides.  Debye's leading term exp(n (tanh a -
//     a))/sqrt(2 pi n tanh a), z = n / cosh a, is an upper bound of J_n(z) and
//     within a third of it there, so where it is a factor 8 off the cutoff
//     either way, it decides; one alps_bessj call at the last node otherwise.
//   * the others test the node nearest J_n's largest maximum (z = n + 0.81
//     n^(1/3)) with one alps_bessj call, which settles nearly all of them.
// Then the orders still open, in increasing order, test every node with the
// whole block, and the first with none above the cutoff is the answer.  Each
// order's decision is the reference's, alps_bessj's values against the cutoff.
// One call of order n costs about 5 (n + sqrt(40 n)) dependent FP64
// operations, and the chain of calls is the time: without the estimate, over
// chunks of 128 orders, 103 us for an answer of 20 to 30 (96 rows), 32 us so.
#define NMAX_CHUNK 128
__device__ void nmax_body(const double* __restrict__ pperp, int N, double kperp, double qs, double bzero, int limit,
                          int* nmax_out, unsigned* settled) {
  const int t = threadIdx.x;
  const double zs = fabs(qs) / kperp, dp = pperp[1] - pperp[0];
  auto zat = [&](int i) { return __ddiv_rn(__dmul_rn(kperp, pperp[i]), qs); };
  auto above = [&](int nn, int i) { return fabs(alps_bessj(nn, zat(i))) > bzero; };
  const float zlast = fabsf((float)zat(N));
  const bool rising = pperp[0] >= 0.0 && dp > 0.0;  // |z| grows with the node
  const float lcut = (bzero >= 1e-290 && bzero <= 1.0) ? (float)log(bzero) : nanf("");
  unsigned* below = settled + NMAX_CHUNK / 32;
  for (int base = 1;; base += NMAX_CHUNK) {
    if (t < NMAX_CHUNK) {  // whole warps (NMAX_CHUNK is a multiple of 32)
      const int nn = base + t;
      bool hit = false, none = false;  // some node above the cutoff; certainly no node
      if (nn < limit) {
        const float x = zlast / (float)nn;
        if (rising && x < 0.95f && x > 1e-30f) {
          const float ta = sqrtf((1.0f - x) * (1.0f + x));
          // n (tanh a - a): a = log((1 + ta)/x)
          const float d = (float)nn * (ta - logf((1.0f + ta) / x)) - 0.5f * logf(6.2831853f * (float)nn * ta) - lcut;
          const float tol = 2.08f + 1e-6f * (float)nn * (1.0f + fabsf(logf(x)));
          if (d > tol) hit = true;
          else if (d < -tol) none = true;
          else hit = above(nn, N), none = !hit;
        } else {
          const double u = ((nn + 0.81 * cbrt((double)nn)) * zs - pperp[0]) / dp;
          const int i0 = (u >= 0.0 && u <= (double)N) ? (int)rint(u) : ((u > 0.0 || u != u) ? N : 0);
          hit = above(nn, i0);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit), q = __ballot_sync(0xffffffffu, none);
      if ((t & 31) == 0) {
        settled[t >> 5] = m;
        below[t >> 5] = q;
      }
    }
    __syncthreads();
    for (int k = 0; k < NMAX_CHUNK; ++k) {
      const int nn = base + k;
      if (nn >= limit) {
        if (t == 0) *nmax_out = limit;
        return;
      }
      if ((settled[k >> 5] >> (k & 31)) & 1u) continue;
      bool hit = false;
      if (!((below[k >> 5] >> (k & 31)) & 1u)) {
        for (int i = t; i <= N && !hit; i += blockDim.x) hit = above(nn, i);
        hit = __syncthreads_or(hit);
      }
      if (!hit) {
        if (t == 0) *nmax_out = nn;
        return;
      }
    }
    __syncthreads();  // settled[] is rewritten by the next chunk
  }
}

__global__ void k_nmax(const double* __restrict__ pperp, int N, double kperp, double qs, double bzero,
                       int limit, int* nmax_out) {
  __shared__ unsigned settled[2 * (NMAX_CHUNK / 32)];
  nmax_body(pperp, N, kperp, qs, bzero, limit, nmax_out, settled);
}

}  // namespace

// determine_nmax of one (context, species) in a batched launch
struct NmaxJob {
  const double* pperp;
  int N;
  double kperp, qs, bzero;
  int* out;
};

namespace {

__global__ void k_nmax_many(const NmaxJob* __restrict__ jobs, int n, int limit) {
  __shared__ unsigned settled[2 * (NMAX_CHUNK / 32)];
  if ((int)blockIdx.x >= n) return;
  const NmaxJob& J = jobs[blockIdx.x];
  nmax_body(J.pperp, J.N, J.kperp, J.qs, J.bzero, limit, J.out, settled);
}

// bessel[(n+1)*(N+1)+i] = J_n(k_perp pperp_i / q), n = -1 .. nmax+1
__global__ void k_bessel_table(const double* __restrict__ pperp, int N, int nmax, double kperp, double qs,
                               double* bessel) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int n = (int)blockIdx.y - 1;
  if (i > N || n > nmax + 1) return;
  double z = __ddiv_rn(__dmul_rn(kperp, pperp[i]), qs);
  bessel[(size_t)(n + 1) * (N + 1) + i] = (n == -1) ? -alps_bessj(1, z) : alps_bessj(n, z);
}

// Rw[(F*(nmax+1) + n)*(N-1) + (i-1)] = w_perp(i) * R_F(n,i), F = 0: J_n^2,
// 1: pperp^2 J_n'^2, 2: pperp J_n J_n' (the three Bessel-product families of
// int_T), w_perp = 2 for i < N-1 and 1 at i = N-1.
__global__ void k_bessel_rows(const double* __restrict__ bessel, const double* __restrict__ pperp, int N,
                              int nmax, double* Rw) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int n = blockIdx.y;
  if (i > N - 1 || n > nmax) return;
  const double* B = bessel;
  int L = N + 1;
  double J = B[(size_t)(n + 1) * L + i];
  double Jp = (n == 0) ? -B[(size_t)2 * L + i] : 0.5 * (B[(size_t)n * L + i] - B[(size_t)(n + 2) * L + i]);
  double w = (i <= N - 2) ? 2.0 : 1.0;
  double p = pperp[i];
  size_t stride = (size_t)(nmax + 1) * (N - 1);
  size_t o = (size_t)n * (N - 1) + (i - 1);
  Rw[o] = w * (J * J);
  Rw[stride + o] = w * ((p * p) * Jp * Jp);
  Rw[2 * stride + o] = w * (p * J * Jp);
}

// C[m][n] = sum_k A[m][k] B[k][n], row-major, FP64, 32x32 tiles, 2x2 per thread.
__global__ void k_dgemm(int Mr, int Nc, int K, const double* __restrict__ A, const double* __restrict__ B,
                        double* C) {
  __shared__ double As[32][17];
  __shared__ double Bs[16][33];
  int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  int row0 = blockIdx.y * 32, col0 = blockIdx.x * 32;
  double acc[2][2] = {{0, 0}, {0, 0}};
  for (int k0 = 0; k0 < K; k0 += 16) {
    for (int t = threadIdx.x; t < 32 * 16; t += 256) {
      int r = t / 16, kk = t % 16;
      int gr = row0 + r, gk = k0 + kk;
      As[r][kk] = (gr < Mr && gk < K) ? A[(size_t)gr * K + gk] : 0.0;
    }
    for (int t = threadIdx.x; t < 16 * 32; t += 256) {
      int kk = t / 32, cc = t % 32;
      int gk = k0 + kk, gc = col0 + cc;
      Bs[kk][cc] = (gk < K && gc < Nc) ? B[(size_t)gk * Nc + gc] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      double a0 = As[ty * 2][kk], a1 = As[ty * 2 + 1][kk];
      double b0 = Bs[kk][tx * 2], b1 = Bs[kk][tx * 2 + 1];
      acc[0][0] = fma(a0, b0, acc[0][0]);
      acc[0][1] = fma(a0, b1, acc[0][1]);
      acc[1][0] = fma(a1, b0, acc[1][0]);
      acc[1][1] = fma(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b) {
      int r = row0 + ty * 2 + a, cidx = col0 + tx * 2 + b;
      if (r < Mr && cidx < Nc) C[(size_t)r * Nc + cidx] = acc[a][b];
    }
}

// V[((n*(M-1)) + (j-1))*12 + 2*e + g] = 2 * c_e(j) * A[F(e)][n][g][j],
// entries e = xx, yy, zz, xy, xz, yz; c = 1, 1, ppar^2, 1, ppar, ppar.
// V of order n (block n) as float pairs scaled by 2^-e, e the exponent of
// max |V[n]|: x 2^-e = hi + lo, hi = float(x 2^-e), lo = float(x 2^-e - hi)
__global__ void k_split_df(const double* __restrict__ V, int M, double* scale, float* Vh, float* Vl) {
  __shared__ double red[256];
  const size_t len = (size_t)(M - 1) * 12;
  const double* v = V + (size_t)blockIdx.x * len;
  double mx = 0.0;
  for (size_t t = threadIdx.x; t < len; t += blockDim.x) mx = fmax(mx, fabs(v[t]));
  red[threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  const int e = (red[0] > 0.0) ? ilogb(red[0]) : 0;
  const double down = ldexp(1.0, -e);
  if (threadIdx.x == 0) scale[blockIdx.x] = ldexp(1.0, e);
  for (size_t t = threadIdx.x; t < len; t += blockDim.x) {
    const double x = v[t] * down;
    const float h = __double2float_rn(x);
    Vh[(size_t)blockIdx.x * len + t] = h;
    Vl[(size_t)blockIdx.x * len + t] = __double2float_rn(x - (double)h);
  }
}

// ppar as float pairs
__global__ void k_split_pp(const double* __restrict__ ppar, int M, float* ph, float* pl) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > M) return;
  const float h = __double2float_rn(ppar[j]);
  ph[j] = h;
  pl[j] = __double2float_rn(ppar[j] - (double)h);
}

__global__ void k_fold_reduced(const double* __restrict__ A, const double* __restrict__ ppar, int M, int nmax,
                               double* V) {
  int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
  int n = blockIdx.y;
  if (j > M - 1 || n > nmax) return;
  size_t ncol = 2 * (size_t)(M - 1);
  auto Aat = [&](int F, int g) { return A[((size_t)F * (nmax + 1) + n) * ncol + (size_t)g * (M - 1) + (j - 1)]; };
  double p = ppar[j];
  double* v = V + ((size_t)n * (M - 1) + (j - 1)) * 12;
  for (int g = 0; g < 2; ++g) {
    double a0 = Aat(0, g), a1 = Aat(1, g), a2 = Aat(2, g);
    v[0 + g] = 2.0 * a0;
    v[2 + g] = 2.0 * a1;
    v[4 + g] = 2.0 * ((p * p) * a0);
    v[6 + g] = 2.0 * a2;
    v[8 + g] = 2.0 * (p * a0);
    v[10 + g] = 2.0 * (p * a2);
  }
}

// X[(j-1)*ALPS_KFAR + k] = x_j^k with x_j = (ppar_j - pcen)/prad, j = 1..M-1,
// each power rounded once (products carried with their error)
__global__ void k_powers(const double* __restrict__ ppar, int M, double pcen, double prad, double* X) {
  int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (j > M - 1) return;
  double x = (ppar[j] - pcen) / prad;
  double p = 1.0, l = 0.0;
  double* o = X + (size_t)(j - 1) * ALPS_KFAR;
  for (int k = 0; k < ALPS_KFAR; ++k) {
    o[k] = p;
    const double h = p * x, e = fma(p, x, -h) + l * x;
    p = h + e;
    l = e - (p - h);
  }
}

// the reduced vectors of the Bessel families F1 = J^2, F2 = pperp^2 J'^2,
// F3 = pperp J J' against g1 and g2 (b = 2 F + g)
__device__ __forceinline__ int base_q(int b) { return b < 4 ? b : b + 2; }

// Laurent moments of the full-range trapezoid pole sum of the base vectors:
// mom[(n*ALPS_KFAR + k)*6 + b] = sum_j f_j V[n][j][base_q(b)] x_j^k, f_j = 1/2
// at j = 1, M-1 and 1 inside (the reduced vectors carry the interior weight
// 2).  For a pole p far from the grid, sum_j f_j V_j / (p - ppar_j) =
//   (1/d) sum_k mom_k (prad/d)^k,  d = p - pcen.
// Bound by the FP64 rate: a warp per 32 powers of one vector, so that the
// warps spread evenly over the SMs (192x384 grid: 33 us; a thread per (n, k,
// q) of all twelve vectors, in blocks of 128, took 70).
__global__ void __launch_bounds__(32) k_moments(const double* __restrict__ V, const double* __restrict__ X, int M,
                                                double* mom) {
  const int k = blockIdx.x * 32 + threadIdx.x, b = blockIdx.y, n = blockIdx.z;
  const double* v = V + (size_t)n * (M - 1) * 12 + base_q(b);
  const double* x = X + k;
  // (four partial sums: a shorter chain, and less rounding)
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j0 = 2; j0 <= M - 2; j0 += 4)
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j0 + u <= M - 2)
        acc[u] = fma(__ldg(v + (size_t)(j0 + u - 1) * 12), __ldg(x + (size_t)(j0 + u - 1) * ALPS_KFAR), acc[u]);
  const double ends = fma(0.5 * v[0], x[0], 0.5 * v[(size_t)(M - 2) * 12] * x[(size_t)(M - 2) * ALPS_KFAR]);
  mom[((size_t)n * ALPS_KFAR + k) * 6 + b] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ends;
}

// C0 v_e(n) in FP64
__global__ void k_plain_fac(int nmax, double z, double kperp, int kperp_norm, double C0, double* pfac) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (nmax + 1) * 6) pfac[t] = fused_factor(t / 6, t % 6, z, kperp, kperp_norm, C0);
}

// Base tables of the fast path's pole sums.  The six T-tensor entries use
// three Bessel families, F1 = J^2 (xx, xz, zz), F2 = pperp^2 J'^2 (yy) and
// F3 = pperp J J' (xy, yz), with the p_par factors 1, p_par, p_par^2.  With
// R_j = 1 / (k_par (zeta - p_j)), zeta the complex resonance momentum,
//   p_j R_j = zeta R_j - 1/k_par,
// so the p_par-weighted sums follow from the family sums and the
// omega-independent sums of the family vectors themselves:
//   sum w F p R   = zeta sum w F R - (1/k_par) sum w F,
//   sum w F p^2 R = zeta sum w F p R - (1/k_par) sum w F p.
// A node or Laurent term then feeds 6 real vectors instead of 12.  The
// vectors are V's q = 0, 1 (F1), 2, 3 (F2), 6, 7 (F3), scaled by
// 1/Vscale[n] (a power of two) and split into float pairs.
// Bt and mBt: hi parts at [rec*12 + b], lo parts at [rec*12 + 6 + b]
__global__ void k_base_pairs(const double* __restrict__ V, const double* __restrict__ mom,
                             const double* __restrict__ Vscale, int M, int nmax, float* Bt, float* mBt) {
  const size_t nv = (size_t)(nmax + 1) * (M - 1) * 6, nm = (size_t)(nmax + 1) * ALPS_KFAR * 6;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nv + nm) return;
  const bool isv = t < nv;
  const size_t u = isv ? t : t - nv;
  const size_t rec = u / 6;
  const int b = (int)(u % 6);
  const int n = isv ? (int)(rec / (M - 1)) : (int)(rec / ALPS_KFAR);
  const double x = (isv ? V[rec * 12 + base_q(b)] : mom[rec * 6 + b]) * (1.0 / Vscale[n]);
  const float h = __double2float_rn(x), l = __double2float_rn(x - (double)h);
  float* o = isv ? Bt : mBt;
  o[rec * 12 + b] = h;
  o[rec * 12 + 6 + b] = l;
}

// Pre[(n*M + j)*6 + c] = sum_{i=1..j} X_c(i), X = V[q]/Vscale[n] for
// q = 0, 1 (F1), 6, 7 (F3), 8, 9 (p_par F1), compensated (two-sum) so that
// each stored prefix is the exact sum rounded once; Cfull[n*6 + c] = the
// trapezoid sum over j = 1..M-1 (ends at weight 1/2).  One warp per (n, c): a
// lane sums a run of nodes with its error, the runs' totals are scanned as
// pairs, and each lane goes over its run again from there (192x384 grid: 119
// us by one thread per (n, c), 12 us so).
__device__ __forceinline__ void comp_add(double& s, double& e, double x) {
  const double y = s + x, b = y - s;
  e += (s - (y - b)) + (x - b);
  s = y;
}
__global__ void __launch_bounds__(64) k_base_consts(const double* __restrict__ V, const double* __restrict__ Vscale,
                                                    int M, int nmax, double* Pre, double* Cfull) {
  const int t = blockIdx.x * 2 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= (nmax + 1) * 6) return;
  const int n = t / 6, c = t % 6;
  const int q = (c < 2) ? c : c + 4;
  const double sc = 1.0 / Vscale[n];
  const double* v = V + (size_t)n * (M - 1) * 12 + q;
  double* P = Pre + (size_t)n * M * 6 + c;
  const int per = (M - 1 + 31) / 32, j0 = 1 + lane * per, j1 = min(M - 1, j0 + per - 1);
  double s = 0.0, e = 0.0;
#pragma unroll 4
  for (int j = j0; j <= j1; ++j) comp_add(s, e, v[(size_t)(j - 1) * 12] * sc);
  for (int off = 1; off < 32; off <<= 1) {
    const double ps = __shfl_up_sync(0xffffffffu, s, off), pe = __shfl_up_sync(0xffffffffu, e, off);
    if (lane >= off) {
      e += pe;
      comp_add(s, e, ps);
    }
  }
  const double ts = __shfl_sync(0xffffffffu, s, 31), te = __shfl_sync(0xffffffffu, e, 31);
  s = __shfl_up_sync(0xffffffffu, s, 1);
  e = __shfl_up_sync(0xffffffffu, e, 1);
  if (lane == 0) {
    s = e = 0.0;
    P[0] = 0.0;
  }
#pragma unroll 4
  for (int j = j0; j <= j1; ++j) {
    comp_add(s, e, v[(size_t)(j - 1) * 12] * sc);
    P[(size_t)j * 6] = s + e;
  }
  if (lane == 0) {
    const double x1 = v[0] * sc, xe = v[(size_t)(M - 2) * 12] * sc;
    Cfull[t] = (ts + te) - 0.5 * (x1 + xe);
  }
}

// bfac and Escale: the order factors C0 v_e(n) Vscale[n] over the power of two
// Escale[e] of the largest, as float pairs.  One block, a thread per (n, e) in
// turn (30 orders: 45 us by a thread per entry, under 12 us so).
__global__ void __launch_bounds__(192) k_base_fac(int nmax, double z, double kperp, int kperp_norm, double C0,
                                                  const double* __restrict__ Vscale, double* Escale, float* bfac) {
  __shared__ unsigned long long mx[6];  // bits of the largest finite-or-not magnitude (ordered as integers)
  if (threadIdx.x < 6) mx[threadIdx.x] = 0;
  __syncthreads();
  const int total = (nmax + 1) * 6;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const double x = fabs(fused_factor(t / 6, t % 6, z, kperp, kperp_norm, C0) * Vscale[t / 6]);
    if (x == x) atomicMax(&mx[t % 6], (unsigned long long)__double_as_longlong(x));
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    const double m = __longlong_as_double((long long)mx[threadIdx.x]);
    Escale[threadIdx.x] = (m > 0.0 && isfinite(m)) ? ldexp(1.0, ilogb(m)) : 1.0;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const double x = fused_factor(t / 6, t % 6, z, kperp, kperp_norm, C0) * Vscale[t / 6] * (1.0 / Escale[t % 6]);
    const float h = __double2float_rn(x);
    bfac[(size_t)t * 2] = h;
    bfac[(size_t)t * 2 + 1] = __double2float_rn(x - (double)h);
  }
}

// omega-independent factors of Maxwellian continuation terms, per row and
// fit: a0 = p1 exp(-pc pperp^2) (the reference's left-to-right product),
// p2, p3, exp(-p2 dppar^2)
__global__ void k_fit_aux(const double* __restrict__ fit, const double* __restrict__ pperp, int N, int nf,
                          double pc0, double pc1, double pc2, double pc3, double dppar, double* aux) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > N) return;
  double pcs[4] = {pc0, pc1, pc2, pc3};
  double p = pperp[i];
  for (int f = 0; f < nf; ++f) {
    double p1 = fit[(i * 5 + 0) * nf + f], p2 = fit[(i * 5 + 1) * nf + f], p3 = fit[(i * 5 + 2) * nf + f];
    double* o = aux + ((size_t)i * nf + f) * 4;
    o[0] = p1 * exp(-pcs[f] * (p * p));
    o[1] = p2;
    o[2] = p3;
    o[3] = exp(-p2 * (dppar * dppar));
  }
}

// Moments of the factorised Landau sums (one Maxwellian term per row,
// f(i,p) = a0_i exp(u_r(p)) exp(delta_i(p)), delta_i = a_i p^2 + b_i p + c_i,
// exp(delta) ~ 1 + delta + delta^2/2 = sum_m kappa_{i,m} p^m, m = 0..4):
//   w = 0: sum_i h_i R_F(n,i) pperp_i a0_i kappa_{i,m}   (the dfpar sum)
//   w = 1: sum_i c_i a0_i kappa_{i,m}, c = the transpose of landau_integrate's
//          p_perp difference operator applied to h_i R_F(n,i)  (the dfperp sum)
// h_i = 1/2 at i = 0, N-1, N and 1 otherwise (src/ALPS_fns.f90:1389-1444).
__global__ void k_landau_moments(const double* __restrict__ bessel, const double* __restrict__ pperp,
                                 const double* __restrict__ aux, int N, int nmax, double dpperp, double* lmom,
                                 float* lmomf) {
  // one warp per (n, F): lanes over the rows, then a warp sum
  const int t = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (t >= (nmax + 1) * 3) return;
  const int n = t / 3, F = t % 3;
  const int L = N + 1;
  auto Rw = [&](int i) {
    double J = bessel[(size_t)(n + 1) * L + i];
    double Jp = (n == 0) ? -bessel[(size_t)2 * L + i]
                         : 0.5 * (bessel[(size_t)n * L + i] - bessel[(size_t)(n + 2) * L + i]);
    double p = pperp[i];
    double h = (i == 0 || i == N - 1 || i == N) ? 0.5 : 1.0;
    double R = (F == 0) ? J * J : (F == 1 ? (p * p) * Jp * Jp : p * J * Jp);
    return h * R;
  };
  const double p2r = aux[1], p3r = aux[2];
  const double i2d = 1.0 / (2.0 * dpperp), i1d = 1.0 / dpperp;
  double m0[5] = {0, 0, 0, 0, 0}, m1[5] = {0, 0, 0, 0, 0};
  for (int i = lane; i <= N; i += 32) {
    const double* ai = aux + (size_t)i * 4;
    double a0 = ai[0], p2 = ai[1], p3 = ai[2];
    double a = -(p2 - p2r), b = 2.0 * (p2 * p3 - p2r * p3r), c = -(p2 * p3 * p3 - p2r * p3r * p3r);
    double k[5] = {1.0 + c + 0.5 * c * c, b * (1.0 + c), a + 0.5 * b * b + a * c, a * b, 0.5 * a * a};
    double w0 = Rw(i) * pperp[i];
    double cc = 0.0;  // transpose of the difference operator at i
    if (i - 1 >= 1 && i - 1 <= N - 1) cc += Rw(i - 1) * i2d;
    if (i + 1 >= 1 && i + 1 <= N - 1) cc -= Rw(i + 1) * i2d;
    if (i == 1) cc += Rw(0) * i1d;
    if (i == 0) cc -= Rw(0) * i1d;
    if (i == N) cc += Rw(N) * i1d;
    if (i == N - 1) cc -= Rw(N) * i1d;
    for (int m = 0; m < 5; ++m) {
      m0[m] += w0 * a0 * k[m];
      m1[m] += cc * a0 * k[m];
    }
  }
  for (int m = 0; m < 5; ++m)
    for (int off = 16; off > 0; off >>= 1) {
      m0[m] += __shfl_xor_sync(0xffffffffu, m0[m], off);
      m1[m] += __shfl_xor_sync(0xffffffffu, m1[m], off);
    }
  if (lane == 0) {
    double* o = lmom + (size_t)t * 10;
    for (int m = 0; m < 5; ++m) {
      o[m] = m0[m];
      o[5 + m] = m1[m];
    }
    // the fast path's copy: float pairs scaled by 2^-e, e the exponent of
    // the largest of the ten (hi at 0..9, lo at 10..19, e at 20)
    double mx = 0.0;
    for (int m = 0; m < 10; ++m) mx = fmax(mx, fabs(o[m]));
    const int e = (mx > 0.0 && isfinite(mx)) ? ilogb(mx) : 0;
    float* f = lmomf + (size_t)t * 24;
    for (int m = 0; m < 10; ++m) {
      const double x = ldexp(o[m], -e);
      const float h = __double2float_rn(x);
      f[m] = h;
      f[10 + m] = __double2float_rn(x - (double)h);
    }
    f[20] = (float)e;
    f[21] = f[22] = f[23] = 0.0f;
  }
}

// grows a table to at least n elements; a regrown table gets a quarter
// more, so a k scan whose nmax rises step by step reallocates (and pays
// cudaFree's device-wide wait) only now and then
template <typename T>
int ensure(T*& ptr, size_t& cap, size_t n) {
  if (n <= cap && ptr) return ALPS_OK;
  const size_t want = ptr ? n + n / 4 : n;
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  cap = 0;
  ALPS_CUDA_TRY(cudaMalloc(&ptr, want * sizeof(T)));
  cap = want;
  return ALPS_OK;
}

// ---------------------------------------------------------------------------
// Chebyshev continuation (ACmethod 2): set_polynomial_basis + determine_GLLS
// + least_squares_fit (src/ALPS_analyt.f90:731-889).  The basis on the
// uniform p_par nodes, and so the normal matrix A^T A, is the same on every
// p_perp row: it is built and LU-factored once (partial pivoting, dgetrf);
// each row then only forms A^T b and back-substitutes.  Sums run over p_par
// in ascending order without contraction.
// ---------------------------------------------------------------------------
__global__ void k_glls_basis(int M, int np, double* A /* [(M+1)][(np+1)] */) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > M) return;
  double yy = __dadd_rn(-1.0, __dmul_rn((double)j, 2.0 / M));
  double* a = A + (size_t)j * (np + 1);
  a[0] = 1.0;
  if (np >= 1) a[1] = yy;
  for (int n = 2; n <= np; ++n) a[n] = __dsub_rn(__dmul_rn(__dmul_rn(2.0, yy), a[n - 1]), a[n - 2]);
}

// alpha = A^T A (column-major m x m), then its LU in place; one block
__global__ void k_glls_normal(const double* __restrict__ A, int M, int np, double* alpha, int* piv, int* status) {
  const int m = np + 1;
  for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
    int k = t % m, l = t / m;
    double acc = 0.0;
    for (int j = 0; j <= M; ++j) acc = __dadd_rn(acc, __dmul_rn(A[(size_t)j * m + k], A[(size_t)j * m + l]));
    alpha[t] = acc;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < m; ++k) {
    int p = k;
    double mx = fabs(alpha[k + m * k]);
    for (int i = k + 1; i < m; ++i)
      if (fabs(alpha[i + m * k]) > mx) {
        mx = fabs(alpha[i + m * k]);
        p = i;
      }
    piv[k] = p;
    if (alpha[p + m * k] == 0.0) {
      *status = ALPS_E_SINGULAR;
      return;
    }
    if (p != k)
      for (int j = 0; j < m; ++j) {
        double tmp = alpha[k + m * j];
        alpha[k + m * j] = alpha[p + m * j];
        alpha[p + m * j] = tmp;
      }
    double dk = alpha[k + m * k];
    for (int i = k + 1; i < m; ++i) alpha[i + m * k] = __ddiv_rn(alpha[i + m * k], dk);
    for (int j = k + 1; j < m; ++j) {
      double f = alpha[k + m * j];
      if (f == 0.0) continue;
      for (int i = k + 1; i < m; ++i) alpha[i + m * j] = __dsub_rn(alpha[i + m * j], __dmul_rn(alpha[i + m * k], f));
    }
  }
}

// one block per p_perp row: b = log10 f0 (zeros replaced by 0.01 x the
// smallest positive value of the row) or f0, w = A^T b, LU solve
__global__ void k_glls_rows(const double* __restrict__ f0, const double* __restrict__ A,
                            const double* __restrict__ alpha, const int* __restrict__ piv, int M, int np, int log_fit,
                            const int* status, double* coeffs) {
  extern __shared__ double sm[];
  double* b = sm;            // [M+1]
  double* w = sm + (M + 1);  // [np+1]
  __shared__ double smin[128], spos[128];
  if (*status) return;
  const int i = blockIdx.x, m = np + 1;
  const double* row = f0 + (size_t)i * (M + 1);
  for (int j = threadIdx.x; j <= M; j += blockDim.x) b[j] = row[j];
  __syncthreads();
  if (log_fit) {
    double mn = 1.0e308, mp = 1.0e308;
    for (int j = threadIdx.x; j <= M; j += blockDim.x) {
      mn = fmin(mn, b[j]);
      if (b[j] > 0.0) mp = fmin(mp, b[j]);
    }
    smin[threadIdx.x] = mn;
    spos[threadIdx.x] = mp;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + s]);
        spos[threadIdx.x] = fmin(spos[threadIdx.x], spos[threadIdx.x + s]);
      }
      __syncthreads();
    }
    const bool fix = !(smin[0] > 0.0);
    const double repl = 0.01 * (spos[0] < 1.0e308 ? spos[0] : 1.0e-40);
    for (int j = threadIdx.x; j <= M; j += blockDim.x) b[j] = log10((fix && b[j] == 0.0) ? repl : b[j]);
    __syncthreads();
  }
  for (int k = threadIdx.x; k < m; k += blockDim.x) {
    double acc = 0.0;
    for (int j = 0; j <= M; ++j) acc = __dadd_rn(acc, __dmul_rn(A[(size_t)j * m + k], b[j]));
    w[k] = acc;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < m; ++k) {
    double t = w[k];
    w[k] = w[piv[k]];
    w[piv[k]] = t;
  }
  for (int j = 0; j < m; ++j)
    for (int r = j + 1; r < m; ++r) w[r] = __dsub_rn(w[r], __dmul_rn(alpha[r + m * j], w[j]));
  for (int j = m - 1; j >= 0; --j) {
    w[j] = __ddiv_rn(w[j], alpha[j + m * j]);
    for (int r = 0; r < j; ++r) w[r] = __dsub_rn(w[r], __dmul_rn(alpha[r + m * j], w[j]));
  }
  for (int k = 0; k < m; ++k) coeffs[(size_t)i * m + k] = w[k];
}

}  // namespace

// ---------------------------------------------------------------------------
int launch_prepare_species(alps_ctx* c, int is) {
  SpeciesHost& S = c->spec[is];
  S.aux_ready = false;  // a new fit: its continuation factors and bounds follow at the next set_k
  if (S.sp.use_bM) return ALPS_OK;  // closed form: nothing to derive or fit
  int N = c->sys.nperp, M = c->sys.npar;
  cudaStream_t st = c->stream;
  size_t nn = (size_t)(N + 1) * (M + 1);
  if (!S.d_g1) ALPS_CUDA_TRY(cudaMalloc(&S.d_g1, nn * sizeof(double)));
  if (!S.d_g2) ALPS_CUDA_TRY(cudaMalloc(&S.d_g2, nn * sizeof(double)));
  if (!S.d_G) ALPS_CUDA_TRY(cudaMalloc(&S.d_G, (size_t)(N - 1) * 2 * (M - 1) * sizeof(double)));
  ALPS_CUDA_TRY(cudaMemsetAsync(S.d_g1, 0, nn * sizeof(double), st));
  ALPS_CUDA_TRY(cudaMemsetAsync(S.d_g2, 0, nn * sizeof(double), st));
  dim3 grid((M - 1 + 127) / 128, N - 1);
  k_derivatives<<<grid, 128, 0, st>>>(S.d_f0, S.d_pperp, S.d_ppar, N, M, S.d_g1, S.d_g2, S.d_G);
  ALPS_CUDA_TRY(cudaGetLastError());
  // ee term: int_ee * 2*pi*q/m * dpperp*dppar/4
  double dpperp = S.pperp[2] - S.pperp[1];
  double dppar = std::fabs(S.ppar[2] - S.ppar[1]);
  double scale = 2.0 * ALPS_PI * S.sp.qs / S.sp.ms * dpperp * dppar * 0.25;
  // per-species device words and fit scratch are kept with the species: a
  // cudaFree here would wait for the whole device, and contexts prepared on
  // several host threads would run one after another
  if (!S.d_words) ALPS_CUDA_TRY(cudaMalloc(&S.d_words, 2 * sizeof(double)));
  double* d_ee = S.d_words;
  int* d_status = reinterpret_cast<int*>(S.d_words + 1);
  k_int_ee<<<EE_BLOCKS, 256, 0, st>>>(S.d_g2, S.d_ppar, N, M, scale, d_ee);
  ALPS_CUDA_TRY(cudaGetLastError());
  // relativistic species: (Gamma, pparbar) grid, f0_rel and its derivatives
  int st_fit = ALPS_OK;
  if (S.sp.relat) st_fit = launch_rel_prepare(c, is);
  // Chebyshev continuation (ACmethod 2)
  if (S.sp.ac_method == 2 && st_fit == ALPS_OK) st_fit = launch_glls(c, is);
  // LM fit of the analytic continuation (ACmethod 1)
  if (S.sp.ac_method == 1 && st_fit == ALPS_OK) {
    FitArgs a;
    a.N = N;
    a.M = M;
    a.nf = S.sp.n_fits;
    a.log_fit = S.sp.log_fit;
    for (int f = 0; f < ALPS_MAX_FITS; ++f) {
      a.fit_type[f] = S.sp.fit_type[f];
      a.pc[f] = S.sp.perp_correction[f];
    }
    a.ms = S.sp.ms;
    a.vA = c->sys.vA;
    a.maxsteps = c->sys.maxsteps_fit;
    a.lambda0 = c->sys.lambda_initial_fit;
    a.lambdafac = c->sys.lambdafac_fit;
    a.eps = c->sys.epsilon_fit;
    a.rel = S.sp.relat ? 1 : 0;
    a.ng = c->sys.ngamma;
    a.np = c->sys.npparbar;
    a.f0rel = S.d_f0rel;
    a.grel = S.d_grel;
    a.prel = S.d_prel;
    int maxpts = a.rel ? a.np : M;
    int rc;
    if ((rc = fit_smem_optin())) return rc;
    const int words = fit_smem_words(a);
    if (!words && (rc = ensure(S.d_fit_scratch, S.fit_scratch_cap, (size_t)(maxpts + 1) * fit_point_words(FIT_MAXP))))
      return rc;
    ALPS_CUDA_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    a.flog = nullptr;
    if (a.log_fit && !a.rel) {
      const size_t nn = (size_t)(N + 1) * (M + 1);
      if ((rc = ensure(S.d_flog, S.flog_cap, nn))) return rc;
      k_fit_logs<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(S.d_f0, nn, S.d_flog);
      ALPS_CUDA_TRY(cudaGetLastError());
      a.flog = S.d_flog;
    }
    k_lm_fit<<<1, FIT_THREADS, words * sizeof(double), st>>>(a, S.d_f0, S.d_pperp, S.d_ppar, S.d_fit, S.d_fit_scratch,
                                                             d_status, words);
    ALPS_CUDA_TRY(cudaGetLastError());
    ALPS_CUDA_TRY(cudaMemcpyAsync(&st_fit, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    ALPS_CUDA_TRY(cudaStreamSynchronize(st));
  }
  double ee = 0.0;
  ALPS_CUDA_TRY(cudaMemcpyAsync(&ee, d_ee, sizeof(double), cudaMemcpyDeviceToHost, st));
  ALPS_CUDA_TRY(cudaStreamSynchronize(st));
  S.int_ee = ee;
  return st_fit;
}

// ---------------------------------------------------------------------------
// Batched preparation of many contexts (alps_prepare_many): the derivative
// and ee kernels of every context on a few streams, then the
// Levenberg-Marquardt fits of every (context, species) in one launch, one
// block each, then one synchronisation.  Relativistic species and the
// Chebyshev continuation take the per-context path.
// ---------------------------------------------------------------------------
static FitArgs fit_args_of(const alps_ctx* c, const SpeciesHost& S) {
  FitArgs a;
  a.N = c->sys.nperp;
  a.M = c->sys.npar;
  a.nf = S.sp.n_fits;
  a.log_fit = S.sp.log_fit;
  for (int f = 0; f < ALPS_MAX_FITS; ++f) {
    a.fit_type[f] = S.sp.fit_type[f];
    a.pc[f] = S.sp.perp_correction[f];
  }
  a.ms = S.sp.ms;
  a.vA = c->sys.vA;
  a.maxsteps = c->sys.maxsteps_fit;
  a.lambda0 = c->sys.lambda_initial_fit;
  a.lambdafac = c->sys.lambdafac_fit;
  a.eps = c->sys.epsilon_fit;
  a.rel = S.sp.relat ? 1 : 0;
  a.ng = c->sys.ngamma;
  a.np = c->sys.npparbar;
  a.f0rel = S.d_f0rel;
  a.grel = S.d_grel;
  a.prel = S.d_prel;
  a.flog = nullptr;
  return a;
}

bool ctx_batch_preparable(const alps_ctx* c) {
  for (const SpeciesHost& S : c->spec)
    if (!S.loaded || S.sp.relat || (!S.sp.use_bM && S.sp.ac_method != 1)) return false;
  return true;
}

int prepare_contexts(alps_ctx* const* ctx, int n, int* status) {
  const int NS = 8;
  cudaStream_t st[NS];
  for (int q = 0; q < NS; ++q) ALPS_CUDA_TRY(cudaStreamCreateWithFlags(&st[q], cudaStreamNonBlocking));
  std::vector<FitJob> jobs;
  std::vector<std::pair<int, int>> who;  // (context, species) of each job
  int rc = fit_smem_optin(), fit_words = 0;
  for (int i = 0; i < n && !rc; ++i) {
    alps_ctx* c = ctx[i];
    cudaStream_t s = st[i % NS];
    const int N = c->sys.nperp, M = c->sys.npar;
    const size_t nn = (size_t)(N + 1) * (M + 1);
    for (int is = 0; is < c->sys.nspec && !rc; ++is) {
      SpeciesHost& S = c->spec[is];
      S.aux_ready = false;
      if (S.sp.use_bM) continue;
      auto fail = [&](cudaError_t e) {
        if (e != cudaSuccess) rc = (e == cudaErrorMemoryAllocation) ? ALPS_E_OOM : ALPS_E_CUDA;
      };
      if (!S.d_g1) fail(cudaMalloc(&S.d_g1, nn * sizeof(double)));
      if (!S.d_g2 && !rc) fail(cudaMalloc(&S.d_g2, nn * sizeof(double)));
      if (!S.d_G && !rc) fail(cudaMalloc(&S.d_G, (size_t)(N - 1) * 2 * (M - 1) * sizeof(double)));
      if (!S.d_words && !rc) fail(cudaMalloc(&S.d_words, 2 * sizeof(double)));
      if (rc) break;
      FitArgs fa = fit_args_of(c, S);
      const int words = fit_smem_words(fa);
      fit_words = std::max(fit_words, words);
      if (!words &&
          (rc = ensure(S.d_fit_scratch, S.fit_scratch_cap, (size_t)(M + 1) * fit_point_words(FIT_MAXP))))
        break;
      if (fa.log_fit && (rc = ensure(S.d_flog, S.flog_cap, nn))) break;
      fail(cudaMemsetAsync(S.d_g1, 0, nn * sizeof(double), s));
      fail(cudaMemsetAsync(S.d_g2, 0, nn * sizeof(double), s));
      fail(cudaMemsetAsync(S.d_words + 1, 0, sizeof(double), s));
      dim3 grid((M - 1 + 127) / 128, N - 1);
      k_derivatives<<<grid, 128, 0, s>>>(S.d_f0, S.d_pperp, S.d_ppar, N, M, S.d_g1, S.d_g2, S.d_G);
      const double dpperp = S.pperp[2] - S.pperp[1], dppar = std::fabs(S.ppar[2] - S.ppar[1]);
      const double scale = 2.0 * ALPS_PI * S.sp.qs / S.sp.ms * dpperp * dppar * 0.25;
      k_int_ee<<<EE_BLOCKS, 256, 0, s>>>(S.d_g2, S.d_ppar, N, M, scale, S.d_words);
      if (fa.log_fit) {
        fa.flog = S.d_flog;
        k_fit_logs<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(S.d_f0, nn, S.d_flog);
      }
      fail(cudaGetLastError());
      FitJob j;
      j.a = fa;
      j.f0 = S.d_f0;
      j.pperp = S.d_pperp;
      j.ppar = S.d_ppar;
      j.fit = S.d_fit;
      j.scratch = S.d_fit_scratch;
      j.status = reinterpret_cast<int*>(S.d_words + 1);
      jobs.push_back(j);
      who.push_back({i, is});
    }
  }
  FitJob* d_jobs = nullptr;
  for (int q = 0; q < NS && !rc; ++q)
    if (cudaStreamSynchronize(st[q]) != cudaSuccess) rc = ALPS_E_CUDA;
  if (!rc && !jobs.empty()) {
    if (cudaMalloc(&d_jobs, jobs.size() * sizeof(FitJob)) != cudaSuccess) rc = ALPS_E_OOM;
    if (!rc && cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(FitJob), cudaMemcpyHostToDevice, st[0]) !=
                   cudaSuccess)
      rc = ALPS_E_CUDA;
    if (!rc) {
      k_lm_fit_many<<<(unsigned)jobs.size(), FIT_THREADS, fit_words * sizeof(double), st[0]>>>(
          d_jobs, (int)jobs.size(), fit_words);
      if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st[0]) != cudaSuccess) rc = ALPS_E_CUDA;
    }
  }
  // ee terms and fit statuses, then the continuation factors (asynchronous)
  for (size_t k = 0; k < who.size() && !rc; ++k) {
    alps_ctx* c = ctx[who[k].first];
    SpeciesHost& S = c->spec[who[k].second];
    double w[2];
    if (cudaMemcpy(w, S.d_words, 2 * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) {
      rc = ALPS_E_CUDA;
      break;
    }
    S.int_ee = w[0];
    int fst = 0;
    memcpy(&fst, &w[1], sizeof(int));
    if (fst && status && !status[who[k].first]) status[who[k].first] = fst;
  }
  for (int q = 0; q < NS; ++q) cudaStreamDestroy(st[q]);
  cudaFree(d_jobs);
  return rc;
}

// determine_nmax of every (non-closed-form) species of every context in one
// launch; nm[i][s] receives the results (closed-form species get 1)
int nmax_contexts(alps_ctx* const* ctx, int n, const double* kperp, std::vector<std::vector<int>>& nm) {
  std::vector<NmaxJob> jobs;
  nm.assign(n, {});
  size_t tot = 0;
  for (int i = 0; i < n; ++i) tot += ctx[i]->sys.nspec;
  // the results and the job table in one stream-ordered allocation on a
  // stream of its own: nothing here waits for other work on the device
  const size_t ob = ((tot ? tot : 1) * sizeof(int) + 15) / 16 * 16;
  size_t njobs = 0;
  for (int i = 0; i < n; ++i)
    for (int is = 0; is < ctx[i]->sys.nspec; ++is) njobs += ctx[i]->spec[is].sp.use_bM ? 0 : 1;
  cudaStream_t st;
  ALPS_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  unsigned char* d_buf = nullptr;
  int rc = ALPS_OK;
  if (cudaMallocAsync(&d_buf, ob + (njobs ? njobs : 1) * sizeof(NmaxJob), st) != cudaSuccess) rc = ALPS_E_OOM;
  int* d_out = reinterpret_cast<int*>(d_buf);
  NmaxJob* d_jobs = reinterpret_cast<NmaxJob*>(d_buf + ob);
  size_t k = 0;
  for (int i = 0; i < n; ++i) {
    nm[i].assign(ctx[i]->sys.nspec, 1);
    for (int is = 0; is < ctx[i]->sys.nspec; ++is, ++k) {
      const SpeciesHost& S = ctx[i]->spec[is];
      if (S.sp.use_bM) continue;
      jobs.push_back(NmaxJob{S.d_pperp, ctx[i]->sys.nperp, kperp[i], S.sp.qs, ctx[i]->sys.Bessel_zero, d_out + k});
    }
  }
  std::vector<int> out(tot ? tot : 1, 0);
  if (!rc && !jobs.empty()) {
    if (cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(NmaxJob), cudaMemcpyHostToDevice, st) !=
        cudaSuccess)
      rc = ALPS_E_CUDA;
    if (!rc) {
      k_nmax_many<<<(unsigned)jobs.size(), 256, 0, st>>>(d_jobs, (int)jobs.size(), 2000);
      if (cudaGetLastError() != cudaSuccess) rc = ALPS_E_CUDA;
    }
    if (!rc && cudaMemcpyAsync(out.data(), d_out, tot * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
      rc = ALPS_E_CUDA;
  }
  if (d_buf) cudaFreeAsync(d_buf, st);
  if (cudaStreamSynchronize(st) != cudaSuccess && !rc) rc = ALPS_E_CUDA;
  cudaStreamDestroy(st);
  k = 0;
  for (int i = 0; i < n && !rc; ++i)
    for (int is = 0; is < ctx[i]->sys.nspec; ++is, ++k)
      if (!ctx[i]->spec[is].sp.use_bM) {
        if (out[k] >= 2000) rc = ALPS_E_INVALID;  // orders beyond 2000 are outside the supported range
        nm[i][is] = out[k];
      }
  return rc;
}

int launch_glls(alps_ctx* c, int is) {
  SpeciesHost& S = c->spec[is];
  const int N = c->sys.nperp, M = c->sys.npar, np = S.sp.poly_order, m = np + 1;
  cudaStream_t st = c->stream;
  double *d_A = nullptr, *d_alpha = nullptr;
  int *d_piv = nullptr, *d_status = nullptr;
  ALPS_CUDA_TRY(cudaMalloc(&d_A, (size_t)(M + 1) * m * sizeof(double)));
  ALPS_CUDA_TRY(cudaMalloc(&d_alpha, (size_t)m * m * sizeof(double)));
  ALPS_CUDA_TRY(cudaMalloc(&d_piv, m * sizeof(int)));
  ALPS_CUDA_TRY(cudaMalloc(&d_status, sizeof(int)));
  ALPS_CUDA_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), st));
  k_glls_basis<<<(M + 1 + 127) / 128, 128, 0, st>>>(M, np, d_A);
  k_glls_normal<<<1, 256, 0, st>>>(d_A, M, np, d_alpha, d_piv, d_status);
  size_t smem = (size_t)(M + 1 + m) * sizeof(double);
  if (smem > 48 * 1024) ALPS_CUDA_TRY(cudaFuncSetAttribute(k_glls_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_glls_rows<<<N + 1, 128, smem, st>>>(S.d_f0, d_A, d_alpha, d_piv, M, np, S.sp.log_fit, d_status, S.d_fit);
  ALPS_CUDA_TRY(cudaGetLastError());
  int status = 0;
  ALPS_CUDA_TRY(cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
  ALPS_CUDA_TRY(cudaStreamSynchronize(st));
  cudaFree(d_A);
  cudaFree(d_alpha);
  cudaFree(d_piv);
  cudaFree(d_status);
  return status;
}

int launch_set_k_species(alps_ctx* c, int is, double kperp, int* nmax_out) {
  SpeciesHost& S = c->spec[is];
  if (S.sp.use_bM) {  // determine_nmax gives a bi-Maxwellian species 1 (src/ALPS_fns.f90:4012-4014)
    *nmax_out = 1;
    return ALPS_OK;
  }
  // a device word kept with the species: no allocation (and no cudaFree,
  // which would wait for the whole device) per k step
  if (!S.d_nmax) ALPS_CUDA_TRY(cudaMalloc(&S.d_nmax, sizeof(int)));
  k_nmax<<<1, 256, 0, c->stream>>>(S.d_pperp, c->sys.nperp, kperp, S.sp.qs, c->sys.Bessel_zero, 2000, S.d_nmax);
  ALPS_CUDA_TRY(cudaGetLastError());
  int nm = 0;
  ALPS_CUDA_TRY(cudaMemcpyAsync(&nm, S.d_nmax, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  ALPS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  if (nm >= 2000) return ALPS_E_INVALID;  // orders beyond 2000 are outside the supported range
  *nmax_out = nm;
  return ALPS_OK;
}

int launch_build_bessel_and_reduced(alps_ctx* c, int is, double kperp) {
  SpeciesHost& S = c->spec[is];
  int N = c->sys.nperp, M = c->sys.npar, nmax = S.nmax;
  cudaStream_t st = c->stream;
  int rc;
  if ((rc = ensure(S.d_bessel, S.bessel_cap, (size_t)(nmax + 3) * (N + 1)))) return rc;
  if ((rc = ensure(S.d_Rw, S.Rw_cap, (size_t)3 * (nmax + 1) * (N - 1)))) return rc;
  if ((rc = ensure(S.d_A, S.A_cap, (size_t)3 * (nmax + 1) * 2 * (M - 1)))) return rc;
  if ((rc = ensure(S.d_V, S.V_cap, (size_t)(nmax + 1) * (M - 1) * 12))) return rc;
  k_bessel_table<<<dim3((N + 1 + 127) / 128, nmax + 3), 128, 0, st>>>(S.d_pperp, N, nmax, kperp, S.sp.qs,
                                                                       S.d_bessel);
  ALPS_CUDA_TRY(cudaGetLastError());
  k_bessel_rows<<<dim3((N - 1 + 127) / 128, nmax + 1), 128, 0, st>>>(S.d_bessel, S.d_pperp, N, nmax, S.d_Rw);
  ALPS_CUDA_TRY(cudaGetLastError());
  int Mr = 3 * (nmax + 1), Nc = 2 * (M - 1), K = N - 1;
  S.tc_used = 0;
  S.tc_fixed = 0;
  if (c->precision == ALPS_PREC_MIXED && K <= 256) {
    // mixed path: the contraction on the tensor cores, FP64-accurate per
    // entry (tc_product_checked recomputes in FP64 whatever its bound does
    // not cover)
    const size_t need = tc_checked_workspace_bytes(Mr, Nc, K);
    if (need > S.tcws_cap) {
      if (S.d_tcws) cudaFree(S.d_tcws);
      S.d_tcws = nullptr;
      S.tcws_cap = 0;
      ALPS_CUDA_TRY(cudaMalloc(&S.d_tcws, need));
      S.tcws_cap = need;
    }
    // (a batched set_k defers the count of FP64-recomputed entries: no sync here)
    if ((rc = tc_product_checked(S.d_Rw, S.d_G, S.d_A, Mr, Nc, K, S.d_tcws, c->defer_sync ? nullptr : &S.tc_fixed,
                                 st)))
      return rc;
    S.tc_used = 1;
  } else {
    k_dgemm<<<dim3((Nc + 31) / 32, (Mr + 31) / 32), 256, 0, st>>>(Mr, Nc, K, S.d_Rw, S.d_G, S.d_A);
    ALPS_CUDA_TRY(cudaGetLastError());
  }
  k_fold_reduced<<<dim3((M - 1 + 127) / 128, nmax + 1), 128, 0, st>>>(S.d_A, S.d_ppar, M, nmax, S.d_V);
  ALPS_CUDA_TRY(cudaGetLastError());
  {
    // the FP32 test for orders far from resonance (both paths' classify):
    // the resonance interval of determine_resonances with a margin of 1e-5
    // of its extent
    const double mi = c->sys.positions_principal * (S.ppar[2] - S.ppar[1]);
    const double rlo = std::min(S.ppar[1] - mi, S.ppar[1]), rhi = std::max(S.ppar[M], S.ppar[M - 1] + mi);
    const double mg = 1e-5 * (std::fabs(rlo) + std::fabs(rhi));
    S.qlo = (float)(rlo - mg);
    S.qhi = (float)(rhi + mg);
    S.qlo_in = (float)(rlo + mg);
    S.qhi_in = (float)(rhi - mg);
  }
  if (!S.d_far) ALPS_CUDA_TRY(cudaMalloc(&S.d_far, (size_t)FAR_LEVELS * FAR_K * 12 * sizeof(double)));
  if ((rc = ensure(S.d_farc, S.farc_cap, (size_t)nmax * FAR_K * 12))) return rc;
  // Laurent moments
  const double pcen = 0.5 * (S.ppar[1] + S.ppar[M - 1]), prad = 0.5 * (S.ppar[M - 1] - S.ppar[1]);
  if (!S.grid_ready) {
    // what depends on the p_par grid alone: powers and float pairs
    if (!S.d_X) ALPS_CUDA_TRY(cudaMalloc(&S.d_X, (size_t)(M - 1) * ALPS_KFAR * sizeof(double)));
    if (!S.d_pph) ALPS_CUDA_TRY(cudaMalloc(&S.d_pph, (M + 1) * sizeof(float)));
    if (!S.d_ppl) ALPS_CUDA_TRY(cudaMalloc(&S.d_ppl, (M + 1) * sizeof(float)));
    k_powers<<<(M - 1 + 127) / 128, 128, 0, st>>>(S.d_ppar, M, pcen, prad, S.d_X);
    ALPS_CUDA_TRY(cudaGetLastError());
    k_split_pp<<<(M + 1 + 127) / 128, 128, 0, st>>>(S.d_ppar, M, S.d_pph, S.d_ppl);
    ALPS_CUDA_TRY(cudaGetLastError());
    S.grid_ready = true;
  }
  if ((rc = ensure(S.d_mom, S.mom_cap, (size_t)(nmax + 1) * ALPS_KFAR * 6))) return rc;
  k_moments<<<dim3(ALPS_KFAR / 32, 6, nmax + 1), 32, 0, st>>>(S.d_V, S.d_X, M, S.d_mom);
  ALPS_CUDA_TRY(cudaGetLastError());
  const double z = c->sys.kperp_norm ? kperp / S.sp.qs : 1.0 / S.sp.qs;
  const double dpperp = S.pperp[2] - S.pperp[1], dppar_abs = std::fabs(S.ppar[2] - S.ppar[1]);
  const double C0 = 2.0 * ALPS_PI * dpperp * dppar_abs * 0.25 * S.sp.qs;
  // the plain path sums nodes and series in FP64 on V and the moments; the
  // float pairs and order-fused tables below serve the mixed path only (a
  // change of path rebuilds the k tables)
  if (c->precision == ALPS_PREC_FP64) {
    if ((rc = ensure(S.d_pfac, S.pfac_cap, (size_t)(nmax + 1) * 6))) return rc;
    k_plain_fac<<<((nmax + 1) * 6 + 127) / 128, 128, 0, st>>>(nmax, z, kperp, c->sys.kperp_norm, C0, S.d_pfac);
    ALPS_CUDA_TRY(cudaGetLastError());
    return ALPS_OK;
  }
  const size_t nvf = (size_t)(nmax + 1) * (M - 1) * 12;
  if ((rc = ensure(S.d_Vh, S.Vf_cap, 2 * nvf))) return rc;  // hi, then lo
  S.d_Vl = S.d_Vh + nvf;
  if ((rc = ensure(S.d_Vscale, S.Vs_cap, (size_t)(nmax + 1)))) return rc;
  k_split_df<<<nmax + 1, 256, 0, st>>>(S.d_V, M, S.d_Vscale, S.d_Vh, S.d_Vl);
  ALPS_CUDA_TRY(cudaGetLastError());
  const size_t nmo = (size_t)(nmax + 1) * ALPS_KFAR * 12;
  // base tables of the fast path's pole sums
  {
    const size_t nm = (size_t)(nmax + 1);
    if ((rc = ensure(S.d_Bt, S.Bt_cap, nvf + nmo + nm * 12))) return rc;  // Bt, mBt, bfac
    if ((rc = ensure(S.d_Bd, S.Bd_cap, 8 + nm * 6 + nm * (size_t)M * 6))) return rc;  // Escale, Cfull, Pre
    const size_t np = (nvf + nmo) / 2;
    k_base_pairs<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(S.d_V, S.d_mom, S.d_Vscale, M, nmax, S.d_Bt,
                                                              S.d_Bt + nvf);
    ALPS_CUDA_TRY(cudaGetLastError());
    k_base_consts<<<(unsigned)((nm * 6 + 1) / 2), 64, 0, st>>>(S.d_V, S.d_Vscale, M, nmax,
                                                                      S.d_Bd + 8 + nm * 6, S.d_Bd + 8);
    ALPS_CUDA_TRY(cudaGetLastError());
    k_base_fac<<<1, 192, 0, st>>>(nmax, z, kperp, c->sys.kperp_norm, C0, S.d_Vscale, S.d_Bd, S.d_Bt + nvf + nmo);
    ALPS_CUDA_TRY(cudaGetLastError());
  }
  return ALPS_OK;
}

int launch_fit_aux(alps_ctx* c, int is) {
  SpeciesHost& S = c->spec[is];
  if (S.aux_ready) return ALPS_OK;  // built for the current fit already
  bool maxw = S.sp.ac_method == 1 && !S.sp.use_bM;
  for (int f = 0; f < S.sp.n_fits && maxw; ++f) maxw = S.sp.fit_type[f] == 1;
  if (!maxw) {
    if (S.d_fit_aux) cudaFree(S.d_fit_aux);
    S.d_fit_aux = nullptr;
    return ALPS_OK;
  }
  int N = c->sys.nperp, nf = S.sp.n_fits;
  if (!S.d_fit_aux) ALPS_CUDA_TRY(cudaMalloc(&S.d_fit_aux, (size_t)(N + 1) * ALPS_MAX_FITS * 4 * sizeof(double)));
  double dppar = std::fabs(S.ppar[2] - S.ppar[1]);
  k_fit_aux<<<(N + 1 + 127) / 128, 128, 0, c->stream>>>(S.d_fit, S.d_pperp, N, nf, S.sp.perp_correction[0],
                                                         S.sp.perp_correction[1], S.sp.perp_correction[2],
                                                         S.sp.perp_correction[3], dppar, S.d_fit_aux);
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}

// Factorised Landau moments for species whose continuation is one Maxwellian
// term; the per-item validity bound uses max |a_i|, |b_i|, |c_i| (host).
int launch_landau_moments(alps_ctx* c, int is) {
  SpeciesHost& S = c->spec[is];
  if (S.aux_ready) {
    // the bounds belong to the fit, not to k: only the moments are per k
    if (!S.lfact) return ALPS_OK;
    int rc;
    if ((rc = ensure(S.d_lmom, S.lmom_cap, (size_t)(S.nmax + 1) * (30 + 36)))) return rc;  // FP64, then the pairs
    const int tot = (S.nmax + 1) * 3;
    k_landau_moments<<<(tot + 3) / 4, 128, 0, c->stream>>>(S.d_bessel, S.d_pperp, S.d_fit_aux, c->sys.nperp,
                                                           S.nmax, S.pperp[2] - S.pperp[1], S.d_lmom,
                                                           reinterpret_cast<float*>(S.d_lmom + (size_t)(S.nmax + 1) * 30));
    ALPS_CUDA_TRY(cudaGetLastError());
    return ALPS_OK;
  }
  S.aux_ready = true;
  S.lfact = false;
  if (!S.d_fit_aux || S.sp.n_fits != 1 || !S.d_bessel) return ALPS_OK;
  int N = c->sys.nperp, nmax = S.nmax;
  std::vector<double> aux((size_t)(N + 1) * 4);
  ALPS_CUDA_TRY(cudaMemcpyAsync(aux.data(), S.d_fit_aux, aux.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                c->stream));
  ALPS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  double p2r = aux[1], p3r = aux[2], la = 0, lb = 0, lc = 0, mina0 = 1e308;
  for (int i = 0; i <= N; ++i) {
    double p2 = aux[i * 4 + 1], p3 = aux[i * 4 + 2];
    la = std::max(la, std::fabs(p2 - p2r));
    lb = std::max(lb, std::fabs(2.0 * (p2 * p3 - p2r * p3r)));
    lc = std::max(lc, std::fabs(p2 * p3 * p3 - p2r * p3r * p3r));
    if (i >= 1) mina0 = std::min(mina0, std::fabs(aux[i * 4 + 0]));
    if (!std::isfinite(p2) || !std::isfinite(p3) || !std::isfinite(aux[i * 4])) return ALPS_OK;
  }
  S.p2r = p2r;
  S.p3r = p3r;
  S.la = la;
  S.lb = lb;
  S.lc = lc;
  S.min_a0 = mina0;
  S.lfact = true;
  int rc;
  if ((rc = ensure(S.d_lmom, S.lmom_cap, (size_t)(nmax + 1) * (30 + 36)))) return rc;  // FP64, then the pairs
  int tot = (nmax + 1) * 3;
  double dpperp = S.pperp[2] - S.pperp[1];
  k_landau_moments<<<(tot + 3) / 4, 128, 0, c->stream>>>(S.d_bessel, S.d_pperp, S.d_fit_aux, N, nmax, dpperp,
                                                         S.d_lmom,
                                                         reinterpret_cast<float*>(S.d_lmom + (size_t)(nmax + 1) * 30));
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}
