// map_value.cuh -- a map point's value, log10 |det D|, with the same bits on the
// host and on the device: a map computed alone finishes on the device, one
// computed by the server on the host, and both are the same map.
//
// |D|^2 = 2^E m is formed as an unevaluated sum of two doubles (error-free
// products and sums), m in [0.7, 1.42]; ln m = 2 atanh((m - 1)/(m + 1)) by the
// Taylor series, its first term in two doubles; log10 |D| = (E log10 2 + log10
// m) / 2.  Within 0.6 units in the last place of log10 of the exact modulus.
#pragma once

#include <cmath>
#include <limits>

#ifdef __CUDA_ARCH__
#define MV_MUL(a, b) __dmul_rn(a, b)
#define MV_ADD(a, b) __dadd_rn(a, b)
#define MV_DIV(a, b) __ddiv_rn(a, b)
#define MV_FMA(a, b, c) __fma_rn(a, b, c)
#else
#define MV_MUL(a, b) ((a) * (b))
#define MV_ADD(a, b) ((a) + (b))
#define MV_DIV(a, b) ((a) / (b))
#define MV_FMA(a, b, c) std::fma(a, b, c)
#endif

__host__ __device__ inline void mv_two_sum(double a, double b, double& s, double& e) {
  s = MV_ADD(a, b);
  const double t = MV_ADD(s, -a);
  e = MV_ADD(MV_ADD(a, -MV_ADD(s, -t)), MV_ADD(b, -t));
}

__host__ __device__ inline double log10_abs(double re, double im) {
  double a = fabs(re), b = fabs(im);
  const double inf = HUGE_VAL;
  if (a == inf || b == inf) return inf;
  if (a != a || b != b) return a + b;
  if (a < b) {
    const double t = a;
    a = b;
    b = t;
  }
  if (a == 0.0) return -inf;
  const int k = ilogb(a);
  a = scalbn(a, -k);
  b = scalbn(b, -k);
  // s = a^2 + b^2 in [1, 8)
  double sh, sl, mh, ml;
  const double p = MV_MUL(a, a), q = MV_MUL(b, b);
  mv_two_sum(p, q, sh, sl);
  sl = MV_ADD(sl, MV_ADD(MV_FMA(a, a, -p), MV_FMA(b, b, -q)));
  mv_two_sum(sh, sl, mh, ml);
  const int j = mh < 1.4142 ? 0 : (mh < 2.8284 ? 1 : (mh < 5.6569 ? 2 : 3));
  const double sc = j == 0 ? 1.0 : (j == 1 ? 0.5 : (j == 2 ? 0.25 : 0.125));
  mh = MV_MUL(mh, sc);
  ml = MV_MUL(ml, sc);
  // w = (m - 1)/(m + 1), |w| < 0.18
  double nh, nl, dh, dl;
  mv_two_sum(mh, -1.0, nh, nl);
  mv_two_sum(mh, 1.0, dh, dl);
  nl = MV_ADD(nl, ml);
  dl = MV_ADD(dl, ml);
  const double w = MV_DIV(nh, dh);
  const double wl = MV_DIV(MV_ADD(MV_ADD(MV_FMA(-w, dh, nh), nl), -MV_MUL(w, dl)), dh);
  const double w2 = MV_MUL(w, w);
  double s = 1.0 / 25.0;
  for (int i = 23; i >= 3; i -= 2) s = MV_FMA(s, w2, 1.0 / (double)i);
  const double c = MV_FMA(MV_MUL(w, w2), s, wl);
  // log10 |D| = E log10(2)/2 + (w + c)/ln 10
  const double kh = 0.4342944819032518, kl = 1.098319650216765e-17;    // 1/ln 10
  const double ch = 0.1505149978319906, cl = -1.4018640638925852e-18;  // log10(2)/2
  const double E = (double)(2 * k + j);
  const double t = MV_MUL(kh, w), g = MV_MUL(ch, E);
  const double te = MV_FMA(kh, c, MV_FMA(kl, w, MV_FMA(kh, w, -t))), ge = MV_FMA(cl, E, MV_FMA(ch, E, -g));
  double r, re2;
  mv_two_sum(g, t, r, re2);
  return MV_ADD(r, MV_ADD(re2, MV_ADD(te, ge)));
}

// the value of det D, which receives map_search's sentinels
// (src/ALPS_fns.f90:3720-3743)
__host__ __device__ inline double map_value(double* re, double* im) {
  const double x = *re;
  double v = log10_abs(x, *im);
  if (*im == 0.0 && x != x) {
    *re = v = 999999.0;
    *im = 0.0;
  }
  if (fabs(x) > 1.0e100) {
    *re = v = 899999.0;
    *im = 0.0;
  }
  return v;
}
