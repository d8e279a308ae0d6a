// disp_kernels.cu -- the omega pass: det D(omega, k) for a batch of
// frequencies (disp, src/ALPS_fns.f90:252-636).
//
// For fixed k the reference's double loop
//     sum_{i,j} w_i w_j resU(i,j) int_T(n,i,j,mode)
// factorises: resU's denominator depends on ppar_j only and its numerator is
// linear in omega, so the p_perp sum was done once per k into the reduced
// vectors V[n][j][12] (setup_kernels.cu).  What is left per omega is a 1-D
// pole sum over ppar per Bessel order:
//     S_{e,g}(n) = sum_j (w_j/2) V_{e,g}(n,j) / (m omega - k_par ppar_j - n q)
// plus, for resonant orders, the principal-value window and the Landau term.
//
// Kernels of one batch (launched on one stream, in this order), each over
// a table of jobs (one per context; a lone batch is one job):
//   k_stage             a lone batch's arguments and job to device memory
//   k_classify_multi    resonant orders of each (omega, species) into
//                       fixed slots, one warp per (omega, species)
//   k_far_orders, k_far_levels  (large batches) coefficients of the power
//                       series in omega that sums a frequency's far orders
//   k_pole_sums_multi   the pole sums over all orders: order chunks x omega
//                       tiles x lanes of a frequency.  Plain path in FP64; fast
//                       path (pole_fused) in double-float on the FP32 pipes,
//                       all orders of a chunk in one set of sums
//   k_resonant_lanes    (mixed batches of 2560 and more) principal value +
//                       Landau per resonant (omega, species, n), an item per
//                       lane; marks the few items it leaves
//   k_resonant_multi    the same for all others: occupied slots gathered into
//                       batches of 32; scalar work one item per lane, the
//                       principal value one item per warp as weights of the
//                       window's nodes (FP64 or double-float)
//   k_finalize_multi    chi, epsilon, wave tensor and det, one thread (or
//                       warp) per omega; sums in a fixed order, so results
//                       do not depend on timing or on the other jobs.
// Small batches run all of it in one launch: k_disp_one, k_disp_many.
//
// Double-float (fast path): a value is a pair of floats h + l (about 46-48
// bits) handled with error-free transformations (device_math.cuh); GB300
// runs FP32 at 64 times its FP64 rate.  Resonance decisions, windows and
// sample points are the reference's on both paths.
#include <algorithm>
#include <array>
#include <atomic>
#include <cstddef>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

#include "alps_internal.cuh"
#include "device_math.cuh"

// what the kernels read of one context (the plasma at its current k)
struct __align__(16) DispArgs {
  SysDev sys;
  SpecDev sp[ALPS_MAX_SPECIES];
  int rcap;      // max resonant slots over species
  int relcap;    // order slots per relativistic species (max nmax + 1), 0 if none
  int has_bm;    // some species go through the NHDS closed form
};

// the shape of one batch: the order chunks of the pole sums and the items
// per warp of k_resonant.  It follows from the batch size and the context
// alone, so a batch sums in the same order wherever it runs.
struct DispShape {
  int js;        // lanes per frequency of the pole sums (a power of two up to 32)
  int wt;        // warps of frequencies: ceil(n js / 32)
  int kmid;      // longest Laurent series that a lane sums alone
  int nchunk;    // order chunks of the species with the most (the stride of the partial sums)
  int nch[ALPS_MAX_SPECIES];  // order chunks of each species (0: no pole sums)
  int ipw;       // resonant-item slots per warp of k_resonant (1..256)
  int fin_warp;  // k_finalize takes a warp per omega (else a thread)
  int far;       // orders beyond the frequency's reach through the far-order series
  int lanes;     // slots per warp of k_resonant_lanes, which takes the items, k_resonant_multi
                 // what it leaves (0: k_resonant_multi takes all)
};

namespace {

// ---------------------------------------------------------------------------
// One warp per (omega, species): the lanes test the orders -nmax..nmax
// and a ballot prefix gives every resonant order its slot in increasing nn,
// so the slot order does not depend on the launch shape.
// whether order nn is resonant: an FP32 estimate of Re p_res settles the
// orders clearly outside or inside the resonance interval (its bounds carry a
// margin of 1e-5 of its extent, the estimate's error is below 2^-22 |p|); the
// FP64 test decides near the interval's ends
__device__ __forceinline__ bool order_resonant(const SysDev& sys, const SpecDev& S, double2 o, int nn, float ikp32) {
  const float x32 = (float)(S.ms * o.x - (double)nn * S.qs) * ikp32;
  const float mg = 9.5367431640625e-7f * fabsf(x32);
  if (x32 < S.qlo - mg || x32 > S.qhi + mg) return false;
  if (x32 > S.qlo_in + mg && x32 < S.qhi_in - mg) return true;
  return res_geometry(S, sys.M_I, o, nn, sys.kpar).res;
}

__device__ __forceinline__ void classify_body(const DispArgs& a, const double2* __restrict__ om, int n_om,
                                              int* count, int* slot_nn, int* flags, long wid) {
  const int lane = threadIdx.x & 31;
  const int S_ = a.sys.nspec;
  if (wid >= (long)n_om * S_) return;
  const int t = (int)(wid / S_), s = (int)(wid % S_);
  const SpecDev& S = a.sp[s];
  if (S.relat || S.bm) {  // relativistic orders run in k_rel_orders, NHDS species in k_nhds
    if (lane == 0) count[(size_t)t * S_ + s] = 0;
    return;
  }
  const double2 o = om[t];
  int* slots = slot_nn + ((size_t)t * S_ + s) * a.rcap;
  int cnt = 0;
  const float ikp32 = (float)a.sys.ikpar;
  for (int base = -S.nmax; base <= S.nmax; base += 32) {
    const int nn = base + lane;
    bool res = false;
    if (nn <= S.nmax) res = order_resonant(a.sys, S, o, nn, ikp32);
    const unsigned m = __ballot_sync(0xffffffffu, res);
    const int at = cnt + __popc(m & ((1u << lane) - 1u));
    if (res && at < a.rcap) slots[at] = nn;
    cnt += __popc(m);
  }
  if (lane == 0) {
    if (cnt > a.rcap) {
      atomicOr(flags, 1);
      cnt = a.rcap;
    }
    count[(size_t)t * S_ + s] = cnt;
  }
}

// ---------------------------------------------------------------------------
// Pole sums.
//
// A warp is 32 / js frequencies by js lanes, js a power of two (32: one
// frequency over the whole warp, for a few of them; 1: one frequency a
// lane, for lattices).  Its unit of work is an order chunk of one species:
// the signed orders nn = -nmax + chunk, + nch, + 2 nch, ...  The stride
// spreads the orders near resonance, which are neighbours and cost a sum
// over the p_par nodes each, over the chunks; contiguous chunks left them
// all in one block, which the others waited for.
//
// The js lanes of a frequency take an order each for what an order's set-up
// needs (the resonance geometry and its FP64 divisions) and for the Laurent
// series of far poles, whose set-up costs more than its few terms; the
// orders left, long series and node sums, then go over the lanes one by
// one, the lanes slicing their terms.  Each lane keeps its own sums and the
// lanes are added once per chunk.
// ---------------------------------------------------------------------------
// Complex double-float helpers of the order-fused pole sums
__device__ __forceinline__ void df_cmul2(dflt ax, dflt ay, dflt bx, dflt by, dflt& rx, dflt& ry) {
  const dflt x = df_add(df_mul(ax, bx), df_neg(df_mul(ay, by)));
  ry = df_add(df_mul(ax, by), df_mul(ay, bx));
  rx = x;
}

// complex double-float values and the combinations of the base sums
struct cdf {
  dflt x, y;
};
__device__ __forceinline__ cdf cdf_mul(cdf a, cdf b) {
  cdf r;
  df_cmul2(a.x, a.y, b.x, b.y, r.x, r.y);
  return r;
}
__device__ __forceinline__ cdf cdf_add(cdf a, cdf b) { return {df_add(a.x, b.x), df_add(a.y, b.y)}; }
__device__ __forceinline__ cdf cdf_rmul(cdf a, dflt s) { return {df_mul(a.x, s), df_mul(a.y, s)}; }
// omega v1 + kappa v2 (v1, v2 complex)
__device__ __forceinline__ cdf om_comb(cdf o, dflt kap, cdf v1, cdf v2) {
  const cdf r = cdf_mul(o, v1);
  return {df_add(r.x, df_mul(kap, v2.x)), df_add(r.y, df_mul(kap, v2.y))};
}
// omega c1 + kappa c2 (c1, c2 real)
__device__ __forceinline__ cdf om_combr(cdf o, dflt kap, dflt c1, dflt c2) {
  return {df_add(df_mul(o.x, c1), df_mul(kap, c2)), df_mul(o.y, c1)};
}

#define FULL_WARP 0xffffffffu

// adds the js adjacent lanes' values by halving: each step hands half of a
// lane's values to its partner, so 12 values over 32 lanes take 13 additions
// a lane and not 60.  On return v[0 .. cnt) holds the totals of components
// first .. first + cnt of the lane's frequency (cnt 0: none).
struct dbl_val {
  double v;
};
__device__ __forceinline__ dbl_val lane_add(dbl_val a, int off) {
  return {a.v + __shfl_xor_sync(FULL_WARP, a.v, off)};
}
__device__ __forceinline__ dflt lane_add(dflt a, int off) {
  return df_add(a, {__shfl_xor_sync(FULL_WARP, a.h, off), __shfl_xor_sync(FULL_WARP, a.l, off)});
}
// keep + the partner's give
__device__ __forceinline__ dbl_val lane_swap_add(dbl_val keep, dbl_val give, int off) {
  return {keep.v + __shfl_xor_sync(FULL_WARP, give.v, off)};
}
__device__ __forceinline__ dflt lane_swap_add(dflt keep, dflt give, int off) {
  return df_add(keep, {__shfl_xor_sync(FULL_WARP, give.h, off), __shfl_xor_sync(FULL_WARP, give.l, off)});
}
template <typename T>
__device__ __forceinline__ void lane_sum12(T v[12], int js, int lane, int& first, int& cnt) {
  first = 0;
  cnt = 12;
  int off = js >> 1;
  if (off == 0) return;
  bool hi = lane & off;
#pragma unroll
  for (int q = 0; q < 6; ++q) v[q] = lane_swap_add(hi ? v[6 + q] : v[q], hi ? v[q] : v[6 + q], off);
  first = hi ? 6 : 0;
  cnt = 6;
  off >>= 1;
  if (off == 0) return;
  hi = lane & off;
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = lane_swap_add(hi ? v[3 + q] : v[q], hi ? v[q] : v[3 + q], off);
  first += hi ? 3 : 0;
  cnt = 3;
  off >>= 1;
  if (off == 0) return;
  // three values: the lower lane keeps two, the upper one (its second is
  // the lower lane's second added to itself, unused)
  hi = lane & off;
  {
    const T k0 = lane_swap_add(hi ? v[2] : v[0], hi ? v[0] : v[2], off);
    v[1] = lane_swap_add(v[1], v[1], off);
    v[0] = k0;
  }
  first += hi ? 2 : 0;
  cnt = hi ? 1 : 2;
  off >>= 1;
  if (off == 0) return;
  const bool two = cnt == 2;  // the same on both partners of the steps below
  hi = lane & off;
  {
    const T s0 = lane_swap_add((hi && two) ? v[1] : v[0], (hi || !two) ? v[0] : v[1], off);
    v[0] = s0;
  }
  if (two) {
    first += hi ? 1 : 0;
    cnt = 1;
  } else {
    cnt = hi ? 0 : 1;
  }
  off >>= 1;
  if (off == 0) return;
  v[0] = lane_add(v[0], off);
  if (lane & off) cnt = 0;
}

// The far-order series (k_far_orders, k_far_levels) at a frequency: with s = m omega and P the
// largest |k_par p| on the grid, the orders |n| >= n0 have poles |n q| - P or
// more away, and their sum is a power series in s / r, r = n0 |q| - P.  n0 is
// the first with |s| <= 0.4 r.  Returns n0, or INT_MAX where fewer than ten
// orders would be left to the series.
struct FarLevel {
  int n0, K, K32;
  double r;
};
__device__ __forceinline__ FarLevel far_level(const SysDev& sys, const SpecDev& S, double2 o, bool on) {
  FarLevel f = {0x7fffffff, 0, 0, 1.0};
  if (!on || !S.farn) return f;
  const float q = fabsf((float)S.qs), P = fabsf((float)sys.kpar) * (fabsf(S.pcen32) + S.prad32);
  const float sx = (float)(S.ms * o.x), sy = (float)(S.ms * o.y), sa = sqrtf(fmaf(sx, sx, sy * sy));
  const float t = (2.5f * sa + P) / q * 1.00001f;
  if (!(t < 1e6f)) return f;
  const int n0 = max(S.farn, (int)ceilf(t));
  if (n0 - S.farn >= FAR_LEVELS || n0 + 4 > S.nmax) return f;
  f.n0 = n0;
  f.r = (double)n0 * fabs(S.qs) - fabs(sys.kpar) * (fabs(S.pcen) + S.prad);
  // rho <= 0.4: terms to 2^-55 of the bound, 2^-33 in double-float
  const float rho = sa / (float)f.r, lr = -__logf(fmaxf(rho, 1e-30f)), l1 = log1pf(-rho);
  f.K = min(FAR_K, (int)ceilf((38.1230949f - l1) / lr) + 1);
  f.K32 = min(f.K, (int)ceilf((22.8738570f - l1) / lr) + 1);
  return f;
}

// what the lanes of a frequency need of one signed order
struct OrderInfo {
  int nn, K, K32;         // K > kfar: node sum; else the Laurent terms (K32 of them in double-float)
  int lo1, hi1, lo2, hi2; // summed node ranges
  int flags;              // 1 resonant, 2 the double-float node sum applies, 4 the far orders
};
__device__ __forceinline__ OrderInfo shfl_info(const OrderInfo& a, int src) {
  OrderInfo r;
  r.nn = __shfl_sync(FULL_WARP, a.nn, src);
  r.K = __shfl_sync(FULL_WARP, a.K, src);
  r.K32 = __shfl_sync(FULL_WARP, a.K32, src);
  r.lo1 = __shfl_sync(FULL_WARP, a.lo1, src);
  r.hi1 = __shfl_sync(FULL_WARP, a.hi1, src);
  r.lo2 = __shfl_sync(FULL_WARP, a.lo2, src);
  r.hi2 = __shfl_sync(FULL_WARP, a.hi2, src);
  r.flags = __shfl_sync(FULL_WARP, a.flags, src);
  return r;
}

// ---------------------------------------------------------------------------
// Fast path, on the base tables: per (omega, signed order) the sums of the
// three Bessel families against g1 and g2 (6 real vectors, complex
// weights), in double-float on the FP32 pipes:
//   * node sums Q = sum_j w_j F_j R_j, R_j = 1/(A - k_par p_j + i D), the
//     p_par-weighted entries from zeta Q - (1/k_par) sum w F (the sums of
//     the family vectors over the summed ranges: full-range table, or FP64
//     prefix sums where a resonance window is cut out);
//   * far poles: the Laurent series Q = f sum_k mom_k t^k, d = p_res - pcen,
//     t = prad/d, f = 1/(k_par d); with T = f sum_{k>=1}, U = f sum_{k>=2}:
//     sum F p R = pcen Q + d T, sum F p^2 R = pcen^2 Q + 2 pcen d T + d^2 U
//     (no cancellation for far poles); the terms from K32 on in FP32;
//   * in large batches, the orders |n| >= n0 in one series of omega (far_level).
// g1 and g2, two nodes' R and two powers of t go side by side through packed
// instructions.  An FP32 test settles orders far from resonance (the FP64 geometry decides
// the rest).  Each order's entries X_e = omega S_{e,1} + kappa S_{e,2} are
// added, times the order factor C0 v_e(n) (sign of -n for xy, xz), to one
// double-float sum per entry; the phase (i for xy, yz) and the entry scale
// are applied once per chunk in FP64.
//
// Bound by FP32 issue on lattices and by the length of one warp's chain of
// instructions on a few frequencies.  One loop body serves every order (a
// lane's own series, then the orders shared by the lanes), which keeps the
// code in the instruction cache.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void pole_fused(const SysDev& sys, const SpecDev& S, double2 o, bool active, int js,
                                           int chunk, int nch, int kmid, bool far, double* out) {
  const int M = S.M, U_ = 2 * S.nmax + 1;
  const FarLevel fl = far_level(sys, S, o, active && far);
  const int lane = threadIdx.x & 31, j = lane & (js - 1), gbase = lane - j;
  const unsigned gmask = (js == 32) ? FULL_WARP : (((1u << js) - 1u) << gbase);
  const double kpar = sys.kpar;
  dflt acc[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) acc[q] = {0.0f, 0.0f};
  const dflt oxd = df_of(o.x), oyd = df_of(o.y), msd = df_of(S.ms), qsd = df_of(S.qs);
  const cdf omd = {oxd, oyd};
  const dflt kap = {S.kaph, S.kapl};
  const dflt kd = df_of(kpar), ikd = df_of(sys.ikpar), pcd = df_of(S.pcen), prd = df_of(S.prad);
  const dflt Dd = df_mul(msd, oyd);  // m omega_i
  const dflt D2 = df_mul(Dd, Dd);
  const dflt dyd = df_mul(Dd, ikd);  // Im p_res
  const dflt mox = df_mul(msd, oxd);
  const float ikp32 = (float)sys.ikpar;
  for (int i0 = 0; chunk + i0 * nch < U_ + (far ? 1 : 0); i0 += js) {
    // ---- this lane's own order: resonance geometry, series or nodes ----
    const int u = chunk + (i0 + j) * nch;
    // (unit U_ is the far orders')
    const bool isfar = fl.n0 != 0x7fffffff && u == U_;
    const bool own = isfar || (active && u < U_ && abs(u - S.nmax) < fl.n0);
    OrderInfo cur = {0, S.kfar + 1, S.kfar + 1, 1, 0, 1, 0, 0};
    if (isfar) {
      cur.K = fl.K;
      cur.K32 = fl.K32;
      cur.flags = 4;
    } else if (own) {
      const int nn = u - S.nmax;
      // A = m omega_r - nn q, the pole's real part times k_par
      const dflt Ad = df_add(mox, df_neg(df_mul({(float)nn, 0.0f}, qsd)));
      const float x32 = Ad.h * ikp32;
      const float mg = 9.5367431640625e-7f * fabsf(x32);  // 2^-20 |x|
      bool res = false;
      float ddf;  // |p_res - pcen|^2 (in FP32 alone for orders far from resonance)
      cur.nn = nn;
      cur.hi1 = M - 1;
      if (x32 < S.qlo - mg || x32 > S.qhi + mg) {
        const float dx = x32 - S.pcen32;
        ddf = fmaf(dx, dx, dyd.h * dyd.h);
      } else {
        const ResGeom g = res_geometry_of(S, sys, o, nn);
        const float dx = (float)(g.pr - S.pcen);
        ddf = fmaf(dx, dx, dyd.h * dyd.h);
        res = g.res;
        cur.lo1 = g.lo1;
        cur.hi1 = g.hi1;
        cur.lo2 = g.lo2;
        cur.hi2 = g.hi2;
      }
      // the series is used up to rho^2 < 0.58, where its K <= kfar terms
      // (checked below) cost less than the node sum
      if (!res && S.prad32 * S.prad32 < 0.58f * ddf) {
        const float rho = S.prad32 * rsqrtf(ddf);
        const float lr = -__logf(rho), l1 = log1pf(-rho);
        cur.K = (int)ceilf((36.7368006f - l1) / lr) + 1;    // 53 ln 2
        cur.K32 = (int)ceilf((22.8738570f - l1) / lr) + 1;  // 33 ln 2
      }
      // the double-float values stay normal floats: |f| = 1/(k_par |d|) for
      // the series, |A - k_par p_j|^2 + D^2 at the summed ranges' ends for
      // the node sum (zero if the pole lies inside a summed range)
      if (cur.K <= S.kfar) {
        const float fm = fabsf(ikp32) * rsqrtf(ddf);
        if (!(fm >= 1e-30f && fm <= 1e30f)) cur.K = cur.K32 = S.kfar + 1;
      }
      bool nodes_df = true;
      if (cur.K > S.kfar) {
        float lo = 3.0e38f, hi = 0.0f;
        const int ends[4] = {cur.lo1, cur.hi1, cur.lo2, cur.hi2};
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
          const int j0 = max(1, ends[2 * r2]), j1 = min(M - 1, ends[2 * r2 + 1]);
          if (j0 > j1) continue;
          const float d0 = Ad.h - kd.h * S.pph[j0], d1 = Ad.h - kd.h * S.pph[j1];
          lo = ((d0 < 0.0f) != (d1 < 0.0f)) ? 0.0f : fminf(lo, fminf(fabsf(d0), fabsf(d1)));
          hi = fmaxf(hi, fmaxf(fabsf(d0), fabsf(d1)));
        }
        const float d2 = D2.h;
        nodes_df = d2 + lo * lo >= 1e-30f && d2 + hi * hi <= 1e30f;
      }
      cur.flags = (res ? 1 : 0) | (nodes_df ? 2 : 0);
    }
    // a lane sums its own order alone if it is a short series (or if it has
    // the frequency to itself); the others go over the frequency's lanes
    const bool solo = own && (js == 1 || cur.K <= kmid);
    unsigned pend = __ballot_sync(FULL_WARP, own && !solo) & gmask;
    bool go = solo;
    int jj = 0, jc = 1;
    const OrderInfo mine = cur;
    for (;;) {
      if (go && (cur.flags & 4)) {
        // the far orders: entries (xx yy zz xy xz yz) against g1, g2 as power
        // series in t = m omega / r, this slice's terms
        const float* __restrict__ cf = reinterpret_cast<const float*>(S.far) + (size_t)(fl.n0 - S.farn) * FAR_K * 24;
        const double ir = 1.0 / fl.r;
        const cdf t1 = {df_of(S.ms * o.x * ir), df_of(S.ms * o.y * ir)};
        cdf tp = {{1.0f, 0.0f}, {0.0f, 0.0f}}, st = t1;
        for (int q = 0; q < jj; ++q) tp = cdf_mul(tp, t1);
        for (int q = jc; q > 1; q >>= 1) st = cdf_mul(st, st);
        dflt2 Xr[6], Xi[6];
#pragma unroll
        for (int e = 0; e < 6; ++e) Xr[e] = Xi[e] = d2_all({0.0f, 0.0f});
        int k = jj;
        for (; k < cur.K32; k += jc) {
          const float4* c4 = reinterpret_cast<const float4*>(cf + (size_t)k * 24);
          const dflt2 x2 = d2_all(tp.x), y2 = d2_all(tp.y);
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const float4 h = __ldg(c4 + e), l = __ldg(c4 + 3 + e);
            d2_mac(Xr[2 * e], make_float2(h.x, h.y), make_float2(l.x, l.y), x2.h, x2.l);
            d2_mac(Xi[2 * e], make_float2(h.x, h.y), make_float2(l.x, l.y), y2.h, y2.l);
            d2_mac(Xr[2 * e + 1], make_float2(h.z, h.w), make_float2(l.z, l.w), x2.h, x2.l);
            d2_mac(Xi[2 * e + 1], make_float2(h.z, h.w), make_float2(l.z, l.w), y2.h, y2.l);
          }
          tp = cdf_mul(tp, st);
        }
        float fx = tp.x.h + tp.x.l, fy = tp.y.h + tp.y.l;
        const float gx = st.x.h + st.x.l, gy = st.y.h + st.y.l;
        for (; k < cur.K; k += jc) {
          const float4* c4 = reinterpret_cast<const float4*>(cf + (size_t)k * 24);
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const float4 h = __ldg(c4 + e);
            Xr[2 * e].l = __ffma2_rn(make_float2(h.x, h.y), f2_all(fx), Xr[2 * e].l);
            Xi[2 * e].l = __ffma2_rn(make_float2(h.x, h.y), f2_all(fy), Xi[2 * e].l);
            Xr[2 * e + 1].l = __ffma2_rn(make_float2(h.z, h.w), f2_all(fx), Xr[2 * e + 1].l);
            Xi[2 * e + 1].l = __ffma2_rn(make_float2(h.z, h.w), f2_all(fy), Xi[2 * e + 1].l);
          }
          const float nx = fx * gx - fy * gy;
          fy = fx * gy + fy * gx;
          fx = nx;
        }
        const dflt z = {0.0f, 0.0f};
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          const cdf x = om_comb(omd, kap, {df_add(d2_x(Xr[e]), z), df_add(d2_x(Xi[e]), z)},
                                {df_add(d2_y(Xr[e]), z), df_add(d2_y(Xi[e]), z)});
          df_acc(acc[2 * e], x.x);
          df_acc(acc[2 * e + 1], x.y);
        }
      } else if (go) {
        const int nn = cur.nn, n = nn < 0 ? -nn : nn, K = cur.K, K32 = cur.K32;
        const dflt Ad = df_add(mox, df_neg(df_mul({(float)nn, 0.0f}, qsd)));
        const float* __restrict__ Bn = S.Bt + (size_t)n * (M - 1) * 12;
        const float* __restrict__ mBn = S.mBt + (size_t)n * ALPS_KFAR * 12;
        cdf X[6];  // the order's entries (xx yy zz xy xz yz), scaled by 1/Vscale[n]
        if (K > S.kfar && !(cur.flags & 2)) {
          // FP64 node sum of this order over V, X_e = omega S_e1 + kappa S_e2
          const double* __restrict__ Vn = S.V + (size_t)n * (M - 1) * 12;
          const double Ar = S.ms * o.x - (double)nn * S.qs, Di = S.ms * o.y;
          double2 Sx[12];
#pragma unroll
          for (int q = 0; q < 12; ++q) Sx[q] = cmk(0.0, 0.0);
          for (int r2 = 0; r2 < 2; ++r2) {
            const int b = r2 ? cur.lo2 : cur.lo1, e = r2 ? cur.hi2 : cur.hi1;
            const int lo = max(1, b), hi = min(M - 1, e);
            for (int jn = lo + ((jj - lo + 1) & (jc - 1)); jn <= hi; jn += jc) {
              const double wgt = (b < e && (jn == b || jn == e)) ? 0.5 : 1.0;
              const double dr = fma(-kpar, S.ppar[jn], Ar);
              const double rr = wgt / fma(dr, dr, Di * Di);
              const double* v = Vn + (size_t)(jn - 1) * 12;
#pragma unroll
              for (int q = 0; q < 12; ++q) {
                Sx[q].x = fma(v[q], dr * rr, Sx[q].x);
                Sx[q].y = fma(v[q], -Di * rr, Sx[q].y);
              }
            }
          }
          const double isc = 1.0 / S.Vscale[n], kapd = S.kappa;
#pragma unroll
          for (int e = 0; e < 6; ++e) {
            const double2 t = cscale(cadd(cmul(o, Sx[2 * e]), cscale(Sx[2 * e + 1], kapd)), isc);
            X[e] = {df_of(t.x), df_of(t.y)};
          }
        } else if (K <= S.kfar) {
          // Laurent series: d = p_res - pcen, t = prad/d, f = 1/(k_par d)
          const int k0 = (jj >= 2) ? jj : jj + jc * ((2 - jj + jc - 1) / jc);  // first k >= 2 of this slice
          const cdf d = {df_add(df_mul(Ad, ikd), df_neg(pcd)), dyd};
          const dflt r = df_rcp_approx(df_add(df_mul(d.x, d.x), df_mul(d.y, d.y)));
          const cdf iv = {df_mul(d.x, r), df_neg(df_mul(d.y, r))};
          const cdf t1 = cdf_rmul(iv, prd), f = cdf_rmul(iv, ikd);
          // U = f sum_{k >= 2} mom_k t^k over this slice's k: powers from f t^k0,
          // step t^jc (both by squaring)
          cdf tp = f, st = t1;
          {
            cdf pw = t1;
            for (int q = k0; q; q >>= 1) {
              if (q & 1) tp = cdf_mul(tp, pw);
              pw = cdf_mul(pw, pw);
            }
            for (int q = jc; q > 1; q >>= 1) st = cdf_mul(st, st);
          }
          // sums over (g1, g2) side by side, real and imaginary parts; two
          // terms' powers side by side, steps of t^2jc
          dflt2 Ur[3], Ui[3];
          float2 Fr[3], Fi[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            Ur[q] = Ui[q] = d2_all({0.0f, 0.0f});
            Fr[q] = Fi[q] = f2_all(0.0f);
          }
          auto term = [&](int k, dflt tx, dflt ty) {
            const float4* m4 = reinterpret_cast<const float4*>(mBn + (size_t)k * 12);
            const float4 a0 = __ldg(m4), a1 = __ldg(m4 + 1), a2 = __ldg(m4 + 2);
            const float2 h[3] = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}};
            const float2 l[3] = {{a1.z, a1.w}, {a2.x, a2.y}, {a2.z, a2.w}};
            const dflt2 x2 = d2_all(tx), y2 = d2_all(ty);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              d2_mac(Ur[q], h[q], l[q], x2.h, x2.l);
              d2_mac(Ui[q], h[q], l[q], y2.h, y2.l);
            }
          };
          int k = k0;
          cdf tl = tp;  // the first power left to the tail
          if (k < K32) {
            const cdf tb = cdf_mul(tp, st), s2 = cdf_mul(st, st);
            dflt2 px = d2_of(tp.x, tb.x), py = d2_of(tp.y, tb.y);
            const dflt2 sx = d2_all(s2.x), sy = d2_all(s2.y);
            for (;;) {
              if (k >= K32) {
                tl = {d2_x(px), d2_x(py)};
                break;
              }
              term(k, d2_x(px), d2_x(py));
              k += jc;
              if (k >= K32) {
                tl = {d2_y(px), d2_y(py)};
                break;
              }
              term(k, d2_y(px), d2_y(py));
              k += jc;
              const dflt2 nx = d2_add(d2_mul(px, sx), d2_neg(d2_mul(py, sy)));
              py = d2_add(d2_mul(px, sy), d2_mul(py, sx));
              px = nx;
            }
          }
          if (k < K) {
            // the tail: terms below 2^-33 of the bound, in FP32
            float fx = tl.x.h + tl.x.l, fy = tl.y.h + tl.y.l;
            const float gx = st.x.h + st.x.l, gy = st.y.h + st.y.l;
            for (; k < K; k += jc) {
              const float4* m4 = reinterpret_cast<const float4*>(mBn + (size_t)k * 12);
              const float4 a0 = __ldg(m4);
              const float2 h[3] = {{a0.x, a0.y}, {a0.z, a0.w}, __ldg(reinterpret_cast<const float2*>(m4 + 1))};
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                Fr[q] = __ffma2_rn(h[q], f2_all(fx), Fr[q]);
                Fi[q] = __ffma2_rn(h[q], f2_all(fy), Fi[q]);
              }
              const float nx = fx * gx - fy * gy;
              fy = fx * gy + fy * gx;
              fx = nx;
            }
          }
          // per family F1, F2, F3: omega U_{F,g1} + kappa U_{F,g2}
          cdf Uw[3];
#pragma unroll
          for (int fm = 0; fm < 3; ++fm) {
            const cdf u1 = {df_add(d2_x(Ur[fm]), {Fr[fm].x, 0.0f}), df_add(d2_x(Ui[fm]), {Fi[fm].x, 0.0f})};
            const cdf u2 = {df_add(d2_y(Ur[fm]), {Fr[fm].y, 0.0f}), df_add(d2_y(Ui[fm]), {Fi[fm].y, 0.0f})};
            Uw[fm] = om_comb(omd, kap, u1, u2);
          }
          // T = f mom_1 t + U, Q = f mom_0 + T on the slices that own k = 1, 0
          cdf T[3] = {Uw[0], Uw[1], Uw[2]};
          auto mterm = [&](int kk, cdf w, cdf* outv) {
            const float* m = mBn + (size_t)kk * 12;
#pragma unroll
            for (int fm = 0; fm < 3; ++fm) {
              const cdf mw = om_combr(omd, kap, {m[2 * fm], m[6 + 2 * fm]}, {m[2 * fm + 1], m[6 + 2 * fm + 1]});
              outv[fm] = cdf_add(outv[fm], cdf_mul(w, mw));
            }
          };
          if (jj == (jc > 1 ? 1 : 0)) mterm(1, cdf_mul(f, t1), T);
          cdf Q[3] = {T[0], T[1], T[2]};
          if (jj == 0) mterm(0, f, Q);
          X[0] = Q[0];
          X[1] = Q[1];
          X[3] = Q[2];
          X[4] = cdf_mul(d, T[0]);
          X[5] = cdf_mul(d, T[2]);
          if (S.pcen32 != 0.0f) {
            // sum F p R = pcen Q + d T, sum F p^2 R = pcen (sum F p R) + d (pcen T + d U)
            X[4] = cdf_add(cdf_rmul(Q[0], pcd), X[4]);
            X[5] = cdf_add(cdf_rmul(Q[2], pcd), X[5]);
            X[2] = cdf_add(cdf_rmul(X[4], pcd), cdf_mul(d, cdf_add(cdf_rmul(T[0], pcd), cdf_mul(d, Uw[0]))));
          } else {
            X[2] = cdf_mul(d, cdf_mul(d, Uw[0]));
          }
        } else {
          // node sum in double-float: Q_b = sum_j w_j B_b(j) / (A - k_par p_j + i D)
          // (g1, g2 side by side; two nodes' R side by side)
          dflt2 Qr[3], Qi[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) Qr[q] = Qi[q] = d2_all({0.0f, 0.0f});
          auto mac = [&](int jn, dflt Rr, dflt Ri) {
            const float4* b4 = reinterpret_cast<const float4*>(Bn + (size_t)(jn - 1) * 12);
            const float4 a0 = __ldg(b4), a1 = __ldg(b4 + 1), a2 = __ldg(b4 + 2);
            const float2 h[3] = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}};
            const float2 l[3] = {{a1.z, a1.w}, {a2.x, a2.y}, {a2.z, a2.w}};
            const dflt2 r2 = d2_all(Rr), i2 = d2_all(Ri);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              d2_mac(Qr[q], h[q], l[q], r2.h, r2.l);
              d2_mac(Qi[q], h[q], l[q], i2.h, i2.l);
            }
          };
          const dflt2 Ad2 = d2_all(Ad), kd2 = d2_all(df_neg(kd)), DD2 = d2_all(D2), nD2 = d2_all(df_neg(Dd));
          // nodes ja and jb (jb < 0: ja alone), weight -1/2 for range ends
          auto nodes = [&](int ja, int jb, bool end) {
            const int jq = jb < 0 ? ja : jb;
            const dflt2 pp = {make_float2(S.pph[ja], S.pph[jq]), make_float2(S.ppl[ja], S.ppl[jq])};
            const dflt2 dr = d2_add(Ad2, d2_mul(kd2, pp));
            const dflt2 r = d2_rcp_approx(d2_add(d2_mul(dr, dr), DD2));
            dflt2 Rr = d2_mul(dr, r), Ri = d2_mul(nD2, r);
            if (end) {
              Rr = {__fmul2_rn(Rr.h, f2_all(-0.5f)), __fmul2_rn(Rr.l, f2_all(-0.5f))};
              Ri = {__fmul2_rn(Ri.h, f2_all(-0.5f)), __fmul2_rn(Ri.l, f2_all(-0.5f))};
            }
            mac(ja, d2_x(Rr), d2_x(Ri));
            if (jb >= 0) mac(jb, d2_y(Rr), d2_y(Ri));
          };
          // the summed ranges (disjoint), each over this slice's nodes
          // jn = 1 + jj (mod jc), then their ends again at weight -1/2
          for (int r2 = 0; r2 < 2; ++r2) {
            const int b = r2 ? cur.lo2 : cur.lo1, e = r2 ? cur.hi2 : cur.hi1;
            const int lo = max(1, b), hi = min(M - 1, e);
            for (int jn = lo + ((jj - lo + 1) & (jc - 1)); jn <= hi; jn += 2 * jc)
              nodes(jn, jn + jc <= hi ? jn + jc : -1, false);
          }
          for (int q = 0; q < 4; ++q) {
            const int b = (q & 2) ? cur.lo2 : cur.lo1, e = (q & 2) ? cur.hi2 : cur.hi1, jn = (q & 1) ? e : b;
            if (b < e && jn >= 1 && jn <= M - 1 && ((jn - 1 - jj) & (jc - 1)) == 0) nodes(jn, -1, true);
          }
          cdf P[3];
#pragma unroll
          for (int fm = 0; fm < 3; ++fm)
            P[fm] = om_comb(omd, kap, {d2_x(Qr[fm]), d2_x(Qi[fm])}, {d2_y(Qr[fm]), d2_y(Qi[fm])});
          const cdf zeta = {df_mul(Ad, ikd), dyd};
          // (1/k_par) times the omega-combined sums of F1, F3 and p_par F1
          // over the summed ranges: six real sums C_c, added once; lane c
          // of the slices forms C_c where there are eight or more of them,
          // the first slice all six otherwise
          auto csum = [&](int c) -> double {
            if (!(cur.flags & 1)) return S.Cfull[(size_t)n * 6 + c];
            const double* __restrict__ P0 = S.Pre + (size_t)n * M * 6;
            const double* __restrict__ Vn = S.V + (size_t)n * (M - 1) * 12;
            const int q = (c < 2) ? c : c + 4;
            const double isc = 1.0 / S.Vscale[n];
            double C = 0.0;
            for (int r2 = 0; r2 < 2; ++r2) {
              const int b = r2 ? cur.lo2 : cur.lo1, e = r2 ? cur.hi2 : cur.hi1;
              const int lo = max(1, b), hi = min(M - 1, e);
              if (lo > hi) continue;
              double v = P0[(size_t)hi * 6 + c] - P0[(size_t)(lo - 1) * 6 + c];
              if (b < e) v -= 0.5 * (Vn[(size_t)(lo - 1) * 12 + q] + Vn[(size_t)(hi - 1) * 12 + q]) * isc;
              C += v;
            }
            return C;
          };
          dflt C[6];
#pragma unroll
          for (int c = 0; c < 6; ++c) C[c] = {0.0f, 0.0f};
          if (jc >= 8) {
            if (jj < 6) {
              const dflt v = df_of(csum(jj));
#pragma unroll
              for (int c = 0; c < 6; ++c)
                if (c == jj) C[c] = v;
            }
          } else if (jj == 0) {
#pragma unroll
            for (int c = 0; c < 6; ++c) C[c] = df_of(csum(c));
          }
          X[0] = P[0];
          X[1] = P[1];
          X[3] = P[2];
          const cdf c1 = cdf_rmul(om_combr(omd, kap, C[0], C[1]), ikd);
          const cdf c3 = cdf_rmul(om_combr(omd, kap, C[2], C[3]), ikd);
          const cdf cp = cdf_rmul(om_combr(omd, kap, C[4], C[5]), ikd);
          cdf xz = cdf_mul(zeta, P[0]), yz = cdf_mul(zeta, P[2]);
          xz = {df_add(xz.x, df_neg(c1.x)), df_add(xz.y, df_neg(c1.y))};
          yz = {df_add(yz.x, df_neg(c3.x)), df_add(yz.y, df_neg(c3.y))};
          const cdf zz = cdf_mul(zeta, xz);
          X[2] = {df_add(zz.x, df_neg(cp.x)), df_add(zz.y, df_neg(cp.y))};
          X[4] = xz;
          X[5] = yz;
        }
        // add the order's entries with its factors C0 v_e(n) (xy and xz odd in n)
        const float* __restrict__ fac = S.bfac + (size_t)n * 12;
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          dflt fe = {fac[2 * e], fac[2 * e + 1]};
          if (nn < 0 && (e == 3 || e == 4)) fe = df_neg(fe);
          df_acc(acc[2 * e], df_mul(fe, X[e].x));
          df_acc(acc[2 * e + 1], df_mul(fe, X[e].y));
        }
      }
      if (!__any_sync(FULL_WARP, pend != 0)) break;
      go = pend != 0;
      const int t = go ? __ffs(pend) - 1 : lane;
      pend &= pend - 1;
      cur = shfl_info(mine, t);
      jj = j;
      jc = js;
    }
  }
  // add the lanes, rescale and apply the phase (i for xy and yz)
  int first, cnt;
  lane_sum12(acc, js, lane, first, cnt);
  if (!active) return;
#pragma unroll
  for (int q = 0; q < 12; ++q)
    if (q < cnt) {
      const int c = first + q, e = c >> 1;
      const double v = df_val(acc[q]) * S.Escale[e];
      if (e == 3 || e == 5) out[c ^ 1] = (c & 1) ? -v : v;  // (x, y) -> (-y, x)
      else out[c] = v;
    }
}

// Plain path, all in FP64: the trapezoid node sum over the reduced vectors for
// orders in or near resonance, the Laurent series about the grid centre to
// 2^-55 of its bound for the others (rho = prad/|d| < 0.76, K terms for the
// 12 vectors' sums; the p_par-weighted entries follow from T and U as in
// pole_fused, without cancellation).  Bound by the FP64 pipe (two lanes a
// clock and SM): a node takes 33 FP64 instructions (24 are the twelve real
// vectors against R_j), a term 16, and most orders need 12 to 30 terms
// instead of 255 nodes: 2867 map frequencies on a 128x256 grid 3180 us by
// nodes alone, 573 us so.
__device__ __forceinline__ void pole_plain(const SysDev& sys, const SpecDev& S, double2 o, bool active, int js,
                                           int chunk, int nch, int kmid, bool far, double* out) {
  const int M = S.M, U_ = 2 * S.nmax + 1;
  const FarLevel fl = far_level(sys, S, o, active && far);
  const int lane = threadIdx.x & 31, j = lane & (js - 1), gbase = lane - j;
  const unsigned gmask = (js == 32) ? FULL_WARP : (((1u << js) - 1u) << gbase);
  const double kpar = sys.kpar, kappa = S.kappa;
  const double Di = S.ms * o.y, Di2 = Di * Di;
  const double* __restrict__ pp = S.ppar;
  const float ikp32 = (float)sys.ikpar, dy32 = (float)Di * ikp32;
  dbl_val acc[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) acc[q] = {0.0};
  for (int i0 = 0; chunk + i0 * nch < U_ + (far ? 1 : 0); i0 += js) {
    const int u = chunk + (i0 + j) * nch;
    const bool isfar = fl.n0 != 0x7fffffff && u == U_;
    const bool own = isfar || (active && u < U_ && abs(u - S.nmax) < fl.n0);
    OrderInfo cur = {0, S.kfar + 1, 0, 1, 0, 1, 0, 0};
    if (isfar) {
      cur.K = fl.K;
      cur.flags = 4;
    } else if (own) {
      cur.nn = u - S.nmax;
      cur.hi1 = M - 1;
      // the FP32 test of k_classify: an order clearly outside the resonance
      // interval sums every node
      const float x32 = (float)(S.ms * o.x - (double)cur.nn * S.qs) * ikp32;
      const float mg = 9.5367431640625e-7f * fabsf(x32);
      bool res = false;
      if (!(x32 < S.qlo - mg || x32 > S.qhi + mg)) {
        const ResGeom g = res_geometry_of(S, sys, o, cur.nn);
        res = g.res;
        cur.lo1 = g.lo1;
        cur.hi1 = g.hi1;
        cur.lo2 = g.lo2;
        cur.hi2 = g.hi2;
      }
      const float dx = x32 - S.pcen32, ddf = fmaf(dx, dx, dy32 * dy32);
      if (!res && S.prad32 * S.prad32 < 0.58f * ddf && ddf < 1e30f && fabsf(ikp32) < 1e30f) {
        const float rho = S.prad32 * rsqrtf(ddf);
        cur.K = (int)ceilf((38.1230949f - log1pf(-rho)) / -__logf(rho)) + 1;  // 55 ln 2
      }
    }
    const bool solo = own && (isfar || cur.K <= S.kfar) && (js == 1 || cur.K <= kmid);
    unsigned pend = __ballot_sync(FULL_WARP, own && !solo) & gmask;
    bool go = solo;
    int jj = 0, jc = 1;
    const OrderInfo mine = cur;
    for (;;) {
      if (go && (cur.flags & 4)) {
        // the far orders as in pole_fused
        const double* __restrict__ cf = reinterpret_cast<const double*>(S.far) + (size_t)(fl.n0 - S.farn) * FAR_K * 12;
        const double ir = 1.0 / fl.r;
        const double2 t1 = cmk(S.ms * o.x * ir, S.ms * o.y * ir);
        double2 tp = cmk(1.0, 0.0), st = t1;
        for (int q = 0; q < jj; ++q) tp = cmul(tp, t1);
        for (int q = jc; q > 1; q >>= 1) st = cmul(st, st);
        double2 X[12];
#pragma unroll
        for (int e = 0; e < 12; ++e) X[e] = cmk(0.0, 0.0);
        for (int k = jj; k < cur.K; k += jc) {
          const double2* c2 = reinterpret_cast<const double2*>(cf + (size_t)k * 12);
#pragma unroll
          for (int e = 0; e < 6; ++e) {
            const double2 c = __ldg(c2 + e);
            X[2 * e].x = fma(c.x, tp.x, X[2 * e].x);
            X[2 * e].y = fma(c.x, tp.y, X[2 * e].y);
            X[2 * e + 1].x = fma(c.y, tp.x, X[2 * e + 1].x);
            X[2 * e + 1].y = fma(c.y, tp.y, X[2 * e + 1].y);
          }
          tp = cmul(tp, st);
        }
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          const double2 x = cadd(cmul(o, X[2 * e]), cscale(X[2 * e + 1], kappa));
          acc[2 * e].v += x.x;
          acc[2 * e + 1].v += x.y;
        }
      } else if (go) {
        const int cn = cur.nn, n = cn < 0 ? -cn : cn, K = cur.K;
        const double Ar = S.ms * o.x - (double)cn * S.qs;
        double2 X[6];  // omega S_e1 + kappa S_e2
        if (K <= S.kfar) {
          // d = p_res - pcen, t = prad/d, f = 1/(k_par d); U = f sum_{k >= 2}
          // mom_k t^k over this slice's k, per family and g
          const double* __restrict__ mn = S.mom + (size_t)n * ALPS_KFAR * 6;
          const int k0 = (jj >= 2) ? jj : jj + jc * ((2 - jj + jc - 1) / jc);
          const double2 d = cmk(fma(Ar, sys.ikpar, -S.pcen), Di * sys.ikpar);
          const double r = rcp_fast(fma(d.x, d.x, d.y * d.y));
          const double2 iv = cmk(d.x * r, -d.y * r), t1 = cscale(iv, S.prad), f = cscale(iv, sys.ikpar);
          double2 tp = f, st = t1;
          {
            double2 pw = t1;
            for (int q = k0; q; q >>= 1) {
              if (q & 1) tp = cmul(tp, pw);
              pw = cmul(pw, pw);
            }
            for (int q = jc; q > 1; q >>= 1) st = cmul(st, st);
          }
          double2 U[6];
#pragma unroll
          for (int b = 0; b < 6; ++b) U[b] = cmk(0.0, 0.0);
          for (int k = k0; k < K; k += jc) {
            const double2* m2 = reinterpret_cast<const double2*>(mn + (size_t)k * 6);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              const double2 m = __ldg(m2 + b);
              U[2 * b].x = fma(m.x, tp.x, U[2 * b].x);
              U[2 * b].y = fma(m.x, tp.y, U[2 * b].y);
              U[2 * b + 1].x = fma(m.y, tp.x, U[2 * b + 1].x);
              U[2 * b + 1].y = fma(m.y, tp.y, U[2 * b + 1].y);
            }
            tp = cmul(tp, st);
          }
          double2 Uw[3];
#pragma unroll
          for (int F = 0; F < 3; ++F) Uw[F] = cadd(cmul(o, U[2 * F]), cscale(U[2 * F + 1], kappa));
          // T = f mom_1 t + U, Q = f mom_0 + T on the slices that own k = 1, 0
          auto mterm = [&](int k, double2 w, double2* to) {
            const double* m = mn + (size_t)k * 6;
#pragma unroll
            for (int F = 0; F < 3; ++F)
              to[F] = cadd(to[F], cmul(w, cmk(fma(o.x, m[2 * F], kappa * m[2 * F + 1]), o.y * m[2 * F])));
          };
          double2 T[3] = {Uw[0], Uw[1], Uw[2]};
          if (jj == (jc > 1 ? 1 : 0)) mterm(1, cmul(f, t1), T);
          double2 Q[3] = {T[0], T[1], T[2]};
          if (jj == 0) mterm(0, f, Q);
          // sum F p R = pcen Q + d T, sum F p^2 R = pcen (sum F p R) + d (pcen T + d U)
          X[0] = Q[0];
          X[1] = Q[1];
          X[3] = Q[2];
          X[4] = cadd(cscale(Q[0], S.pcen), cmul(d, T[0]));
          X[5] = cadd(cscale(Q[2], S.pcen), cmul(d, T[2]));
          X[2] = cadd(cscale(X[4], S.pcen), cmul(d, cadd(cscale(T[0], S.pcen), cmul(d, Uw[0]))));
        } else {
          const double* __restrict__ Vn = S.V + (size_t)n * (M - 1) * 12;
          double2 Sx[12];
#pragma unroll
          for (int q = 0; q < 12; ++q) Sx[q] = cmk(0.0, 0.0);
          // a range's two ends carry weight 1/2 (a range of a single node none:
          // integrate(a,a) weighs it fully)
          for (int r2 = 0; r2 < 2; ++r2) {
            const int b = r2 ? cur.lo2 : cur.lo1, e = r2 ? cur.hi2 : cur.hi1;
            const int lo = max(1, b), hi = min(M - 1, e);
            for (int jn = lo + ((jj - lo + 1) & (jc - 1)); jn <= hi; jn += jc) {
              const double dr = fma(-kpar, pp[jn], Ar);
              double r = rcp_fast(fma(dr, dr, Di2));
              if (b < e && (jn == b || jn == e)) r *= 0.5;
              const double Rr = dr * r, Ri = -Di * r;
              const double2* v2 = reinterpret_cast<const double2*>(Vn + (size_t)(jn - 1) * 12);
#pragma unroll
              for (int q = 0; q < 6; ++q) {
                const double2 v = __ldg(v2 + q);
                Sx[2 * q].x = fma(v.x, Rr, Sx[2 * q].x);
                Sx[2 * q].y = fma(v.x, Ri, Sx[2 * q].y);
                Sx[2 * q + 1].x = fma(v.y, Rr, Sx[2 * q + 1].x);
                Sx[2 * q + 1].y = fma(v.y, Ri, Sx[2 * q + 1].y);
              }
            }
          }
#pragma unroll
          for (int e = 0; e < 6; ++e) X[e] = cadd(cmul(o, Sx[2 * e]), cscale(Sx[2 * e + 1], kappa));
        }
        // integrate = C0 pref X (xy and xz odd in n); xy and yz carry the
        // factor i, applied at the end
        const double* __restrict__ fac = S.pfac + (size_t)n * 6;
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          if (n == 0 && (e == 0 || e == 3 || e == 4)) continue;
          const double f = (cn < 0 && (e == 3 || e == 4)) ? -fac[e] : fac[e];
          acc[2 * e].v = fma(f, X[e].x, acc[2 * e].v);
          acc[2 * e + 1].v = fma(f, X[e].y, acc[2 * e + 1].v);
        }
      }
      if (!__any_sync(FULL_WARP, pend != 0)) break;
      go = pend != 0;
      const int t = go ? __ffs(pend) - 1 : lane;
      pend &= pend - 1;
      cur = shfl_info(mine, t);
      jj = j;
      jc = js;
    }
  }
  int first, cnt;
  lane_sum12(acc, js, lane, first, cnt);
  if (!active) return;
#pragma unroll
  for (int q = 0; q < 12; ++q)
    if (q < cnt) {
      const int c = first + q, e = c >> 1;
      const double v = acc[q].v;
      if (e == 3 || e == 5) out[c ^ 1] = (c & 1) ? -v : v;
      else out[c] = v;
    }
}

// one warp's unit: an order chunk of species s for a tile of 32 / js
// frequencies; its entries go to part[(w S + s) nchunk + chunk]
__device__ __noinline__ void pole_body(const SysDev& sys, const SpecDev& S, const DispShape& sh,
                                          const double2* __restrict__ om, int n_om, double2* part, int s, long unit) {
  const int chunk = (int)(unit / sh.wt), tile = (int)(unit % sh.wt);
  const int js = sh.js, lane = threadIdx.x & 31;
  const int w = tile * (32 / js) + lane / js;
  const bool active = w < n_om;
  if (tile * (32 / js) >= n_om) return;
  const double2 o = active ? om[w] : cmk(0.0, 0.0);
  double* out = active ? reinterpret_cast<double*>(part + (((size_t)w * sys.nspec + s) * sh.nchunk + chunk) * 6) : nullptr;
  if (S.df_sums)
    pole_fused(sys, S, o, active, js, chunk, sh.nch[s], sh.kmid, sh.far != 0, out);
  else
    pole_plain(sys, S, o, active, js, chunk, sh.nch[s], sh.kmid, sh.far != 0, out);
}

// ---------------------------------------------------------------------------
// Analytic continuation f(pperp_i, complex ppar) (eval_fit,
// src/ALPS_analyt.f90:32-181; fit_function :185-266).
// ---------------------------------------------------------------------------
// fit_function_poly (src/ALPS_analyt.f90:268-363): Chebyshev series in
// t = (p - centre)/half-width, zero for |t| > 1; with log_fit the series is
// log10 f, cut to zero beyond +-poly_log_max
__device__ double2 eval_fit_poly(const SpecDev& S, int iperp, double2 p) {
  const int np = S.poly_order;
  const double* c = S.fit + (size_t)iperp * (np + 1);
  const double n1 = 5.0e-1 * (S.ppar_hi + S.ppar_lo), n2 = 5.0e-1 * (S.ppar_hi - S.ppar_lo);
  double2 t = cmk((p.x - n1) / n2, p.y / n2);
  if (cabs_(t) > 1.0) return cmk(0.0, 0.0);
  double2 b0 = cmk(1.0, 0.0), b1 = t;
  double2 f = cadd(cscale(b0, c[0]), cscale(b1, c[1]));
  for (int n = 2; n <= np; ++n) {
    double2 b2 = csub(cmul(cscale(t, 2.0), b1), b0);
    f = cadd(f, cscale(b2, c[n]));
    b0 = b1;
    b1 = b2;
  }
  if (S.log_fit) {
    const double L = S.poly_log_max;
    if ((f.x < -L) || (f.y < -L) || (f.x > L) || (f.y > L)) return cmk(0.0, 0.0);
    f = cexp_d(cscale(f, 2.302585092994045684));  // 10^f = exp(f ln 10)
  }
  return f;
}

// term f of the continuation at row iperp
__device__ __forceinline__ double2 fit_term_d(const SpecDev& S, double vA, int iperp, int f, double2 p) {
  const double pperp = S.pperp[iperp];
  const double* fit = S.fit;
  const int nf = S.nf, t = S.fit_type[f];
  const double pc = S.perp_corr[f];
  auto P = [&](int k) { return fit[(iperp * 5 + k) * nf + f]; };
  double2 d = csub(p, cmk(P(2), 0.0));
  double2 d2 = cmul(d, d);
  if (t == 1) {
    double a0 = P(0) * exp(-pc * (pperp * pperp));
    return cscale(cexp_d(cscale(d2, -P(1))), a0);
  }
  if (t == 2) {
    double2 kp = cadd(cmk(1.0, 0.0), cadd(cscale(d2, P(1)), cmk(pc * P(4) * (pperp * pperp), 0.0)));
    return cscale(cexp_d(cscale(clog_d(kp), P(3))), P(0));
  }
  if (t == 3) {
    double2 in = cadd(cmk(1.0, 0.0), cscale(cadd(cmk(pperp * pperp, 0.0), d2), vA * vA / (S.ms * S.ms)));
    double2 sq = csqrt_d(in);
    return cscale(cexp_d(cscale(sq, -P(1))), P(0));
  }
  if (t == 6) {
    double2 q = cadd(cmk(P(3) * pc * (pperp * pperp), 0.0), cscale(d2, P(1)));
    double2 arg = cscale(csub(q, cexp_d(q)), 0.5);
    return cscale(cexp_d(arg), P(0));
  }
  return cmk(0.0, 0.0);
}

__device__ double2 eval_fit_d(const SpecDev& S, double vA, int iperp, double2 p) {
  if (S.ac_method == 2) return eval_fit_poly(S, iperp, p);
  double pperp = S.pperp[iperp];
  if (S.ac_method == 0) {
    // distribution_analyt (distribution/distribution_analyt.f90:59-79)
    double ms;
    if (S.species_index == 1) ms = 1.0;
    else if (S.species_index == 2) ms = 1.0 / 1836.0;
    else return cmk(0.0, 0.0);
    double norm = pow(ALPS_PI, -1.5) / pow(ms * 1.0, 1.5);
    double2 p2 = cmul(p, p);
    double2 arg = cmk(-(p2.x / ms + (pperp * pperp) / ms), -(p2.y / ms));
    return cscale(cexp_d(arg), norm);
  }
  double2 ff = cmk(0.0, 0.0);
  for (int f = 0; f < S.nf; ++f) ff = cadd(ff, fit_term_d(S, vA, iperp, f, p));
  return ff;
}

// The continuation at p, p + pd and p - pd.  A kappa term P0 z^K, z = 1 + P1
// (p - P2)^2 + ...: with zb = z(p) + P1 pd^2,
//   z(p +- pd) = zb (1 +- u), u = 2 P1 (p - P2) pd / zb,   z(p) = zb (1 - b), b = P1 pd^2 / zb,
// so one complex power and two short binomial series (to 2^-58) give all
// three, where |u| (|K| + 1) <= 1/2 and none of them crosses the logarithm's
// cut.  Bound by the FP64 pipe: the resonant kernel of 700 frequencies on a
// 193x385 grid 386 us with three powers a row, 336 us so.
__device__ void eval_fit3_d(const SpecDev& S, double vA, int iperp, double2 p, double pd, double2& f0, double2& fp,
                            double2& fm) {
  const double2 pu = cadd(p, cmk(pd, 0.0)), pl = csub(p, cmk(pd, 0.0));
  if (S.ac_method != 1) {
    f0 = eval_fit_d(S, vA, iperp, p);
    fp = eval_fit_d(S, vA, iperp, pu);
    fm = eval_fit_d(S, vA, iperp, pl);
    return;
  }
  f0 = fp = fm = cmk(0.0, 0.0);
  for (int f = 0; f < S.nf; ++f) {
    if (S.fit_type[f] == 2) {
      const double pperp = S.pperp[iperp];
      auto P = [&](int k) { return S.fit[(iperp * 5 + k) * S.nf + f]; };
      const double P1 = P(1), K = P(3);
      const double2 d = cmk(p.x - P(2), p.y), d2 = cmul(d, d);
      const double2 zb = cmk(1.0 + (P1 * (d2.x + pd * pd) + S.perp_corr[f] * P(4) * (pperp * pperp)), P1 * d2.y);
      const double r = rcp_fast(fma(zb.x, zb.x, zb.y * zb.y));
      const double2 iz = cmk(zb.x * r, -zb.y * r);
      const double2 u = cscale(cmul(iz, d), 2.0 * P1 * pd), b = cscale(iz, -(P1 * (pd * pd)));  // b: minus b
      const float ka = fabsf((float)K), ua = sqrtf((float)fma(u.x, u.x, u.y * u.y)),
                  ba = sqrtf((float)fma(b.x, b.x, b.y * b.y));
      if (ua * (ka + 1.0f) <= 0.5f && ua <= 0.1f && ba * (ka + 1.0f) <= 0.1f && ba <= 0.02f && ka < 64.0f &&
          (zb.x > 0.0 || fabs(zb.y) > -0.25 * zb.x)) {
        const double2 w = cscale(cexp_d(cscale(clog_d(zb), K)), P(0));
        // even and odd parts of (1 + u)^K
        double2 ev = cmk(1.0, 0.0), od = cscale(u, K), t = od;
        float mag = ka * ua;
        for (int n = 1; n < 64 && mag > 3.5e-18f; ++n) {
          const double g = (K - (double)n) * rcp_fast((double)(n + 1));
          mag *= ua * (ka + (float)n) / (float)(n + 1);
          t = cscale(cmul(t, u), g);
          if (n & 1) ev = cadd(ev, t);
          else od = cadd(od, t);
        }
        double2 e0 = cadd(cmk(1.0, 0.0), cscale(b, K));
        t = cscale(b, K);
        mag = ka * ba;
        for (int n = 1; n < 64 && mag > 3.5e-18f; ++n) {
          mag *= ba * (ka + (float)n) / (float)(n + 1);
          t = cscale(cmul(t, b), (K - (double)n) * rcp_fast((double)(n + 1)));
          e0 = cadd(e0, t);
        }
        fp = cadd(fp, cmul(w, cadd(ev, od)));
        fm = cadd(fm, cmul(w, csub(ev, od)));
        f0 = cadd(f0, cmul(w, e0));
        continue;
      }
    }
    f0 = cadd(f0, fit_term_d(S, vA, iperp, f, p));
    fp = cadd(fp, fit_term_d(S, vA, iperp, f, pu));
    fm = cadd(fm, fit_term_d(S, vA, iperp, f, pl));
  }
}

// ---------------------------------------------------------------------------
// Resonant items: the principal-value part of integrate_res
// (src/ALPS_fns.f90:1000-1236) and landau_integrate (:1327-1452) for one
// (omega, species, n).
//
// Principal value.  Summed over iperp, funct_g (:1243-1321) is the linear
// interpolation H_e(p) = h_e(jc) + s_e(jc) (p - ppar_jc) on the node values
// h_e(j) = omega V_{e,1}(j) + kappa V_{e,2}(j) with the centred slope
// s_e(j) = (h_e(j+1) - h_e(j-1)) / (2 dppar).  The sum over samples
//   T_e = sum_k w_k [ H_e(p_k) / (dx_k - i y) - H_e(2 p_res - p_k) / (dx_k + i y) ],
// dx_k = p_k - p_res, y = Im p_res, therefore needs of each piece jc only the
// sums over its samples of w r dx, w r and w r dx^2, r = 1/(dx^2 + y^2): they
// give the weights' sum A and first moment B, and with them T_e is a weighted
// sum over a few nodes, W_j = A_j + (B_{j-1} - B_{j+1}) / (2 dppar),
//   T_e = sum_j (omega V_{e,1}(j) + kappa V_{e,2}(j)) W_j.
// Both sides of the window share the sums: they are running (prefix) sums
// over k, cut where a side moves to its next piece.
//
// The cuts are the reference's decisions.  An FP32 estimate in units of a
// spacing, measured from the node next to p_res, settles each to 5e-6 of a
// spacing (more where it is far from p_res, or the grid long: pv_cut); nearer,
// the search over the reference's own sample points does.
// Exactly half-way its rounded distances may exceed half a spacing to both
// nodes: funct_g then falls back to the grid's second node, and such an item
// is summed sample by sample (pv_direct).
//
// Landau: for Maxwellian fit terms the three continuation values a row needs
// share one Gaussian, exp(-p2 (d +- D)^2) = exp(-p2 d^2) exp(-+2 p2 D d)
// exp(-p2 D^2), so a row costs two complex exponentials; the omega-independent
// factors come from k_fit_aux.
//
// Two kernels:
//   k_resonant_lanes  an item per lane: lattices on the mixed path.  No
//     exchange between lanes; items that need the FP64 sums, the Landau
//     rows, or a shape that a lane does not take (PVL_SAMPLES samples, pieces
//     at the grid's ends) are left to the other kernel, which sums them as in
//     a smaller batch.
//   k_resonant_multi  an item per warp (the per-item set-up still one per
//     lane): everything else.
// ---------------------------------------------------------------------------
#define RES_WARPS 4
#define PV_CHUNK 128   // samples a warp sums between two looks at the cuts
#define PV_TOL 5e-6f   // a cut nearer than this (in spacings; SpecDev::ptol on long grids) to a sample is
                       // decided by the search, and a distance's rounding more
#define PV_DIST 4e-7f  // of a cut far from p_res, per spacing

// scalar arithmetic of the principal-value sums: FP64 or double-float
__device__ __forceinline__ double sc_add(double a, double b) { return a + b; }
__device__ __forceinline__ dflt sc_add(dflt a, dflt b) { return df_add(a, b); }
__device__ __forceinline__ double sc_neg(double a) { return -a; }
__device__ __forceinline__ dflt sc_neg(dflt a) { return df_neg(a); }
__device__ __forceinline__ double sc_mul(double a, double b) { return a * b; }
__device__ __forceinline__ dflt sc_mul(dflt a, dflt b) { return df_mul(a, b); }
__device__ __forceinline__ double sc_rcp(double a) { return rcp_fast(a); }
__device__ __forceinline__ dflt sc_rcp(dflt a) { return df_rcp_approx(a); }
__device__ __forceinline__ double sc_scale(double a, float s) { return a * (double)s; }  // s a power of 2
__device__ __forceinline__ dflt sc_scale(dflt a, float s) { return df_scale(a, s); }
__device__ __forceinline__ void sc_acc(double& a, double c) { a += c; }
__device__ __forceinline__ void sc_acc(dflt& a, dflt c) { df_acc(a, c); }
__device__ __forceinline__ void sc_mac(double& a, double v, double r) { a = fma(v, r, a); }
__device__ __forceinline__ void sc_mac(dflt& a, dflt v, dflt r) { df_mac(a, v.h, v.l, r); }
__device__ __forceinline__ double sc_val(double a) { return a; }
__device__ __forceinline__ double sc_val(dflt a) { return df_val(a); }
__device__ __forceinline__ double sc_shfl(double a, int src) { return __shfl_sync(FULL_WARP, a, src); }
__device__ __forceinline__ dflt sc_shfl(dflt a, int src) {
  return {__shfl_sync(FULL_WARP, a.h, src), __shfl_sync(FULL_WARP, a.l, src)};
}
__device__ __forceinline__ double sc_up(double a, int o) { return __shfl_up_sync(FULL_WARP, a, o); }
__device__ __forceinline__ dflt sc_up(dflt a, int o) {
  return {__shfl_up_sync(FULL_WARP, a.h, o), __shfl_up_sync(FULL_WARP, a.l, o)};
}
__device__ __forceinline__ bool sc_is_df(double) { return false; }
__device__ __forceinline__ bool sc_is_df(dflt) { return true; }
template <typename T>
__device__ __forceinline__ T sc_of(double x);
template <>
__device__ __forceinline__ double sc_of<double>(double x) { return x; }
template <>
__device__ __forceinline__ dflt sc_of<dflt>(double x) { return df_of(x); }

// a species' constants and nodes in either arithmetic (the float pairs are
// formed once on the host: a conversion is FP64 work for the whole warp)
template <typename T>
struct ScSpec;
template <>
struct ScSpec<double> {
  static __device__ __forceinline__ double kap(const SpecDev& S) { return S.kappa; }
  static __device__ __forceinline__ double hid(const SpecDev& S) { return S.hidpa; }
  static __device__ __forceinline__ double dpp(const SpecDev& S) { return S.dppar; }
  static __device__ __forceinline__ double idp(const SpecDev& S) { return S.idppar; }
  static __device__ __forceinline__ double node(const SpecDev& S, int j) { return S.ppar[j]; }
  static __device__ __forceinline__ double v(const SpecDev& S, size_t at) { return S.V[at]; }
  static __device__ __forceinline__ double half_turn(const SysDev& y, const SpecDev&, double cap) {
    return 2.0 * ALPS_PI * (double)y.M_P * rcp_fast(cap);
  }
};
template <>
struct ScSpec<dflt> {
  static __device__ __forceinline__ dflt kap(const SpecDev& S) { return {S.kaph, S.kapl}; }
  static __device__ __forceinline__ dflt hid(const SpecDev& S) { return {S.hidh, S.hidl}; }
  static __device__ __forceinline__ dflt dpp(const SpecDev& S) { return {S.dpph, S.dppl}; }
  static __device__ __forceinline__ dflt idp(const SpecDev& S) { return {S.idph, S.idpl}; }
  static __device__ __forceinline__ dflt node(const SpecDev& S, int j) { return {S.pph[j], S.ppl[j]}; }
  static __device__ __forceinline__ dflt v(const SpecDev& S, size_t at) { return {S.Vh[at], S.Vl[at]}; }
  static __device__ __forceinline__ dflt half_turn(const SysDev&, const SpecDev& S, dflt cap) {
    return df_mul({S.tpmh, S.tpml}, df_rcp_approx(cap));
  }
};

// sums over samples of w r dx, w r, w r dx^2
template <typename T>
struct PvSums {
  T s1, s2, s3;
};
template <typename T>
__device__ __forceinline__ PvSums<T> pv_diff(PvSums<T> a, PvSums<T> b) {
  return {sc_add(a.s1, sc_neg(b.s1)), sc_add(a.s2, sc_neg(b.s2)), sc_add(a.s3, sc_neg(b.s3))};
}

// the principal-value constants of an item (integrate_res,
// src/ALPS_fns.f90:1000-1040): capDelta, smdelta, the tiny rest's count and
// spacing, and the samples' places in spacings from node j0, next to p_res
// (jt0: next to the first sample of the tiny rest)
struct PvItem {
  double pr, pim;
  double cap, sm, cor;   // capDelta, smdelta, the tiny rest's correction
  dflt capd, smd, cord, pimd, oxd, oyd;  // and the double-float path's pairs
  float f0, du, ft0, dut;
  int j0, jt0, ntiny;
  int lower, upper, nn;
  int direct;            // some sample lies half-way between nodes and funct_g's search may find neither
};

// the reference's own sample points, for the search near half-way points
struct PvExact {
  double pr, cap, sm, cor;
  int M_P;
  __device__ double sym(int k) const {
    return k == 0 ? pr : (k == M_P ? __dadd_rn(pr, cap) : __dadd_rn(pr, __dmul_rn(sm, (double)k)));
  }
  __device__ double tiny(int k) const {
    return k == 0 ? __dadd_rn(pr, cap) : __dadd_rn(__dadd_rn(pr, cap), __dmul_rn(__dmul_rn(cor, sm), (double)k));
  }
};
__device__ __noinline__ PvExact pv_exact(const SpecDev& S, const SysDev& sys, const PvItem& it, double omr) {
  PvExact x;
  x.M_P = sys.M_P;
  x.pr = pres_real(S, omr, it.nn, sys.kpar);
  x.cap = x.pr - S.ppar[it.lower];
  x.sm = x.cap / (1.0 * sys.M_P);
  x.cor = it.ntiny > 0 ? ((S.ppar[it.upper] - x.pr - x.cap) / (1.0 * it.ntiny)) / x.sm : 0.0;
  return x;
}
// funct_g's search: the last node in 1..M-1 within half a spacing of p, 0 if none
__device__ __noinline__ int pv_search(const SpecDev& S, double p) {
  const int M = S.M;
  const double jd = floor((p - S.ppar[0]) * fabs(S.idppar) + 0.5), half = 0.5 * S.dppar_abs;
  if (jd > -10.0 && jd < (double)M + 10.0) {
    const int j = (int)jd;
    for (int jj = min(j + 2, M - 1); jj >= max(j - 2, 1); --jj)
      if (fabs(S.ppar[jj] - p) <= half) return jj;
  }
  return 0;
}

__device__ __forceinline__ void pv_setup(const SpecDev& S, const SysDev& sys, const ResGeom& g, int nn, double omr,
                                         PvItem& it) {
  it.pr = g.pr;
  it.pim = g.pi;
  it.lower = g.lower;
  it.upper = g.upper;
  it.nn = nn;
  const double cap = g.pr - S.ppar[g.lower];
  it.cap = cap;
  it.sm = cap * sys.iM_P;
  // ntiny = floor(rest / smdelta); the reference's own quotient near integers
  const double rest = S.ppar[g.upper] - g.pr - cap, q = rest * rcp_fast(it.sm);
  int nt = rest_samples(q);
  if (!(fabs(q - rint(q)) > 1e-6)) {
    it.ntiny = 0;
    const PvExact x = pv_exact(S, sys, it, omr);
    nt = rest_samples((S.ppar[g.upper] - x.pr - x.cap) / x.sm);
  }
  it.ntiny = nt;
  it.cor = nt > 0 ? q * rcp_fast((double)nt) : 0.0;
  const double u = 1.0 + (g.pr - S.ppar[1]) * S.idppar;
  it.j0 = (int)rint(u);
  it.f0 = (float)(u - (double)it.j0);
  it.du = (float)(it.sm * S.idppar);
  const double ut = u + cap * S.idppar;
  it.jt0 = (int)rint(ut);
  it.ft0 = (float)(ut - (double)it.jt0);
  it.dut = it.du * (float)it.cor;
  it.direct = 0;
  if (fabsf(it.f0) > 0.5f - S.ptol || (nt > 0 && fabsf(it.ft0) > 0.5f - S.ptol)) {
    // the sample at p_res (or the tiny rest's first) half-way between nodes
    const PvExact x = pv_exact(S, sys, it, omr);
    const int j = pv_search(S, x.sym(0)), jt = pv_search(S, x.tiny(0));
    if (j == 0 || (nt > 0 && jt == 0) || fabs(it.pim) <= sys.Tlim) it.direct = 1;
    if (j > 0 && j != it.j0) {
      it.f0 += (float)(it.j0 - j);
      it.j0 = j;
    }
    if (jt > 0 && jt != it.jt0) {
      it.ft0 += (float)(it.jt0 - jt);
      it.jt0 = jt;
    }
  }
}

// First sample k beyond piece i of a side (0: p_k upwards from p_res, 1: the
// mirrored points downwards, 2: the tiny rest upwards): i + 1/2 spacings from
// the side's first node.  A point half-way belongs to the upper node; lost: to
// none.  FAR: a cut may lie more than a dozen spacings from p_res.
template <bool FAR>
__device__ __forceinline__ int pv_cut(const SpecDev& S, const SysDev& sys, const PvItem& it, double omr, int side,
                                      int i, bool& lost) {
  const int K = side == 2 ? it.ntiny : sys.M_P;
  const float f = side == 2 ? it.ft0 : it.f0, du = side == 2 ? it.dut : it.du;
  const float dist = (float)i + (side == 1 ? 0.5f + f : 0.5f - f);
  const float t = dist / du;
  if (!(t < (float)K + 1.0f)) return K + 1;
  const float tr = rintf(t);
  int k = (side == 1) ? (int)floorf(t) + 1 : (int)ceilf(t);
  if (fabsf(t - tr) * du < (FAR ? fmaf(PV_DIST, dist, S.ptol) : S.ptol)) {
    k = (int)tr;
    const PvExact x = pv_exact(S, sys, it, omr);
    const int j = pv_search(S, side == 0 ? x.sym(k) : (side == 1 ? 2.0 * x.pr - x.sym(k) : x.tiny(k)));
    if (j == 0 && k <= K) lost = true;
    const bool beyond = side == 0 ? j >= it.j0 + i + 1 : (side == 1 ? j <= it.j0 - i - 1 : j >= it.jt0 + i + 1);
    if (!beyond) ++k;
  }
  return max(0, min(K + 1, k));
}

// what the sums need of an item, in their arithmetic
template <typename T>
struct PvScal {
  T sm, cap, csd, cor, y, y2;
};
template <typename T>
__device__ __forceinline__ PvScal<T> pv_scal(const PvItem& it);
template <>
__device__ __forceinline__ PvScal<double> pv_scal<double>(const PvItem& it) {
  return {it.sm, it.cap, it.cor * it.sm, it.cor, it.pim, it.pim * it.pim};
}
template <>
__device__ __forceinline__ PvScal<dflt> pv_scal<dflt>(const PvItem& it) {
  return {it.smd, it.capd, df_mul(it.cord, it.smd), it.cord, it.pimd, df_mul(it.pimd, it.pimd)};
}
__device__ __forceinline__ double sc_times(double a, int k) { return a * (double)k; }
__device__ __forceinline__ dflt sc_times(dflt a, int k) { return df_mul(a, {(float)k, 0.0f}); }

// adds sample k of the symmetric window (tiny: of the tiny rest, without its
// correction); sym: the first sample counts
template <typename T>
__device__ __forceinline__ void pv_sample(PvSums<T>& s, const PvScal<T>& c, int k, int K, bool tiny, bool sym) {
  T dx = sc_times(tiny ? c.csd : c.sm, k);
  if (tiny) dx = sc_add(c.cap, dx);
  else if (k == K) dx = c.cap;
  T r = sc_scale(sc_rcp(sc_add(sc_mul(dx, dx), c.y2)), (k == 0 || k == K) ? 1.0f : 2.0f);
  if (k == 0 && !sym) r = sc_of<T>(0.0);
  const T t = sc_mul(dx, r);
  sc_acc(s.s1, t);
  sc_acc(s.s2, r);
  sc_mac(s.s3, dx, t);
}

// a piece's A and first moment about p_res from its sums (side as pv_cut)
template <typename T>
__device__ __forceinline__ void pv_moment(const PvSums<T>& s, const PvScal<T>& c, int side, T& Ax, T& Ay, T& Cx, T& Cy) {
  Ax = side == 1 ? sc_neg(s.s1) : s.s1;
  Ay = sc_mul(c.y, s.s2);
  Cx = s.s3;
  Cy = sc_mul(c.y, s.s1);
  if (side == 1) Cy = sc_neg(Cy);
  if (side == 2) {
    Ax = sc_mul(Ax, c.cor);
    Ay = sc_mul(Ay, c.cor);
    Cx = sc_mul(Cx, c.cor);
    Cy = sc_mul(Cy, c.cor);
  }
}

// ---------------------------------------------------------------------------
// One item's principal-value sum by a warp
// ---------------------------------------------------------------------------
template <typename T>
struct __align__(16) PvPiece {
  T Ax, Ay, Bx, By;
  int a, pad[3];
};
// Windows of more than PV_WIDE nodes to a side are summed sample by sample
// (pv_direct): a piece then holds two samples or fewer of the usual 100, the
// weights of a window's nodes cost its square, and past 354 nodes they would
// not fit a block's shared memory.  Mixed and FP64, 64x256 grid, 700
// frequencies, us by pieces and by samples: 24 nodes 333 and 388, 633 and 621;
// 48: 461 and 334, 771 and 555; 100: 517 and 272, 774 and 423; 4096
// frequencies: 24: 871 and 1446, 2160 and 2357; 48: 1114 and 1156, 2504 and
// 1992; 100: 1181 and 705, 2278 and 1429.
#define PV_WIDE 48
// pieces at most: both sides of the window, the tiny rest
__host__ __device__ inline int pv_max_pieces(int M_I) { return 2 * ((M_I < PV_WIDE ? M_I : PV_WIDE) + 4) + 8; }
// double2 words per warp: prefix sums of a chunk, pieces, node weights (as many as pieces)
__host__ __device__ inline size_t pv_warp_words(int M_I) {
  const size_t np = (size_t)pv_max_pieces(M_I);
  return (PV_CHUNK * 24 + 15) / 16 + np * (sizeof(PvPiece<double>) / 16) + np;
}

// prefix sums at the lane's cut kc (see pv_sample); pre: PV_CHUNK PvSums (a
// chunk's first sample is unsigned: the last chunk of the most samples ends
// past the largest int)
template <typename T>
__device__ __forceinline__ PvSums<T> pv_cut_sums(const PvScal<T>& c, int K, bool tiny, bool sym, int kc,
                                                 PvSums<T>* pre, int lane) {
  const T z = sc_of<T>(0.0);
  PvSums<T> out = {z, z, z}, carry = {z, z, z};
  for (unsigned k0 = 0; k0 <= (unsigned)K; k0 += PV_CHUNK) {
    const int n = (int)min((unsigned)PV_CHUNK, (unsigned)K + 1u - k0), per = (n + 31) / 32;
    const int b = min(n, lane * per), e = min(n, b + per);
    PvSums<T> loc = {z, z, z};
    for (int j = b; j < e; ++j) {
      pre[j] = loc;
      pv_sample(loc, c, (int)k0 + j, K, tiny, sym);
    }
    PvSums<T> inc = loc;
    for (int o = 1; o < 32; o <<= 1) {
      const T a = sc_up(inc.s1, o), d = sc_up(inc.s2, o), f = sc_up(inc.s3, o);
      if (lane >= o) {
        inc.s1 = sc_add(inc.s1, a);
        inc.s2 = sc_add(inc.s2, d);
        inc.s3 = sc_add(inc.s3, f);
      }
    }
    PvSums<T> bef;
    bef.s1 = sc_up(inc.s1, 1);
    bef.s2 = sc_up(inc.s2, 1);
    bef.s3 = sc_up(inc.s3, 1);
    if (lane == 0) bef = {z, z, z};
    bef = {sc_add(carry.s1, bef.s1), sc_add(carry.s2, bef.s2), sc_add(carry.s3, bef.s3)};
    for (int j = b; j < e; ++j)
      pre[j] = {sc_add(pre[j].s1, bef.s1), sc_add(pre[j].s2, bef.s2), sc_add(pre[j].s3, bef.s3)};
    carry = {sc_add(carry.s1, sc_shfl(inc.s1, 31)), sc_add(carry.s2, sc_shfl(inc.s2, 31)),
             sc_add(carry.s3, sc_shfl(inc.s3, 31))};
    __syncwarp();
    const int at = kc - (int)k0;
    if (at >= 0 && at < n) out = pre[at];
    __syncwarp();
  }
  if (kc > K) out = carry;
  return out;
}

// The weights W of the nodes a0 .. a0 + cnt - 1 in wts (FP64 or double-float
// pairs of 16 bytes); false if the item has to be summed directly
template <typename T>
__device__ bool pv_warp_weights(const SpecDev& S, const SysDev& sys, const PvItem& it, double omr, PvSums<T>* pre,
                                PvPiece<T>* rec, T* wts, int lane, int& a0, int& cnt) {
  const int M = S.M, M_P = sys.M_P, cap_rec = pv_max_pieces(sys.M_I);
  const PvScal<T> c = pv_scal<T>(it);
  typedef ScSpec<T> SS;
  const T z = sc_of<T>(0.0), plo = SS::node(S, it.lower);
  const bool sym = fabs(it.pim) > sys.Tlim;
  auto clampj = [&](int j) { return (j >= M - 1) ? M - 2 : ((j <= 1) ? 2 : j); };
  auto put = [&](int slot, int j, T Ax, T Ay, T Cx, T Cy) {
    PvPiece<T> p;
    p.a = clampj(j);
    // p_res - p_a = capDelta + (p_lower - p_a)
    const T del = sc_add(c.cap, sc_add(plo, sc_neg(SS::node(S, p.a))));
    p.Ax = Ax;
    p.Ay = Ay;
    p.Bx = sc_add(Cx, sc_mul(del, Ax));
    p.By = sc_add(Cy, sc_mul(del, Ay));
    rec[slot] = p;
  };
  int nrec = 0;
  bool lost = it.direct;
  if (sym) {
    // pieces of both sides, side by side over the lanes: even slots up, odd down
    const int most = 2 * (sys.M_I + 4);
    for (int t0 = 0; t0 < most; t0 += 32) {
      const int t = t0 + lane, side = t & 1, i = t >> 1;
      const int kb = i == 0 ? 0 : pv_cut<true>(S, sys, it, omr, side, i - 1, lost);
      const int ke = pv_cut<true>(S, sys, it, omr, side, i, lost);
      const bool has = t < most && kb <= M_P;
      const PvSums<T> se = pv_cut_sums(c, M_P, false, true, has ? ke : 0, pre, lane);
      PvSums<T> sb;
      sb.s1 = sc_up(se.s1, 2);
      sb.s2 = sc_up(se.s2, 2);
      sb.s3 = sc_up(se.s3, 2);
      if (t0 > 0 && __any_sync(FULL_WARP, has && lane < 2)) {
        const PvSums<T> s0 = pv_cut_sums(c, M_P, false, true, kb, pre, lane);
        if (lane < 2) sb = s0;
      }
      if (i == 0) sb = {z, z, z};
      const unsigned m = __ballot_sync(FULL_WARP, has);
      if (has) {
        T Ax, Ay, Cx, Cy;
        pv_moment(pv_diff(se, sb), c, side, Ax, Ay, Cx, Cy);
        const int slot = nrec + __popc(m & ((1u << lane) - 1u));
        if (slot < cap_rec) put(slot, side ? it.j0 - i : it.j0 + i, Ax, Ay, Cx, Cy);
      }
      nrec += __popc(m);
      if (!m) break;
    }
  } else {
    // Tlim branch: g' sum_k w_k dx^2/(dx^2 + y^2) + sign(y) i pi G(p_res)/smdelta
    const PvSums<T> s = pv_cut_sums(c, M_P, false, false, M_P + 1, pre, lane);
    if (lane < 3) {
      // H at p_res + dppar, p_res - dppar and p_res
      const int d = lane == 0 ? 1 : (lane == 1 ? -1 : 0), j = it.j0 + d;
      T Ax = z, Ay = z;
      if (d != 0) {
        // g' 2 sum = (H1 - H2) sum / dppar
        Ax = sc_mul(s.s3, SS::idp(S));
        if (d < 0) Ax = sc_neg(Ax);
      } else {
        Ay = sc_scale(SS::half_turn(sys, S, c.cap), it.pim > 0.0 ? 1.0f : (it.pim < 0.0 ? -1.0f : 0.0f));
      }
      const T off = sc_scale(SS::dpp(S), (float)d);
      put(lane, j, Ax, Ay, sc_mul(off, Ax), sc_mul(off, Ay));
    }
    nrec = 3;
  }
  if (it.ntiny > 0) {
    const int i = lane;
    const int ke = pv_cut<true>(S, sys, it, omr, 2, i, lost), kb = i == 0 ? 0 : pv_cut<true>(S, sys, it, omr, 2, i - 1, lost);
    const bool has = i < 6 && kb <= it.ntiny;
    const PvSums<T> se = pv_cut_sums(c, it.ntiny, true, true, has ? ke : 0, pre, lane);
    PvSums<T> sb;
    sb.s1 = sc_up(se.s1, 1);
    sb.s2 = sc_up(se.s2, 1);
    sb.s3 = sc_up(se.s3, 1);
    if (i == 0) sb = {z, z, z};
    const unsigned m = __ballot_sync(FULL_WARP, has);
    if (has && nrec + i < cap_rec) {
      T Ax, Ay, Cx, Cy;
      pv_moment(pv_diff(se, sb), c, 2, Ax, Ay, Cx, Cy);
      put(nrec + i, it.jt0 + i, Ax, Ay, Cx, Cy);
    }
    nrec += __popc(m);
  }
  if (__any_sync(FULL_WARP, lost)) return false;
  nrec = min(nrec, cap_rec);
  __syncwarp();
  int lo = M, hi = 0;
  for (int t = lane; t < nrec; t += 32) {
    lo = min(lo, rec[t].a);
    hi = max(hi, rec[t].a);
  }
  a0 = __reduce_min_sync(FULL_WARP, lo) - 1;
  cnt = min(__reduce_max_sync(FULL_WARP, hi) + 1 - a0 + 1, cap_rec);
  const T hid = SS::hid(S);
  for (int t = lane; t < cnt; t += 32) {
    T Wx = z, Wy = z, Dx = z, Dy = z;
    for (int q = 0; q < nrec; ++q) {
      const int d = a0 + t - rec[q].a;
      if (d == 0) {
        Wx = sc_add(Wx, rec[q].Ax);
        Wy = sc_add(Wy, rec[q].Ay);
      } else if (d == 1 || d == -1) {
        Dx = sc_add(Dx, d > 0 ? rec[q].Bx : sc_neg(rec[q].Bx));
        Dy = sc_add(Dy, d > 0 ? rec[q].By : sc_neg(rec[q].By));
      }
    }
    wts[2 * t] = sc_add(Wx, sc_mul(hid, Dx));
    wts[2 * t + 1] = sc_add(Wy, sc_mul(hid, Dy));
  }
  __syncwarp();
  return true;
}

// adds component c of T_e times the window's scale to the output row; xy and
// yz have imaginary prefactors: (x, y) -> pe (-y, x)
__device__ __forceinline__ void pv_add_out(double2* out, const double* pref, int n, int e, int c, double v) {
  if (n == 0 && (e == 0 || e == 3 || e == 4)) return;
  double* d = reinterpret_cast<double*>(out + e);
  v *= pref[e];
  if (e == 3 || e == 5) d[c ^ 1] += c ? -v : v;
  else d[c] += v;
}

// The same sum sample by sample over the reference's own points, in FP64: for
// items with a sample that funct_g's search finds no node for, and for
// windows of more than PV_WIDE nodes to a side.
__device__ __noinline__ void pv_direct(const SpecDev& S, const SysDev& sys, const PvItem& it, double2 o,
                                       const double* pref, double2* out) {
  const int lane = threadIdx.x & 31, M = S.M, M_P = sys.M_P, n = it.nn < 0 ? -it.nn : it.nn;
  const PvExact x = pv_exact(S, sys, it, o.x);
  const double y = it.pim, y2 = y * y;
  dbl_val T[12];
  for (int q = 0; q < 12; ++q) T[q].v = 0.0;
  // T += f H(p)
  auto add = [&](double p, double2 f) {
    int j = pv_search(S, p);
    j = (j >= M - 1) ? M - 2 : ((j <= 1) ? 2 : j);
    const double* v = S.V + ((size_t)n * (M - 1) + (j - 1)) * 12;
    const double dx = (p - S.ppar[j]) * S.hidpa;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const double v1 = fma(v[12 + 2 * e] - v[2 * e - 12], dx, v[2 * e]);
      const double v2 = fma(v[13 + 2 * e] - v[2 * e - 11], dx, v[2 * e + 1]);
      const double2 t = cmul(cmk(fma(o.x, v1, S.kappa * v2), o.y * v1), f);
      T[2 * e].v += t.x;
      T[2 * e + 1].v += t.y;
    }
  };
  if (fabs(y) > sys.Tlim) {
    for (unsigned k = lane; k <= (unsigned)M_P; k += 32) {
      const double p = x.sym((int)k), dx = p - x.pr;
      const double r = ((k == 0 || k == (unsigned)M_P) ? 1.0 : 2.0) * rcp_fast(fma(dx, dx, y2));
      add(p, cmk(dx * r, y * r));
      add(2.0 * x.pr - p, cmk(-dx * r, y * r));
    }
  } else {
    double fr = 0.0;
    for (unsigned k = 1 + lane; k <= (unsigned)M_P; k += 32) {
      const double d = x.sym((int)k) - x.pr;
      fr += (k == (unsigned)M_P ? 1.0 : 2.0) * ((d * d) / (d * d + y2));
    }
    for (int off = 16; off > 0; off >>= 1) fr += __shfl_xor_sync(FULL_WARP, fr, off);
    const double c = fr * S.idppar;
    if (lane == 0) add(x.pr + S.dppar, cmk(c, 0.0));
    if (lane == 1) add(x.pr - S.dppar, cmk(-c, 0.0));
    if (lane == 2 && y != 0.0) add(x.pr, cmk(0.0, (y > 0.0 ? 2.0 : -2.0) * ALPS_PI / x.sm));
  }
  for (unsigned k = lane; k <= (unsigned)it.ntiny && it.ntiny > 0; k += 32) {
    const double p = x.tiny((int)k), dx = p - x.pr;
    const double r = ((k == 0 || k == (unsigned)it.ntiny) ? 1.0 : 2.0) * x.cor * rcp_fast(fma(dx, dx, y2));
    add(p, cmk(dx * r, y * r));
  }
  int first, cnt;
  lane_sum12(T, 32, lane, first, cnt);
  if (cnt) pv_add_out(out, pref, n, first >> 1, first & 1, T[0].v * (x.sm * S.pvc));
  __syncwarp();
}

__device__ __forceinline__ void pv_omega(const PvItem&, double2 o, double& x, double& y) {
  x = o.x;
  y = o.y;
}
__device__ __forceinline__ void pv_omega(const PvItem& it, double2, dflt& x, dflt& y) {
  x = it.oxd;
  y = it.oyd;
}

// adds an item's principal-value part to its output row; pv_scal<dflt> needs
// values that stay normal floats (df_ok of the item)
template <typename T>
__device__ __noinline__ void pv_warp(const SpecDev& S, const SysDev& sys, const PvItem& it, double2 o,
                                     const double* pref, double2* wk, double2* out) {
  const int lane = threadIdx.x & 31, M = S.M, n = it.nn < 0 ? -it.nn : it.nn;
  PvSums<T>* pre = reinterpret_cast<PvSums<T>*>(wk);
  PvPiece<T>* rec = reinterpret_cast<PvPiece<T>*>(wk + (PV_CHUNK * 24 + 15) / 16);
  T* wts = reinterpret_cast<T*>(wk + (PV_CHUNK * 24 + 15) / 16 + pv_max_pieces(sys.M_I) * (sizeof(PvPiece<double>) / 16));
  int a0, cnt;
  if (sys.M_I > PV_WIDE || !pv_warp_weights<T>(S, sys, it, o.x, pre, rec, wts, lane, a0, cnt)) {
    pv_direct(S, sys, it, o, pref, out);
    return;
  }
  // lane 4 e + 2 g + c: component c of sum_j V_{e,g}(j) W_j
  T s = sc_of<T>(0.0);
  if (lane < 24) {
    const size_t base = ((size_t)n * (M - 1) + (a0 - 1)) * 12 + (lane >> 1);
    for (int t = 0; t < cnt; ++t) {
      const int j = a0 + t;
      if (j < 1 || j > M - 1) continue;
      sc_mac(s, ScSpec<T>::v(S, base + (size_t)t * 12), wts[2 * t + (lane & 1)]);
    }
  }
  s = sc_add(s, sc_of<T>(0.0));  // (normalises a double-float accumulator)
  const T other = sc_shfl(s, lane ^ 1), g2 = sc_shfl(s, (lane + 2) & 31);
  T ox, oy;
  pv_omega(it, o, ox, oy);
  const T kap = ScSpec<T>::kap(S);
  const bool im = lane & 1;
  const T x = sc_add(sc_add(sc_mul(ox, s), im ? sc_mul(oy, other) : sc_neg(sc_mul(oy, other))), sc_mul(kap, g2));
  // G = K_e H with K_e = -(q/kpar) pref_e / 2; result 2 pi T smdelta dpperp/4
  if (lane < 24 && !(lane & 2))
    pv_add_out(out, pref, n, lane >> 2, im ? 1 : 0, sc_val(x) * (it.sm * S.pvc * (sc_is_df(s) ? S.Vscale[n] : 1.0)));
  __syncwarp();
}

// ---------------------------------------------------------------------------
// The factorised Landau term of one item on one lane: res_e for entries
// xx yy zz xy xz yz.  Valid when the rows' deviation |delta_i(p')| <= 1e-5 for
// p' = p, p +- dppar (second-order remainder <= 1.7e-16); the bound in FP32
// with a margin (an item just inside it takes the rows).
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool landau_factorises(const SpecDev& S, double2 p) {
  if (!S.lmom) return false;
  const float ap = sqrtf(fmaf((float)p.x, (float)p.x, (float)p.y * (float)p.y)) * 1.00001f + (float)S.dppar_abs;
  return fmaf(fmaf(S.la32, ap, S.lb32), ap, S.lc32) <= 0.999e-5f;
}
// m 2^e as a double: m's exponent moved in its bits where the result stays a
// normal number (no FP64 operation), two products otherwise
__device__ __forceinline__ double scale_exp(double m, int e) {
  const int hi = __double2hiint(m), x = (hi >> 20) & 0x7ff, y = x + e;
  if (x != 0 && x != 0x7ff && y > 0 && y < 0x7ff) return __hiloint2double(hi + (e << 20), __double2loint(m));
  const int e1 = max(-1000, min(1000, e / 2)), e2 = max(-1000, min(1000, e - e1));
  return m * __hiloint2double((1023 + e1) << 20, 0) * __hiloint2double((1023 + e2) << 20, 0);
}
// WARP: every lane has the same item; the exponentials, the three points and
// the entries go over the lanes, and res[0] receives entry min(lane, 5).
__device__ __forceinline__ dflt df_from(dflt v, int src) {
  return {__shfl_sync(FULL_WARP, v.h, src), __shfl_sync(FULL_WARP, v.l, src)};
}
__device__ __forceinline__ cdf cdf_from(cdf v, int src) { return {df_from(v.x, src), df_from(v.y, src)}; }
template <bool WARP>
__device__ __forceinline__ void landau_lane(const SpecDev& S, cdf omd, double2 p, int lf, int n, const dflt* prefd,
                                            double2* res) {
  const int lane = threadIdx.x & 31;
  // Row Gaussian G(x) = exp(-p2r (x - p3r)^2) at x = p, p +- dppar:
  // G(p +- pd) = lgc G(p) X^{+-1}, X = exp(-2 p2r pd (p - p3r)).  In
  // double-float with powers of two kept apart: G(p) = 2^k0 g0,
  // X = 2^kx xm.  With P_F, Q_F the moment polynomials of family F,
  //   Spar  = (G(p+pd) P_F(p+pd) - G(p-pd) P_F(p-pd)) / (2 pd)
  //         = lgc/(2 pd) G(p) (X P_F(p+pd) - X^-1 P_F(p-pd)),
  //   Sperp = G(p) Q_F(p),
  //   sum_F = (q/|k_par|) (kappa Spar + (omega - kappa p) Sperp).
  const double dx = p.x - S.p3r, dy = p.y;
  int k0 = 0, kx = 0;
  cdf g0 = {{0.0f, 0.0f}, {0.0f, 0.0f}}, xm = g0, xi = g0;
#pragma unroll 1
  for (int u = WARP ? (lane & 1) : 0; u < 2; u += WARP ? 2 : 1) {
    int e;
    dflt cs, sn;
    const dflt m = df_exp_scaled(u ? S.lcx * dx : -S.p2r * ((dx - dy) * (dx + dy)), e);
    df_cis(u ? S.lcx * dy : -2.0 * S.p2r * dx * dy, cs, sn);
    const cdf v = {df_mul(m, cs), df_mul(m, sn)};
    if (u) {
      const dflt im = df_rcp_approx(m);
      xm = v;
      xi = {df_mul(im, cs), df_neg(df_mul(im, sn))};
      kx = e;
    } else {
      g0 = v;
      k0 = e;
    }
  }
  if (WARP) {
    g0 = cdf_from(g0, 0);
    xm = cdf_from(xm, 1);
    xi = cdf_from(xi, 1);
    k0 = __shfl_sync(FULL_WARP, k0, 0);
    kx = __shfl_sync(FULL_WARP, kx, 1);
  }
  // an underflowing Gaussian (|G| min_a0 below the FP64 range at any of the
  // three points) leaves the term zero, as in FP64
  const int akx = kx < 0 ? -kx : kx;
  if ((k0 + S.lze < -1072) || (k0 - akx + S.lge + S.lze < -1072)) return;
  // X P+ - X^-1 P- = 2^|kx| (a P+ - b P-): (a, b) = (xm, 2^-2kx xi) for
  // kx >= 0, (2^2kx xm, xi) otherwise (a term below 2^-126 of the other is
  // dropped); Sperp enters with 2^-|kx| of it
  const float sc = akx <= 63 ? ldexpf(1.0f, -2 * akx) : 0.0f, sp = akx <= 126 ? ldexpf(1.0f, -akx) : 0.0f;
  if (kx >= 0) xi = {df_scale(xi.x, sc), df_scale(xi.y, sc)};
  else xm = {df_scale(xm.x, sc), df_scale(xm.y, sc)};
  const cdf pz = {df_of(p.x), df_of(p.y)};
  const dflt pdd = {S.pdh, S.pdl}, kapd = {S.kaph, S.kapl};
  const dflt lk = df_mul({S.lgch, S.lgcl}, df_mul(kapd, df_rcp_approx(df_scale(pdd, 2.0f))));  // kappa lgc / (2 pd)
  const float* lm0 = S.lmomf + (size_t)n * 72;
  const dflt z = {0.0f, 0.0f};
  cdf sum[3] = {{z, z}, {z, z}, {z, z}};  // per family: kappa Spar + (omega - kappa p) Sperp over G
#pragma unroll 1
  for (int u = WARP ? min(lane, 2) : 0; u < 3; u += WARP ? 3 : 1) {
    // the moment polynomials at p + pd, p - pd (P_F) and p (Q_F), each times
    // its factor
    cdf zu = pz, f;
    if (u == 0) {
      zu.x = df_add(pz.x, pdd);
      f = cdf_rmul(xm, lk);
    } else if (u == 1) {
      zu.x = df_add(pz.x, df_neg(pdd));
      f = cdf_rmul(xi, df_neg(lk));
    } else {
      f = {df_scale(df_add(omd.x, df_neg(df_mul(kapd, pz.x))), sp),
           df_scale(df_add(omd.y, df_neg(df_mul(kapd, pz.y))), sp)};
    }
    const cdf z2 = cdf_mul(zu, zu), z3 = cdf_mul(z2, zu), z4 = cdf_mul(z2, z2);
#pragma unroll
    for (int F = 0; F < 3; ++F) {
      const float* cf = lm0 + F * 24 + (u == 2 ? 5 : 0);
      cdf q = {{cf[0], cf[10]}, z};
      q = cdf_add(q, cdf_rmul(zu, {cf[1], cf[11]}));
      q = cdf_add(q, cdf_rmul(z2, {cf[2], cf[12]}));
      q = cdf_add(q, cdf_rmul(z3, {cf[3], cf[13]}));
      q = cdf_add(q, cdf_rmul(z4, {cf[4], cf[14]}));
      sum[F] = cdf_add(sum[F], cdf_mul(f, q));
    }
  }
  if (WARP)
    for (int F = 0; F < 3; ++F)
      sum[F] = cdf_add(cdf_add(cdf_from(sum[F], 0), cdf_from(sum[F], 1)), cdf_from(sum[F], 2));
  // res_e = pref_e c_e sum_F(e) ifac, c_e = 1, p or p^2; ifac =
  // -i dpperp 2 pi^2 lf, pref_e real (imaginary for xy, yz); with q / |k_par|
  const cdf gq = cdf_rmul(g0, df_mul({S.qlh, S.qll}, df_scale({S.lih, S.lil}, (float)lf)));
#pragma unroll
  for (int t = 0; t < (WARP ? 1 : 6); ++t) {
    const int e = WARP ? min(lane, 5) : t, fam = (e == 1) ? 1 : ((e == 3 || e == 5) ? 2 : 0);
    const int ex = k0 + akx + (int)lm0[fam * 24 + 20];
    cdf v = cdf_mul(gq, fam == 0 ? sum[0] : (fam == 1 ? sum[1] : sum[2]));
    if (e == 2 || e == 4 || e == 5) v = cdf_mul(v, pz);
    if (e == 2) v = cdf_mul(v, pz);
    // pref ifac: real pref -> i pref fi; imaginary i pref -> -(pref fi)
    const bool im = (e == 3 || e == 5);
    dflt pf = prefd[0];
#pragma unroll
    for (int q = 1; q < 6; ++q)
      if (e == q) pf = prefd[q];
    const double vx = scale_exp(df_val(df_mul(v.x, pf)), ex), vy = scale_exp(df_val(df_mul(v.y, pf)), ex);
    res[t] = im ? cmk(-vx, -vy) : cmk(-vy, vx);
  }
}

__device__ inline double2 crcp(double2 z) {
  double r = 1.0 / (z.x * z.x + z.y * z.y);
  return cmk(z.x * r, -z.y * r);
}

// The same term in FP64 (plain path): false if the neighbours' Gaussians leave
// exp's range and the rows have to be summed one by one.  Some 350 FP64
// instructions for 32 items at once, where the rows' two exponentials each
// take 180 per 32 rows of one item: 2867 map frequencies 1008 us by rows,
// 321 us so (k_resonant_multi); a single frequency 47 and 33 us.
__device__ __forceinline__ double2 cmul_rn(double2 a, double2 b) {
  return cmk(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 c_from(double2 v, int src) {
  return cmk(__shfl_sync(FULL_WARP, v.x, src), __shfl_sync(FULL_WARP, v.y, src));
}
// (operations rounded one by one: both forms give the same bits)
template <bool WARP>
__device__ __noinline__ bool landau_lane_fp64(const SpecDev& S, double2 o, double2 p, int lf, int n,
                                              const double* pref, double2* res) {
  const int lane = threadIdx.x & 31;
  const double pd = S.dppar_abs, dx = p.x - S.p3r, dy = p.y;
  const double e0 = __dmul_rn(-S.p2r, __dmul_rn(dx - dy, dx + dy)), ex = __dmul_rn(S.lcx, dx);
  if (!(fabs(ex) < 600.0)) return false;
  // an underflowing Gaussian leaves the term zero (landau_lane's test)
  const double L2E = 1.4426950408889634;
  const double k0 = rint(e0 * L2E), akx = fabs(rint(ex * L2E));
  if (k0 + (double)S.lze < -1072.0 || k0 - akx + (double)(S.lge + S.lze) < -1072.0) return true;
  double2 G = cmk(0.0, 0.0), X = G;
#pragma unroll 1
  for (int u = WARP ? (lane & 1) : 0; u < 2; u += WARP ? 2 : 1) {
    const double2 v = cexp_d(u ? cmk(ex, __dmul_rn(S.lcx, dy)) : cmk(e0, __dmul_rn(__dmul_rn(-2.0 * S.p2r, dx), dy)));
    if (u) X = v;
    else G = v;
  }
  if (WARP) {
    G = c_from(G, 0);
    X = c_from(X, 1);
  }
  const double ql = S.qs / fabs(S.kappa * S.ms), lk = S.lgc * S.kappa / (2.0 * pd);
  const double* __restrict__ lm = S.lmom + (size_t)n * 30;
  double2 sum[3] = {cmk(0.0, 0.0), cmk(0.0, 0.0), cmk(0.0, 0.0)};
#pragma unroll 1
  for (int u = WARP ? min(lane, 2) : 0; u < 3; u += WARP ? 3 : 1) {
    double2 z = p, f;
    if (u == 0) {
      z.x = __dadd_rn(z.x, pd);
      f = cmk(__dmul_rn(X.x, lk), __dmul_rn(X.y, lk));
    } else if (u == 1) {
      z.x = __dadd_rn(z.x, -pd);
      const double r = __ddiv_rn(-lk, __fma_rn(X.x, X.x, __dmul_rn(X.y, X.y)));
      f = cmk(__dmul_rn(X.x, r), __dmul_rn(-X.y, r));
    } else {
      f = cmk(__fma_rn(-S.kappa, p.x, o.x), __fma_rn(-S.kappa, p.y, o.y));
    }
    f = cmul_rn(f, G);
    const double2 z2 = cmul_rn(z, z), z3 = cmul_rn(z2, z), z4 = cmul_rn(z2, z2);
#pragma unroll
    for (int F = 0; F < 3; ++F) {
      const double* c = lm + F * 10 + (u == 2 ? 5 : 0);
      const double2 q =
          cmk(__fma_rn(c[4], z4.x, __fma_rn(c[3], z3.x, __fma_rn(c[2], z2.x, __fma_rn(c[1], z.x, c[0])))),
              __fma_rn(c[4], z4.y, __fma_rn(c[3], z3.y, __fma_rn(c[2], z2.y, __dmul_rn(c[1], z.y)))));
      const double2 t = cmul_rn(f, q);
      sum[F] = cmk(__dadd_rn(sum[F].x, t.x), __dadd_rn(sum[F].y, t.y));
    }
  }
  if (WARP)
    for (int F = 0; F < 3; ++F) {
      const double2 t0 = c_from(sum[F], 0), t1 = c_from(sum[F], 1), t2 = c_from(sum[F], 2);
      sum[F] = cmk(__dadd_rn(__dadd_rn(t0.x, t1.x), t2.x), __dadd_rn(__dadd_rn(t0.y, t1.y), t2.y));
    }
  const double fi = -S.dpperp * ALPS_PI * 2.0 * ALPS_PI * (double)lf * ql;
#pragma unroll
  for (int t = 0; t < (WARP ? 1 : 6); ++t) {
    const int e = WARP ? min(lane, 5) : t, fam = (e == 1) ? 1 : ((e == 3 || e == 5) ? 2 : 0);
    double pf = pref[0];
#pragma unroll
    for (int q = 1; q < 6; ++q)
      if (e == q) pf = pref[q];
    pf = __dmul_rn(pf, fi);
    const double2 sf = fam == 0 ? sum[0] : (fam == 1 ? sum[1] : sum[2]);
    double2 v = cmk(__dmul_rn(sf.x, pf), __dmul_rn(sf.y, pf));
    if (e == 2 || e == 4 || e == 5) v = cmul_rn(v, p);
    if (e == 2) v = cmul_rn(v, p);
    // pref ifac: real pref -> i pref fi; imaginary i pref -> -(pref fi)
    res[t] = (e == 3 || e == 5) ? cmk(-v.x, -v.y) : cmk(-v.y, v.x);
  }
  return true;
}

// what the warp phase of k_resonant_multi needs of one item
struct __align__(16) ResItem {
  PvItem pv;
  double pref[6];     // T-tensor prefactors: imaginary for xy and yz, else real
  int work;           // 1 principal value, 2 Landau rows, 4 the sums in double-float; lf << 3
  int w, s, pad;      // omega, species
  long long slot;     // the item's slot (its output row)
};
// An item's geometry, prefactors and principal-value constants.  Returns the
// work left (ResItem; 8: a Landau term that factorises).
__device__ __forceinline__ int res_core(const DispArgs& a, const SpecDev& S, double2 o, int nn, PvItem& pv,
                                        double pref[6], int& lf) {
  {
    // t_prefactors' nonzero parts, with 1/z
    const double dz = (double)nn * S.iz;
    const double k2 = a.sys.kperp_norm ? 1.0 : a.sys.kperp * a.sys.kperp, k1 = a.sys.kperp_norm ? 1.0 : a.sys.kperp;
    pref[0] = dz * dz;
    pref[1] = pref[2] = k2;
    pref[3] = pref[4] = k1 * dz;
    pref[5] = -k2;
  }
  const ResGeom g = res_geometry_of(S, a.sys, o, nn);
  lf = (o.y < 0.0) ? 2 : ((o.y == 0.0) ? 1 : 0);
  int work = 0;
  pv.pr = g.pr;
  pv.pim = g.pi;
  pv.nn = nn;
  if (g.kind == 3) {
    pv_setup(S, a.sys, g, nn, o.x, pv);
    work = 1;
    if (S.df_sums) {
      // a spacing, window or |p_im| outside 1e-12 .. 1e12 would leave the
      // normal floats: those items take the FP64 sums
      auto inr = [](float x) { return x >= 1e-12f && x <= 1e12f; };
      const float sm = (float)pv.sm, pim = fabsf((float)pv.pim);
      if (inr(sm) && inr((float)pv.cap) && pim <= 1e12f && (pim <= (float)a.sys.Tlim || inr(pim)) &&
          (pv.ntiny <= 0 || inr((float)pv.cor * sm)))
        work |= 4;
      pv.capd = df_of(pv.cap);
      pv.smd = df_of(pv.sm);
      pv.cord = df_of(pv.cor);
      pv.pimd = df_of(pv.pim);
    }
  }
  if (S.df_sums) {
    pv.oxd = df_of(o.x);
    pv.oyd = df_of(o.y);
  }
  if (lf > 0) work |= landau_factorises(S, cmk(g.pr, g.pi)) ? 8 : 2;
  return work;
}
// compiled once for the forms that have to agree bit for bit
__device__ __noinline__ int res_core_call(const DispArgs& a, const SpecDev& S, double2 o, int nn, PvItem& pv,
                                          double pref[6], int& lf) {
  return res_core(a, S, o, nn, pv, pref, lf);
}
// the factorised Landau term of an item (landau_lane); false: by rows
template <bool WARP>
__device__ __forceinline__ bool res_landau(const DispArgs& a, const SpecDev& S, double2 o, const PvItem& pv, int lf,
                                           const double pref[6], double2* res) {
  const int nn = pv.nn, n = nn < 0 ? -nn : nn;
  const double2 p = cmk(pv.pr, pv.pim);
  if (S.df_sums) {
    const dflt izd = {S.izh, S.izl}, dzd = df_mul({(float)nn, 0.0f}, izd);
    const dflt k2d = {a.sys.k2h, a.sys.k2l}, xyd = df_mul({a.sys.k1h, a.sys.k1l}, dzd);
    const dflt prefd[6] = {df_mul(dzd, dzd), k2d, k2d, xyd, xyd, df_neg(k2d)};
    landau_lane<WARP>(S, {pv.oxd, pv.oyd}, p, lf, n, prefd, res);
  } else if (!landau_lane_fp64<WARP>(S, o, p, lf, n, pref, res)) {
    return false;
  }
  if (n == 0) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int t = 0; t < (WARP ? 1 : 6); ++t) {
      const int e = WARP ? min(lane, 5) : t;
      if (e == 0 || e == 3 || e == 4) res[t] = cmk(0.0, 0.0);
    }
  }
  return true;
}
// an item's per-lane part: the above and the Landau term where it factorises
// (in res).  Returns the work left.
template <bool ONCE>
__device__ __forceinline__ int res_item(const DispArgs& a, const SpecDev& S, double2 o, int nn, PvItem& pv,
                                        double pref[6], double2 res[6], int& lf) {
#pragma unroll
  for (int e = 0; e < 6; ++e) res[e] = cmk(0.0, 0.0);
  const int work = ONCE ? res_core_call(a, S, o, nn, pv, pref, lf) : res_core(a, S, o, nn, pv, pref, lf);
  const bool rows = (work & 8) && !res_landau<false>(a, S, o, pv, lf, pref, res);
  return (work & 7) | (rows ? 2 : 0);
}

// a slot's order in k_resonant_multi's list mode: the order and the work that
// k_resonant_lanes left
#define FLAG_TODO 256  // bit of a job's error word while such work is left
__device__ __forceinline__ int todo_slot(int nn, int work) { return (nn & 0xffff) | (work << 16); }

// Walks a warp's slots slot0 .. slot0 + ipw - 1.  Most slots of a large batch
// are empty (an (omega, species) fills count of its rcap slots), so the
// occupied ones are gathered, in slot order, into batches of up to 32 items;
// body(nb, item, mine) runs with the batch's items one per lane.  Which batch
// or lane an item lands on does not change its result.
template <typename F, typename G>
__device__ __forceinline__ void res_batches(const DispArgs& a, int ipw, int n_om, const int* __restrict__ count,
                                            long slot0, int* queue, F want, G body) {
  const int lane = threadIdx.x & 31, S_ = a.sys.nspec;
  const long total = (long)n_om * S_ * a.rcap;
  const unsigned lt = (1u << lane) - 1u;
  int qn = 0;
  for (int c0 = 0; c0 < ipw; c0 += 32) {
    {
      const long sl = slot0 + c0 + lane;
      bool occ = false;
      if (c0 + lane < ipw && sl < total) {
        const unsigned u = (unsigned)(sl / a.rcap), r = (unsigned)(sl - (long)u * a.rcap);  // u = w S + s
        occ = (int)r < count[u] && want(sl);
      }
      const unsigned m = __ballot_sync(FULL_WARP, occ);
      if (occ) queue[qn + __popc(m & lt)] = c0 + lane;
      qn += __popc(m);
      __syncwarp();
    }
    const bool last = c0 + 32 >= ipw;
    while (qn >= 32 || (last && qn > 0)) {
      const int nb = qn < 32 ? qn : 32;
      const long item = (lane < nb) ? slot0 + queue[lane] : -1;
      body(nb, item);
      // the items beyond this batch move to the front of the queue
      const int rest = qn - nb;
      const int keep = (lane < rest) ? queue[nb + lane] : 0;
      __syncwarp();
      if (lane < rest) queue[lane] = keep;
      __syncwarp();
      qn = rest;
    }
  }
}

// the warp's region for principal-value work, then for the Landau rows, in double2
__host__ __device__ inline size_t res_region(int N, int M_I) {
  const size_t rows = 3 * (size_t)(N + 1), pv = pv_warp_words(M_I);
  return rows > pv ? rows : pv;
}
// per-warp shared memory in double2: the region, the warp's 32 items, 3
// values handed to lanes 0-5 and the queue of occupied slots (64 ints)
__host__ __device__ inline size_t res_warp_smem(int N, int M_I) {
  return res_region(N, M_I) + 32 * (sizeof(ResItem) / sizeof(double2)) + 3 + 16;
}

// Slots per warp: small batches spread their items over many warps (a single
// omega's few resonant orders run side by side, as latency wants), large ones
// take up to 256 slots per warp.
inline int res_items_per_warp(long nslots, int warps_per_sm = 12) {
  const long warps_wanted = 152L * warps_per_sm;  // SMs x resident warps of k_resonant
  long ipw = nslots / warps_wanted;
  return (int)(ipw < 1 ? 1 : (ipw > 256 ? 256 : ipw));
}


// The Landau term of one item by its rows, over the warp: added to out
__device__ __noinline__ void landau_rows(const DispArgs& a, const SpecDev& S, double2 o, double2 p, int nn, int lf,
                                         const double* pref, double2* wk, double2* out) {
  const int lane = threadIdx.x % 32, N = S.N, n = nn < 0 ? -nn : nn;
  const double kpar = a.sys.kpar;
  double2* frow = wk;                  // f(i, p_res)
  double2* fpr = frow + (N + 1);       // f(i, p_res + dppar)
  double2* fmr = fpr + (N + 1);        // f(i, p_res - dppar)
  double2* tb = wk + res_region(N, a.sys.M_I) + 32 * (sizeof(ResItem) / sizeof(double2));  // values handed to lanes 0-5
    const double pd = S.dppar_abs, dpp = S.dpperp;
    const double vA = a.sys.vA;
    if (S.fit_aux) {
      // Maxwellian terms: f = sum_f a0 exp(-p2 (p - p3)^2)
      const int nf = S.nf;
      for (int i = lane; i <= N; i += 32) {
        double2 f0 = cmk(0, 0), fp = cmk(0, 0), fm = cmk(0, 0);
        for (int f = 0; f < nf; ++f) {
          const double* aux = S.fit_aux + ((size_t)i * nf + f) * 4;  // a0, p2, p3, exp(-p2 D^2)
          double p2 = aux[1];
          double2 d = cmk(p.x - aux[2], p.y);
          double2 E0 = cexp_d(cscale(cmul(d, d), -p2));
          double2 G = cscale(E0, aux[0]);
          double2 ax = cscale(d, -2.0 * p2 * pd);
          double2 X, Xi;
          if (fabs(ax.x) < 600.0) {
            X = cexp_d(ax);
            Xi = crcp(X);
            double2 Gc = cscale(G, aux[3]);
            fp = cadd(fp, cmul(Gc, X));
            fm = cadd(fm, cmul(Gc, Xi));
          } else {
            double2 dp = cadd(d, cmk(pd, 0.0)), dm = csub(d, cmk(pd, 0.0));
            fp = cadd(fp, cscale(cexp_d(cscale(cmul(dp, dp), -p2)), aux[0]));
            fm = cadd(fm, cscale(cexp_d(cscale(cmul(dm, dm), -p2)), aux[0]));
          }
          f0 = cadd(f0, G);
        }
        frow[i] = f0;
        fpr[i] = fp;
        fmr[i] = fm;
      }
    } else {
      for (int i = lane; i <= N; i += 32) {
        eval_fit3_d(S, vA, i, p, pd, frow[i], fpr[i], fmr[i]);
      }
    }
    __syncwarp();
    bool zero = false;
    double2 sums[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
    const double ql = S.qs / fabs(kpar);
    const int L = N + 1;
    for (int i = lane; i <= N; i += 32) {
      double2 fpi = fpr[i], fpf = fmr[i];
      double2 dfperp, dfpar;
      double h;
      if (i == 0) {
        dfperp = cscale(csub(frow[1], frow[0]), 1.0 / dpp);
        h = 0.5;
      } else if (i == N) {
        dfperp = cscale(csub(frow[N], frow[N - 1]), 1.0 / dpp);
        h = 0.5;
      } else {
        // |f| = 0 exactly when both parts are
        auto nil = [](double2 x) { return x.x == 0.0 && x.y == 0.0; };
        if (nil(fpi) || nil(fpf) || nil(frow[i + 1])) zero = true;
        dfperp = cscale(csub(frow[i + 1], frow[i - 1]), 1.0 / (2.0 * dpp));
        h = (i == N - 1) ? 0.5 : 1.0;
      }
      dfpar = cscale(csub(fpi, fpf), 1.0 / (2.0 * pd));
      double pp_i = S.pperp[i];
      // (q/|kpar|) ((pperp dfpar - p dfperp) kpar/m + omega dfperp)
      double2 Lv = cscale(cadd(cscale(csub(cscale(dfpar, pp_i), cmul(p, dfperp)), kpar / S.ms), cmul(o, dfperp)),
                          ql);
      double J = S.bessel[(size_t)(n + 1) * L + i];
      double Jp = (n == 0) ? -S.bessel[(size_t)2 * L + i]
                           : 0.5 * (S.bessel[(size_t)n * L + i] - S.bessel[(size_t)(n + 2) * L + i]);
      sums[0] = cadd(sums[0], cscale(Lv, h * (J * J)));
      sums[1] = cadd(sums[1], cscale(Lv, h * ((pp_i * pp_i) * Jp * Jp)));
      sums[2] = cadd(sums[2], cscale(Lv, h * (pp_i * J * Jp)));
    }
    zero = __any_sync(0xffffffffu, zero);
    for (int F = 0; F < 3; ++F)
      for (int off = 16; off > 0; off >>= 1) {
        sums[F].x += __shfl_xor_sync(0xffffffffu, sums[F].x, off);
        sums[F].y += __shfl_xor_sync(0xffffffffu, sums[F].y, off);
      }
    if (!zero) {
      // landau_e = -pref_e c_e(p) Sigma_F(e) * i dpperp 2 pi^2, lanes 0-5
      if (lane == 0)
        for (int F = 0; F < 3; ++F) tb[F] = sums[F];
      __syncwarp();
      if (lane < 6 && !(n == 0 && (lane == 0 || lane == 3 || lane == 4))) {
        const int e = lane;
        const double2 ce = (e == 2) ? cmul(p, p) : ((e == 4 || e == 5) ? p : cmk(1.0, 0.0));
        const int fam = (e == 1) ? 1 : ((e == 3 || e == 5) ? 2 : 0);
        const double2 ifac = cmk(0.0, -dpp * ALPS_PI * 2.0 * ALPS_PI * (double)lf);
        const double2 land = cmul(cmul((e == 3 || e == 5 ? cmk(0.0, pref[e]) : cmk(pref[e], 0.0)), ce), tb[fam]);
        out[e] = cadd(out[e], cmul(land, ifac));
      }
      __syncwarp();
    }
}

// Up to 32 resonant items, one per lane (item < 0: none): the per-lane part,
// then the principal-value sums and Landau rows item by item over the warp.
// sv is the item's order (list: what k_resonant_lanes left of it), wk the
// warp's shared memory.
__device__ __noinline__ void resonant_group(const DispArgs& a, const double2* __restrict__ om, double2* items,
                                               double2* wk, long item, int sv, bool list) {
  const int lane = threadIdx.x % 32;
  const int S_ = a.sys.nspec;
  const int N = a.sp[0].N;  // every species has the same p_perp grid
  ResItem* ri = reinterpret_cast<ResItem*>(wk + res_region(N, a.sys.M_I));
  // ---- one item per lane ----
  int work = 0;
  if (item >= 0) {
    const int u = (int)(item / a.rcap), s = u % S_, w = u / S_;
    const SpecDev& S = a.sp[s];
    const int nn = list ? (int)(short)(sv & 0xffff) : sv;
    const double2 o = om[w];
    ResItem& it = ri[lane];
    double2 res[6];
    double pref[6];
    PvItem pv;
    int lf;
    work = res_item<true>(a, S, o, nn, pv, pref, res, lf);
    double2* out = items + item * 6;
    if (list) work &= sv >> 16;
    else
      for (int e = 0; e < 6; ++e) out[e] = res[e];
    it.pv = pv;
    it.work = work | (lf << 3);
    it.w = w;
    it.s = s;
    it.slot = item;
    for (int e = 0; e < 6; ++e) it.pref[e] = pref[e];
  }
  __syncwarp();

  // ---- one item per warp: the principal-value sums and the Landau rows ----
  unsigned pend = __ballot_sync(FULL_WARP, (work & 3) != 0);
  while (pend) {
    const int il = __ffs(pend) - 1;
    pend &= pend - 1;
    const ResItem& it = ri[il];
    const int s = it.s, w = it.w, nn = it.pv.nn;
    const int wkk = it.work & 7, lf = it.work >> 3;
    const SpecDev& S = a.sp[s];
    const double2 o = om[w];
    double2* out = items + it.slot * 6;

    if (wkk & 1) {
      if (wkk & 4) pv_warp<dflt>(S, a.sys, it.pv, o, it.pref, wk, out);
      else pv_warp<double>(S, a.sys, it.pv, o, it.pref, wk, out);
    }

    if (wkk & 2) landau_rows(a, S, o, cmk(it.pv.pr, it.pv.pim), nn, lf, it.pref, wk, out);
    __syncwarp();  // the next item reuses the region
  }
}

// One item by a warp of its own (small batches): what resonant_group does for
// it, with the factorised Landau term's parts over the lanes too.
__device__ __noinline__ void resonant_one(const DispArgs& a, const SpecDev& S, double2 o, int nn, double2* wk,
                                          double2* out) {
  const int lane = threadIdx.x & 31;
  PvItem pv;
  double pref[6];
  int lf;
  int work = res_core_call(a, S, o, nn, pv, pref, lf);
  double2 res = cmk(0.0, 0.0);
  if ((work & 8) && !res_landau<true>(a, S, o, pv, lf, pref, &res)) work |= 2;
  if (lane < 6) out[lane] = res;
  __syncwarp();
  if (work & 1) {
    if (work & 4) pv_warp<dflt>(S, a.sys, pv, o, pref, wk, out);
    else pv_warp<double>(S, a.sys, pv, o, pref, wk, out);
  }
  if (work & 2) landau_rows(a, S, o, cmk(pv.pr, pv.pim), nn, lf, pref, wk, out);
}

__device__ __forceinline__ void resonant_body(const DispArgs& a, const DispShape& sh, const double2* __restrict__ om,
                                              int n_om, const int* __restrict__ count,
                                              const int* __restrict__ slot_nn, double2* items, long block) {
  extern __shared__ double2 sm[];
  const int warp = threadIdx.x / 32;
  const int N = a.sp[0].N;
  double2* wk = sm + (size_t)warp * res_warp_smem(N, a.sys.M_I);
  // occupied slots, offsets from slot0
  int* queue = reinterpret_cast<int*>(wk + res_region(N, a.sys.M_I) + 32 * (sizeof(ResItem) / sizeof(double2)) + 3);
  const long slot0 = (block * RES_WARPS + warp) * (long)sh.ipw;
  if (slot0 >= (long)n_om * a.sys.nspec * a.rcap) return;
  const bool list = sh.lanes;  // only what k_resonant_lanes left
  res_batches(
      a, sh.ipw, n_om, count, slot0, queue, [&](long sl) { return !list || (slot_nn[sl] >> 16) != 0; },
      [&](int, long item) { resonant_group(a, om, items, wk, item, item >= 0 ? slot_nn[item] : 0, list); });
}

// ---------------------------------------------------------------------------
// One item per lane (mixed path, lattices).  A lane sums its item's samples
// in turn and leaves the running sums at the cuts in its column of shared
// memory; the cuts are the bytes of a word per side.  Then it walks the
// window's nodes, forming each node's weight from the pieces beside it and
// adding the node's base vectors.  Bound by issue (some 800 warp instructions
// an item, against 3300 when a warp shared an item's samples and merged its
// lanes' pieces) and by the instruction cache: the loops over cuts, sample
// runs, sides and the Landau term's points are kept rolled, which took the
// kernel from 1847 to 1539 us.  512x512 map, 1.2 M items: 7330 us by warps,
// 1539 us so; 8192 frequencies 384 and 119 us.
// ---------------------------------------------------------------------------
#define PVL_TINY 4  // cuts of the tiny rest at most
#define PVL_SAMPLES 128  // samples of a run below this (a cut is a byte); more go by warps
__host__ __device__ inline int pvl_side(int M_I) { return M_I + 3; }  // cuts of a side at most (eight)
__host__ __device__ inline int pvl_slots(int M_I) { return 2 * pvl_side(M_I) + PVL_TINY; }
// bytes per block: two float pairs and a weight per cut and lane, the warps' queues
__host__ __device__ inline size_t pvl_smem(int M_I) {
  return (size_t)pvl_slots(M_I) * 20 * (RES_WARPS * 32) + RES_WARPS * 64 * sizeof(int);
}
// running sums of w r dx, w r and w, half the weights of PvSums
struct PvRun {
  dflt s1, s2;
  float w;
};
struct PvCols {
  float4* a;   // s1, s2 at [slot * 128 + thread]
  float* b;    // w
  __device__ __forceinline__ void put(int slot, const PvRun& s) const {
    a[slot * (RES_WARPS * 32) + threadIdx.x] = make_float4(s.s1.h, s.s1.l, s.s2.h, s.s2.l);
    b[slot * (RES_WARPS * 32) + threadIdx.x] = s.w;
  }
  __device__ __forceinline__ PvRun get(int slot) const {
    const float4 x = a[slot * (RES_WARPS * 32) + threadIdx.x];
    return {{x.x, x.y}, {x.z, x.w}, b[slot * (RES_WARPS * 32) + threadIdx.x]};
  }
};
// adds a sample at dx with half its weight, w = 1 or 1/2: r = w / (dx^2 + y2).
// The pairs stay unnormalised between the steps (low parts below 2^-21 of the
// high ones), which the sums' error-free additions take: 44 operations.
__device__ __forceinline__ void pvl_add(PvRun& s, dflt dx, dflt y2, float w) {
  const float p = __fmul_rn(dx.h, dx.h);
  const float pl = __fmaf_rn(__fadd_rn(dx.h, dx.h), dx.l, __fmaf_rn(dx.h, dx.h, -p));
  const dflt d = df_two_sum(p, y2.h);
  dflt r = df_rcp_approx({d.h, __fadd_rn(d.l, __fadd_rn(pl, y2.l))});
  if (w != 1.0f) r = df_scale(r, w);
  const float t = __fmul_rn(dx.h, r.h);
  const float tl = __fmaf_rn(dx.h, r.l, __fmaf_rn(dx.l, r.h, __fmaf_rn(dx.h, r.h, -t)));
  df_acc(s.s1, {t, tl});
  df_acc(s.s2, r);
  s.w += w;
}
__device__ __forceinline__ dflt pvl_times(dflt a, float k) {
  const float p = __fmul_rn(a.h, k);
  return df_quick(p, __fmaf_rn(a.l, k, __fmaf_rn(a.h, k, -p)));
}

// T_e times scale into X (xx yy zz xy xz yz, divided by Vscale[n]); false if
// the item's shape is not one of the fast form's
__device__ __forceinline__ bool pv_lane(const SpecDev& S, const SysDev& sys, const PvItem& it, double2 o, PvCols col,
                                        cdf X[6]) {
  const int M = S.M, M_P = sys.M_P, n = it.nn < 0 ? -it.nn : it.nn;
  const int side_max = pvl_side(sys.M_I);
  const bool sym = fabs(it.pim) > sys.Tlim;
  // the cuts of the three runs of samples (up, down, tiny rest), a byte each
  unsigned long long cu = ~0ull, cd = ~0ull, ct = ~0ull;
  bool ok = M_P < PVL_SAMPLES && it.ntiny < PVL_SAMPLES, lost = it.direct;
  int nu = 2, nd = 2, nt = 0;  // pieces (without sym: H at p_res and a spacing to either side)
#pragma unroll 1
  for (int sd = 0; sd < 3; ++sd) {
    if (sd == 2 ? it.ntiny <= 0 : !sym) continue;
    const int K = sd == 2 ? it.ntiny : M_P, most = sd == 2 ? PVL_TINY : side_max;
    int np = 1, last = 0;
    unsigned long long pk = ~0ull;
#pragma unroll 1
    for (int i = 0; i <= most; ++i) {
      const int k = pv_cut<false>(S, sys, it, o.x, sd, i, lost);  // (at most pvl_side's eight spacings)
      if (k > K) break;
      ok = ok && k > last && i < most;
      last = k;
      np = i + 2;
      if (i < 8) pk ^= (unsigned long long)(0xff ^ (k & 0xff)) << (8 * i);
    }
    if (sd == 0) {
      cu = pk;
      nu = np;
    } else if (sd == 1) {
      cd = pk;
      nd = np;
    } else {
      ct = pk;
      nt = np;
    }
  }
  // (a piece M - 1 takes node M - 2's interpolant)
  const int jlo = it.j0 - (nd - 1), jtop = max(it.j0 + nu - 1, nt ? it.jt0 + nt - 1 : 0), jhi = min(jtop, M - 2);
  ok = ok && !lost && jlo >= 2 && jtop <= M - 1;
  if (!ok) return false;
  const PvScal<dflt> c = pv_scal<dflt>(it);
  const dflt z = {0.0f, 0.0f};
  PvRun end = {z, z, 0.0f}, endt = end;
#pragma unroll 1
  for (int rep = 0; rep < (nt ? 2 : 1); ++rep) {  // the window, the tiny rest
    const int K = rep ? it.ntiny : M_P;
    const dflt step = rep ? c.csd : c.sm;
    unsigned long long pa = rep ? ct : cu, pb = rep ? ~0ull : cd;
    int ia = rep ? 2 * side_max : 0, ib = side_max;
    PvRun s = {z, z, 0.0f};
#pragma unroll 1
    for (int k = (rep || sym) ? 0 : 1; k <= K; ++k) {
      if ((int)(pa & 0xff) == k && k) {
        col.put(ia++, s);
        pa >>= 8;
      }
      if ((int)(pb & 0xff) == k && k) {
        col.put(ib++, s);
        pb >>= 8;
      }
      dflt dx = pvl_times(step, (float)k);
      if (rep) dx = df_add(c.cap, dx);
      else if (k == K) dx = c.cap;
      pvl_add(s, dx, c.y2, (k == 0 || k == K) ? 0.5f : 1.0f);
    }
    if (rep) endt = s;
    else end = s;
  }
  // piece j's A and moment B about node j; sums of side sd, run of cuts at
  // slot b0, piece i of ni, total tot
  const dflt plo = {S.pph[it.lower], S.ppl[it.lower]};
  auto part = [&](int sd, int b0, int i, int ni, const PvRun& tot, cdf& A, cdf& C) {
    PvRun e = (i + 1 < ni) ? col.get(b0 + i) : tot;
    if (i > 0) {
      const PvRun b = col.get(b0 + i - 1);
      e = {df_add(e.s1, df_neg(b.s1)), df_add(e.s2, df_neg(b.s2)), e.w - b.w};
    } else {
      e = {df_add(e.s1, z), df_add(e.s2, z), e.w};
    }
    // sum of w r dx^2 = sum of w - y^2 sum of w r
    PvSums<dflt> s = {df_scale(e.s1, 2.0f), df_scale(e.s2, 2.0f), z};
    s.s3 = df_add({2.0f * e.w, 0.0f}, df_neg(df_mul(c.y2, s.s2)));
    dflt Ax, Ay, Cx, Cy;
    pv_moment(s, c, sd, Ax, Ay, Cx, Cy);
    A = cdf_add(A, {Ax, Ay});
    C = cdf_add(C, {Cx, Cy});
  };
  auto piece = [&](int j, cdf& A, cdf& B) {
    A = {z, z};
    cdf C = {z, z};
#pragma unroll 1
    for (int jj = j; jj <= (j == jhi ? jtop : j); ++jj) {
      const int i = jj - it.j0;
#pragma unroll 1
      for (int sd = sym ? 0 : 2; sd < 3; ++sd) {
        const int q = sd == 0 ? i : (sd == 1 ? -i : jj - it.jt0), nq = sd == 0 ? nu : (sd == 1 ? nd : nt);
        if (q >= 0 && q < nq) part(sd, sd * side_max, q, nq, sd == 2 ? endt : end, A, C);
      }
      if (!sym && i >= -1 && i <= 1) {
        if (i != 0) {
          // g' sum_k w_k dx^2/(dx^2 + y^2)
          const dflt s3 = df_add({2.0f * end.w, 0.0f}, df_neg(df_mul(c.y2, df_scale(df_add(end.s2, z), 2.0f))));
          dflt x = df_mul(s3, {S.idph, S.idpl});
          if (i < 0) x = df_neg(x);
          A.x = df_add(A.x, x);
          C.x = df_add(C.x, df_mul(df_scale({S.dpph, S.dppl}, (float)i), x));
        } else {
          const float sgn = (it.pim > 0.0) ? 1.0f : ((it.pim < 0.0) ? -1.0f : 0.0f);
          A.y = df_add(A.y, df_scale(df_mul({S.tpmh, S.tpml}, df_rcp_approx(c.cap)), sgn));
        }
      }
    }
    // p_res - p_j = capDelta + (p_lower - p_j)
    const dflt del = df_add(c.cap, df_add(plo, df_neg({S.pph[j], S.ppl[j]})));
    B = cdf_add(C, cdf_rmul(A, del));
  };
  dflt2 Sr[6], Si[6];  // per entry, (g1, g2) side by side
#pragma unroll
  for (int q = 0; q < 6; ++q) Sr[q] = Si[q] = d2_all(z);
  const dflt hid = {S.hidh, S.hidl};
  cdf Aj = {z, z}, Bp = {z, z}, Bj = {z, z};
#pragma unroll 1
  for (int j = jlo - 1; j <= jhi + 1; ++j) {
    cdf An = {z, z}, Bn = {z, z};
    if (j + 1 <= jhi) piece(j + 1, An, Bn);
    // W_j = A_j + (B_{j-1} - B_{j+1}) / (2 dppar)
    const cdf W = cdf_add(Aj, cdf_rmul({df_add(Bp.x, df_neg(Bn.x)), df_add(Bp.y, df_neg(Bn.y))}, hid));
    const dflt pj = {S.pph[j], S.ppl[j]};
    const cdf Wp = cdf_rmul(W, pj), Wpp = cdf_rmul(Wp, pj);
    const float4* b4 = reinterpret_cast<const float4*>(S.Bt + ((size_t)n * (M - 1) + (j - 1)) * 12);
    const float4 a0 = __ldg(b4), a1 = __ldg(b4 + 1), a2 = __ldg(b4 + 2);
    const float2 hb[3] = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}}, lb[3] = {{a1.z, a1.w}, {a2.x, a2.y}, {a2.z, a2.w}};
    // entries xx yy zz xy xz yz: vectors (F1, F2, F1 p^2, F3, F1 p, F3 p)
    auto add = [&](int e, int f, cdf v) {
      const dflt2 x2 = d2_all(v.x), y2 = d2_all(v.y);
      d2_mac(Sr[e], hb[f], lb[f], x2.h, x2.l);
      d2_mac(Si[e], hb[f], lb[f], y2.h, y2.l);
    };
    add(0, 0, W);
    add(1, 1, W);
    add(2, 0, Wpp);
    add(3, 2, W);
    add(4, 0, Wp);
    add(5, 2, Wp);
    Bp = Bj;
    Aj = An;
    Bj = Bn;
  }
  const cdf omd = {it.oxd, it.oyd};
  const dflt kap = {S.kaph, S.kapl};
#pragma unroll
  for (int e = 0; e < 6; ++e)
    X[e] = om_comb(omd, kap, {df_add(d2_x(Sr[e]), z), df_add(d2_x(Si[e]), z)},
                   {df_add(d2_y(Sr[e]), z), df_add(d2_y(Si[e]), z)});
  return true;
}

__device__ __forceinline__ void lanes_body(const DispArgs& a, const DispShape& sh, const double2* __restrict__ om,
                                           int n_om, const int* __restrict__ count, int* slot_nn, double2* items,
                                           int* flags, long block) {
  extern __shared__ double2 sm[];
  const int warp = threadIdx.x / 32, S_ = a.sys.nspec;
  PvCols col;
  const int slots = pvl_slots(a.sys.M_I);
  col.a = reinterpret_cast<float4*>(sm);
  col.b = reinterpret_cast<float*>(col.a + slots * RES_WARPS * 32);
  int* queue = reinterpret_cast<int*>(col.b + slots * RES_WARPS * 32) + warp * 64;
  const long slot0 = (block * RES_WARPS + warp) * (long)sh.lanes;
  if (slot0 >= (long)n_om * S_ * a.rcap) return;
  res_batches(
      a, sh.lanes, n_om, count, slot0, queue, [](long) { return true; },
      [&](int nb, long item) {
        if (item >= 0) {
          const int u = (int)(item / a.rcap), s = u % S_, w = u / S_;
          const SpecDev& S = a.sp[s];
          const int nn = slot_nn[item], n = nn < 0 ? -nn : nn;
          const double2 o = om[w];
          double2 res[6];
          double pref[6];
          PvItem pv;
          int lf;
          int work = res_item<false>(a, S, o, nn, pv, pref, res, lf);
          cdf X[6];
          if ((work & 5) == 5 && pv_lane(S, a.sys, pv, o, col, X)) {
            const double scale = S.Vscale[n] * pv.sm * S.pvc;
#pragma unroll
            for (int e = 0; e < 6; ++e) {
              if (n == 0 && (e == 0 || e == 3 || e == 4)) continue;
              const double f = scale * pref[e], x = df_val(X[e].x) * f, y = df_val(X[e].y) * f;
              if (e == 3 || e == 5) res[e] = cadd(res[e], cmk(-y, x));
              else res[e] = cadd(res[e], cmk(x, y));
            }
            work &= ~1;
          }
          double2* out = items + item * 6;
#pragma unroll
          for (int e = 0; e < 6; ++e) out[e] = res[e];
          slot_nn[item] = todo_slot(nn, (work & 3) ? work : 0);
          if (work & 3) atomicOr(flags, FLAG_TODO);
        }
      });
}

// ---------------------------------------------------------------------------
// chi, epsilon, wave tensor, det (src/ALPS_fns.f90:500-626)
//
// Two forms: a thread per omega for lattices, where the FP64 pipe is the
// bound, and a warp per omega for everything smaller, where one thread's
// chain of some 600 FP64 operations was (24 us for 31 frequencies, 87 us for
// 2999).  There lane c + 12 h holds component c (re, im of xx yy zz xy xz yz)
// of half h of the sums, and the products of the determinant go side by side.
// ---------------------------------------------------------------------------
// the wave tensor's entries w11 w22 w33 w12 w13 w23 from eps
__device__ __forceinline__ void wave_entries(const SysDev& sy, double2 o, const double2 eps[6], double2 w[6]) {
  const double kperp = sy.kperp, kpar = sy.kpar, vA = sy.vA;
  const double2 ov = sy.kperp_norm ? cscale(o, vA) : cscale(cscale(o, kperp), vA);
  const double2 unit = cmul(ov, ov);
  double enx2, enz2, enxnz;
  if (sy.kperp_norm) {
    enx2 = kperp * kperp;
    enz2 = kpar * kpar;
    enxnz = kpar * kperp;
  } else {
    enx2 = kperp * kperp * kperp * kperp;
    enz2 = kpar * kpar * kperp * kperp;
    enxnz = kpar * kperp * kperp * kperp;
  }
  w[0] = csub(cadd(eps[0], unit), cmk(enz2, 0.0));
  w[1] = csub(csub(cadd(eps[1], unit), cmk(enz2, 0.0)), cmk(enx2, 0.0));
  w[2] = csub(cadd(eps[2], unit), cmk(enx2, 0.0));
  w[3] = eps[3];
  w[4] = cadd(eps[4], cmk(enxnz, 0.0));
  w[5] = eps[5];
}

// one thread per omega (no tensors, plain species, few chunks)
__device__ __forceinline__ void finalize_thread(const DispArgs& a, const DispShape& sh, const double2* __restrict__ om,
                                                int n_om, const double2* __restrict__ part,
                                                const int* __restrict__ count, const double2* __restrict__ items,
                                                double2* D, int w) {
  if (w >= n_om) return;
  const int S_ = a.sys.nspec;
  const double2 o = om[w];
  const double kperp = a.sys.kperp;
  double2 eps[6];
  for (int e = 0; e < 6; ++e) eps[e] = cmk(0.0, 0.0);
  for (int s = 0; s < S_; ++s) {
    const SpecDev& S = a.sp[s];
    double2 chi[6];
    for (int e = 0; e < 6; ++e) chi[e] = cmk(0.0, 0.0);
    const size_t ws = (size_t)w * S_ + s, base = ws * sh.nchunk;
    for (int ch = 0; ch < sh.nch[s]; ++ch)
      for (int e = 0; e < 6; ++e) chi[e] = cadd(chi[e], part[(base + ch) * 6 + e]);
    const int cnt = count[ws];
    for (int r = 0; r < cnt; ++r)
      for (int e = 0; e < 6; ++e) chi[e] = cadd(chi[e], items[(ws * a.rcap + r) * 6 + e]);
    chi[2].x += a.sys.kperp_norm ? S.int_ee : kperp * kperp * S.int_ee;
    const double norm = S.ns * S.qs;
    for (int e = 0; e < 6; ++e) eps[e] = cmk(fma(norm, chi[e].x, eps[e].x), fma(norm, chi[e].y, eps[e].y));
  }
  double2 q[6];
  wave_entries(a.sys, o, eps, q);
  // w11 (w22 w33 + w23^2) + 2 w12 w23 w13 - w13^2 w22 + w12^2 w33
  D[w] = cadd(csub(cadd(cmul(q[0], cadd(cmul(q[1], q[2]), cmul(q[5], q[5]))), cscale(cmul(cmul(q[3], q[5]), q[4]), 2.0)),
                   cmul(cmul(q[4], q[4]), q[1])),
              cmul(cmul(q[3], q[3]), q[2]));
}

// one warp per omega; all lanes take part.  With ext the order chunks are
// single orders, from which the n = -1, 0, 1 parts follow.  Partial sums and
// items are read through L2: k_disp_one and k_disp_many write them in the
// same launch.
__device__ __noinline__ void finalize_warp(const DispArgs& a, const DispShape& sh, const double2* __restrict__ om,
                                              int n_om, const double2* part, const int* count, const int* slot_nn,
                                              const double2* items, const double2* __restrict__ rel,
                                              const double2* __restrict__ bmres, double2* D, double2* ext, long w) {
  if (w >= n_om) return;
  const int lane = threadIdx.x & 31, h = lane / 12, c = lane % 12, e = c >> 1;
  const int S_ = a.sys.nspec;
  const double2 o = om[w];
  const double kperp = a.sys.kperp, vA = a.sys.vA;
  double2 denom = cmk(1.0, 0.0);
  if (ext) {
    denom = cmul(o, o);
    denom = a.sys.kperp_norm ? cscale(cscale(denom, vA), vA)
                             : cscale(cscale(cscale(cscale(denom, vA), vA), kperp), kperp);
  }
  double eps = 0.0;  // component c of the sum over species (lanes 0..11)
  const int cnts = lane < S_ ? __ldcg(count + (size_t)w * S_ + lane) : 0;
  for (int s = 0; s < S_; ++s) {
    const SpecDev& S = a.sp[s];
    const size_t ws = (size_t)w * S_ + s, base = ws * sh.nchunk;
    double v = 0.0, lw[3] = {0.0, 0.0, 0.0};
    if (h < 2) {
      const int nch = sh.nch[s], cnt = __shfl_sync(0xffffffu, cnts, s);
      const double* pt = reinterpret_cast<const double*>(part + base * 6) + c;
      const double* it = reinterpret_cast<const double*>(items + ws * a.rcap * 6) + c;
      // up to eight chunks and four items of a lane are in flight together
      for (int ch = h; ch < nch; ch += 16) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = ch + 2 * u < nch ? __ldcg(pt + (size_t)(ch + 2 * u) * 12) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          v += x[u];
          if (ext)
            for (int l = 0; l < 3; ++l)
              if (ch + 2 * u - S.nmax == l - 1) lw[l] += x[u];
        }
      }
      for (int r = h; r < cnt; r += 8) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = r + 2 * u < cnt ? __ldcg(it + (size_t)(r + 2 * u) * 12) : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          v += x[u];
          if (ext && r + 2 * u < cnt) {
            const int nn = __ldcg(slot_nn + ws * a.rcap + r + 2 * u);
            for (int l = 0; l < 3; ++l)
              if (nn == l - 1) lw[l] += x[u];
          }
        }
      }
      if (S.relat) {
        // the row blocks' partial sums of +n and -n; n = 0 adds yy, zz, yz only
        const bool in0 = e == 1 || e == 2 || e == 5;
        for (int n = h; n <= S.nmax; n += 2) {
          const double* __restrict__ b = reinterpret_cast<const double*>(rel + (ws * a.relcap + n) * 2 * REL_RB * 6) + c;
          double pl = 0.0, mi = 0.0;
#pragma unroll
          for (int q = 0; q < REL_RB; ++q) {
            pl += b[q * 12];
            if (n > 0) mi += b[(REL_RB + q) * 12];
          }
          if (n == 0) {
            if (in0) {
              v += pl;
              lw[1] += pl;
            }
          } else {
            v += pl + mi;
            if (n == 1) {
              lw[2] += pl;
              lw[0] += mi;
            }
          }
        }
      }
    }
    const double ov = __shfl_down_sync(FULL_WARP, v, 12);
    v += ov;
    if (ext)
      for (int l = 0; l < 3; ++l) lw[l] += __shfl_down_sync(FULL_WARP, lw[l], 12);
    if (S.bm) {
      // NHDS chi, divided by n q before the common normalisation as in disp
      // (src/ALPS_fns.f90:344-358); no ee term
      const double* b = reinterpret_cast<const double*>(bmres + ws * 24);
      const double nq = S.ns * S.qs;
      v += b[c] / nq;
      if (ext)
        for (int l = 0; l < 3; ++l) lw[l] = b[12 + 12 * l + c] / nq;
    } else {
      // the ee term; a relativistic species' goes into chi alone
      // (src/ALPS_fns.f90:461-497)
      double ee = S.relat ? S.int_ee_rel : S.int_ee;
      if (!a.sys.kperp_norm) ee *= kperp * kperp;
      if (c == 4) {
        v += ee;
        if (!S.relat) lw[1] += ee;
      }
    }
    const double norm = S.ns * S.qs;
    v *= norm;
    eps += v;
    if (ext) {
      // chi0 (S x 3 x 3) and chi0_low (S x 3 x 3 x 3): lane 6 q + entry takes
      // one division, q = 0 chi, q = 1..3 the n = -1, 0, 1 parts
      for (int l = 0; l < 3; ++l) lw[l] *= norm;
      const int q = lane / 6, en = lane % 6;
      double x = __shfl_sync(FULL_WARP, v, 2 * en), y = __shfl_sync(FULL_WARP, v, 2 * en + 1);
      for (int l = 0; l < 3; ++l) {
        const double lx = __shfl_sync(FULL_WARP, lw[l], 2 * en), ly = __shfl_sync(FULL_WARP, lw[l], 2 * en + 1);
        if (q == l + 1) {
          x = lx;
          y = ly;
        }
      }
      if (q < 4) {
        const double2 t = cdiv(cmk(x, y), denom);
        double2* dst = ext + (size_t)w * (S_ * 36 + 9) + (q == 0 ? s * 9 : S_ * 9 + s * 27 + (q - 1) * 9);
        const int ii[6] = {0, 1, 2, 0, 0, 1}, jj[6] = {0, 1, 2, 1, 2, 2};
        dst[3 * ii[en] + jj[en]] = t;
        if (en >= 3) dst[3 * jj[en] + ii[en]] = (en == 4) ? t : cneg(t);
      }
    }
  }
  double2 ep[6], q[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    ep[k].x = __shfl_sync(FULL_WARP, eps, 2 * k);
    ep[k].y = __shfl_sync(FULL_WARP, eps, 2 * k + 1);
  }
  wave_entries(a.sys, o, ep, q);  // w11 w22 w33 w12 w13 w23
  // det = w11 (w22 w33 + w23^2) + 2 w12 w23 w13 - w13^2 w22 + w12^2 w33: first
  // the pair products on lanes 0..4, then the four terms on lanes 0..3
  auto from = [&](double2 v, int src) {
    return cmk(__shfl_sync(FULL_WARP, v.x, src), __shfl_sync(FULL_WARP, v.y, src));
  };
  const double2 p = cmul(lane == 0 ? q[1] : (lane == 1 ? q[5] : (lane == 3 ? q[4] : q[3])),
                         lane == 0 ? q[2] : (lane == 1 || lane == 2 ? q[5] : (lane == 3 ? q[4] : q[3])));
  const double2 p1 = from(p, 1), pn = from(p, lane + 1);
  double2 t = cmul(lane == 0 ? cadd(p, p1) : pn, lane == 0 ? q[0] : (lane == 1 ? q[4] : (lane == 2 ? q[1] : q[2])));
  if (lane == 1) t = cscale(t, 2.0);
  const double2 t1 = from(t, 1), t2 = from(t, 2), t3 = from(t, 3);
  if (lane == 0) D[w] = cadd(csub(cadd(t, t1), t2), t3);
  if (ext && lane < 9) {
    // the wave tensor: w12, w13, w23 above the diagonal
    const int m[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
    double2 x = q[0];
#pragma unroll
    for (int k = 1; k < 6; ++k)
      if (m[lane] == k) x = q[k];
    if (lane == 3 || lane == 7) x = cneg(x);
    ext[(size_t)w * (S_ * 36 + 9) + S_ * 36 + lane] = x;
  }
}

// ---------------------------------------------------------------------------
// Jobs.  Every batch, of one context or fused over many, runs the same
// kernels over a table of jobs in device memory: each kernel's grid is the
// concatenation of the jobs' own grids, and a block finds its job by the
// first block of each job.  A job's arguments (the context at its k) and its
// launch shape are those of a lone batch of its size, and small batches in
// one launch give the bits of the kernels apart (k_disp_one), so a context's
// results do not depend on what it was batched with, bit for bit.
// ---------------------------------------------------------------------------
struct DispJob {
  const DispArgs* a;  // the context's arguments (device copy)
  DispShape sh;
  int n, S;
  int nslots;         // resonant slots of the prepared size
  // first block of the job in classify, pole sums, resonant, finalize,
  // resonant lanes, and in k_disp_many
  long blk[6];
  const double2* om;
  double2* D;
  double2* part;
  int* count;
  int* slot_nn;
  double2* items;
  int* flags;
  int* arrive;        // k_disp_one, k_disp_many: units done per frequency, zero between launches
  int* hflag;         // host word that receives a non-zero error word, or null (k_disp_one)
  double2* ext;       // chi0, chi0_low, wave per omega, or null
  const double2* rel; // relativistic orders, or null
  const double2* bm;  // closed-form species, or null
};

#define DISP_JOB_BYTES sizeof(DispJob)

// stores a lone batch's arguments and job where its kernels read them
__global__ void k_stage(DispArgs a, DispJob j, DispArgs* da, DispJob* dj) {
  const int4* src = reinterpret_cast<const int4*>(&a);
  int4* dst = reinterpret_cast<int4*>(da);
  for (int q = threadIdx.x; q < (int)(sizeof(DispArgs) / sizeof(int4)); q += blockDim.x) dst[q] = src[q];
  if (threadIdx.x == 0) {
    j.a = da;
    *dj = j;
  }
}

__device__ __forceinline__ const DispJob& job_of(const DispJob* jobs, int nj, long b, int k) {
  int lo = 0, hi = nj - 1;  // last job whose first block is <= b
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].blk[k] <= b) lo = mid;
    else hi = mid - 1;
  }
  return jobs[lo];
}

// blocks of k_pole_sums_multi: four warps a block, whole blocks per species
__host__ __device__ inline long pole_blocks(const DispShape& sh, int s) { return ((long)sh.nch[s] * sh.wt + 3) / 4; }
inline long pole_blocks_all(const DispShape& sh, int S_) {
  long b = 0;
  for (int s = 0; s < S_; ++s) b += pole_blocks(sh, s);
  return b;
}

// k_finalize: one warp per omega up to FIN_WARP_MAX of them, where its
// blocks still fill the chip a few times over; one thread per omega beyond
__host__ __device__ inline long fin_blocks(const DispShape& sh, int n) {
  return sh.fin_warp ? (n + 3) / 4 : (n + 127) / 128;
}

// A block's job is one context: its arguments go to shared memory once, and
// every thread reads them there.
__device__ __forceinline__ const DispArgs& stage_args(const DispArgs* src, DispArgs& dst) {
  const int4* s4 = reinterpret_cast<const int4*>(src);
  int4* d4 = reinterpret_cast<int4*>(&dst);
  for (int q = threadIdx.x; q < (int)(sizeof(DispArgs) / sizeof(int4)); q += blockDim.x) d4[q] = s4[q];
  __syncthreads();
  return dst;
}

#define CLS_PER_WARP 8
// blocks of 128 threads of k_classify_multi for n omegas and S species
__host__ __device__ inline long cls_blocks(long n, int S_) { return (n * S_ + 4 * CLS_PER_WARP - 1) / (4 * CLS_PER_WARP); }

__global__ void k_classify_multi(const DispJob* __restrict__ jobs, int nj) {
  __shared__ DispArgs sa;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 0);
  const DispArgs& a = stage_args(J.a, sa);
  const long lb = (long)blockIdx.x - J.blk[0];
  // CLS_PER_WARP (omega, species) pairs per warp: the block's argument
  // staging is shared by more pairs
  const long w0 = ((lb * blockDim.x + threadIdx.x) >> 5) * CLS_PER_WARP;
  for (int q = 0; q < CLS_PER_WARP; ++q) classify_body(a, J.om, J.n, J.count, J.slot_nn, J.flags, w0 + q);
}

// copies n bytes (a multiple of 16) from global to shared memory
__device__ __forceinline__ void stage_bytes(const void* src, void* dst, int n) {
  const int4* s4 = reinterpret_cast<const int4*>(src);
  int4* d4 = reinterpret_cast<int4*>(dst);
  for (int q = threadIdx.x; q < n / 16; q += blockDim.x) d4[q] = s4[q];
}

// Coefficients of the far-order series.  For the orders nn = +-n with n |q| >=
// 2.5 P (P the largest |k_par p| on the grid) and s = m omega,
//   sum_j w_j F_j / (s - nn q - k_par p_j) = sum_l s^l c_l(nn),
//   c_l = -sum_k binom(l + k, k) (-k_par prad)^k A^-(l+k+1) mom_k,  A = nn q +
//   k_par pcen,
// with the Laurent moments mom_k of the family vectors (k_moments); the
// p_par-weighted entries take the moments of p F = pcen F + prad x F.  Times
// the order factors: farc[(n - farn) FAR_K + l][entry][g], the two orders +-n
// together.  A warp per term l and eight n, four lanes per n over quarters of
// the k; bound by the FP64 pipe (some 35 instructions a term k).
__global__ void __launch_bounds__(32) k_far_orders(const DispJob* __restrict__ jobs) {
  __shared__ double ratio[ALPS_KFAR];
  const DispJob& J = jobs[blockIdx.z];
  const int l = blockIdx.x % FAR_K, grp = blockIdx.x / FAR_K, s = blockIdx.y, lane = threadIdx.x;
  if (!J.sh.far || s >= J.S) return;
  const SpecDev& S = J.a->sp[s];
  const SysDev& sys = J.a->sys;
  const int n1 = S.farn, n = n1 + grp * 8 + (lane & 7), k0 = (lane >> 3) * (ALPS_KFAR / 4);
  if (!n1 || n1 + grp * 8 > S.nmax) return;
  for (int k = lane; k < ALPS_KFAR; k += 32) ratio[k] = (double)(l + k + 1) * rcp_fast((double)(k + 1));
  __syncwarp();
  // binom(l + k0, k0) at the quarters' starts: products of four, then over the lanes
  double bin = ratio[4 * lane] * ratio[4 * lane + 1] * ratio[4 * lane + 2] * ratio[4 * lane + 3];
  for (int off = 1; off < 32; off <<= 1) {
    const double t = __shfl_up_sync(FULL_WARP, bin, off);
    if (lane >= off) bin *= t;
  }
  bin = __shfl_sync(FULL_WARP, bin, max(0, k0 / 4 - 1));
  if (k0 == 0) bin = 1.0;
  const double kpar = sys.kpar, pc = S.pcen, pr = S.prad;
  auto power = [](double x, int e) {
    double y = 1.0;
    for (; e; e >>= 1) {
      if (e & 1) y *= x;
      x *= x;
    }
    return y;
  };
  double2 v[6];  // entries xx yy zz xy xz yz, (g1, g2)
#pragma unroll
  for (int e = 0; e < 6; ++e) v[e] = cmk(0.0, 0.0);
  if (n <= S.nmax) {
    const double r1 = (double)n1 * fabs(S.qs) - fabs(kpar) * (fabs(pc) + pr);
    const double ip = 1.0 / ((double)n * S.qs + kpar * pc), im = 1.0 / (-(double)n * S.qs + kpar * pc);
    const double cp = -kpar * pr * ip, cm = -kpar * pr * im;
    double wp = -ip * power(r1 * ip, l) * power(cp, k0) * bin, wm = -im * power(r1 * im, l) * power(cm, k0) * bin;
    const double2* __restrict__ m = reinterpret_cast<const double2*>(S.mom + ((size_t)n * ALPS_KFAR + k0) * 6);
    double2 a0 = __ldg(m), a1 = __ldg(m + 3), b0 = __ldg(m + 2), b1 = __ldg(m + 5);
    const int ke = min(k0 + ALPS_KFAR / 4, ALPS_KFAR - 2);
#pragma unroll 4
    for (int k = k0; k < ke; ++k, m += 3) {
      const double2 a2 = __ldg(m + 6), b2 = __ldg(m + 8), f2 = __ldg(m + 1);
      const double we = wp + wm, wo = wp - wm;
      const double2 ap = cmk(fma(pc, a0.x, pr * a1.x), fma(pc, a0.y, pr * a1.y));
      const double2 aq = cmk(fma(pc, a1.x, pr * a2.x), fma(pc, a1.y, pr * a2.y));
      v[0] = cmk(fma(we, a0.x, v[0].x), fma(we, a0.y, v[0].y));
      v[1] = cmk(fma(we, f2.x, v[1].x), fma(we, f2.y, v[1].y));
      v[2] = cmk(fma(we, fma(pc, ap.x, pr * aq.x), v[2].x), fma(we, fma(pc, ap.y, pr * aq.y), v[2].y));
      v[3] = cmk(fma(wo, b0.x, v[3].x), fma(wo, b0.y, v[3].y));
      v[4] = cmk(fma(wo, ap.x, v[4].x), fma(wo, ap.y, v[4].y));
      v[5] = cmk(fma(we, fma(pc, b0.x, pr * b1.x), v[5].x), fma(we, fma(pc, b0.y, pr * b1.y), v[5].y));
      wp *= cp * ratio[k];
      wm *= cm * ratio[k];
      a0 = a1;
      a1 = a2;
      b0 = b1;
      b1 = b2;
    }
  }
#pragma unroll
  for (int e = 0; e < 6; ++e)
    for (int off = 8; off < 32; off <<= 1) {
      v[e].x += __shfl_xor_sync(FULL_WARP, v[e].x, off);
      v[e].y += __shfl_xor_sync(FULL_WARP, v[e].y, off);
    }
  if (lane < 8 && n <= S.nmax) {
    const double C0 = 2.0 * ALPS_PI * S.dpperp * S.dppar_abs * 0.25 * S.qs;
    const double z = sys.kperp_norm ? sys.kperp / S.qs : 1.0 / S.qs;
    double2* o = reinterpret_cast<double2*>(S.farc + ((size_t)(n - n1) * FAR_K + l) * 12);
    double2 pref[6];
    t_prefactors(n, z, sys.kperp, sys.kperp_norm, pref);
#pragma unroll
    for (int e = 0; e < 6; ++e) o[e] = cscale(v[e], C0 * ((e == 3 || e == 5) ? pref[e].y : pref[e].x));
  }
}

// Summed from the highest order down and scaled to t = s / r: the series of all
// orders |n| >= n0 for the levels n0 = farn .. farn + FAR_LEVELS - 1, FP64 or
// float pairs.  A warp per term and species, a lane per entry and g for the
// running sums, then one per coefficient in turn.  Both kernels together take
// 58 us for 30 + 7 orders.
__global__ void __launch_bounds__(32) k_far_levels(const DispJob* __restrict__ jobs) {
  __shared__ double sum[FAR_LEVELS][12];
  const DispJob& J = jobs[blockIdx.z];
  const int l = blockIdx.x, s = blockIdx.y;
  if (!J.sh.far || s >= J.S) return;
  const SpecDev& S = J.a->sp[s];
  const int n1 = S.farn, nl = min(FAR_LEVELS, S.nmax - n1 + 1);
  if (!n1) return;
  if (threadIdx.x < 12) {
    const double* c = S.farc + (size_t)l * 12 + threadIdx.x;
    double acc = 0.0;
#pragma unroll 8
    for (int n = S.nmax - n1; n >= 0; --n) {
      acc += __ldg(c + (size_t)n * FAR_K * 12);
      if (n < FAR_LEVELS) sum[n][threadIdx.x] = acc;
    }
  }
  __syncthreads();
  const double qa = fabs(S.qs), P = fabs(J.a->sys.kpar) * (fabs(S.pcen) + S.prad), i1 = 1.0 / ((double)n1 * qa - P);
  for (int t = threadIdx.x; t < nl * 12; t += blockDim.x) {
    const int n = t / 12, q = t % 12;
    double y = sum[n][q], x = ((double)(n + n1) * qa - P) * i1;
    if (S.df_sums) y *= 1.0 / S.Escale[q >> 1];
    for (int e = l; e; e >>= 1) {
      if (e & 1) y *= x;
      x *= x;
    }
    const size_t at = (size_t)n * FAR_K + l;
    if (S.df_sums) {
      float* o = reinterpret_cast<float*>(S.far) + at * 24 + q;
      const float h = __double2float_rn(y);
      o[0] = h;
      o[12] = __double2float_rn(y - (double)h);
    } else {
      reinterpret_cast<double*>(S.far)[at * 12 + q] = y;
    }
  }
}

// A pole-sums block works on one species: it stages the system constants
// and that species' constants only (an eighth of DispArgs), which matters
// when a fused round has many small jobs, each of many small blocks.
__global__ void __launch_bounds__(128, 4) k_pole_sums_multi(const DispJob* __restrict__ jobs, int nj) {
  __shared__ __align__(16) SysDev ssys;
  __shared__ __align__(16) SpecDev sspec;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 1);
  long lb = (long)blockIdx.x - J.blk[1];
  int s = 0;
  for (; s + 1 < J.S; ++s) {
    const long nb = pole_blocks(J.sh, s);
    if (lb < nb) break;
    lb -= nb;
  }
  stage_bytes(&J.a->sys, &ssys, sizeof(SysDev));
  stage_bytes(&J.a->sp[s], &sspec, sizeof(SpecDev));
  __syncthreads();
  const long unit = lb * 4 + (threadIdx.x >> 5);
  if (unit < (long)J.sh.nch[s] * J.sh.wt) pole_body(ssys, sspec, J.sh, J.om, J.n, J.part, s, unit);
}

__global__ void __launch_bounds__(RES_WARPS * 32, 3) k_resonant_multi(const DispJob* __restrict__ jobs, int nj) {
  __shared__ DispArgs sa;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 2);
  if (J.sh.lanes && !(*J.flags & FLAG_TODO)) return;
  const DispArgs& a = stage_args(J.a, sa);
  resonant_body(a, J.sh, J.om, J.n, J.count, J.slot_nn, J.items, (long)blockIdx.x - J.blk[2]);
}

__global__ void __launch_bounds__(RES_WARPS * 32, 3) k_resonant_lanes(const DispJob* __restrict__ jobs, int nj) {
  __shared__ DispArgs sa;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 4);
  const DispArgs& a = stage_args(J.a, sa);
  lanes_body(a, J.sh, J.om, J.n, J.count, J.slot_nn, J.items, J.flags, (long)blockIdx.x - J.blk[4]);
}

__global__ void k_finalize_multi(const DispJob* __restrict__ jobs, int nj) {
  __shared__ DispArgs sa;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 3);
  const DispArgs& a = stage_args(J.a, sa);
  const long lb = (long)blockIdx.x - J.blk[3];
  if (J.sh.lanes && lb == 0 && threadIdx.x == 0) atomicAnd(J.flags, ~FLAG_TODO);
  if (J.sh.fin_warp)
    finalize_warp(a, J.sh, J.om, J.n, J.part, J.count, J.slot_nn, J.items, J.rel, J.bm, J.D, J.ext,
                  lb * (blockDim.x / 32) + threadIdx.x / 32);
  else
    finalize_thread(a, J.sh, J.om, J.n, J.part, J.count, J.items, J.D, (int)(lb * blockDim.x + threadIdx.x));
}

// ---------------------------------------------------------------------------
// Small batches in one launch.  The batches of root searches and scans are a
// few frequencies: every kernel above is then one chain of dependent
// instructions, and the sum of the chains and of the gaps between the
// launches is the time of an evaluation.  Here the pole-sum units and the
// resonant slots run side by side, a warp each (a slot's warp finds its
// order itself), and the warp that brings a frequency its last unit goes on
// to that frequency's det D: nothing waits on anything.  The sums are those of
// the kernels above, in the same order.  One frequency, mixed path, 60x120
// grid: 67 us in five kernels, 38 us so; a call from the host 110 and 62 us.
// The bodies both forms share (pole_body, res_core_call, pv_warp, pv_direct,
// landau_rows, finalize_warp) are compiled once (noinline), and the factorised
// Landau terms, of which resonant_one spreads one over the lanes, round every
// operation by itself, so a frequency's det D is the same bit for bit in
// either form.
// ---------------------------------------------------------------------------
// the slot's order (the r-th resonant order of its (omega, species)) and its
// item; returns the slot's frequency, -1 beyond the batch
__device__ __forceinline__ int small_slot(const DispArgs& a, const DispJob& J, double2* wk, int slot) {
  const int lane = threadIdx.x & 31, S_ = a.sys.nspec;
  const int u = slot / a.rcap, r = slot - u * a.rcap, s = u % S_, w = u / S_;
  if (w >= J.n) return -1;
  const SpecDev& S = a.sp[s];
  const double2 o = J.om[w];
  const float ikp32 = (float)a.sys.ikpar;
  int cnt = 0, nn = 0;
  bool found = false;
  for (int base = -S.nmax; base <= S.nmax; base += 32) {
    const bool res = base + lane <= S.nmax && order_resonant(a.sys, S, o, base + lane, ikp32);
    const unsigned m = __ballot_sync(FULL_WARP, res);
    const unsigned hit = __ballot_sync(FULL_WARP, res && cnt + __popc(m & ((1u << lane) - 1u)) == r);
    if (hit) {
      found = true;
      nn = base + __ffs(hit) - 1;
    }
    cnt += __popc(m);
  }
  if (r == 0 && lane == 0) {
    if (cnt > a.rcap) atomicOr(J.flags, 1);
    J.count[u] = min(cnt, a.rcap);
  }
  if (found) {
    if (lane == 0) J.slot_nn[slot] = nn;
    resonant_one(a, S, o, nn, wk, J.items + (size_t)slot * 6);
  }
  return w;
}

// A lane with has brings frequency w one unit; whoever brings the last one
// finishes it.
__device__ __forceinline__ void small_arrive(const DispArgs& a, const DispJob& J, int w, bool has) {
  const int lane = threadIdx.x & 31;
  int need = a.sys.nspec * a.rcap;
  for (int s = 0; s < a.sys.nspec; ++s) need += J.sh.nch[s];
  __threadfence();
  __syncwarp();
  const bool last = has && atomicAdd(J.arrive + w, 1) == need - 1;
  unsigned m = __ballot_sync(FULL_WARP, last);
  if (m) __threadfence();
  while (m) {
    const int t = __ffs(m) - 1;
    m &= m - 1;
    const int wt = __shfl_sync(FULL_WARP, w, t);
    finalize_warp(a, J.sh, J.om, J.n, J.part, J.count, J.slot_nn, J.items, nullptr, nullptr, J.D, J.ext, wt);
    if (lane == 0) {
      J.arrive[wt] = 0;
      if (J.hflag) {
        const int f = atomicOr(J.flags, 0);
        if (f) *J.hflag = f;
      }
    }
  }
}

__host__ __device__ inline int small_slot_blocks(int nslots) { return (nslots + RES_WARPS - 1) / RES_WARPS; }

__device__ __forceinline__ void small_body(const DispArgs& a, const DispJob& J, long lb) {
  extern __shared__ double2 sm[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int nsb = small_slot_blocks(J.nslots);
  if (lb < nsb) {
    const int slot = (int)lb * RES_WARPS + warp;
    if (slot >= J.nslots) return;
    const int w = small_slot(a, J, sm + (size_t)warp * res_warp_smem(a.sp[0].N, a.sys.M_I), slot);
    if (w >= 0) small_arrive(a, J, w, lane == 0);
    return;
  }
  lb -= nsb;
  int s = 0;
  for (; s + 1 < J.S; ++s) {
    const long nb = pole_blocks(J.sh, s);
    if (lb < nb) break;
    lb -= nb;
  }
  const long unit = lb * 4 + warp;
  if (unit >= (long)J.sh.nch[s] * J.sh.wt) return;
  pole_body(a.sys, a.sp[s], J.sh, J.om, J.n, J.part, s, unit);
  const int js = J.sh.js, w = (int)(unit % J.sh.wt) * (32 / js) + lane / js;
  __syncwarp();
  small_arrive(a, J, w, w < J.n && (lane & (js - 1)) == 0);
}

static_assert(RES_WARPS == 4, "pole sums and slots share blocks of 128 threads");
__global__ void __launch_bounds__(128, 3) k_disp_one(const __grid_constant__ DispArgs pa,
                                                     const __grid_constant__ DispJob pj) {
  __shared__ DispArgs sa;
  const DispArgs& a = stage_args(&pa, sa);
  small_body(a, pj, blockIdx.x);
}
__global__ void __launch_bounds__(128, 3) k_disp_many(const DispJob* __restrict__ jobs, int nj) {
  __shared__ DispArgs sa;
  const DispJob& J = job_of(jobs, nj, blockIdx.x, 5);
  const DispArgs& a = stage_args(J.a, sa);
  small_body(a, J, (long)blockIdx.x - J.blk[5]);
}

template <typename T>
int ensure_buf(T*& ptr, size_t& cap, size_t n) {
  if (n <= cap && ptr) return ALPS_OK;
  // a buffer that grows again grows by half its size at least: each
  // regrowth frees the old buffer, and cudaFree waits for the whole device
  // (in the request server, for every request in flight)
  const size_t want = ptr ? std::max(n, cap + cap / 2) : n;
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  cap = 0;
  ALPS_CUDA_TRY(cudaMalloc(&ptr, (want ? want : 1) * sizeof(T)));
  cap = want;
  return ALPS_OK;
}

}  // namespace

void fill_sys_dev(const alps_ctx* c, SysDev* o) {
  o->nspec = c->sys.nspec;
  o->kperp_norm = c->sys.kperp_norm;
  o->M_I = c->sys.positions_principal;
  o->M_P = c->sys.n_resonance_interval;
  o->iM_P = 1.0 / c->sys.n_resonance_interval;
  o->Tlim = c->sys.Tlim;
  o->vA = c->sys.vA;
  o->kperp = c->kperp;
  o->kpar = c->kpar;
  o->ikpar = 1.0 / c->kpar;
  const double k1 = c->sys.kperp_norm ? 1.0 : c->kperp, k2 = c->sys.kperp_norm ? 1.0 : c->kperp * c->kperp;
  o->k1h = (float)k1;
  o->k1l = (float)(k1 - (double)o->k1h);
  o->k2h = (float)k2;
  o->k2l = (float)(k2 - (double)o->k2h);
}

void fill_spec_dev(const alps_ctx* c, int is, SpecDev* o) {
  const SpeciesHost& S = c->spec[is];
  o->N = c->sys.nperp;
  o->M = c->sys.npar;
  o->nmax = S.nmax;
  o->nf = S.sp.ac_method == 1 ? S.sp.n_fits : 1;
  o->ac_method = S.sp.ac_method;
  o->log_fit = S.sp.log_fit;
  for (int f = 0; f < ALPS_MAX_FITS; ++f) {
    o->fit_type[f] = S.sp.fit_type[f];
    o->perp_corr[f] = S.sp.perp_correction[f];
  }
  o->qs = S.sp.qs;
  o->ms = S.sp.ms;
  o->ns = S.sp.ns;
  const bool bm = S.sp.use_bM != 0;
  o->dpperp = bm ? 0.0 : S.pperp[2] - S.pperp[1];
  o->dppar = bm ? 0.0 : S.ppar[2] - S.ppar[1];
  o->dppar_abs = std::fabs(o->dppar);
  o->idppar = bm ? 0.0 : 1.0 / o->dppar;
  o->hidpa = bm ? 0.0 : 0.5 / o->dppar_abs;
  o->qk = S.sp.qs / c->kpar;
  o->species_index = is + 1;
  o->int_ee = S.int_ee;
  o->pperp = S.d_pperp;
  o->ppar = S.d_ppar;
  o->f0 = S.d_f0;
  o->g1 = S.d_g1;
  o->g2 = S.d_g2;
  o->fit = S.d_fit;
  o->bessel = S.d_bessel;
  o->V = S.d_V;
  o->mom = S.d_mom;
  o->pfac = S.d_pfac;
  o->Vh = S.d_Vh;
  o->Vl = S.d_Vl;
  o->Vscale = S.d_Vscale;
  o->pph = S.d_pph;
  o->ppl = S.d_ppl;
  o->df_sums = (c->precision != ALPS_PREC_FP64 && S.d_Vh) ? 1 : 0;
  {
    const size_t nm = (size_t)(S.nmax + 1), M = (size_t)c->sys.npar;
    const size_t nvf = nm * (M - 1) * 12, nmo = nm * ALPS_KFAR * 12;
    const bool fz = S.d_Bt != nullptr && S.d_Bd != nullptr;
    o->Bt = fz ? S.d_Bt : nullptr;
    o->mBt = fz ? S.d_Bt + nvf : nullptr;
    o->bfac = fz ? S.d_Bt + nvf + nmo : nullptr;
    o->Escale = fz ? S.d_Bd : nullptr;
    o->Cfull = fz ? S.d_Bd + 8 : nullptr;
    o->Pre = fz ? S.d_Bd + 8 + nm * 6 : nullptr;
    o->qlo = S.qlo;
    o->qhi = S.qhi;
    o->qlo_in = S.qlo_in;
    o->qhi_in = S.qhi_in;
  }
  {
    const double kap = c->kpar / S.sp.ms;
    o->kaph = (float)kap;  // round to nearest, as __double2float_rn
    o->kapl = (float)(kap - (double)o->kaph);
    o->hidh = (float)o->hidpa;
    o->hidl = (float)(o->hidpa - (double)o->hidh);
    o->kappa = kap;
    o->dpph = (float)o->dppar;
    o->dppl = (float)(o->dppar - (double)o->dpph);
    o->idph = (float)o->idppar;
    o->idpl = (float)(o->idppar - (double)o->idph);
    const double tpm = 2.0 * ALPS_PI * c->sys.n_resonance_interval;
    o->tpmh = (float)tpm;
    o->tpml = (float)(tpm - (double)o->tpmh);
    o->pvc = 2.0 * ALPS_PI * o->dpperp * 0.25 * (-o->qk * 0.5);
    auto pair = [](double x, float* h, float* l) {
      *h = (float)x;
      *l = (float)(x - (double)*h);
    };
    const double z = c->sys.kperp_norm ? c->kperp / S.sp.qs : 1.0 / S.sp.qs;
    o->iz = 1.0 / z;
    pair(o->iz, &o->izh, &o->izl);
    pair(o->dppar_abs, &o->pdh, &o->pdl);
    pair(c->kpar < 0.0 ? -o->qk : o->qk, &o->qlh, &o->qll);
    pair(-o->dpperp * ALPS_PI * 2.0 * ALPS_PI, &o->lih, &o->lil);
  }
  o->pcen = bm ? 0.0 : 0.5 * (S.ppar[1] + S.ppar[c->sys.npar - 1]);
  o->prad = bm ? 0.0 : 0.5 * (S.ppar[c->sys.npar - 1] - S.ppar[1]);
  o->pcen32 = (float)o->pcen;
  o->prad32 = (float)o->prad;
  const float drift = 4e-9f * (float)c->sys.npar;
  o->gtol = std::max(1e-5f, drift);
  o->ptol = std::max(PV_TOL, drift);
  // the series is used only where it is cheaper than the node sum
  o->kfar = std::min(ALPS_KFAR, (int)(0.8 * (c->sys.npar - 1)));
  o->far = S.d_far;
  o->farc = S.d_farc;
  {
    // far orders: n |q| >= 2.5 P; the window beyond the grid's ends lies well
    // inside their distance on grids of a few windows
    const double P = std::fabs(c->kpar) * (std::fabs(o->pcen) + o->prad), n1 = std::ceil(2.5 * P / std::fabs(S.sp.qs));
    o->farn = (!bm && S.d_far && S.sp.qs != 0.0 && n1 + 4.0 <= (double)S.nmax &&
               c->sys.npar >= 4 * (c->sys.positions_principal + 2))
                  ? std::max(1, (int)n1)
                  : 0;
  }
  o->rcap = S.rcap;
  o->fit_aux = S.d_fit_aux;
  o->lmom = S.lfact ? S.d_lmom : nullptr;
  o->p2r = S.p2r;
  o->p3r = S.p3r;
  o->la = S.la;
  o->lb = S.lb;
  o->lc = S.lc;
  o->lgc = std::exp(-S.p2r * o->dppar * o->dppar);  // dppar is 0 for closed-form species (no grid)
  o->lmomf = o->lmom ? reinterpret_cast<const float*>(S.d_lmom + (size_t)(S.nmax + 1) * 30) : nullptr;
  o->la32 = (float)S.la;
  o->lb32 = (float)S.lb;
  o->lc32 = (float)S.lc;
  o->lgch = (float)o->lgc;
  o->lgcl = (float)(o->lgc - (double)o->lgch);
  o->lcx = -2.0 * S.p2r * o->dppar_abs;
  // (a row of amplitude zero leaves the Landau term zero at every frequency)
  o->lze = S.min_a0 > 0.0 ? std::ilogb(S.min_a0) : -1000000;
  o->lge = (o->lgc > 0.0) ? std::ilogb(o->lgc) : -2000;
  o->relat = S.sp.relat ? 1 : 0;
  o->ng = c->sys.ngamma;
  o->np = c->sys.npparbar;
  o->grel = S.d_grel;
  o->prel = S.d_prel;
  o->f0rel = S.d_f0rel;
  o->dfr1 = S.d_dfr1;
  o->dfr2 = S.d_dfr2;
  o->relfam = S.d_relfam;
  o->relcoef = S.d_relcoef;
  {
    const size_t nn = (size_t)(c->sys.nperp + 1) * (c->sys.npar + 1);
    o->relgam = S.d_relgam;
    o->relg2g = S.d_relgam ? S.d_relgam + nn : nullptr;
    o->relgf = S.d_relgam ? reinterpret_cast<const float*>(S.d_relgam + 2 * nn) : nullptr;
  }
  o->Rw = S.d_Rw;
  o->cone = S.d_cone;
  o->int_ee_rel = S.int_ee_rel;
  o->poly_order = S.sp.poly_order;
  o->poly_log_max = S.sp.poly_log_max;
  o->ppar_lo = bm ? 0.0 : S.ppar[0];
  o->ppar_hi = bm ? 0.0 : S.ppar[c->sys.npar];
  o->bm = bm ? 1 : 0;
  o->bm_nrun = S.bm_nrun;
  o->bm_beta = S.sp.bM_betas;
  o->bm_alpha = S.sp.bM_alphas;
  o->bm_pdrift = S.sp.bM_pdrifts;
  o->bmI = S.d_bmI;
}

bool any_bm(const alps_ctx* c) {
  for (int s = 0; s < c->sys.nspec; ++s)
    if (c->spec[s].sp.use_bM) return true;
  return false;
}

// order slots of the relativistic per-order results (0 when no species is)
int rel_capacity(const alps_ctx* c) {
  int cap = 0;
  for (int s = 0; s < c->sys.nspec; ++s)
    if (c->spec[s].sp.relat) cap = std::max(cap, c->spec[s].nmax + 1);
  return cap;
}

int collect_profile(alps_ctx* c) {
  for (auto& ev : c->ev_pending) {
    ALPS_CUDA_TRY(cudaEventSynchronize(ev[4]));
    for (int q = 0; q < 4; ++q) {
      float ms = 0.f;
      ALPS_CUDA_TRY(cudaEventElapsedTime(&ms, ev[q], ev[q + 1]));
      c->prof_ms[q] += ms;
    }
    c->prof_batches++;
    for (auto e : ev) c->ev_pool.push_back(e);
  }
  c->ev_pending.clear();
  return ALPS_OK;
}

// Runs the four kernels of one batch on stream st.
// the arguments of one context at its current k; *maxn = largest nmax
void build_disp_args(const alps_ctx* c, DispArgs* a, int* maxn) {
  fill_sys_dev(c, &a->sys);
  int mx = 0, rc = 1;
  for (int s = 0; s < c->sys.nspec; ++s) {
    fill_spec_dev(c, s, &a->sp[s]);
    mx = std::max(mx, c->spec[s].nmax);
    rc = std::max(rc, c->spec[s].rcap);
  }
  a->rcap = rc;
  a->relcap = rel_capacity(c);
  a->has_bm = any_bm(c) ? 1 : 0;
  *maxn = mx;
}

// ---------------------------------------------------------------------------
// Launch-shape table of the autotuner (alps_autotune).  Per bucket of
// (N_perp, N_par, nmax + 1, batch size), each rounded up to a power of two,
// species count and precision path: the tuned j slices per omega, pole-sum
// blocks per SM and resonant warps per SM.  Batches outside the table take
// the default rule of batch_geom.  A change of the table moves the tuning
// epoch, which retires the server's captured graphs.
// ---------------------------------------------------------------------------
namespace {
std::mutex g_tune_mu;
std::map<std::array<int, 6>, TuneShape> g_tune;
std::atomic<uint64_t> g_tune_epoch{0};
thread_local const TuneShape* t_tune_force = nullptr;  // the autotuner's candidate
int ceil_log2(long v) {
  int b = 0;
  while ((1L << b) < v) ++b;
  return b;
}
std::array<int, 6> tune_key(const alps_ctx* c, int n, int maxn) {
  return {ceil_log2(c->sys.nperp), ceil_log2(c->sys.npar), ceil_log2(maxn + 1), ceil_log2(n), c->sys.nspec,
          c->precision};
}
TuneShape tune_lookup(const alps_ctx* c, int n, int maxn) {
  if (t_tune_force) return *t_tune_force;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (g_tune.empty()) return TuneShape{};
  auto it = g_tune.find(tune_key(c, n, maxn));
  return it == g_tune.end() ? TuneShape{} : it->second;
}
}  // namespace

uint64_t tune_epoch() { return g_tune_epoch.load(); }

// The default lanes per frequency and signed orders per chunk of a batch of
// u = n orders / 32 warps of single orders at one lane each: more lanes where
// one lane's sum over the nodes would be the longest chain, fewer where the
// lanes' own set-up counts.  Within a class the shape is the same for every
// n, and so are a frequency's sums (csize 0: as many orders as leave twice 32
// warps per SM, where a batch has warps to spare).  The lines lie where the
// next form measured faster.  Small batches, the one launch in us (lanes/
// orders): mixed 128x256 grid, 73 signed orders, n = 1: 33 with 32/4, 38 with
// 32/8; 31: 39 with 32/4, 45 with 32/8; 60x120 grid, 113 orders, 31: 41 with
// 32/8, 45 with 32/4; 64: 52 with 32/8, 68 with 32/4; FP64, 120x240 grid, 138
// orders, n = 1: 38 with 32/1, 44 with 32/2; 8: 42 with 32/4, 69 with 32/1;
// 31: 64 with 32/8, 78 with 32/4; 64: 87 with 32/16, 97 with 16/8.  Larger
// ones, the pole sums in us, 128x256 grid: mixed n = 512: 59 with 8 lanes, 72
// with 16, 80 with 4; 2048: 150 with 8 or 4, 167 with 2; 4096: 256 with 1, 262
// with 2, 269 with 4; about one order per lane is best (512, 8 lanes: 59 with
// 8 orders, 64 with 4, 81 with 2).  FP64 n = 256: 138 with 16/8, 163 with 8/8;
// 2048: 579 with 8/8, 627 with 16/16, 699 with 4/8; 16384: 3535 with 8/64,
// 4388 with 8/16, 4606 with 1/16.
void default_shape(long u, bool mixed, int* lanes, long* csize) {
  if (mixed) {
    *lanes = u < 300 ? 32 : (u < 440 ? 16 : (u < 3000 ? 8 : (u < 7700 ? 4 : 1)));
    *csize = u < 100 ? 4 : (u < 3000 ? 8 : (u < 7700 ? 4 : 0));
  } else {
    *lanes = u < 400 ? 32 : (u < 600 ? 16 : 8);
    *csize = u < 8 ? 1 : (u < 50 ? 4 : (u < 180 ? 8 : (u < 400 ? 16 : (u < 20000 ? 8 : 64))));
  }
}

// Lanes per frequency of a batch with tensors (u as above), whose chunks are
// single orders: one lane of a frequency takes its order's series, so more of
// them pay only where the batch leaves the chip idle and the node sums are the
// longest chain.  calc_eigen on a 96x192 grid, mixed, us with 32/16/8/4/2/1
// lanes: u = 80: 113, 121, 170, 282, 491, 874; 208: 196, 175, 216, 350, 631,
// 1123; 832: 345, 273, 235, 255, 701, 1225; 1181: 622, 537, 488, 463, 479, 509;
// 2418: 851, 660, 547, 512, 487, 539; 24187: 6911, 4929, 3872, 3293, 3009,
// 2874; FP64: 80: 141, 145, 229, ..; 832: 710, 480, 386, 427, ..; 2418: 1891,
// 1303, 1000, 886, 870, 1130; 8062: 5841, 3903, 2835, 2265, 2126, 2079.
int tensor_lanes(long u) { return u < 100 ? 32 : (u < 300 ? 16 : (u < 900 ? 8 : (u < 1500 ? 4 : (u < 7000 ? 2 : 1)))); }

// launch shape of a batch of n omegas on a context (default rule, or the
// autotuner's shape for the batch's bucket).  The shape depends on n, the
// context and the table only: the lanes and chunks fix the summation order.
// tensors: the batch writes chi_low, so every order is a chunk of its own.
#define FIN_WARP_MAX 4096
// an item per lane takes 97 us at any size up to some 4096 frequencies (one
// lane's chain), a warp per item 116 us at 1024 and 208 us at 2999; where a
// species' Landau terms are left to the warps (kappa electrons, 128x256 grid, 2600
// frequencies) a batch takes 957 us with the lanes, 1045 without
#define RES_LANES_MIN 2560
// Slots per warp of k_resonant_multi at most where it only takes what the lanes
// left.  Where the Landau terms do not factorise that is every damped order by
// its rows, and the warps' times differ: two Maxwellians on a 64x128 grid,
// 2600, 16384 and 150000 frequencies, us in all: 32 slots 1093, 5221, 39396;
// 64: 1093, 5438, 39746; 128: 1090, 5944, 40635; 256 and more 3969, 7154, 40521.
// With nothing left the blocks end at once, which very many of them feel: sixteen
// times what the chip holds at most.
inline int res_left_per_warp(long nslots) { return (int)std::max(32L, std::min(256L, nslots / (152L * 12 * 16))); }
// The far-order series takes the orders |n| >= n0 of a frequency (some two
// thirds of them) in 44 terms; its coefficients are built for each batch.
// Pole sums by single orders and so, with the 58 us of the coefficients (128x256
// grid, 73 signed orders): 12000 frequencies 481 and 465 us, 16384: 636 and
// 546, 32768: 1141 and 926, 262144: 5145 and 3140; FP64, 16384: 3643 and 3317.
#define FAR_MIN 25000
#define ALPS_NOALLOC_SCRATCH_BYTES (16u << 20)

// 256-byte aligned carve-out of n bytes from a scratch array
inline size_t carve(size_t& off, size_t bytes) {
  size_t at = (off + 255) & ~(size_t)255;
  off = at + bytes;
  return at;
}

// doubles of a species' far-order tables: by level (far), then by order (farc)
size_t far_words(const SpeciesHost& S) { return (size_t)(FAR_LEVELS + S.nmax) * FAR_K * 12; }

// the scratch of a batch in one array: error word, counts, slots, items,
// relativistic and closed-form results, arguments, job, far-order tables
// (far: the batch takes that series), and last the partial sums (part_bytes
// of them); off[] receives the offsets
enum { SC_FLAGS, SC_COUNT, SC_SLOTS, SC_ITEMS, SC_REL, SC_BM, SC_ARGS, SC_JOB, SC_FAR, SC_PART, SC_N };
size_t scratch_layout(const alps_ctx* c, size_t n, size_t nslots, size_t part_bytes, bool far, size_t* off) {
  const size_t S_ = c->sys.nspec;
  size_t farw = 0;
  for (size_t s = 0; s < S_ && far; ++s) farw += far_words(c->spec[s]);
  size_t end = 0;
  off[SC_FLAGS] = carve(end, sizeof(int));
  off[SC_COUNT] = carve(end, n * S_ * sizeof(int));
  off[SC_SLOTS] = carve(end, nslots * sizeof(int));
  off[SC_ITEMS] = carve(end, nslots * 6 * sizeof(double2));
  off[SC_REL] = carve(end, n * S_ * rel_capacity(c) * 2 * REL_RB * 6 * sizeof(double2));
  off[SC_BM] = carve(end, n * S_ * (any_bm(c) ? 24 : 0) * sizeof(double2));
  off[SC_ARGS] = carve(end, sizeof(DispArgs));
  off[SC_JOB] = carve(end, DISP_JOB_BYTES);
  off[SC_FAR] = carve(end, farw * sizeof(double));
  off[SC_PART] = carve(end, part_bytes);
  return end;
}

// The order chunks that alps_disp_batch_noalloc has always had room for: one
// for about every four warps per SM of 128-frequency tiles.  A batch that
// fits its static array with so many chunks has to fit it with the shape
// chosen here, which is the same for every entry point.
long noalloc_chunks(int n, int S_, int maxn) {
  const int js = n < 32 ? 32 : (n < 64 ? 4 : (n < 128 ? 2 : 1)), tw = 128 / js;
  const long tiles = (long)((n + tw - 1) / tw) * S_;
  const long nchunk = std::max(1L, std::min(maxn + 1L, (152L * 4 + tiles - 1) / tiles));
  long csize = (maxn + nchunk) / nchunk;
  if (n < 32) csize = std::max(csize, (long)std::min(maxn + 1, 16 / std::max(1, n)));
  return (maxn + csize) / csize;
}

struct BatchGeom {
  size_t nslots;
  DispShape sh;
};
BatchGeom batch_geom(const alps_ctx* c, int n, int S_, int maxn, int rcap, bool tensors) {
  BatchGeom b;
  const TuneShape ts = tune_lookup(c, n, maxn);
  const bool mixed = c->precision != ALPS_PREC_FP64;
  DispShape& sh = b.sh;
  long orders = 0;
  for (int s = 0; s < S_; ++s)
    if (!c->spec[s].sp.relat && !c->spec[s].sp.use_bM) orders += 2 * c->spec[s].nmax + 1;
  long csize = 0;
  default_shape((long)n * orders / 32, mixed, &sh.js, &csize);
  if (tensors) sh.js = tensor_lanes((long)n * orders / 32);
  else if (ts.js) sh.js = ts.js;
  sh.wt = (int)(((long)n * sh.js + 31) / 32);
  if (ts.blocks_per_sm || csize == 0) {
    const long want = ts.blocks_per_sm ? 152L * 4 * ts.blocks_per_sm : 152L * 64;
    csize = (orders * sh.wt + want - 1) / want;
  }
  if (tensors) csize = 1;
  csize = std::max(csize, 1L);
  b.nslots = (size_t)n * S_ * rcap;
  sh.far = (!tensors && (long)n * orders / 32 >= FAR_MIN) ? 1 : 0;
  if (!tensors) {
    size_t off[SC_N];
    const size_t row = (size_t)n * S_ * 6 * sizeof(double2), part = row * noalloc_chunks(n, S_, maxn);
    if (scratch_layout(c, n, b.nslots, part, false, off) <= ALPS_NOALLOC_SCRATCH_BYTES) {
      // (a batch that fits without the far-order tables alone does without
      // the series, through every entry point)
      if (sh.far && scratch_layout(c, n, b.nslots, part, true, off) > ALPS_NOALLOC_SCRATCH_BYTES) {
        sh.far = 0;
        scratch_layout(c, n, b.nslots, part, false, off);
      }
      const long room = (long)((ALPS_NOALLOC_SCRATCH_BYTES - off[SC_PART]) / row);
      csize = std::max(csize, (2L * maxn + room) / room);
    }
  }
  sh.nchunk = 1;
  for (int s = 0; s < ALPS_MAX_SPECIES; ++s) {
    const bool has = s < S_ && !c->spec[s].sp.relat && !c->spec[s].sp.use_bM;
    sh.nch[s] = has ? (int)((2 * c->spec[s].nmax + 1 + csize - 1) / csize) : 0;
    sh.nchunk = std::max(sh.nchunk, sh.nch[s]);
  }
  // a lane sums a series alone while its terms cost less than the slices of
  // a node sum
  sh.kmid = (int)(0.8 * (c->sys.npar - 1) / sh.js) + 16;
  sh.ipw = res_items_per_warp((long)b.nslots, ts.warps_per_sm ? ts.warps_per_sm : 12);
  sh.lanes = 0;
  if (mixed && !tensors && n >= RES_LANES_MIN && pvl_side(c->sys.positions_principal) <= 8 &&
      c->sys.n_resonance_interval < PVL_SAMPLES) {
    // about a third of the slots is occupied: 96 fill a warp's lanes once
    const long per = ((long)b.nslots / (152 * 12) + 31) / 32 * 32;
    sh.lanes = (int)std::max(96L, std::min(256L, per));
    sh.ipw = std::min(sh.ipw, res_left_per_warp((long)b.nslots));
  }
  sh.fin_warp = (n <= FIN_WARP_MAX || tensors || rel_capacity(c) || any_bm(c)) ? 1 : 0;
  return b;
}

namespace {

// the job of a lone batch (first blocks at 0)
DispJob lone_job(const DispShape& sh, int n, int S_, const double2* om, double2* D, double2* part,
                 int* count, int* slots, double2* items, int* flags) {
  DispJob j;
  j.a = nullptr;
  j.sh = sh;
  j.n = n;
  j.S = S_;
  j.nslots = 0;
  for (int k = 0; k < 6; ++k) j.blk[k] = 0;
  j.arrive = nullptr;
  j.hflag = nullptr;
  j.om = om;
  j.D = D;
  j.part = part;
  j.count = count;
  j.slot_nn = slots;
  j.items = items;
  j.flags = flags;
  j.ext = nullptr;
  j.rel = nullptr;
  j.bm = nullptr;
  return j;
}

// dynamic shared memory of k_resonant_multi for a context, and the opt-in
// above 48 KB (per kernel, once per size)
size_t res_smem(const alps_ctx* c) {
  return (size_t)RES_WARPS * res_warp_smem(c->sys.nperp, c->sys.positions_principal) * sizeof(double2);
}
std::mutex g_res_smem_mu;
size_t g_res_smem_set[4] = {0, 0, 0, 0};  // k_resonant_multi, k_resonant_lanes, k_disp_one, k_disp_many
int res_smem_optin(size_t smem, size_t lanes_smem, bool small = false) {
  const size_t want[4] = {small ? 0 : smem, lanes_smem, small ? smem : 0, small ? smem : 0};
  auto set = [](int q, int bytes) {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    return q == 0 ? cudaFuncSetAttribute(k_resonant_multi, at, bytes)
                  : (q == 1 ? cudaFuncSetAttribute(k_resonant_lanes, at, bytes)
                            : (q == 2 ? cudaFuncSetAttribute(k_disp_one, at, bytes)
                                      : cudaFuncSetAttribute(k_disp_many, at, bytes)));
  };
  std::lock_guard<std::mutex> lk(g_res_smem_mu);
  for (int q = 0; q < 4; ++q)
    if (want[q] > 40 * 1024 && g_res_smem_set[q] < want[q]) {
      ALPS_CUDA_TRY(set(q, (int)want[q]));
      g_res_smem_set[q] = want[q];
    }
  return ALPS_OK;
}
// Batches that run in one launch (k_disp_one, k_disp_many): as many warps as
// the chip holds twice over at most.  Beyond, the warps of empty slots and
// the kernel's larger frame cost more than the gaps between the launches (60x120
// grid, us in one launch and apart: 31 frequencies 53 and 82, 128: 100 and
// 113, 256: 141 and 125).
#define SMALL_WARPS (152 * 12 * 2)
#define MANY_WARPS (152 * 12 * 4)
long pole_warps(const DispShape& sh, int S_) { return 4 * pole_blocks_all(sh, S_); }
bool small_batch(const alps_ctx* c, const BatchGeom& bg) {
  return !c->profiling && !rel_capacity(c) && !any_bm(c) && bg.sh.fin_warp && !bg.sh.lanes && !bg.sh.far &&
         (long)bg.nslots + pole_warps(bg.sh, c->sys.nspec) <= SMALL_WARPS;
}
int launch_one(const alps_ctx* c, const DispArgs& a, const DispShape& sh, const DispJob& job, cudaStream_t st) {
  const size_t smem = res_smem(c);
  int rc = res_smem_optin(smem, 0, true);
  if (rc) return rc;
  const long blocks = small_slot_blocks(job.nslots) + pole_blocks_all(sh, c->sys.nspec);
  k_disp_one<<<(unsigned)blocks, 128, smem, st>>>(a, job);
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}
int far_groups(int maxn) { return (maxn + 7) / 8; }
void launch_far(const DispJob* jobs, int groups, int species, int nj, cudaStream_t st) {
  k_far_orders<<<dim3(FAR_K * groups, species, nj), 32, 0, st>>>(jobs);
  k_far_levels<<<dim3(FAR_K, species, nj), 32, 0, st>>>(jobs);
}
long lanes_blocks(const BatchGeom& bg) {
  const long per = (long)RES_WARPS * bg.sh.lanes;
  return per ? ((long)bg.nslots + per - 1) / per : 0;
}

}  // namespace

// first: the first part of a batch, which clears its error word
static int launch_disp_part(alps_ctx* c, int n, const double2* d_om, double2* d_D, double2* d_ext, cudaStream_t st,
                            int* hflag, bool* flag_there, bool first) {
  const int S_ = c->sys.nspec;
  DispArgs a;
  int maxn = 0;
  build_disp_args(c, &a, &maxn);
  const BatchGeom bg = batch_geom(c, n, S_, maxn, a.rcap, d_ext != nullptr);
  const DispShape sh = bg.sh;
  const size_t nslots = bg.nslots;
  int rcode;
  const void* before[7] = {c->d_part, c->d_count, c->d_slot_nn, c->d_items, c->d_rel, c->d_bm, c->d_flags};
  if ((rcode = ensure_buf(c->d_part, c->part_cap, (size_t)n * S_ * sh.nchunk * 6))) return rcode;
  if ((rcode = ensure_buf(c->d_count, c->count_cap, (size_t)n * S_))) return rcode;
  if (nslots * 6 > c->items_cap || !c->d_slot_nn) {
    // the slot table holds items_cap / 6 entries (one per item row of six)
    if ((rcode = ensure_buf(c->d_items, c->items_cap, nslots * 6))) return rcode;
    if (c->d_slot_nn) cudaFree(c->d_slot_nn);
    c->d_slot_nn = nullptr;
    ALPS_CUDA_TRY(cudaMalloc(&c->d_slot_nn, (c->items_cap / 6) * sizeof(int)));
  }
  if (a.relcap)
    if ((rcode = ensure_buf(c->d_rel, c->rel_cap, (size_t)n * S_ * a.relcap * 2 * REL_RB * 6))) return rcode;
  if (a.has_bm)
    if ((rcode = ensure_buf(c->d_bm, c->bm_cap, (size_t)n * S_ * 24))) return rcode;
  if (!c->d_flags) {
    // the error word, and a counter per frequency of a small batch (zero
    // between launches)
    ALPS_CUDA_TRY(cudaMalloc(&c->d_flags, (1 + SMALL_WARPS) * sizeof(int)));
    ALPS_CUDA_TRY(cudaMemsetAsync(c->d_flags, 0, (1 + SMALL_WARPS) * sizeof(int), st));
  }
  const void* after[7] = {c->d_part, c->d_count, c->d_slot_nn, c->d_items, c->d_rel, c->d_bm, c->d_flags};
  for (int q = 0; q < 7; ++q)
    if (before[q] != after[q]) c->gen++;  // buffer addresses changed: cached graphs are stale
  const bool small = small_batch(c, bg);
  int* flags = c->d_flags;
  if (small && hflag) {
    // a word and counters of their own: these batches are over when their call
    // returns, so nothing that a caller leaves running reaches them, and the
    // word is zero while none reported
    if (!c->d_hflags) {
      ALPS_CUDA_TRY(cudaMalloc(&c->d_hflags, (1 + SMALL_WARPS) * sizeof(int)));
      ALPS_CUDA_TRY(cudaMemsetAsync(c->d_hflags, 0, (1 + SMALL_WARPS) * sizeof(int), st));
      c->flags_dirty = false;
    }
    flags = c->d_hflags;
    if (c->flags_dirty) ALPS_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int), st));
    c->flags_dirty = false;
  } else if (first) {
    // (with the counters: calls that a caller let overlap, against the
    // contract, leave nothing behind)
    ALPS_CUDA_TRY(cudaMemsetAsync(flags, 0, (small ? 1 + n : 1) * sizeof(int), st));
  }
  if (small) {
    DispJob job = lone_job(sh, n, S_, d_om, d_D, c->d_part, c->d_count, c->d_slot_nn, c->d_items, flags);
    job.ext = d_ext;
    job.nslots = (int)nslots;
    job.arrive = flags + 1;
    job.hflag = hflag;
    if ((rcode = launch_one(c, a, sh, job, st))) return rcode;
    if (flag_there) *flag_there = hflag != nullptr;
    c->stats.n_eval = n;
    c->stats.n_eval_total += n;
    c->stats.kernels_launched = 1;
    return ALPS_OK;
  }

  std::vector<cudaEvent_t> ev;
  if (c->profiling) {
    for (int q = 0; q < 5; ++q) {
      cudaEvent_t e;
      if (!c->ev_pool.empty()) {
        e = c->ev_pool.back();
        c->ev_pool.pop_back();
      } else {
        ALPS_CUDA_TRY(cudaEventCreate(&e));
      }
      ev.push_back(e);
    }
    ALPS_CUDA_TRY(cudaEventRecord(ev[0], st));
  }
  if (!c->d_args) {
    ALPS_CUDA_TRY(cudaMalloc(&c->d_args, sizeof(DispArgs)));
    ALPS_CUDA_TRY(cudaMallocHost(&c->h_args, sizeof(DispArgs)));
  }
  if (!c->d_job) ALPS_CUDA_TRY(cudaMalloc(&c->d_job, sizeof(DispJob)));
  DispJob job = lone_job(sh, n, S_, d_om, d_D, c->d_part, c->d_count, c->d_slot_nn, c->d_items, c->d_flags);
  job.ext = d_ext;
  job.rel = a.relcap ? c->d_rel : nullptr;
  job.bm = a.has_bm ? c->d_bm : nullptr;
  const DispJob* dj = static_cast<const DispJob*>(c->d_job);
  k_stage<<<1, 128, 0, st>>>(a, job, static_cast<DispArgs*>(c->d_args), static_cast<DispJob*>(c->d_job));
  ALPS_CUDA_TRY(cudaGetLastError());
  c->args_gen = c->gen;  // the device copy is the context at its current state
  c->args_maxn = maxn;
  c->args_rcap = a.rcap;
  k_classify_multi<<<(unsigned)cls_blocks(n, S_), 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (c->profiling) ALPS_CUDA_TRY(cudaEventRecord(ev[1], st));
  const long g2 = pole_blocks_all(sh, S_);
  const size_t smem = res_smem(c);
  const size_t lsmem = pvl_smem(c->sys.positions_principal);
  const long lblocks = lanes_blocks(bg);
  if ((rcode = res_smem_optin(smem, lblocks ? lsmem : 0))) return rcode;
  long blocks = ((long)nslots + RES_WARPS * sh.ipw - 1) / (RES_WARPS * sh.ipw);
  if (sh.far) launch_far(dj, far_groups(maxn), S_, 1, st);
  if (g2 > 0) k_pole_sums_multi<<<(unsigned)g2, 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (c->profiling) ALPS_CUDA_TRY(cudaEventRecord(ev[2], st));
  if (lblocks) k_resonant_lanes<<<(unsigned)lblocks, RES_WARPS * 32, lsmem, st>>>(dj, 1);
  k_resonant_multi<<<(unsigned)blocks, RES_WARPS * 32, smem, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (a.relcap && (rcode = launch_rel_orders(a.sys, a.sp, a.relcap, n, d_om, c->d_rel, c->d_flags, st)))
    return rcode;
  if (a.has_bm && (rcode = launch_nhds(a.sys, a.sp, n, d_om, c->d_bm, st))) return rcode;
  if (c->profiling) ALPS_CUDA_TRY(cudaEventRecord(ev[3], st));
  k_finalize_multi<<<(unsigned)fin_blocks(sh, n), 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (c->profiling) {
    ALPS_CUDA_TRY(cudaEventRecord(ev[4], st));
    c->ev_pending.push_back(ev);
  }
  c->stats.n_eval = n;
  c->stats.n_eval_total += n;
  // k_stage and the four; the far orders' two and k_resonant_lanes for large batches
  c->stats.kernels_launched = 5 + (sh.far ? 2 : 0) + (lblocks ? 1 : 0) + (a.relcap ? 1 : 0) + (a.has_bm ? 1 : 0);
  return ALPS_OK;
}

// The partial sums of a batch with tensors, one per order, are held for at most
// so many bytes of frequencies at a time: each part still has some 22 000 warps
// of orders, twelve times what the chip holds.
#define TENSOR_PART_BYTES (64L << 20)

int launch_disp_batch(alps_ctx* c, int n, const double2* d_om, double2* d_D, double2* d_ext, cudaStream_t st,
                      int* hflag, bool* flag_there) {
  if (flag_there) *flag_there = false;
  if (n <= 0) return ALPS_OK;
  long parts = 1;
  if (d_ext) {
    long orders = 1;
    for (const SpeciesHost& S : c->spec)
      if (!S.sp.relat && !S.sp.use_bM) orders = std::max(orders, 2L * S.nmax + 1);
    const long bytes = orders * c->sys.nspec * 6 * (long)sizeof(double2);
    parts = std::min((long)n, (n * bytes + TENSOR_PART_BYTES - 1) / TENSOR_PART_BYTES);
  }
  if (parts <= 1) return launch_disp_part(c, n, d_om, d_D, d_ext, st, hflag, flag_there, true);
  // (even parts: one launch shape for all)
  auto launched = c->stats.kernels_launched;
  launched = 0;
  for (int p = 0, o = 0; p < (int)parts; ++p) {
    const int m = n / (int)parts + (p < n % (int)parts ? 1 : 0);
    const int rc = launch_disp_part(c, m, d_om + o, d_D + o, d_ext + (size_t)o * (c->sys.nspec * 36 + 9), st, nullptr,
                                    nullptr, p == 0);
    if (rc) return rc;
    launched += c->stats.kernels_launched;
    o += m;
  }
  c->stats.n_eval = n;
  c->stats.kernels_launched = launched;
  return ALPS_OK;
}

// ---------------------------------------------------------------------------
// Fused batches of several contexts (the request server's rounds)
// ---------------------------------------------------------------------------
struct MultiScratch {
  DispJob* d_jobs = nullptr;
  DispJob* h_jobs = nullptr;  // pinned
  size_t jobs_cap = 0;
  double2* part = nullptr;
  size_t part_cap = 0;
  int* count = nullptr;
  size_t count_cap = 0;
  int* slots = nullptr;
  size_t slots_cap = 0;
  double2* items = nullptr;
  size_t items_cap = 0;
  int* arrive = nullptr;  // units done per frequency, zero between launches
  size_t arrive_cap = 0;
};

void multi_scratch_free(MultiScratch* m) {
  if (!m) return;
  cudaFree(m->d_jobs);
  cudaFreeHost(m->h_jobs);
  cudaFree(m->part);
  cudaFree(m->count);
  cudaFree(m->slots);
  cudaFree(m->items);
  cudaFree(m->arrive);
  delete m;
}

bool ctx_fusable(const alps_ctx* c) { return !rel_capacity(c) && !any_bm(c) && !c->profiling; }

namespace {

// the context's kernel arguments on the device, rebuilt when the plasma, k,
// precision or a table moved (alps_ctx::gen)
int ctx_device_args(alps_ctx* c, cudaStream_t st, const DispArgs** out) {
  if (!c->d_args) {
    ALPS_CUDA_TRY(cudaMalloc(&c->d_args, sizeof(DispArgs)));
    ALPS_CUDA_TRY(cudaMallocHost(&c->h_args, sizeof(DispArgs)));
    c->args_gen = 0;
  }
  if (c->args_gen != c->gen) {
    DispArgs* h = static_cast<DispArgs*>(c->h_args);
    build_disp_args(c, h, &c->args_maxn);
    c->args_rcap = h->rcap;
    ALPS_CUDA_TRY(cudaMemcpyAsync(c->d_args, h, sizeof(DispArgs), cudaMemcpyHostToDevice, st));
    c->args_gen = c->gen;
  }
  *out = static_cast<const DispArgs*>(c->d_args);
  return ALPS_OK;
}

}  // namespace

int launch_disp_multi(alps_ctx* const* ctx, const int* n, int nj, const double2* d_om, double2* d_D, int* d_flags,
                      MultiScratch** scratch, cudaStream_t st) {
  if (nj <= 0) return ALPS_OK;
  MultiLaunch ml;
  int rc = prepare_disp_multi(ctx, n, nj, d_om, d_D, d_flags, scratch, st, &ml);
  if (rc) return rc;
  return run_disp_multi(ml, st);
}

int prepare_disp_multi(alps_ctx* const* ctx, const int* n, int nj, const double2* d_om, double2* d_D, int* d_flags,
                       MultiScratch** scratch, cudaStream_t st, MultiLaunch* out) {
  MultiScratch* m = *scratch;
  if (!m) *scratch = m = new MultiScratch();
  if ((size_t)nj > m->jobs_cap) {
    cudaFree(m->d_jobs);
    cudaFreeHost(m->h_jobs);
    m->d_jobs = nullptr;
    m->h_jobs = nullptr;
    m->jobs_cap = 0;
    ALPS_CUDA_TRY(cudaMalloc(&m->d_jobs, (size_t)nj * sizeof(DispJob)));
    ALPS_CUDA_TRY(cudaMallocHost(&m->h_jobs, (size_t)nj * sizeof(DispJob)));
    m->jobs_cap = nj;
  }
  // shapes, grid offsets and scratch offsets of every job
  std::vector<size_t> o_part(nj), o_count(nj), o_slots(nj);
  size_t part_n = 0, count_n = 0, slots_n = 0, om_off = 0, smem = 0, lsmem = 0;
  long blk[6] = {0, 0, 0, 0, 0, 0}, warps = 0;
  bool small = true;
  for (int j = 0; j < nj; ++j) {
    alps_ctx* c = ctx[j];
    const DispArgs* da = nullptr;
    int rcode = ctx_device_args(c, st, &da);
    if (rcode) return rcode;
    const int S_ = c->sys.nspec;
    const BatchGeom bg = batch_geom(c, n[j], S_, c->args_maxn, c->args_rcap, false);
    DispJob& J = m->h_jobs[j];
    J.a = da;
    J.sh = bg.sh;
    J.n = n[j];
    J.S = S_;
    J.blk[0] = blk[0];
    blk[0] += cls_blocks(n[j], S_);
    J.blk[1] = blk[1];
    blk[1] += pole_blocks_all(bg.sh, S_);
    J.blk[2] = blk[2];
    blk[2] += ((long)bg.nslots + RES_WARPS * bg.sh.ipw - 1) / (RES_WARPS * bg.sh.ipw);
    J.blk[3] = blk[3];
    blk[3] += fin_blocks(bg.sh, n[j]);
    J.blk[4] = blk[4];
    blk[4] += lanes_blocks(bg);
    J.nslots = (int)bg.nslots;
    J.blk[5] = blk[5];
    blk[5] += small_slot_blocks(J.nslots) + pole_blocks_all(bg.sh, S_);
    small = small && small_batch(c, bg);
    warps += (long)bg.nslots + pole_warps(bg.sh, S_);
    J.hflag = nullptr;
    if (bg.sh.lanes) lsmem = std::max(lsmem, pvl_smem(c->sys.positions_principal));
    J.om = d_om + om_off;
    J.D = d_D + om_off;
    J.flags = d_flags + j;
    J.ext = nullptr;
    J.rel = nullptr;
    J.bm = nullptr;
    om_off += n[j];
    o_part[j] = part_n;
    part_n += (size_t)n[j] * S_ * bg.sh.nchunk * 6;
    o_count[j] = count_n;
    count_n += (size_t)n[j] * S_;
    o_slots[j] = slots_n;
    slots_n += bg.nslots;
    smem = std::max(smem, res_smem(c));
  }
  // items per warp of k_resonant from the whole round (it does not change sums)
  const int ipw = res_items_per_warp((long)slots_n);
  blk[2] = 0;
  for (int j = 0; j < nj; ++j) {
    DispJob& J = m->h_jobs[j];
    const long nsl = (long)((j + 1 < nj ? o_slots[j + 1] : slots_n) - o_slots[j]);
    J.sh.ipw = J.sh.lanes ? std::min(ipw, res_left_per_warp(nsl)) : ipw;
    J.blk[2] = blk[2];
    blk[2] += (nsl + RES_WARPS * J.sh.ipw - 1) / (RES_WARPS * J.sh.ipw);
  }
  int rcode;
  if (om_off > m->arrive_cap) {
    if ((rcode = ensure_buf(m->arrive, m->arrive_cap, om_off))) return rcode;
    ALPS_CUDA_TRY(cudaMemsetAsync(m->arrive, 0, m->arrive_cap * sizeof(int), st));
  }
  if ((rcode = ensure_buf(m->part, m->part_cap, part_n))) return rcode;
  if ((rcode = ensure_buf(m->count, m->count_cap, count_n))) return rcode;
  if ((rcode = ensure_buf(m->slots, m->slots_cap, slots_n))) return rcode;
  if ((rcode = ensure_buf(m->items, m->items_cap, slots_n * 6))) return rcode;
  for (int j = 0; j < nj; ++j) {
    DispJob& J = m->h_jobs[j];
    J.part = m->part + o_part[j];
    J.count = m->count + o_count[j];
    J.slot_nn = m->slots + o_slots[j];
    J.items = m->items + o_slots[j] * 6;
    J.arrive = m->arrive + (J.om - d_om);
  }
  ALPS_CUDA_TRY(cudaMemcpyAsync(m->d_jobs, m->h_jobs, (size_t)nj * sizeof(DispJob), cudaMemcpyHostToDevice, st));
  small = small && warps <= MANY_WARPS;
  if ((rcode = res_smem_optin(smem, lsmem, small))) return rcode;
  out->small = small;
  out->far = 0;
  for (int j = 0; j < nj; ++j)
    if (m->h_jobs[j].sh.far) out->far = std::max(out->far, far_groups(ctx[j]->args_maxn));
  out->jobs = m->d_jobs;
  out->nj = nj;
  for (int k = 0; k < 6; ++k) out->blocks[k] = blk[k];
  out->smem = smem;
  out->lanes_smem = lsmem;
  out->flags = d_flags;
  return ALPS_OK;
}

// Where a job's frequency count sits in the device job table: a caller that
// lowers it between launches (alps_solve_many: roots asking for one
// frequency, or finished) makes the kernels skip the other slots, while the
// job's launch shape, and so its sums, stay those of the prepared size.
void disp_job_layout(size_t* stride, size_t* n_offset) {
  *stride = sizeof(DispJob);
  *n_offset = offsetof(DispJob, n);
}

// The kernels of a prepared fused batch (no host work: capturable, also
// inside a conditional graph body).
int run_disp_multi(const MultiLaunch& ml, cudaStream_t st) {
  const DispJob* jobs = static_cast<const DispJob*>(ml.jobs);
  ALPS_CUDA_TRY(cudaMemsetAsync(ml.flags, 0, (size_t)ml.nj * sizeof(int), st));
  if (ml.small) {
    k_disp_many<<<(unsigned)ml.blocks[5], 128, ml.smem, st>>>(jobs, ml.nj);
    ALPS_CUDA_TRY(cudaGetLastError());
    return ALPS_OK;
  }
  k_classify_multi<<<(unsigned)ml.blocks[0], 128, 0, st>>>(jobs, ml.nj);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (ml.far) launch_far(jobs, ml.far, ALPS_MAX_SPECIES, ml.nj, st);
  k_pole_sums_multi<<<(unsigned)ml.blocks[1], 128, 0, st>>>(jobs, ml.nj);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (ml.blocks[4]) k_resonant_lanes<<<(unsigned)ml.blocks[4], RES_WARPS * 32, ml.lanes_smem, st>>>(jobs, ml.nj);
  k_resonant_multi<<<(unsigned)ml.blocks[2], RES_WARPS * 32, ml.smem, st>>>(jobs, ml.nj);
  ALPS_CUDA_TRY(cudaGetLastError());
  k_finalize_multi<<<(unsigned)ml.blocks[3], 128, 0, st>>>(jobs, ml.nj);
  ALPS_CUDA_TRY(cudaGetLastError());
  return ALPS_OK;
}

// ===========================================================================
// det D batch without any device allocation.
//
// Some callers cannot let this library allocate device memory while they
// run: a host application whose own caching allocator owns the device heap
// and must see every byte, a real-time loop that cannot afford the implicit
// device-wide synchronisation of cudaMalloc/cudaFree, or a plugin host that
// forbids plugins from creating allocations behind its back.  For them,
// alps_disp_batch_noalloc runs the same kernels as
// alps_disp_batch_device with all of their scratch (partial sums,
// resonant-order slots, resonant results, far-order tables, error flag)
// carved from the file-scope device array below instead of context buffers:
// a call may overlap the context's other batches.
//
// The array is ALPS_NOALLOC_SCRATCH_BYTES (16 MiB) and lives on every device
// that loads this library until the process exits.  Its device address is
// looked up once per device with cudaGetSymbolAddress, by the first call on
// that device (with that device current); make that first call before any
// stream capture.  Every call shares the one array: two calls whose kernels
// overlap on the GPU (different streams, or different host threads) race on
// it and must be ordered by the caller.  The error flag and a small batch's
// counters are cleared at the start of every call; every other word a call
// reads it writes first.  The
// flag word's device address is recorded in the context, so
// alps_batch_status reports the call's device errors (read it before the
// next call on the device clears the word).
// ===========================================================================
#define ALPS_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) unsigned char g_noalloc_scratch[ALPS_NOALLOC_SCRATCH_BYTES];
static __device__ int g_noalloc_arrive[SMALL_WARPS];  // counters of a small batch

namespace {
std::mutex g_noalloc_mu;
void* g_noalloc_addr[ALPS_NOALLOC_MAX_DEVICES] = {nullptr};
void* g_noalloc_cnt[ALPS_NOALLOC_MAX_DEVICES] = {nullptr};
}  // namespace

extern "C" int alps_disp_batch_noalloc(alps_ctx* c, int n, const alps_complex* d_om, alps_complex* d_D,
                                       void* stream, size_t* scratch_bytes) {
  if (!c || n < 0 || !c->kset) return ALPS_E_INVALID;
  if (n == 0) return ALPS_OK;
  if (!d_om || !d_D) return ALPS_E_INVALID;
  int dev = -1;
  ALPS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= ALPS_NOALLOC_MAX_DEVICES) return ALPS_E_INVALID;
  void *base = nullptr, *cnt = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&g_noalloc_cnt[dev], g_noalloc_arrive);
      if (e == cudaSuccess) e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        alps_set_last_cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
        return ALPS_E_CUDA;
      }
      g_noalloc_addr[dev] = p;
    }
    base = g_noalloc_addr[dev];
    cnt = g_noalloc_cnt[dev];
  }
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  const int S_ = c->sys.nspec;
  DispArgs a;
  int maxn = 0;
  build_disp_args(c, &a, &maxn);
  const BatchGeom bg = batch_geom(c, n, S_, maxn, a.rcap, false);
  const DispShape sh = bg.sh;
  size_t off[SC_N];
  const size_t nslots = bg.nslots;
  const size_t total = scratch_layout(c, n, nslots, (size_t)n * S_ * sh.nchunk * 6 * sizeof(double2), sh.far != 0, off);
  if (scratch_bytes) *scratch_bytes = total;
  if (total > ALPS_NOALLOC_SCRATCH_BYTES) return ALPS_E_INVALID;  // batch too large for the static scratch
  unsigned char* b = static_cast<unsigned char*>(base);
  int* flags = reinterpret_cast<int*>(b + off[SC_FLAGS]);
  int* count = reinterpret_cast<int*>(b + off[SC_COUNT]);
  int* slots = reinterpret_cast<int*>(b + off[SC_SLOTS]);
  double2* part = reinterpret_cast<double2*>(b + off[SC_PART]);
  double2* items = reinterpret_cast<double2*>(b + off[SC_ITEMS]);
  double2* relb = reinterpret_cast<double2*>(b + off[SC_REL]);
  double2* bmb = reinterpret_cast<double2*>(b + off[SC_BM]);
  const double2* om = reinterpret_cast<const double2*>(d_om);
  double2* D = reinterpret_cast<double2*>(d_D);
  ALPS_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int), st));
  DispJob job = lone_job(sh, n, S_, om, D, part, count, slots, items, flags);
  job.rel = a.relcap ? relb : nullptr;
  job.bm = a.has_bm ? bmb : nullptr;
  if (small_batch(c, bg)) {
    ALPS_CUDA_TRY(cudaMemsetAsync(cnt, 0, n * sizeof(int), st));
    job.nslots = (int)nslots;
    job.arrive = static_cast<int*>(cnt);
    const int rc = launch_one(c, a, sh, job, st);
    if (rc) return rc;
    c->async_flags = flags;
    return ALPS_OK;
  }
  DispArgs* da = reinterpret_cast<DispArgs*>(b + off[SC_ARGS]);
  DispJob* dj = reinterpret_cast<DispJob*>(b + off[SC_JOB]);
  if (sh.far) {
    // the coefficients belong to this batch's k_par: the context's own tables
    // may serve another batch of it at another k_par meanwhile
    double* f = reinterpret_cast<double*>(b + off[SC_FAR]);
    for (int s = 0; s < S_; ++s) {
      a.sp[s].far = f;
      a.sp[s].farc = f + (size_t)FAR_LEVELS * FAR_K * 12;
      f += far_words(c->spec[s]);
    }
  }
  k_stage<<<1, 128, 0, st>>>(a, job, da, dj);
  ALPS_CUDA_TRY(cudaGetLastError());
  k_classify_multi<<<(unsigned)cls_blocks(n, S_), 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  const long g2 = pole_blocks_all(sh, S_);
  if (sh.far) launch_far(dj, far_groups(maxn), S_, 1, st);
  if (g2 > 0) k_pole_sums_multi<<<(unsigned)g2, 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  const size_t smem = res_smem(c);
  const size_t lsmem = pvl_smem(c->sys.positions_principal);
  const long lblocks = lanes_blocks(bg);
  int rcode0 = res_smem_optin(smem, lblocks ? lsmem : 0);
  if (rcode0) return rcode0;
  if (lblocks) k_resonant_lanes<<<(unsigned)lblocks, RES_WARPS * 32, lsmem, st>>>(dj, 1);
  long blocks = ((long)nslots + RES_WARPS * sh.ipw - 1) / (RES_WARPS * sh.ipw);
  k_resonant_multi<<<(unsigned)blocks, RES_WARPS * 32, smem, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  if (a.relcap) {
    int rcode = launch_rel_orders(a.sys, a.sp, a.relcap, n, om, relb, flags, st);
    if (rcode) return rcode;
  }
  if (a.has_bm) {
    int rcode = launch_nhds(a.sys, a.sp, n, om, bmb, st);
    if (rcode) return rcode;
  }
  k_finalize_multi<<<(unsigned)fin_blocks(sh, n), 128, 0, st>>>(dj, 1);
  ALPS_CUDA_TRY(cudaGetLastError());
  c->async_flags = flags;  // alps_batch_status reads the word before the next call clears it
  return ALPS_OK;
}

// ---------------------------------------------------------------------------
// The autotuner: times the candidate launch shapes of a batch of n omegas
// on this context (at its k and precision path) and keeps the fastest for
// the batch's bucket.  Candidates: j slices per omega 1, 2, 4, 8, 16, 32 x
// pole-sum blocks per SM 2, 4, 8 x resonant warps per SM 6, 12, 24, each
// the best of two timed launches after a warm-up on the context's stream.
// A shape changes only the summation order of the pole sums (slices and
// order chunks), never which terms are summed.
// ---------------------------------------------------------------------------
extern "C" int alps_autotune(alps_ctx* c, int n, const alps_complex* d_om_in, alps_tune_result* out) {
  if (!c || !c->kset || n <= 0 || !out) return ALPS_E_INVALID;
  std::memset(out, 0, sizeof(*out));
  double2* d_D = nullptr;
  double2* d_omb = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = ALPS_OK;
  auto fail = [&](int code) {
    rc = code;
    return code;
  };
  const double2* d_om = reinterpret_cast<const double2*>(d_om_in);
  if (cudaMalloc(&d_D, (size_t)n * sizeof(double2)) != cudaSuccess) return ALPS_E_OOM;
  if (!d_om) {
    // a lattice over Re omega in [0.05, 2.5], Im omega in [-0.4, 0.05]
    const int nr = std::max(1, (int)std::ceil(std::sqrt((double)n)));
    std::vector<double2> h(n);
    for (int i = 0; i < n; ++i) {
      const int ir = i % nr, ii = i / nr;
      h[i] = make_double2(0.05 + 2.45 * (ir + 0.5) / nr, -0.4 + 0.45 * (ii + 0.5) / std::max(1, (n + nr - 1) / nr));
    }
    if (cudaMalloc(&d_omb, (size_t)n * sizeof(double2)) != cudaSuccess) {
      cudaFree(d_D);
      return ALPS_E_OOM;
    }
    if (cudaMemcpy(d_omb, h.data(), (size_t)n * sizeof(double2), cudaMemcpyHostToDevice) != cudaSuccess)
      fail(ALPS_E_CUDA);
    d_om = d_omb;
  }
  if (!rc && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) fail(ALPS_E_CUDA);
  DispArgs a;
  int maxn = 0;
  build_disp_args(c, &a, &maxn);
  // best of two timed launches of one shape (nullptr: the default rule)
  auto time_shape = [&](const TuneShape* sh, float* ms) -> int {
    t_tune_force = sh;
    int st = launch_disp_batch(c, n, d_om, d_D, nullptr, c->stream);
    float best = 3.0e38f;
    for (int r = 0; r < 2 && !st; ++r) {
      if (cudaEventRecord(e0, c->stream) != cudaSuccess) st = ALPS_E_CUDA;
      if (!st) st = launch_disp_batch(c, n, d_om, d_D, nullptr, c->stream);
      if (!st && cudaEventRecord(e1, c->stream) != cudaSuccess) st = ALPS_E_CUDA;
      if (!st && cudaEventSynchronize(e1) != cudaSuccess) st = ALPS_E_CUDA;
      float t = 0.0f;
      if (!st && cudaEventElapsedTime(&t, e0, e1) != cudaSuccess) st = ALPS_E_CUDA;
      if (!st) best = std::min(best, t);
    }
    t_tune_force = nullptr;
    *ms = best;
    return st;
  };
  TuneShape best{};
  float t_def = 0.0f, t_best = 3.0e38f;
  if (!rc) rc = time_shape(nullptr, &t_def);
  if (!rc) {
    t_best = t_def;
    const int jsv[6] = {1, 2, 4, 8, 16, 32}, bpv[3] = {2, 4, 8}, wpv[3] = {6, 12, 24};
    for (int x = 0; x < 6 && !rc; ++x)
      for (int y = 0; y < 3 && !rc; ++y)
        for (int z = 0; z < 3 && !rc; ++z) {
          TuneShape cand;
          cand.js = jsv[x];
          cand.blocks_per_sm = bpv[y];
          cand.warps_per_sm = wpv[z];
          float t = 0.0f;
          rc = time_shape(&cand, &t);
          out->candidates++;
          // a candidate replaces the default only when it is 3 % faster
          if (!rc && t < t_best && t < 0.97f * t_def) {
            t_best = t;
            best = cand;
          }
        }
  }
  if (!rc) {
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      g_tune[tune_key(c, n, maxn)] = best;
    }
    g_tune_epoch++;
    const BatchGeom bg = batch_geom(c, n, c->sys.nspec, maxn, a.rcap, false);
    out->js = bg.sh.js;
    // (the default rule has no fixed number of either: nominal figures)
    out->blocks_per_sm = best.blocks_per_sm ? best.blocks_per_sm : 4;
    out->warps_per_sm = best.warps_per_sm ? best.warps_per_sm : 12;
    out->tuned = best.js != 0;
    out->ms_default = t_def;
    out->ms_best = t_best;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(d_D);
  if (d_omb) cudaFree(d_omb);
  return rc;
}

extern "C" int alps_tune_clear(void) {
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune.clear();
  }
  g_tune_epoch++;
  return ALPS_OK;
}
