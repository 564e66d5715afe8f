// Frequency-integral tables of ComputeTs (ComputeTs.c:517-664) on the device:
// per shell the frequency of unit optical depth (nu_tau_one,
// XRayHeatingFunctions.c:229-375), then for every x_HII node the heating,
// ionisation and Ly-alpha integrals over frequency (integrate_over_nu,
// :672-800).  All in FP64 with the quadrature (QUADPACK QAG, 61 points) and
// the root finder (Brent) of host_physics.cpp, so that the same intervals are
// bisected and the same root is stepped to; build_freq_integrals there is
// the same computation on host threads, for tables whose adaptive intervals
// outgrow FREQ_INTERVALS (FreqDevResult::fail).
//
//   k_tau_lower       a block per shell: the 61 nodes of tau_X(nu) in 61
//                     threads; their redshift factors do not depend on nu and
//                     are kept over the steps of the root finder.
//   k_freq_integrals  a block per (shell, table, x_HII node), the two halves
//                     of a bisected interval in its two pairs of warps.
//
// Shells below unit optical depth at E0 share their lower limit, so their
// integrals are the same numbers: the first of them is computed for all.
//
// On 16 host threads the tables took 8.4 ms per snapshot, longer than the
// shells' transforms of any grid below 512^3.  Here (40 shells, one E0)
// k_tau_lower takes 134 us, 20 steps one after another, and k_freq_integrals
// 297 us, the bisections of the longest integral (30 and more rounds), both bound by
// the FP64 unit's latency (its pipe is 30 to 45% busy on the longest SM).  173 and
// 366 us with one thread keeping the interval list, an FP64 error estimate for every
// tau_X and the species one after another; 360 and 986 us with the cross sections'
// formulas instead of their polynomials.
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "freq_tables.cuh"
#include "gk61.h"

namespace mx {

namespace {
// per host thread: a call counts its own launches when contexts run concurrently
thread_local int freq_launches = 0;

constexpr int TAU_THREADS = 64;
constexpr int INT_THREADS = 128;

// Node and weight of the 61-point rule for thread j < 61 of a panel: 0..29
// below the centre, 30..59 above, 60 the centre (x = 0).
struct Rule
{
  double x, wk, wg;
};

__constant__ Gk61 c_rule = GK61;

__device__ __forceinline__ Rule rule_of(int j)
{
  Rule r{ 0.0, 0.0, 0.0 };
  if (j < 61) {
    const int i = j < 30 ? j : (j < 60 ? j - 30 : 30);
    r.x = j < 30 ? -c_rule.x[i] : (j < 60 ? c_rule.x[i] : 0.0);
    r.wk = c_rule.wk[i];
    r.wg = (i & 1) ? c_rule.wg[i >> 1] : 0.0;  // i = 30 has no Gauss weight
  }
  return r;
}

struct Panel
{
  double result, abserr, resabs, resasc;
};

// The sums of one panel: Kronrod, Gauss, Kronrod of |f|, and Kronrod of
// |f - mean|, two warps' parts each.
struct PanelSums
{
  double part[2][4], asc[2];
};

// Sums of v[0..3] over a warp, sum i in the lanes with (lane & 3) == i: the
// first two exchanges halve the values that a lane carries, so that the four
// sums take six additions (at 16 cycles each per warp) instead of twenty.
__device__ __forceinline__ double warp_sum4(const double (&v)[4])
{
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 2, odd = lane & 1;
  double a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 2);
  b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 2);
  double s = odd ? b : a;
  s += __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
    s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The panel's sums from the integrand values f of its 64 threads (0 in the
// last three), in p; the block calls it for all its panels together.  The
// sums may be read after the next block barrier.
__device__ __forceinline__ void panel_sums(double f, const Rule& w, PanelSums& p)
{
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 1;
  const double s = warp_sum4({ w.wk * f, w.wg * f, w.wk * fabs(f), 0.0 });
  if (lane < 4)
    p.part[warp][lane] = s;
  __syncthreads();
  const double mean = (p.part[0][0] + p.part[1][0]) * 0.5;
  double c = w.wk * fabs(f - mean);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0)
    p.asc[warp] = c;
}

// QUADPACK's error estimate: asc (200 err / asc)^1.5 up to asc, as a product
// with one reciprocal root (a quotient and a root one after the other take twice
// as long).
__device__ double rescale_err(double err, double res_abs, double res_asc)
{
  err = fabs(err);
  if (res_asc != 0 && err != 0) {
    const double x = 200 * err, m = x * res_asc;
    if (!(x < res_asc))
      err = res_asc;
    else if (m > 1e-280)
      err = x * x * rsqrt(m);
    else
      err = x * sqrt(x / res_asc);
  }
  if (res_abs > DBL_MIN / (50 * DBL_EPSILON)) {
    const double min_err = 50 * DBL_EPSILON * res_abs;
    if (min_err > err)
      err = min_err;
  }
  return err;
}

__device__ Panel panel_of(const PanelSums& s, double a, double b)
{
  const double half = 0.5 * (b - a), ahalf = fabs(half);
  const double rk = s.part[0][0] + s.part[1][0], rg = s.part[0][1] + s.part[1][1];
  Panel p;
  p.result = rk * half;
  p.resabs = (s.part[0][2] + s.part[1][2]) * ahalf;
  p.resasc = (s.asc[0] + s.asc[1]) * ahalf;
  p.abserr = rescale_err((rk - rg) * half, p.resabs, p.resasc);
  return p;
}

// One panel of 64 threads whose error is clearly within eps of its result
// (the estimate, taken in floats, a hundredth below the tolerance): *result is
// the Kronrod sum.  false: the panel's sums decide.
struct FastSums
{
  double part[2][2];
  float asc[2], abs[2];
};
__device__ __forceinline__ bool settled(double f, const Rule& w, FastSums& p, double half, double eps, double* result)
{
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 1;
  const bool odd = lane & 1;
  double s = odd ? w.wg * f : w.wk * f;
  s += __shfl_xor_sync(0xffffffffu, odd ? w.wk * f : w.wg * f, 1);
#pragma unroll
  for (int o = 2; o < 32; o <<= 1)
    s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane < 2)
    p.part[warp][lane] = s;
  __syncthreads();
  const double rk = p.part[0][0] + p.part[1][0], rg = p.part[0][1] + p.part[1][1];
  const float wk = (float)w.wk;
  float asc = wk * fabsf((float)(f - rk * 0.5)), abs = wk * fabsf((float)f);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    asc += __shfl_xor_sync(0xffffffffu, asc, o);
    abs += __shfl_xor_sync(0xffffffffu, abs, o);
  }
  if (lane == 0) {
    p.asc[warp] = asc;
    p.abs[warp] = abs;
  }
  __syncthreads();
  *result = rk * half;
  const float h = fabsf((float)half), tol = 0.99f * (float)(eps * fabs(*result));
  asc = (p.asc[0] + p.asc[1]) * h;
  const float least = 1.2e-14f * (p.abs[0] + p.abs[1]) * h;  // 50 epsilon, rounded up
  const float x = 200.0f * fabsf((float)((rk - rg) * half));
  return x < 0.9f * asc && x * sqrtf(x / asc) < tol && least < 0.5f * asc && least < tol && asc > 1e-30f;
}

// Interval list in QUADPACK's order of errors (qpsrt, whole list) and the running
// state of one adaptive integral, kept by warp 0 of the block.
struct Qag
{
  double a[FREQ_INTERVALS], b[FREQ_INTERVALS], r[FREQ_INTERVALS], e[FREQ_INTERVALS];
  int order[FREQ_INTERVALS];
  int size, i, rt1, rt2, more;
  double area, errsum, epsrel, result;
  PanelSums sums[2];

  // The list after interval imax = order[0] became imax (error emax) and n
  // (error emin <= emax): emax goes behind the larger ones, emin before those
  // that are not larger than it.  Errors are not negative: as integers they
  // compare in the same order.  All lanes of a warp.
  __device__ void sort_errors(int imax, int n, double emax, double emin)
  {
    const int lane = threadIdx.x & 31;
    const long long hi = __double_as_longlong(emax), lo = __double_as_longlong(emin);
    int idx[FREQ_INTERVALS / 32], to[FREQ_INTERVALS / 32], larger = 0, between = 0;
#pragma unroll
    for (int c = 0; c < FREQ_INTERVALS / 32; c++) {
      to[c] = -1;
      if (32 * c < n - 1) {
        const int t = 32 * c + lane;
        const bool in = t < n - 1;
        idx[c] = in ? order[t + 1] : 0;
        const long long x = __double_as_longlong(e[idx[c]]);
        larger += __popc(__ballot_sync(0xffffffffu, in && x > hi));
        between += __popc(__ballot_sync(0xffffffffu, in && x <= hi && x > lo));
        if (in)
          to[c] = x > hi ? t : t + 1 + (lo >= x);
      }
    }
    __syncwarp();
    const bool tie = n >= 2 && lo >= hi;
#pragma unroll
    for (int c = 0; c < FREQ_INTERVALS / 32; c++)
      if (to[c] >= 0)
        order[to[c]] = idx[c];
    if (lane == 0) {
      order[larger + tie] = imax;
      order[tie ? larger : larger + 1 + between] = n;
      i = larger ? idx[0] : (tie ? n : imax);
    }
  }

  // after the first panel (its sums in sums[0]); more: bisect on.  Warp 0.
  __device__ void begin(double lo, double hi, double eps)
  {
    const Panel p = panel_of(sums[0], lo, hi);
    if ((threadIdx.x & 31) == 0) {
      const double tol = eps * fabs(p.result);
      epsrel = eps;
      result = p.result;
      more = 1;
      const double round_off = 50 * DBL_EPSILON * p.resabs;
      if ((p.abserr <= round_off && p.abserr > tol) || (p.abserr <= tol && p.abserr != p.resasc) || p.abserr == 0.0)
        more = 0;
      a[0] = lo;
      b[0] = hi;
      r[0] = p.result;
      e[0] = p.abserr;
      order[0] = 0;
      size = 1;
      i = rt1 = rt2 = 0;
      area = p.result;
      errsum = p.abserr;
    }
  }

  // the two halves of interval i, their sums in sums[0] and sums[1].  Warp 0:
  // its even lanes estimate the error of the one and its odd lanes of the other.
  __device__ void step(double ai, double b1, double bi, int limit, int* fail)
  {
    const int lane = threadIdx.x & 31, odd = lane & 1;
    const Panel p = panel_of(sums[odd], odd ? b1 : ai, odd ? bi : b1);
    auto of = [](double v, int l) { return __shfl_sync(0xffffffffu, v, l); };
    const double r1 = of(p.result, 0), r2 = of(p.result, 1), e1 = of(p.abserr, 0), e2 = of(p.abserr, 1);
    const unsigned limited = __ballot_sync(0xffffffffu, p.resasc == p.abserr) & 3u;
    const int im = i, n = size;
    const double ri = r[im], ei = e[im], area12 = r1 + r2, err12 = e1 + e2;
    const double sum = errsum + (err12 - ei), whole = area + (area12 - ri);
    int t1 = rt1, t2 = rt2;
    if (!limited) {
      if (fabs(ri - area12) <= 1.0e-5 * fabs(area12) && err12 >= 0.99 * ei)
        t1++;
      if (n >= 10 && err12 > ei)
        t2++;
    }
    bool on = sum > epsrel * fabs(whole);
    if (on) {
      const double tmp = (1 + 100 * DBL_EPSILON) * (fabs(b1) + 1000 * DBL_MIN);
      if (t1 >= 6 || t2 >= 20 || (fabs(ai) <= tmp && fabs(bi) <= tmp))
        on = false;
    }
    if (on && n + 1 >= limit) {
      if (lane == 0)
        *fail = 1;
      on = false;
    }
    const bool swap = e2 > e1;
    __syncwarp();  // every lane has read the state
    if (lane == 0) {
      errsum = sum;
      area = whole;
      rt1 = t1;
      rt2 = t2;
      size = n + 1;
      more = on;
      a[im] = swap ? b1 : ai;
      b[im] = swap ? bi : b1;
      r[im] = swap ? r2 : r1;
      e[im] = swap ? e2 : e1;
      a[n] = swap ? ai : b1;
      b[n] = swap ? b1 : bi;
      r[n] = swap ? r1 : r2;
      e[n] = swap ? e1 : e2;
    }
    if (on) {
      sort_errors(im, n, swap ? e2 : e1, swap ? e1 : e2);
    } else if (lane == 0) {
      double s = 0;
      for (int q = 0; q <= n; q++)
        s += r[q];
      result = s;
    }
  }
};

// ---------------------------------------------------------- cross sections
// The formulas (XRayHeatingFunctions.c:823-900; eps = sqrt(nu / nu0 - 1)), for
// frequencies near and below a threshold.
__device__ double xs_hydrogenic(double nu, double nu0, double sigma)
{
  if (nu < nu0)
    return 0;
  if (nu == nu0)
    nu += k::TINY;
  const double q = nu0 / nu, q2 = q * q;
  const double eps = sqrt(nu / nu0 - 1), ieps = 1.0 / eps;
  return sigma * (q2 * q2) * exp(4 - (4 * atan(eps) * ieps)) / (1 - exp(-2 * k::PI * ieps));
}
__device__ __noinline__ double xs_formula(int q, double nu)
{
  if (q != 1)
    return q == 0 ? xs_hydrogenic(nu, k::NU_HI, k::SIGMA_HI) : xs_hydrogenic(nu, k::NU_HEII, 6.3e-18 / 4);
  if (nu < k::NU_HEI)
    return 0;
  const double x = nu * (1.0 / k::NU_OVER_EV / 13.61) - 0.4434;
  const double y = sqrt(x * x + 2.136 * 2.136);
  // y^(0.5 * 3.188 - 5.5) (1 + sqrt(y / 1.469))^-3.188
  return 9.492e-16 * ((x - 1) * (x - 1) + 2.039 * 2.039) *
         exp((0.5 * 3.188 - 5.5) * log(y) - 3.188 * log(1.0 + sqrt(y * (1.0 / 1.469))));
}

// Interval and local coordinate of nu in the polynomial tables.  The tables
// agree with the formulas to 4e-16 of the value, at 9 multiply-adds instead
// of roots, exponentials, logarithms and an arctangent (several hundred
// operations at the FP64 rate).
struct XsAt
{
  int i;
  double t;
};
__device__ __forceinline__ XsAt xs_at(double nu)
{
  const double x = nu * (1.0 / k::NU_HI);
  const int hi = __double2hiint(x);
  const int sub = (hi >> 16) & (XS_SUB - 1);  // leading mantissa bits
  XsAt p;
  p.i = ((hi >> 20) - 1023) * XS_SUB + sub;  // x > 0: the sign bit is clear
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
  p.t = (m - (1.0 + (sub + 0.5) / XS_SUB)) * (2.0 * XS_SUB);
  return p;
}
// first interval at or above 1.5 thresholds: x = 1.5, 2.7122 (2.75), 6
__device__ __forceinline__ bool xs_in_table(int q, int i)
{
  return i >= (q == 0 ? XS_SUB / 2 : (q == 1 ? XS_SUB + 3 * XS_SUB / 8 : 2 * XS_SUB + XS_SUB / 2)) && i < XS_INTERVALS;
}
// The three species' values at p from tab, or formula(q) below their tables.
// Above 6 NU_HI all three are polynomials, evaluated side by side in pairs of
// terms: the FP64 unit's latency, not its rate, bounds a chain of nine.
template <class F>
__device__ __forceinline__ void xs_values(const double (&tab)[3][XS_INTERVALS][XS_N], const XsAt& p, double (&s)[3],
                                          const F& formula)
{
  static_assert(XS_N == 10);
  const double t2 = p.t * p.t, t4 = t2 * t2, t8 = t4 * t4;
  auto poly = [&](int q) {
    const double2* c = reinterpret_cast<const double2*>(tab[q][p.i]);
    double v[5];
#pragma unroll
    for (int j = 0; j < 5; j++) {
      const double2 u = __ldg(c + j);
      v[j] = fma(u.y, p.t, u.x);
    }
    return fma(v[4], t8, fma(fma(v[3], t2, v[2]), t4, fma(v[1], t2, v[0])));
  };
  if (xs_in_table(2, p.i)) {
#pragma unroll
    for (int q = 0; q < 3; q++)
      s[q] = poly(q);
  } else {
#pragma unroll 1
    for (int q = 0; q < 3; q++) {
      const double v = xs_in_table(q, p.i) ? poly(q) : formula(q);
      s[0] = q == 0 ? v : s[0];
      s[1] = q == 1 ? v : s[1];
      s[2] = q == 2 ? v : s[2];
    }
  }
}

// ---------------------------------------------------------- optical depth
// dtdz (XRayHeatingFunctions.c:377-392) times C n HI at redshift zhat
__device__ double tau_factor(const FreqArgs& a, double zhat, double fcoll1, double x_e_ave)
{
  const double opz = (double)(1 + (float)zhat);
  const double s = sqrt(a.ol / a.om), ir = 1.0 / (opz * sqrt(opz));
  const double x = s * ir, dxdz = s * (ir / opz) * (-3.0 / 2.0);
  const double root = sqrt(x * x + 1);
  const double const1 = 2 * sqrt(1 + a.om / a.ol) / (3.0 * k::HUBBLE * a.hubble_h);
  const double dtdz = const1 * (dxdz * (1 + x / root)) / (x + root);
  const double o = 1 + zhat;
  const double n = a.n_b0 * (o * o * o);
  double fc = fcoll1;
  if (!a.first_snapshot)
    fc = a.fcoll0 + (zhat - a.z0) * (fcoll1 - a.fcoll0) / (a.z1 - a.z0);
  if (fc < 0.0)
    fc = 0.0;
  double HI = fc < 1e-20 ? 1 : 1 - (a.eff * fc) / (1.0 - x_e_ave);
  if (HI < 1e-4)
    HI = 1e-4;
  return k::C * dtdz * n * HI;
}

__global__ void __launch_bounds__(TAU_THREADS) k_tau_lower(const __grid_constant__ FreqArgs a)
{
  __shared__ Qag q;
  __shared__ FastSums fast;
  const int r = blockIdx.x, j = threadIdx.x;
  const double x_e = a.sums[1] / a.total, fcoll1 = a.sums[0] / a.total;
  if (x_e > 0.9999) {
    if (j == 0)
      a.out->nu1[r] = -1.0;
    return;
  }
  const Rule w = rule_of(j);
  const double zpp = a.zpp[r], zp = a.zp;
  const double z0 = 0.5 * (zpp + zp) + 0.5 * (zp - zpp) * w.x;
  const double factor0 = j < 61 ? tau_factor(a, z0, fcoll1, x_e) : 0.0;
  const double share[3] = { a.f_h * (1 - x_e), a.f_he * (1 - x_e), a.f_he * x_e };
  // tau_X(nu): the integral from zpp to zp
  auto tau = [&](double nu) {
    const double nu0 = nu / (1 + zp);
    auto value = [&](double zhat, double factor) {
      if (j >= 61)
        return 0.0;
      const double nuhat = nu0 * (1 + zhat);
      double xs[3];
      xs_values(a.tables->xs, xs_at(nuhat), xs, [&](int q) { return xs_formula(q, nuhat); });
      return factor * fma(share[2], xs[2], fma(share[1], xs[1], share[0] * xs[0]));
    };
    const double f = value(z0, factor0);
    double first;
    if (settled(f, w, fast, 0.5 * (zp - zpp), 0.005, &first))
      return first;
    panel_sums(f, w, q.sums[0]);
    __syncthreads();
    if (j < 32)
      q.begin(zpp, zp, 0.005);
    __syncthreads();
    while (q.more) {
      const double lo = q.a[q.i], hi = q.b[q.i], mid = 0.5 * (lo + hi);
#pragma unroll 1
      for (int h = 0; h < 2; h++) {
        const double pa = h ? mid : lo, pb = h ? hi : mid;
        const double z = 0.5 * (pa + pb) + 0.5 * (pb - pa) * w.x;
        panel_sums(value(z, tau_factor(a, z, fcoll1, x_e)), w, q.sums[h]);
      }
      __syncthreads();
      if (j < 32)
        q.step(lo, mid, hi, a.intervals, &a.out->fail);
      __syncthreads();
    }
    return q.result;
  };
  // nu_tau_one: every thread steps the same bracket (the same sums in each)
  double root = k::NU_HEI;
  const double f_lo = tau(k::NU_HEI);
  if (!(f_lo < 1)) {
    double xa = k::NU_HEI, xb = 1e6 * k::NU_OVER_EV, fa = f_lo - 1, fb = tau(xb) - 1;
    double xc = xb, fc = fb, d = xb - xa, e = d, xl = xa, xu = xb;
    root = 0.5 * (xa + xb);
    for (int iter = 1; iter <= 100; iter++) {
      bool two_points = false;
      if ((fb < 0 && fc < 0) || (fb > 0 && fc > 0)) {
        two_points = true;
        xc = xa;
        fc = fa;
        d = e = xb - xa;
      }
      if (fabs(fc) < fabs(fb)) {
        two_points = true;
        xa = xb;
        xb = xc;
        xc = xa;
        fa = fb;
        fb = fc;
        fc = fa;
      }
      const double tol = 0.5 * DBL_EPSILON * fabs(xb), m = 0.5 * (xc - xb);
      if (fb == 0) {
        root = xl = xu = xb;
        break;
      }
      if (fabs(m) <= tol) {
        root = xb;
        break;
      }
      if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
        d = e = m;
      } else {
        const double s = fb / fa;
        double pp, qq;
        if (two_points) {
          pp = 2 * m * s;
          qq = 1 - s;
        } else {
          const double t = fa / fc, rr = fb / fc;
          pp = s * (2 * m * t * (t - rr) - (xb - xa) * (rr - 1));
          qq = (t - 1) * (rr - 1) * (s - 1);
        }
        if (pp > 0)
          qq = -qq;
        else
          pp = -pp;
        if (2 * pp < fmin(3 * m * qq - fabs(tol * qq), fabs(e * qq))) {
          e = d;
          d = pp / qq;
        } else {
          d = e = m;
        }
      }
      xa = xb;
      fa = fb;
      xb += fabs(d) > tol ? d : (m > 0 ? tol : -tol);
      fb = tau(xb) - 1;
      root = xb;
      double other = xc;
      if ((fb < 0 && fc < 0) || (fb > 0 && fc > 0))
        other = xa;
      xl = fmin(xb, other);
      xu = fmax(xb, other);
      const double min_abs = (xl > 0 && xu > 0) || (xl < 0 && xu < 0) ? fmin(fabs(xl), fabs(xu)) : 0.0;
      if (fabs(xu - xl) < 0.02 * min_abs)
        break;
    }
  }
  if (j == 0)
    a.out->nu1[r] = root;
}

// ----------------------------------------------------- frequency integrals
// interp_tab (XRayHeatingFunctions.c:914-1190): the energy's bin and the float
// interpolation in it, then (at the last x_HII node only, which is looked up
// just below itself) between two x_HII rows.
struct EnergyBin
{
  int n;
  float dE;
  bool below;  // below the table
};
// The bins of the three species' energies: a guess from the logarithm, one step
// off at most where the table's steps round, and then the exact edges.
__device__ __forceinline__ void energy_bins(const FreqDevTables& t, float (&En)[3], EnergyBin (&b)[3])
{
  float4 at[3];
  bool off = false;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    if (En[q] > t.energy_cap)
      En[q] = t.energy_top;
    b[q].below = En[q] < t.bin[0].z;
    const bool fine = En[q] < 1008.88f;
    const float l = logf(En[q] * (fine ? 0.1f : (float)(1 / 1008.88)));
    const int n = fine ? (int)(l * (float)(1 / 1.98026273e-2)) : 232 + (int)(l * (float)(1 / 9.53101798e-2));
    b[q].n = min(max(n, 0), k::NENERGY - 2);
    at[q] = __ldg(&t.bin[b[q].n]);
    off |= (b[q].n > 0 && En[q] < at[q].x) || (b[q].n < k::NENERGY - 2 && En[q] >= at[q].y);
  }
  if (off) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      int n = b[q].n;
      while (n > 0 && En[q] < t.bin[n].x)
        n--;
      while (n < k::NENERGY - 2 && En[q] >= t.bin[n].y)
        n++;
      b[q].n = n;
      at[q] = t.bin[n];
    }
  }
#pragma unroll
  for (int q = 0; q < 3; q++)
    b[q].dE = En[q] - at[q].z;
}
__device__ __forceinline__ float in_energy(const float2* row, const EnergyBin& b)
{
  const float2 v = __ldg(row + b.n);
  return fmaf(v.y, b.dE, v.x);
}
__device__ __forceinline__ float interp(const FreqDevTables& t, const float2 (*tab)[k::NENERGY], float below,
                                        const EnergyBin& b, int xi)
{
  float v;
  if (xi < k::NXHII - 1) {
    v = in_energy(tab[xi], b);
  } else {
    const int m0 = k::NXHII - 2;
    const float x = (float)(t.xhii[k::NXHII - 1] * 0.999);
    const float lo = in_energy(tab[m0], b), hi = in_energy(tab[m0 + 1], b);
    v = (hi - lo) / (t.xhii[m0 + 1] - t.xhii[m0]);
    v *= x - t.xhii[m0];
    v += lo;
  }
  return b.below ? below : v;
}

__device__ __forceinline__ double integrand(const FreqArgs& a, double nu, int flag, int xi, double spec)
{
  const FreqDevTables& t = *a.tables;
  const double xe = t.xhii[xi];
  const double nus[3] = { k::NU_HI, k::NU_HEI, k::NU_HEII };
  const double share[3] = { a.f_h * (1 - xe), a.f_he * (1 - xe), a.f_he * xe };
  const double eV = nu * (1.0 / k::NU_OVER_EV);
  float En[3];
#pragma unroll
  for (int q = 0; q < 3; q++)
    En[q] = (float)(eV - nus[q] / k::NU_OVER_EV);
  EnergyBin b[3];
  energy_bins(t, En, b);
  double c[3], xs[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    if (flag == 0)
      c[q] = (double)interp(t, t.fheat, 1.0f, b[q], xi) * (nu - nus[q]);
    else if (flag == 1)
      c[q] = (double)(interp(t, t.nion[0], 0.0f, b[q], xi) + interp(t, t.nion[1], 0.0f, b[q], xi) +
                      interp(t, t.nion[2], 0.0f, b[q], xi) + 1);
    else
      c[q] = (double)interp(t, t.nlya, 0.0f, b[q], xi);
    c[q] *= share[q];
  }
  xs_values(t.xs_spec, xs_at(nu), xs,
            [&](int q) { return xs_formula(q, nu) * exp((-a.alpha - 1) * log(nu * (1.0 / k::NU_HI))); });
  return fma(c[2], xs[2], fma(c[1], xs[1], c[0] * xs[0])) * spec;
}

__global__ void __launch_bounds__(INT_THREADS) k_freq_integrals(const __grid_constant__ FreqArgs a)
{
  __shared__ Qag q;
  // the Ly-alpha tables of the most ionised nodes bisect longest: first
  int blk = blockIdx.x;
  const int r = blk % a.S;
  blk /= a.S;
  const int set = blk % a.n_sets;
  blk /= a.n_sets;
  const int xi = k::NXHII - 1 - blk % k::NXHII, flag = 2 - blk / k::NXHII;
  const double E0nu = a.E0[set] * k::NU_OVER_EV;
  // shells whose lower limit is E0 share their integrals: the first computes
  const bool at_E0 = !(a.out->nu1[r] > E0nu);
  if (at_E0)
    for (int o = 0; o < r; o++)
      if (!(a.out->nu1[o] > E0nu))
        return;
  const double lower = at_E0 ? E0nu : a.out->nu1[r];
  const int j = threadIdx.x & 63, h = threadIdx.x >> 6;
  const Rule w = rule_of(j);
  // the factors that do not depend on nu or the species
  const double spec = a.spec[set] * (flag == 0 ? k::PLANCK : 1.0);
  auto sums = [&](double pa, double pb) {
    const double f = j < 61 ? integrand(a, 0.5 * (pa + pb) + 0.5 * (pb - pa) * w.x, flag, xi, spec) : 0.0;
    panel_sums(f, w, q.sums[h]);
    __syncthreads();
  };
  sums(lower, a.numax);
  if (threadIdx.x < 32)
    q.begin(lower, a.numax, 0.01);
  __syncthreads();
  while (q.more) {
    const double lo = q.a[q.i], hi = q.b[q.i], mid = 0.5 * (lo + hi);
    sums(h ? mid : lo, h ? hi : mid);
    if (threadIdx.x < 32)
      q.step(lo, mid, hi, a.intervals, &a.out->fail);
    __syncthreads();
  }
  if (threadIdx.x < a.S) {
    const int o = threadIdx.x;
    double res = q.result;
    if (flag == 2)
      res = res * k::C / (4 * k::PI) / k::LYA_HZ / a.hubble;
    if (o == r || (at_E0 && !(a.out->nu1[o] > E0nu)))
      a.out->tab[set][(flag * k::NXHII + xi) * a.S + o] = res;
  }
}
}  // namespace

// Interpolation at the Chebyshev nodes of each interval, as powers of the local
// coordinate.
static void fill_xs(double alpha, FreqDevTables* t)
{
  double (*xs[3])(double) = { xs_HI, xs_HeI, xs_HeII };
  double node[XS_N], dct[XS_N][XS_N], cheb[XS_N][XS_N] = {};  // cheb[j]: powers of T_j
  for (int n = 0; n < XS_N; n++) {
    node[n] = std::cos(k::PI * (n + 0.5) / XS_N);
    for (int j = 0; j < XS_N; j++)
      dct[j][n] = std::cos(k::PI * j * (n + 0.5) / XS_N) * (j ? 2.0 : 1.0) / XS_N;
  }
  cheb[0][0] = cheb[1][1] = 1.0;
  for (int j = 2; j < XS_N; j++)
    for (int m = 0; m < XS_N; m++)
      cheb[j][m] = (m ? 2.0 * cheb[j - 1][m - 1] : 0.0) - cheb[j - 2][m];
  for (int i = 0; i < XS_INTERVALS; i++)
    for (int q = 0; q < 3; q++) {
      double v[2][XS_N];
      for (int n = 0; n < XS_N; n++) {
        const double x = std::ldexp(1.0 + (i % XS_SUB + 0.5 + 0.5 * node[n]) / XS_SUB, i / XS_SUB);
        v[0][n] = xs[q](x * k::NU_HI);
        v[1][n] = v[0][n] * std::pow(x, -alpha - 1);
      }
      double (*out[2])[XS_N] = { &t->xs[q][i], &t->xs_spec[q][i] };
      for (int w = 0; w < 2; w++) {
        for (int m = 0; m < XS_N; m++)
          (*out[w])[m] = 0.0;
        for (int j = 0; j < XS_N; j++) {
          double c = 0.0;
          for (int n = 0; n < XS_N; n++)
            c += v[w][n] * dct[j][n];
          for (int m = 0; m <= j; m++)
            (*out[w])[m] += c * cheb[j][m];
        }
      }
    }
}

void fill_freq_dev_tables(const HeatTables& ht, double alpha, FreqDevTables* t)
{
  fill_xs(alpha, t);
  std::memcpy(t->xhii, ht.xhii, sizeof(t->xhii));
  // a value and the slope to the next one, as interp_tab forms it
  auto rows = [&](const float (&v)[k::NXHII][k::NENERGY], float2 (&out)[k::NXHII][k::NENERGY]) {
    for (int x = 0; x < k::NXHII; x++)
      for (int n = 0; n < k::NENERGY; n++) {
        out[x][n].x = v[x][n];
        out[x][n].y = n + 1 < k::NENERGY ? (v[x][n + 1] - v[x][n]) / (ht.energy[n + 1] - ht.energy[n]) : 0.0f;
      }
  };
  rows(ht.fheat, t->fheat);
  rows(ht.nlya, t->nlya);
  rows(ht.nion_hi, t->nion[0]);
  rows(ht.nion_hei, t->nion[1]);
  rows(ht.nion_heii, t->nion[2]);
  // the last energy's 0.999 as interp_tab compares (in double) and takes it:
  // the largest float not above it, and its float
  const double cap = 0.999 * ht.energy[k::NENERGY - 1];
  t->energy_top = (float)(ht.energy[k::NENERGY - 1] * 0.999);
  t->energy_cap = (double)(float)cap > cap ? std::nextafter((float)cap, 0.0f) : (float)cap;
  // loc_energy does not decrease with the energy: bisect the float at which
  // it reaches n
  const float top = ht.energy[k::NENERGY - 1];
  std::vector<float> edge(k::NENERGY + 1, 0.0f);
  for (int n = 1; n <= k::NENERGY; n++) {
    if (loc_energy(top) < n) {
      edge[n] = INFINITY;
      continue;
    }
    float lo = ht.energy[0], hi = top;
    if (loc_energy(lo) >= n)
      hi = lo;
    while (std::nextafter(lo, hi) < hi) {
      const float mid = lo + 0.5f * (hi - lo);
      (loc_energy(mid) >= n ? hi : lo) = mid;
    }
    edge[n] = hi;
  }
  for (int n = 0; n < k::NENERGY; n++)
    t->bin[n] = make_float4(edge[n], edge[n + 1], ht.energy[n], 0.0f);
}

FreqArgs make_freq_args(const mx_params& p, const Derived& d, const std::vector<double>& zz, const double* stored_fcoll,
                        int snapshot, const ShellPlan& sp)
{
  FreqArgs a{};
  a.S = sp.S;

  a.zp = zz[snapshot];
  for (int r = 0; r < sp.S; r++)
    a.zpp[r] = shell_redshift(sp, a.zp, r);
  a.alpha = p.spec_index_xray_gal;
  a.numax = p.nu_xray_max * k::NU_OVER_EV;
  a.hubble = hubble(p, (float)a.zp);
  a.om = p.omega_m;
  a.ol = p.omega_lambda;
  a.hubble_h = p.hubble_h;
  a.n_b0 = d.n_b0;
  a.f_h = d.f_h;
  a.f_he = d.f_he;
  a.eff = p.reion_efficiency;
  a.first_snapshot = snapshot == 0;
  if (snapshot > 0) {
    a.fcoll0 = stored_fcoll[snapshot - 1];
    a.z0 = zz[snapshot - 1];
  }
  a.z1 = a.zp;
  return a;
}

void launch_freq_tables(const FreqArgs& a, cudaStream_t s)
{
  cudaMemsetAsync(&a.out->fail, 0, sizeof(int), s);
  k_tau_lower<<<a.S, TAU_THREADS, 0, s>>>(a);
  k_freq_integrals<<<a.S * a.n_sets * FREQ_TAB, INT_THREADS, 0, s>>>(a);
  freq_launches += 2;
}

int freq_kernel_launches() { return freq_launches; }

}  // namespace mx
