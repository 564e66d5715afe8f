// Peculiar-velocity corrections of the 21 cm brightness temperature
// (BrightnessTemperature.c:158-509, velocity_gradient reionization.c:2172-2187),
// used when the spin temperature is on and Flag_IncludePecVelsFor21cm is 1-3:
//
//   k_vel_convert    velocity units in place (trees convention, to comoving
//                    Mpc/s), rounded to float after each factor like the
//                    reference;
//   (cuFFT R2C of vel, in mx_reion.cu)
//   k_vel_grad_k     1/N and h scale, times i k_z (k from BoxSize in Mpc/h);
//   (cuFFT C2R in place: dv/dx on the padded layout)
//   k_pecvel_cells   mode 1: divide by (dv/dx / H + 1) with |dv/dx| capped at
//                    0.2 H; modes 2-3: optical-depth form
//                    (1 - exp(-tau / |dv/dx / H + 1|)) 1000 (T_S - T_CMB) / (1+z);
//   k_rsd_columns    mode 3: the line-of-sight remap along z of the reference's
//                    50 sub-cells per cell, a thread per cell (fixed point,
//                    order-independent deposits).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "pecvel.cuh"

namespace mx {

namespace {
// per host thread: a call counts its own launches when contexts run concurrently
thread_local int pv_launches = 0;
constexpr double FRACT_FLOAT_ERR_D = 1e-7;
constexpr double MPC_CM = 3.086e24;

// Products of a float with double factors one after another, each rounded to float.
// A factor is held as two floats and a power of two, c = (hi + lo) 2^e with hi in
// [1/2, 1]: the product is one rounding of the exact x hi + x lo but for the last place
// of x lo, so it equals (float)(c * (double)x) unless that lies within 2^-48 of a tie.
// That holds while x lo and the products are normal floats (the powers of two wait for
// the end): for `least` <= |x| <= `most` on the way in (1e-19 to 1e37 km/s for the
// units, from 1e-29 for the gradient).  Zeros are kept, and what lies outside
// (infinities and NaN too) takes the products in FP64, out of line.  Two FP32 operations
// a factor instead of two conversions and a product at the FP64 rate (the FP64 form took
// 0.50 ms in k_vel_convert and, with its quotient, 0.41 ms in k_vel_grad_k at 256^3, this
// one 79 and 31 us).
template <int N>
struct Scales
{
  float hi[N], lo[N], pow2, least = 0.0f, most = FLT_MAX;
  double c[N];

  __host__ explicit Scales(const double (&factors)[N])
  {
    double product = 1.0, mantissas = 1.0;
    int exponents = 0;
    for (int i = 0; i < N; i++) {
      int e;
      const double m = std::frexp(factors[i], &e);
      c[i] = factors[i];
      hi[i] = (float)m;
      lo[i] = (float)(m - (double)hi[i]);
      product *= c[i];
      mantissas *= m;
      exponents += e;
      // lo is 2^-26 of hi or nothing, and every product is within the floats
      least = std::max({ least, (float)(0x1p-99 / mantissas), (float)(0x1p-125 / product) });
      most = std::min(most, (float)std::min(0x1p127 / product, (double)FLT_MAX));
    }
    pow2 = std::ldexp(1.0f, exponents);
  }
  __device__ __forceinline__ bool takes(float x) const
  {
    const float a = fabsf(x);
    return (a >= least && a <= most) || x == 0.0f;
  }
  __device__ __forceinline__ float operator()(float x) const
  {
#pragma unroll
    for (int i = 0; i < N; i++)
      x = __fmaf_rn(x, hi[i], __fmul_rn(x, lo[i]));
    return __fmul_rn(x, pow2);
  }
};
template <int N>
__device__ __noinline__ float scales_fp64(const Scales<N>& s, float x)
{
  for (int i = 0; i < N; i++)
    x = (float)(s.c[i] * (double)x);
  return x;
}

// the unit factors in the reference's order
template <int NF>
__global__ void k_vel_convert(float* vel, const __grid_constant__ Scales<NF> units, int D, int H, long long N)
{
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    const long long ip = row * 2LL * H + (ir - row * D);
    const float v = vel[ip];
    vel[ip] = units.takes(v) ? units(v) : scales_fp64(units, v);
  }
}

// c /= N; c *= h (each rounded to float); c *= (0 + i k_z) as a float complex
// product
__global__ void k_vel_grad_k(float2* spec, int H, long long C, const __grid_constant__ Scales<2> scales, float delta_k)
{
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < C; i += (long long)gridDim.x * blockDim.x) {
    float2 v = spec[i];
    if (scales.takes(v.x) && scales.takes(v.y))
      v = make_float2(scales(v.x), scales(v.y));
    else
      v = make_float2(scales_fp64(scales, v.x), scales_fp64(scales, v.y));
    const int nz = (int)(i % H);
    const float kz = __fmul_rn((float)nz, delta_k);
    // (a + i b)(0 + i k): real a*0 - b*k, imaginary a*k + b*0
    const float re = __fsub_rn(__fmul_rn(v.x, 0.0f), __fmul_rn(v.y, kz));
    const float im = __fadd_rn(__fmul_rn(v.x, kz), __fmul_rn(v.y, 0.0f));
    spec[i] = make_float2(re, im);
  }
}

// An unevaluated sum of two floats, |lo| at most half an ulp of hi: about 2^-44
// of the value, on the FP32 pipe (64 times the FP64 rate).
struct Pair
{
  float hi, lo;
};
__device__ __forceinline__ Pair fast_two_sum(float a, float b)  // |a| >= |b|
{
  const float s = __fadd_rn(a, b);
  return { s, __fsub_rn(b, __fsub_rn(s, a)) };
}
__device__ __forceinline__ Pair two_sum(float a, float b)
{
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return { s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t)) };
}
__device__ __forceinline__ Pair mul(Pair a, Pair b)
{
  const float p = __fmul_rn(a.hi, b.hi);
  const float e = __fmaf_rn(a.hi, b.hi, -p) + (__fmul_rn(a.hi, b.lo) + __fmul_rn(a.lo, b.hi));
  return fast_two_sum(p, e);
}
// a / b for a float a
__device__ __forceinline__ Pair div(float a, Pair b)
{
  const float r = __fdividef(1.0f, b.hi), q = __fmul_rn(a, r);
  const float rest = __fmaf_rn(-q, b.hi, a) - __fmul_rn(q, b.lo);
  return fast_two_sum(q, __fmul_rn(rest, r));
}

// x (1 - x/2 + x^2/6 - ...) = 1 - exp(-x) for |x| < 1/8: 1 - x/2 in pairs, the
// rest (below 2^-8.6, the last term left out below 2^-36) in float, whose rounding
// is the result's error: 2^-32.6 at x = 1/8, 2^-37 at 0.03
constexpr float SMALL_TAU = 0.125f;
__device__ __forceinline__ Pair one_minus_exp_small(Pair x)
{
  float s = 1.0f / 40320.0f;
  s = fmaf(-s, x.hi, 1.0f / 5040.0f);
  s = fmaf(-s, x.hi, 1.0f / 720.0f);
  s = fmaf(-s, x.hi, 1.0f / 120.0f);
  s = fmaf(-s, x.hi, 1.0f / 24.0f);
  s = fmaf(-s, x.hi, 1.0f / 6.0f);
  const Pair p = fast_two_sum(1.0f, -0.5f * x.hi);
  return mul(x, fast_two_sum(p.hi, p.lo + fmaf(s * x.hi, x.hi, -0.5f * x.lo)));
}

// The cells of BrightnessTemperature.c:219-320.  The reference works in FP64;
// here pairs of floats carry the same sums to eight bits and more beyond the float
// result (one_minus_exp_small), and cells outside their range (a gradient near -H,
// optical depths of 1/8 and more, values beyond 1e15, infinities, NaN) take the FP64
// form.  The error against 64 bits is that of the FP64 form in modes 1 and 2 (96
// boxes of 24^3 to 256^3: the same maximum, rms and quantiles).  In
// FP64 throughout, its issue rate bound the pass: 1.97 ms at 256^3 with the
// reference's quotients, 1.31 ms with one.
__device__ __noinline__ float pecvel_cell_fp64(const PecvelArgs& a, float dT, float grad, float TS)
{
  const double g = (double)grad;
  if (a.mode == 1) {
    double dvdx = g;
    if (fabs(dvdx) > a.max_v_deriv)
      dvdx = dvdx < 0 ? -a.max_v_deriv : a.max_v_deriv;
    return (float)((double)dT / (dvdx * a.inv_H + 1.0));
  }
  const double gc = fabs(g * a.inv_H + 1.0);
  const double scale = ((double)TS - a.T_rad) * a.mK;
  if (gc < FRACT_FLOAT_ERR_D)
    return (float)scale;
  return (float)((1. - exp(-(double)dT / gc)) * scale);
}

__global__ void k_pecvel_cells(PecvelArgs a, int D, int H, long long N)
{
  // 1/H is 1e17 s and more: powers of two keep the pairs' products in range
  const Pair invH = { (float)(a.inv_H * 0x1p-60), (float)(a.inv_H * 0x1p-60 - (double)(float)(a.inv_H * 0x1p-60)) };
  const Pair T_rad = { (float)a.T_rad, (float)(a.T_rad - (double)(float)a.T_rad) };
  const Pair mK = { (float)a.mK, (float)(a.mK - (double)(float)a.mK) };
  const float cap = (float)(a.max_v_deriv * 0x1p60);
  // 1 + dv/dx / H at the caps
  const double up = 1.0 + a.max_v_deriv * a.inv_H, down = 1.0 - a.max_v_deriv * a.inv_H;
  const Pair cap_up = { (float)up, (float)(up - (double)(float)up) };
  const Pair cap_down = { (float)down, (float)(down - (double)(float)down) };
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    const float grad = a.grad[row * 2LL * H + (ir - row * D)], dT = a.delta_T[ir];
    const float TS = a.mode == 1 ? 0.0f : a.TS[ir];
    const float g = grad * 0x1p60f;
    // 1 + dv/dx / H
    const float q = __fmul_rn(g, invH.hi);
    const Pair t = two_sum(1.0f, q);
    const Pair one_g = fast_two_sum(t.hi, t.lo + (__fmaf_rn(g, invH.hi, -q) + __fmul_rn(g, invH.lo)));
    float out;
    bool good;
    if (a.mode == 1) {
      // capped at +- max_v_deriv; FP64 decides near the cap
      const Pair r = div(dT, fabsf(g) > cap ? (g < 0.0f ? cap_down : cap_up) : one_g);
      out = r.hi + r.lo;
      good = fabsf(fabsf(g) - cap) > 1e-5f * cap && fabsf(dT) < 1e15f && fabsf(dT) > 1e-15f;
    } else {
      const Pair gc = one_g.hi < 0.0f ? Pair{ -one_g.hi, -one_g.lo } : one_g;
      const Pair x = div(dT, gc);
      const Pair d = two_sum(TS, -T_rad.hi);
      const Pair scale = mul(fast_two_sum(d.hi, d.lo - T_rad.lo), mK);
      const Pair r = mul(one_minus_exp_small(x), scale);
      out = r.hi + r.lo;
      good = gc.hi > 1e-4f && gc.hi < 1e6f && fabsf(x.hi) < SMALL_TAU && (fabsf(dT) > 1e-15f || dT == 0.0f) &&
             fabsf(TS) < 1e15f;
    }
    a.delta_T[ir] = good ? out : pecvel_cell_fp64(a, dT, grad, TS);
  }
}

// Target cell index of a deposit.  The reference's index arithmetic assumes
// a displacement below one box length; wrapping keeps every access inside the
// column in any case and is the identity whenever the reference's index is
// valid.
__device__ __forceinline__ int wrap(int t, int D) { return ((t % D) + D) % D; }

// BrightnessTemperature.c:325-499 for one z column, sub-cell by sub-cell into
// los: the columns that hold a value which the closed form below cannot take.
__device__ __noinline__ void rsd_column_sequential(const RsdArgs& a, long long col, int D, int H)
{
  const float* vel = a.vel + col * 2LL * H;
  const float* dTc = a.delta_T + col * D;
  const float* xHc = a.xH + col * D;
  float* los = a.los + col * D;
  const int NS = RSD_STEPS;
  const double cw = a.box / (float)D;  // BoxSize / (float)ReionGridDim
  const double sw = a.subcell_width;
  const float H_z = a.H_z;
  for (int kk = 0; kk < D; kk++)
    los[kk] = 0.0f;
  for (int kk = 0; kk < D; kk++) {
    const float dT = dTc[kk];
    if (!((fabs((double)dT) >= FRACT_FLOAT_ERR_D) && ((double)xHc[kk] >= FRACT_FLOAT_ERR_D)))
      continue;
    // displacements: float divisions assigned to doubles, as in the reference
    double d1_low, d2_low, d1_high, d2_high;
    if (kk == 0) {
      d1_low = __fdiv_rn(vel[D - 1], H_z);
      d2_low = __fdiv_rn(vel[kk], H_z);
    } else {
      d1_low = __fdiv_rn(vel[kk - 1], H_z);
      d2_low = __fdiv_rn(vel[kk], H_z);
    }
    if (kk == D - 1) {
      d1_high = __fdiv_rn(vel[kk], H_z);
      d2_high = __fdiv_rn(vel[0], H_z);
    } else {
      d1_high = __fdiv_rn(vel[kk], H_z);
      d2_high = __fdiv_rn(vel[kk + 1], H_z);
    }
    const float share = __fdiv_rn(dT, (float)NS);  // delta_T / (float)N_RSD_STEPS
    for (int iii = 0; iii < NS; iii++) {
      const float xp = a.x_pos[iii];
      double disp;
      if (xp <= 0.5f)
        disp = d1_low + (((double)xp + 0.5) - 0.) * (d2_low - d1_low) / (1. - 0.);
      else
        disp = d1_high + (((double)xp - 0.5) - 0.) * (d2_high - d1_high) / (1. - 0.);
      const double pos = ((double)a.x_pos_offset[iii] + disp) / cw;
      const double lo = pos - (sw / 2.) / cw;
      const double hi = pos + (sw / 2.) / cw;
      if (lo >= 0.0 && hi < 1.0) {
        los[kk] = __fadd_rn(los[kk], share);
      } else if (lo < 0.0 && hi < 0.0) {
        const double cell_distance = ceil(fabs(lo)) - 1.;
        const int cd = (int)cell_distance;
        if (fabs(hi) > cell_distance) {
          const int t = wrap(kk < cd + 1 ? kk - (cd + 1) + D : kk - (cd + 1), D);
          los[t] = __fadd_rn(los[t], share);
        } else {
          const double fo = (fabs(lo) - cell_distance) / (sw / cw);
          const double fw = 1. - fo;
          const int t1 = wrap(kk < cd ? kk - cd + D : kk - cd, D);
          los[t1] = (float)((double)los[t1] + fw * (double)dT / (double)(float)NS);
          const int t2 = wrap(kk < cd + 1 ? kk - (cd + 1) + D : kk - (cd + 1), D);
          los[t2] = (float)((double)los[t2] + fo * (double)dT / (double)(float)NS);
        }
      } else if (lo < 0.0 && (hi > 0.0 && hi < 1.0)) {
        const double fw = hi / (sw / cw);
        const double fo = 1. - fw;
        const int t1 = kk == 0 ? D - 1 : kk - 1;
        los[t1] = (float)((double)los[t1] + fo * (double)dT / (double)(float)NS);
        los[kk] = (float)((double)los[kk] + fw * (double)dT / (double)(float)NS);
      } else if ((lo >= 0.0 && lo < 1.0) && (hi >= 1.0)) {
        const double fo = (hi - 1.) / (sw / cw);
        const double fw = 1. - fo;
        const int t2 = kk == D - 1 ? 0 : kk + 1;
        los[kk] = (float)((double)los[kk] + fw * (double)dT / (double)(float)NS);
        los[t2] = (float)((double)los[t2] + fo * (double)dT / (double)(float)NS);
      } else {
        const double cell_distance = floor(fabs(hi));
        const int cd = (int)cell_distance;
        if (lo >= cell_distance) {
          const int t = wrap(kk > D - 1 - cd ? kk + cd - D : kk + cd, D);
          los[t] = __fadd_rn(los[t], share);
        } else {
          const double fo = (hi - cell_distance) / (sw / cw);
          const double fw = 1. - fo;
          const int t1 = wrap(kk > D - 1 - (cd - 1) ? kk + cd - 1 - D : kk + cd - 1, D);
          los[t1] = (float)((double)los[t1] + fw * (double)dT / (double)(float)NS);
          const int t2 = wrap(kk > D - 1 - cd ? kk + cd - D : kk + cd, D);
          los[t2] = (float)((double)los[t2] + fo * (double)dT / (double)(float)NS);
        }
      }
    }
  }
}

// The remap of BrightnessTemperature.c:325-499.  The reference moves fifty
// sub-cells of a cell by the velocity interpolated between the cell's
// neighbours and shares each over the unit cells it overlaps.  In each half of
// a cell (25 sub-cells) the interpolation is linear, so the sub-cells' lower
// edges are lo + i B / 50, and what lands below a cell boundary b is
//   sum_i clamp(U - |B| i, 0, 1),  U = 50 (b - lowest edge),
// an arithmetic series: n1 whole sub-cells and n2 - n1 partial ones.  A half
// needs one such sum per boundary that it crosses (one or two) instead of 25
// positions with three FP64 quotients each, and every cell is a thread of its
// own.
//
// Everything is fixed point: 100 x position in units of 2^-40 cells (in which
// the sub-cells' offsets and widths are whole), sub-cells to 2^-(33 - log2 D) and
// 24-bit sources, relative to the column's largest.  The sums are exact but for
// the last of these roundings (1e-9 of a source at 256 cells), a column's
// deposits stay below 2^63, and the result does not depend on their order.  n1
// and n2 come from FP32: the series is continuous where they step, and a count off
// by one within rounding of a step moves 1.5e-6 |B| of a sub-cell.  Where the
// sub-cells lie more than two widths apart (|B| > 2; up to 8192 between
// neighbours of opposite far displacements, which would move 1e-2), one exact
// comparison each mends the counts.
// A column with an infinite source or a displacement of RSD_FAR cells or more
// (or NaN) takes the sequential routine.
//
// Bound by integer issue and shared-memory atomics.  At 256^3: one thread per
// column with the sequential loop 88.1 ms; the series in FP64 2.1 ms.
constexpr int RSD_THREADS = 256;
constexpr int RSD_CELLS = 1024;   // cells of a block: whole columns, at least one
constexpr double RSD_FAR = 4096.0;
constexpr long long RSD_ONE = 1LL << 40, RSD_CELL = 100 * RSD_ONE;

// floor(x / RSD_CELL)
__device__ __forceinline__ int rsd_cell_of(long long x)
{
  int c = (int)floorf((float)x * (float)(1.0 / (double)RSD_CELL));
  while (x < c * RSD_CELL)
    c--;
  while (x >= (c + 1) * RSD_CELL)
    c++;
  return c;
}

// The 25 sub-cells of half a cell: lower edge of the first (100 x cells, 2^-40)
// and B (2^-40); source mantissa, right shift, and bits per sub-cell.
__device__ __forceinline__ void rsd_half(unsigned long long* acc, int kk, int D, long long lo0, long long B, int mant,
                                         int shift, int bits)
{
  constexpr int n = RSD_STEPS / 2;
  const long long step = B < 0 ? -B : B;
  const long long lo = B < 0 ? lo0 + 2 * (n - 1) * B : lo0;
  const int first = rsd_cell_of(lo), last = rsd_cell_of(lo + 2 * (n - 1) * step + 2 * RSD_ONE - 1);
  int t = kk + first;
  if (t < 0 || t >= D)
    t = wrap(t, D);
  auto add = [&](int mass) { atomicAdd(acc + t, (unsigned long long)(((long long)mass * mant) >> shift)); };
  int done = 0;
  if (first < last) {
    const float inv_step = __fdividef(1.0f, fmaxf((float)step * 0x1p-40f, 1e-20f));
    for (int c = first; c < last; c++) {
      // sub-cells below the boundary c + 1
      const long long U = ((c + 1) * RSD_CELL - lo) >> 1;
      const float u = (float)U * 0x1p-40f;
      int n1 = (int)fminf(fmaxf(floorf((u - 1.0f) * inv_step) + 1.0f, 0.0f), (float)n);
      int n2 = (int)fminf(fmaxf(ceilf(u * inv_step), 0.0f), (float)n);
      if (step > 2 * RSD_ONE) {
        // whole: U - i step >= 1; at least partly below: U - i step > 0
        if (n1 < n && U - n1 * step >= RSD_ONE)
          n1++;
        else if (n1 > 0 && U - (n1 - 1) * step < RSD_ONE)
          n1--;
        if (n2 < n && U - n2 * step > 0)
          n2++;
        else if (n2 > 0 && U - (n2 - 1) * step <= 0)
          n2--;
      }
      n2 = max(n1, n2);
      const int m = n2 - n1;
      const long long below = n1 * RSD_ONE + (m * U - ((n1 + n2 - 1) * m / 2) * step);
      const int mass = (int)((below + (1LL << (39 - bits))) >> (40 - bits));
      add(mass - done);
      done = mass;
      t = t + 1 == D ? 0 : t + 1;
    }
  }
  add((n << bits) - done);
}

// Block: `cols` whole columns.  Shared memory: displacement (2^-40 cells) and
// deposit of each cell; `bits` per sub-cell.
__global__ void __launch_bounds__(RSD_THREADS)
  k_rsd_columns(const __grid_constant__ RsdArgs a, int D, int H, int cols, int bits)
{
  extern __shared__ long long rsd_sm[];
  long long* disp = rsd_sm;
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(rsd_sm + cols * D);
  int* top = reinterpret_cast<int*>(acc + cols * D);  // per column: bits of the largest |source|
  int* bad = top + cols;
  const long long col0 = (long long)blockIdx.x * cols;
  const int nc = (int)min((long long)cols, (long long)D * D - col0);
  const int cells = nc * D;
  for (int i = threadIdx.x; i < nc; i += RSD_THREADS)
    top[i] = bad[i] = 0;
  __syncthreads();
  auto source = [&](int i) {
    const float dT = a.delta_T[col0 * D + i];
    const bool on = fabs((double)dT) >= FRACT_FLOAT_ERR_D && (double)a.xH[col0 * D + i] >= FRACT_FLOAT_ERR_D;
    return on ? dT : 0.0f;
  };
  for (int i = threadIdx.x; i < cells; i += RSD_THREADS) {
    const int c = i / D;
    const double d = (double)__fdiv_rn(a.vel[(col0 + c) * 2LL * H + (i - c * D)], a.H_z) * a.inv_cell;
    const bool near = fabs(d) < RSD_FAR;
    disp[i] = near ? __double2ll_rn(d * (double)RSD_ONE) : 0;
    acc[i] = 0;
    const int top_bits = __float_as_int(fabsf(source(i)));
    if (top_bits)
      atomicMax(top + c, top_bits);
    if (!near)
      bad[c] = 1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cells; i += RSD_THREADS) {
    const int c = i / D, kk = i - c * D;
    const int b = __float_as_int(source(i));
    if (b << 1 == 0 || bad[c] || top[c] >= 0x7f800000)
      continue;
    // a source is at least 1e-7: a normal float
    const int mant = ((b & 0x7fffff) | 0x800000) * (b < 0 ? -1 : 1);
    const int shift = min((top[c] >> 23) - (b >> 23 & 0xff), 62);
    const long long* d = disp + c * D;
    const long long here = d[kk], lo_d = here - d[kk == 0 ? D - 1 : kk - 1], hi_d = d[kk == D - 1 ? 0 : kk + 1] - here;
    // first half: from the lower neighbour's velocity at x = -1/2 to this
    // cell's at 1/2 (sub-cell centres 0.01 ... 0.49); second half: from this
    // cell's at 1/2 to the upper neighbour's at 3/2 (0.51 ... 0.99)
    rsd_half(acc + c * D, kk, D, 100 * here - 49 * lo_d, RSD_ONE + lo_d, mant, shift, bits);
    rsd_half(acc + c * D, kk, D, 50 * RSD_ONE + 100 * here + hi_d, RSD_ONE + hi_d, mant, shift, bits);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cells; i += RSD_THREADS) {
    const int c = i / D;
    if (bad[c] || top[c] >= 0x7f800000)
      continue;
    // 2^(e - 23 - bits) / 50 per unit, e the exponent of the largest source
    const int e = (top[c] >> 23) - 127 - 23 - bits;
    a.delta_T_out[col0 * D + i] =
      (float)((double)(long long)acc[i] * (__hiloint2double((1023 + e) << 20, 0) * (1.0 / RSD_STEPS)));
  }
  for (int c = threadIdx.x; c < nc; c += RSD_THREADS)
    if (bad[c] || top[c] >= 0x7f800000) {
      rsd_column_sequential(a, col0 + c, D, H);
      const float* los = a.los + (col0 + c) * D;
      for (int kk = 0; kk < D; kk++)
        a.delta_T_out[(col0 + c) * D + kk] = los[kk];
    }
}
}  // namespace

void launch_vel_convert(float* vel, int trees_id, float redshift, const GridDims& gd, cudaStream_t s)
{
  const double first = trees_id == 1 ? std::sqrt(1. / (1. + redshift)) / 1000. : 1. + redshift;
  const double mpc = 1000. * 100. / MPC_CM, comoving = 1. / (1. / (1. + redshift));
  if (trees_id >= 0 && trees_id <= 2)
    k_vel_convert<<<RED_BLOCKS, RED_THREADS, 0, s>>>(vel, Scales<3>({ first, mpc, comoving }), gd.D, gd.H, gd.N);
  else
    k_vel_convert<<<RED_BLOCKS, RED_THREADS, 0, s>>>(vel, Scales<2>({ mpc, comoving }), gd.D, gd.H, gd.N);
  pv_launches++;
}

void launch_vel_grad_k(float2* spec, const GridDims& gd, double hubble_h, float delta_k, cudaStream_t s)
{
  k_vel_grad_k<<<RED_BLOCKS, RED_THREADS, 0, s>>>(spec, gd.H, gd.C, Scales<2>({ 1.0 / (double)gd.N, hubble_h }), delta_k);
  pv_launches++;
}

void launch_pecvel_cells(const PecvelArgs& a, const GridDims& gd, cudaStream_t s)
{
  k_pecvel_cells<<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, gd.D, gd.H, gd.N);
  pv_launches++;
}

void launch_rsd(const RsdArgs& a, const GridDims& gd, cudaStream_t s)
{
  const long long columns = (long long)gd.D * gd.D;
  const int cols = (int)std::max(1, RSD_CELLS / gd.D);
  const size_t smem = (size_t)cols * (gd.D * (sizeof(double) + sizeof(unsigned long long)) + 2 * sizeof(int));
  int log2_D = 1;
  while ((1 << log2_D) < gd.D)
    log2_D++;
  k_rsd_columns<<<(unsigned)((columns + cols - 1) / cols), RSD_THREADS, smem, s>>>(a, gd.D, gd.H, cols,
                                                                                    std::min(25, 33 - log2_D));
  pv_launches++;
}

int pecvel_kernel_launches() { return pv_launches; }

}  // namespace mx
