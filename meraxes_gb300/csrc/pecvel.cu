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
//                    50 sub-cells per cell, a thread per cell (FP64 positions
//                    and sums, order-independent deposits).
#include <algorithm>
#include <cmath>

#include "pecvel.cuh"

namespace mx {

namespace {
// per host thread: a call counts its own launches when contexts run concurrently
thread_local int pv_launches = 0;
constexpr double FRACT_FLOAT_ERR_D = 1e-7;
constexpr double MPC_CM = 3.086e24;

// The float nearest to c x, c a double held as two floats (c = hi + lo): one
// rounding of the exact x hi + x lo but for the last place of x lo, so the
// result equals (float)(c * (double)x) unless that lies within 2^-48 of a tie.
// Two FP32 operations instead of two conversions and a product at the FP64
// rate (the FP64 form took 0.50 ms in k_vel_convert and, with its quotient,
// 0.41 ms in k_vel_grad_k at 256^3).
struct Scale2
{
  float hi, lo;
  Scale2() = default;
  __host__ explicit Scale2(double c) : hi((float)c), lo((float)(c - (double)(float)c)) {}
  __device__ __forceinline__ float operator()(float x) const { return __fmaf_rn(x, hi, __fmul_rn(x, lo)); }
};

// The unit factors in the reference's order, each rounded to float.
struct VelScales
{
  Scale2 f[3];
  int n;
};

__global__ void k_vel_convert(float* vel, VelScales sc, int D, int H, long long N)
{
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    const long long ip = row * 2LL * H + (ir - row * D);
    float v = vel[ip];
    for (int i = 0; i < sc.n; i++)
      v = sc.f[i](v);
    vel[ip] = v;
  }
}

// c /= N; c *= h (each rounded to float); c *= (0 + i k_z) as a float complex
// product.  1/N = inv_n * pow2 with inv_n in [1, 2), so that the low part of
// the factor stays a normal float.
__global__ void k_vel_grad_k(float2* spec, int H, long long C, Scale2 inv_n, float pow2, Scale2 hubble_h, float delta_k)
{
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < C; i += (long long)gridDim.x * blockDim.x) {
    float2 v = spec[i];
    v.x = hubble_h(inv_n(v.x) * pow2);
    v.y = hubble_h(inv_n(v.y) * pow2);
    const int nz = (int)(i % H);
    const float kz = __fmul_rn((float)nz, delta_k);
    // (a + i b)(0 + i k): real a*0 - b*k, imaginary a*k + b*0
    const float re = __fsub_rn(__fmul_rn(v.x, 0.0f), __fmul_rn(v.y, kz));
    const float im = __fadd_rn(__fmul_rn(v.x, kz), __fmul_rn(v.y, 0.0f));
    spec[i] = make_float2(re, im);
  }
}

// 1 - exp(-x).  Optical depths are small: below 1/32 nine terms of the series
// reach FP64 rounding (x^9 / 9! < 1e-19 of x) without the cancellation.
__device__ __forceinline__ double one_minus_exp(double x)
{
  if (!(fabs(x) < 0.03125))
    return 1. - exp(-x);
  double s = 1.0 - x * (1.0 / 9);
  s = 1.0 - x * (1.0 / 8) * s;
  s = 1.0 - x * (1.0 / 7) * s;
  s = 1.0 - x * (1.0 / 6) * s;
  s = 1.0 - x * (1.0 / 5) * s;
  s = 1.0 - x * (1.0 / 4) * s;
  s = 1.0 - x * (1.0 / 3) * s;
  s = 1.0 - x * (1.0 / 2) * s;
  return x * s;
}

// FP64 per cell, like the reference, with the constants' quotients taken once
// on the host (FP64 issue bounds the kernel; 1.97 ms at 256^3 with a quotient
// each).
__global__ void k_pecvel_cells(PecvelArgs a, int D, int H, long long N)
{
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    const long long ip = row * 2LL * H + (ir - row * D);
    const double g = (double)a.grad[ip];
    if (a.mode == 1) {
      double dvdx = g;
      if (fabs(dvdx) > a.max_v_deriv)
        dvdx = dvdx < 0 ? -a.max_v_deriv : a.max_v_deriv;
      a.delta_T[ir] = (float)((double)a.delta_T[ir] / (dvdx * a.inv_H + 1.0));
    } else {
      const double gc = fabs(g * a.inv_H + 1.0);
      const double scale = ((double)a.TS[ir] - a.T_rad) * a.mK;
      if (gc < FRACT_FLOAT_ERR_D)
        a.delta_T[ir] = (float)scale;
      else
        a.delta_T[ir] = (float)(one_minus_exp((double)a.delta_T[ir] / gc) * scale);
    }
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
// own.  Positions, sums and deposits are FP64; n1 and n2 may come from FP32,
// because the series is continuous where they step (a count off by one within
// rounding of a step moves 1e-6 of a sub-cell).
//
// Deposits of different source cells meet in shared memory as 64-bit fixed
// point (2^-50 of the column's largest source), so that the result does not
// depend on their order.  D <= 2048 sources of 2^50 stay below 2^63.
// A column with an infinite source or a displacement of RSD_FAR cells or more
// (or NaN) takes the sequential routine.
//
// Bound by FP64 issue (about 50 operations per cell; 2 lanes per clock and
// SM).  One thread per column with the sequential loop took 88.1 ms at 256^3.
constexpr int RSD_THREADS = 256;
constexpr int RSD_CELLS = 1024;   // cells of a block: whole columns, at least one
constexpr double RSD_FAR = 4096.0;

struct RsdSeries
{
  double lo, step;  // lowest lower edge [cells], |B|
  float inv_step;
  __device__ __forceinline__ RsdSeries(double lo0, double B)
  {
    constexpr int n = RSD_STEPS / 2;
    lo = B < 0 ? lo0 + B * ((n - 1) * (1.0 / RSD_STEPS)) : lo0;
    step = fabs(B);
    inv_step = __fdividef(1.0f, fmaxf((float)step, 1e-20f));
  }
  // sub-cells below boundary b
  __device__ __forceinline__ double below(int b) const
  {
    constexpr float n = RSD_STEPS / 2;
    const double U = ((double)b - lo) * (double)RSD_STEPS;
    const float u = (float)U;
    const int n1 = (int)fminf(fmaxf(floorf((u - 1.0f) * inv_step) + 1.0f, 0.0f), n);
    const int n2 = max(n1, (int)fminf(fmaxf(ceilf(u * inv_step), 0.0f), n));
    const int m = n2 - n1;
    return (double)n1 + ((double)m * U - (double)((n1 + n2 - 1) * m / 2) * step);
  }
};

__device__ __forceinline__ void rsd_half(unsigned long long* acc, int kk, int D, double lo0, double B, double q)
{
  constexpr double n = RSD_STEPS / 2;
  const RsdSeries s(lo0, B);
  const int first = (int)floor(s.lo);
  const int last = (int)ceil(s.lo + s.step * ((n - 1) / RSD_STEPS) + 1.0 / RSD_STEPS) - 1;
  double done = 0.0;
  int t = kk + first;
  if (t < 0 || t >= D)
    t = wrap(t, D);
  for (int c = first; c < last; c++) {
    const double m = s.below(c + 1);
    atomicAdd(acc + t, (unsigned long long)__double2ll_rn((m - done) * q));
    done = m;
    t = t + 1 == D ? 0 : t + 1;
  }
  atomicAdd(acc + t, (unsigned long long)__double2ll_rn((n - done) * q));
}

// Block: `cols` whole columns.  Shared memory: displacement [cells] and
// deposit of each cell.
__global__ void __launch_bounds__(RSD_THREADS) k_rsd_columns(const __grid_constant__ RsdArgs a, int D, int H, int cols)
{
  extern __shared__ double rsd_sm[];
  double* disp = rsd_sm;
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
    disp[i] = d;
    acc[i] = 0;
    const int bits = __float_as_int(fabsf(source(i)));
    if (bits)
      atomicMax(top + c, bits);
    if (!(fabs(d) < RSD_FAR))
      bad[c] = 1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cells; i += RSD_THREADS) {
    const int c = i / D, kk = i - c * D;
    const float dT = source(i);
    if (dT == 0.0f || bad[c] || top[c] >= 0x7f800000)
      continue;
    // |largest source| * 2^shift in [2^49, 2^50)
    const int shift = 49 - ((top[c] >> 23) - 127);
    const double q = (double)dT * __hiloint2double((1023 + shift) << 20, 0) * (1.0 / RSD_STEPS);
    const double* d = disp + c * D;
    const double here = d[kk], lo_d = here - d[kk == 0 ? D - 1 : kk - 1], hi_d = d[kk == D - 1 ? 0 : kk + 1] - here;
    // first half: from the lower neighbour's velocity at x = -1/2 to this
    // cell's at 1/2 (sub-cell centres 0.01 ... 0.49); second half: from this
    // cell's at 1/2 to the upper neighbour's at 3/2 (0.51 ... 0.99)
    rsd_half(acc + c * D, kk, D, here - 0.49 * lo_d, 1.0 + lo_d, q);
    rsd_half(acc + c * D, kk, D, 0.5 + here + 0.01 * hi_d, 1.0 + hi_d, q);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cells; i += RSD_THREADS) {
    const int c = i / D;
    if (bad[c] || top[c] >= 0x7f800000)
      continue;
    const int shift = 49 - ((top[c] >> 23) - 127);
    a.delta_T_out[col0 * D + i] = (float)((double)(long long)acc[i] * __hiloint2double((1023 - shift) << 20, 0));
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
  VelScales sc{};
  if (trees_id == 1)
    sc.f[sc.n++] = Scale2(std::sqrt(1. / (1. + redshift)) / 1000.);
  else if (trees_id == 0 || trees_id == 2)
    sc.f[sc.n++] = Scale2(1. + redshift);
  sc.f[sc.n++] = Scale2(1000. * 100. / MPC_CM);
  sc.f[sc.n++] = Scale2(1. / (1. / (1. + redshift)));
  k_vel_convert<<<RED_BLOCKS, RED_THREADS, 0, s>>>(vel, sc, gd.D, gd.H, gd.N);
  pv_launches++;
}

void launch_vel_grad_k(float2* spec, const GridDims& gd, double hubble_h, float delta_k, cudaStream_t s)
{
  int e;
  const double m = std::frexp(1.0 / (double)gd.N, &e);
  k_vel_grad_k<<<RED_BLOCKS, RED_THREADS, 0, s>>>(spec, gd.H, gd.C, Scale2(2.0 * m), std::ldexp(1.0f, e - 1),
                                                  Scale2(hubble_h), delta_k);
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
  k_rsd_columns<<<(unsigned)((columns + cols - 1) / cols), RSD_THREADS, smem, s>>>(a, gd.D, gd.H, cols);
  pv_launches++;
}

int pecvel_kernel_launches() { return pv_launches; }

}  // namespace mx
