// Per-cell spin-temperature update (FP32 fast path with FP64 fallback).
//
// ComputeTs.c:743-900 with evolveInt (XRayHeatingFunctions.c:1241-1435) and
// get_Ts (XRayHeatingFunctions.c:1513-1882).  GB300's FP64 rate is a small
// fraction of its FP32 rate, so the per-cell arithmetic runs in FP32 on
// host-prepared, range-scaled coefficients; FP64 is kept for the frequency
// tables (host), the volume averages, and the spin-temperature fixed point
// of the rare cells whose FP32 stopping test lands within 1e-5 of the
// reference's 1e-3 criterion (those cells are recomputed in FP64 so that they
// stop after the same iteration as the reference).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "bulk.cuh"
#include "kernels.cuh"

namespace mx {

namespace {
constexpr int NXHII = 14;
constexpr double TCMB = 2.728;
constexpr double T21 = 0.0628;
constexpr double A10 = 2.85e-15;
constexpr float MAX_TK = 5e4f;
constexpr double FRACT_FLOAT_ERR = 1e-7;
constexpr int TS_MAX_ITER = 10000;

// per host thread: a call counts its own launches when contexts run concurrently
thread_local int ts_launches = 0;

template <int NV>
__device__ void block_sum_store(double (&v)[NV], double* partials)
{
  __shared__ double sh[NV][RED_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; q++) {
    double x = v[q];
    for (int o = 16; o > 0; o >>= 1)
      x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0)
      sh[q][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
    for (int w = 0; w < RED_THREADS / 32; w++)
      s += sh[threadIdx.x][w];
    partials[(long long)blockIdx.x * NV + threadIdx.x] = s;
  }
}

// floats of the frequency tables at the start of the evolve kernel's shared
// memory (one float4 per x_HII node and shell), whole 16-byte units for the
// shell ring behind them
__host__ __device__ constexpr int ev_tables_floats(int S) { return 4 * NXHII * S; }

__device__ __forceinline__ long long pad_index(long long ir, int D, int H)
{
  const long long row = row_of(ir, D);
  return ir - row * D + row * 2LL * H;
}

// -------------------------------------------------------- FP64 (fallback)
__device__ double spline_d(const double* x, const double* y, const double* c, int n, double xv)
{
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (x[mid] > xv)
      hi = mid;
    else
      lo = mid;
  }
  const double h = x[lo + 1] - x[lo];
  const double dx = xv - x[lo];
  const double b = (y[lo + 1] - y[lo]) / h - h * (c[lo + 1] + 2.0 * c[lo]) / 3.0;
  const double d = (c[lo + 1] - c[lo]) / (3.0 * h);
  return y[lo] + dx * (b + dx * (c[lo] + dx * d));
}

// kappa_10 (which 0, power law above the table) and kappa_10_elec /
// kappa_10_pH (1, 2: linear extrapolation in logs), XRayHeatingFunctions.c:1686-1839
__device__ double kappa_d(const TsDevConst& c, int which, double T)
{
  const int n = c.nk[which];
  const double* x = c.kx[which];
  const double* y = c.ky[which];
  const double lt = log(T);
  double ans;
  if (lt < x[0])
    ans = y[0];
  else if (lt > x[n - 1])
    ans = which == 0 ? log(exp(y[n - 1]) * pow(T / exp(x[n - 1]), 0.381))
                     : y[n - 1] + ((y[n - 1] - y[n - 2]) / (x[n - 1] - x[n - 2]) * (lt - x[n - 1]));
  else
    ans = spline_d(x, y, c.kc[which], n, lt);
  return exp(ans);
}

__device__ __noinline__ float get_Ts_d(const TsDevConst& c, float z, float delta, float TK, float xe, float Jalpha, float* xalpha,
                          unsigned int* err)
{
  const double zd = z, TKd = TK, dd = delta, xd = xe;
  const double Trad = TCMB * (1.0 + zd);
  const double p3 = pow(1.0 + zd, 3.0);
  const double xc = T21 / Trad * ((1.0 - xd) * c.no * p3 * (1.0 + dd)) * kappa_d(c, 0, TKd) / A10 +
                    T21 / Trad * (xd * c.n_b0 * p3 * (1.0 + dd)) * kappa_d(c, 1, TKd) / A10 +
                    T21 / Trad * (xd * c.no * p3 * (1.0 + dd)) * kappa_d(c, 2, TKd) / A10;
  double TS, xa = 0;
  if (Jalpha > 1.0e-20) {
    TS = Trad;
    double TSold = 0.0;
    const double tgp = 1.342881e-7 / c.hubble_z * c.no * pow(1 + zd, 3) * (1.0 + dd) * (1.0 - xd);
    const double xi = pow(1.0e-7 * tgp / TKd / TKd, 1.0 / 3.0);
    int it = 0;
    while (fabs(TS - TSold) / TS > 1.0e-3) {
      if (++it > TS_MAX_ITER) {
        atomicOr(err, 1u);
        break;
      }
      TSold = TS;
      double St = 1.0 - 0.0631789 / TKd + 0.115995 / TKd / TKd - 0.401403 / TS / TKd;
      St += 0.336463 / TS / TKd / TKd;
      St /= 1.0 + 2.98394 * xi + 1.53583 * xi * xi + 3.85289 * xi * xi * xi;
      xa = 1.66e11 / (1.0 + zd) * St * (double)Jalpha;
      const double Tceff = 1.0 / (1.0 / TKd + 0.405535 / TKd * (1.0 / TS - 1.0 / TKd));
      TS = 1.0 / ((1.0 / Trad + xa / Tceff + xc / TKd) / (1.0 + xa + xc));
    }
    *xalpha = (float)xa;
  } else {
    TS = 1.0 / ((1.0 / Trad + xc / TKd) / (1.0 + xc));
    *xalpha = 0;
  }
  return (float)fabs(TS);
}

// --------------------------------------------------------------- FP32 path
__device__ float spline_f(const float* x, const float* y, const float* c, int n, float xv)
{
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (x[mid] > xv)
      hi = mid;
    else
      lo = mid;
  }
  const float h = x[lo + 1] - x[lo];
  const float ih = __fdividef(1.0f, h);
  const float dx = xv - x[lo];
  const float b = (y[lo + 1] - y[lo]) * ih - h * (c[lo + 1] + 2.0f * c[lo]) * (1.0f / 3.0f);
  const float d = (c[lo + 1] - c[lo]) * ih * (1.0f / 3.0f);
  return y[lo] + dx * (b + dx * (c[lo] + dx * d));
}

__device__ float kappa_f(const TsDevConst& c, int which, float T)
{
  const int n = c.nk[which];
  const float* x = c.fkx[which];
  const float* y = c.fky[which];
  const float lt = logf(T);
  float ans;
  if (lt < x[0])
    ans = y[0];
  else if (lt > x[n - 1])
    ans = which == 0 ? y[n - 1] + 0.381f * (lt - x[n - 1])
                     : y[n - 1] + ((y[n - 1] - y[n - 2]) / (x[n - 1] - x[n - 2]) * (lt - x[n - 1]));
  else
    ans = spline_f(x, y, c.fkc[which], n, lt);
  return expf(ans);
}

// The kappa splines in shared memory, the cubic of each interval beside its node
// and, for 64 steps of ln T, the interval that a step begins in: three binary
// searches through global memory took a fifth of the per-cell update's time.
struct KappaTab
{
  static constexpr int STEPS = 64, NODES = 27;
  float4 p[3][NODES];  // y, and the coefficients of dx, dx^2, dx^3
  float x[3][NODES + 1];
  float x_last[3], y_last[3], slope[3], step[3];  // slope of the extrapolation above, steps per ln T
  int last[3];                                    // last interval
  unsigned char begin[3][STEPS];
};
__device__ void fill_kappa(KappaTab& t, const TsDevConst& c)
{
  for (int i = threadIdx.x; i < 3 * KappaTab::NODES; i += blockDim.x) {
    const int w = i / KappaTab::NODES, q = i % KappaTab::NODES, n = c.nk[w];
    const float *x = c.fkx[w], *y = c.fky[w], *cc = c.fkc[w];
    if (q < n)
      t.x[w][q] = x[q];
    if (q < n - 1) {
      const float h = x[q + 1] - x[q];
      const float ih = __fdividef(1.0f, h);
      const float b = (y[q + 1] - y[q]) * ih - h * (cc[q + 1] + 2.0f * cc[q]) * (1.0f / 3.0f);
      t.p[w][q] = make_float4(y[q], b, cc[q], (cc[q + 1] - cc[q]) * ih * (1.0f / 3.0f));
    }
    if (q == n - 1) {
      t.x_last[w] = x[q];
      t.y_last[w] = y[q];
      t.slope[w] = w == 0 ? 0.381f : (y[q] - y[q - 1]) / (x[q] - x[q - 1]);
      t.step[w] = KappaTab::STEPS / (x[q] - x[0]);
      t.last[w] = n - 2;
    }
  }
  for (int i = threadIdx.x; i < 3 * KappaTab::STEPS; i += blockDim.x) {
    const int w = i / KappaTab::STEPS, q = i % KappaTab::STEPS, n = c.nk[w];
    const float* x = c.fkx[w];
    // a hundredth of a step early, for the rounding of the step's number
    const float from = x[0] + (x[n - 1] - x[0]) * ((q - 0.01f) / KappaTab::STEPS);
    int lo = 0;
    while (lo < n - 2 && x[lo + 1] <= from)
      lo++;
    t.begin[w][q] = (unsigned char)lo;
  }
}
// kappa at lt = ln T as kappa_f, and d ln kappa / d ln T (the spline's derivative
// inside the table, the extrapolations' slopes outside it)
template <bool GRAD = false>
__device__ __forceinline__ float kappa_s(const KappaTab& t, int w, float lt, float* dln = nullptr)
{
  const float x0 = t.x[w][0];
  int lo = t.begin[w][(int)fminf(fmaxf((lt - x0) * t.step[w], 0.0f), (float)(KappaTab::STEPS - 1))];
  while (lo < t.last[w] && t.x[w][lo + 1] <= lt)
    lo++;
  const float4 p = t.p[w][lo];
  const float dx = lt - t.x[w][lo];
  float ans = p.x + dx * (p.y + dx * (p.z + dx * p.w));
  if constexpr (GRAD)
    *dln = p.y + dx * (2.0f * p.z + 3.0f * p.w * dx);
  if (lt < x0) {
    ans = t.p[w][0].x;
    if constexpr (GRAD)
      *dln = 0.0f;
  } else if (lt > t.x_last[w]) {
    ans = t.y_last[w] + t.slope[w] * (lt - t.x_last[w]);
    if constexpr (GRAD)
      *dln = t.slope[w];
  }
  return expf(ans);
}

// a * b + c of both halves, each rounded as fmaf
__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c)
{
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%5, %6};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// Node below xcall in the x_HII table, whose bracket the tables are taken in
// (ComputeTs.c:761-773).  Upwards: the gas outside ionised regions is nearly
// neutral, and the table's lower nodes are its.
__device__ __forceinline__ int xhii_node(const float* xhii, float xcall)
{
  int lo = 0;
  while (lo < NXHII - 2 && xcall >= xhii[lo + 1])
    lo++;
  return lo;
}

// alpha_A (Abel et al. 1997 fit), XRayHeatingFunctions.c:1450-1458, in Horner form
__device__ float alpha_A_f(float T)
{
  const float l = logf(T * (1.0f / 1.1604505e4f));
  float p = -3.07113524e-9f;
  p = p * l - 1.85676704e-8f;
  p = p * l + 5.75561414e-7f;
  p = p * l + 4.98910892e-6f;
  p = p * l - 1.42150291e-5f;
  p = p * l - 3.21260521e-4f;
  p = p * l - 2.38086188e-3f;
  p = p * l - 2.02604473e-2f;
  p = p * l - 0.72411256f;
  p = p * l - 28.6130338f;
  return expf(p);
}

// get_Ts in FP32; returns false when a stopping test is too close to the
// reference's 1e-3 criterion for FP32 to decide it like FP64 would.  Its
// quotients are reciprocals or quotients of __fdividef (2 ulp), well inside
// that 1e-5 band around the criterion; get_Ts_grad repeats the same
// operations, so the adjoint runs the forward's iteration count.
template <class K>
__device__ bool get_Ts_f(const TsDevConst& c, const K& kappa, float delta, float TK, float xe, float Jalpha,
                         float* TS_out, float* xalpha)
{
  const float Trad = c.ftrad;
  const float opd = 1.0f + delta;
  const float xc = c.fxc[0] * ((1.0f - xe) * opd) * kappa(0) + c.fxc[1] * (xe * opd) * kappa(1) +
                   c.fxc[2] * (xe * opd) * kappa(2);
  float TS, xa = 0.0f;
  const float iTK = __fdividef(1.0f, TK);
  const float iTrad = __fdividef(1.0f, Trad);
  if (Jalpha > 1.0e-20f) {
    TS = Trad;
    float TSold = 0.0f;
    const float tgp = c.ftgp * opd * (1.0f - xe);
    const float xi = cbrtf(1.0e-7f * tgp * iTK * iTK);
    const float den = 1.0f + 2.98394f * xi + 1.53583f * xi * xi + 3.85289f * xi * xi * xi;
    const float iden = __fdividef(1.0f, den);
    int it = 0;
    for (;;) {
      const float iTS = __fdividef(1.0f, TS);
      const float rel = fabsf(TS - TSold) * iTS;
      if (fabsf(rel - 1.0e-3f) < 1.0e-5f)
        return false;
      if (!(rel > 1.0e-3f))
        break;
      if (++it > TS_MAX_ITER)
        return false;
      TSold = TS;
      const float St =
        (1.0f - 0.0631789f * iTK + 0.115995f * iTK * iTK - 0.401403f * iTS * iTK + 0.336463f * iTS * iTK * iTK) * iden;
      xa = c.fxa * St * Jalpha;
      // 1 / Tceff = iTK + 0.405535 iTK (iTS - iTK)
      const float iTceff = iTK + 0.405535f * iTK * (iTS - iTK);
      TS = __fdividef(1.0f + xa + xc, iTrad + xa * iTceff + xc * iTK);
    }
    *xalpha = xa;
  } else {
    TS = __fdividef(1.0f + xc, iTrad + xc * iTK);
    *xalpha = 0.0f;
  }
  *TS_out = fabsf(TS);
  return true;
}
}  // namespace

// Per-cell update.  A block owns tiles of EV_TILE consecutive cells (one per
// thread), tile k at cell (blockIdx.x + k gridDim.x) EV_TILE.  The 40 shell
// values of a tile (40 rows of EV_TILE floats, one per shell) are streamed
// into shared memory by bulk copies through a two-stage ring, so the shell
// reads do not depend on how many loads each thread keeps in flight; the next
// tile's copies run while the current tile is computed.
// With a tensor map of the shells (cells x shells) a tile's S rows arrive
// by one tiled tensor copy of the box (EV_TILE cells, S shells); the copy
// engine's cost per copy made the S separate row copies the bound of the
// ring.  The map applies when every tile is whole, the cell coordinate fits
// a signed 32-bit index and S fits a box dimension.
//
// Bound by the latency and the shared-memory loads of its arithmetic at 16 warps
// per SM (the two tables' rows for each shell and cell), then by HBM: 40 shells at
// 256^3 take 1.41 ms (2.2 TB/s), at 512^3 11.2 ms.  With the kappa splines and the
// x_HII table searched in global memory 1.70 and 13.6 ms; with those in shared memory
// and scalar multiply-adds 1.53 and 12.1 ms.
constexpr int EV_TILE = RED_THREADS;

bool ev_shell_map_ok(long long N, int S) { return N % EV_TILE == 0 && N < (1LL << 31) && S >= 1 && S <= 256; }

// shared-memory offset (floats) of the shell ring of k_evolve_f32: after the
// tables, on a 128-byte boundary for the tensor copies
__host__ __device__ constexpr int ev_ring_offset(int S) { return (ev_tables_floats(S) + 31) / 32 * 32; }

template <int STAGES = 2>
__device__ __forceinline__ void ev_issue(uint64_t* bars, float* stages, const float* shells, const bulk::TensorMap* map,
                                         int S, long long N, long long tile, int k)
{
  const long long c0 = tile * EV_TILE;
  float* st = stages + (size_t)(k % STAGES) * S * EV_TILE;
  uint64_t* bar = &bars[k % STAGES];
  if (map) {
    bulk::mbar_arm(bar, (unsigned)(sizeof(float) * EV_TILE * S));
    bulk::bulk_tensor_2d(st, map, (int)c0, 0, bar);
    return;
  }
  const int n = (int)((N - c0) < EV_TILE ? (N - c0) : EV_TILE);
  bulk::mbar_arm(bar, (unsigned)(sizeof(float) * n * S));
  for (int r = 0; r < S; r++)
    bulk::bulk_copy(st + r * EV_TILE, shells + (long long)r * N + c0, (unsigned)(sizeof(float) * n), bar);
}

// STAGES shell-ring stages (2: a tile in flight while one is summed).  One
// stage (half the shared memory, three blocks per SM at 80 registers with
// spills) measured slower: 11.9 against 11.2 ms at 512^3.
template <int STAGES>
__global__ void __launch_bounds__(RED_THREADS, 2)
  k_evolve_f32(EvolveArgs a, int D, int H, long long N, const __grid_constant__ bulk::TensorMap shell_map, int use_map)
{
  const bulk::TensorMap* map = use_map ? &shell_map : nullptr;
  const TsDevConst& c = *a.cst;
  const int S = c.S;
  // frequency tables times the shell coefficients, P[x][r] = (K_H tab_H,
  // K_I tab_I, K_L tab_L, K_S) at node x of the x_HII table, then the shell
  // ring.  The interpolation in x_HII is linear, so a cell's sums are
  // (1 - w) sum_r shell_r P[lo][r] + w sum_r shell_r P[hi][r].
  extern __shared__ __align__(128) float sm[];
  float4* s_P = reinterpret_cast<float4*>(sm);  // NXHII * S
  float* stages = sm + ev_ring_offset(S);       // 2 * S * EV_TILE
  __shared__ uint64_t bars[STAGES];
  __shared__ KappaTab s_kappa;
  __shared__ float s_xhii[NXHII];
  fill_kappa(s_kappa, c);
  if (threadIdx.x < NXHII)
    s_xhii[threadIdx.x] = c.xhii[threadIdx.x];
  for (int i = threadIdx.x; i < NXHII * S; i += blockDim.x) {
    const int x = i / S, r = i % S;
    s_P[i] = make_float4(c.fKH[r] * c.ftab[0][x][r], c.fKI[r] * c.ftab[1][x][r], c.fKL[r] * c.ftab[2][x][r],
                         c.fKS[r]);
  }
  const long long ntiles = (N + EV_TILE - 1) / EV_TILE;
  const int my_tiles = blockIdx.x < ntiles ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  const bool light = !c.no_light;
  const bool full = bulk::full_waits();
  if (threadIdx.x == 0 && light) {
    for (int b = 0; b < STAGES; b++)
      bulk::mbar_init(&bars[b], 1);
    bulk::mbar_init_fence();
  }
  __syncthreads();
  if (threadIdx.x == 0 && light)
    for (int k = 0; k < STAGES && k < my_tiles; k++)
      ev_issue<STAGES>(bars, stages, a.shells, map, S, N, blockIdx.x + (long long)k * gridDim.x, k);
  CSum sum[4];
  // the cell state of tile k + 1 is read while tile k is computed
  float n_delta = 0.f, n_xe = 0.f, n_T = 1.f;
  long long n_ip = 0;
  auto read_state = [&](int k) {
    const long long ir = (blockIdx.x + (long long)k * gridDim.x) * EV_TILE + threadIdx.x;
    if (k < my_tiles && ir < N) {
      n_ip = pad_index(ir, D, H);
      n_delta = a.deltax[n_ip];
      n_xe = a.x_e_prev[n_ip];
      n_T = a.Tk[ir];
    }
  };
  read_state(0);
  for (int k = 0; k < my_tiles; k++) {
    const long long tile = blockIdx.x + (long long)k * gridDim.x;
    const long long ir = tile * EV_TILE + threadIdx.x;
    const bool valid = ir < N;
    const long long ip = n_ip;
    float delta = 0.f, xe = 0.f, T = 1.f;
    if (valid) {
      delta = n_delta;
      xe = n_xe;
      T = n_T;
    }
    read_state(k + 1);
    // interpolation bracket in x_HII (ComputeTs.c:761-773)
    float xcall = xe;
    if (xcall > s_xhii[NXHII - 1] * 0.999f)
      xcall = s_xhii[NXHII - 1] * 0.999f;
    else if (xcall < s_xhii[0])
      xcall = 1.001f * s_xhii[0];
    const int lo = xhii_node(s_xhii, xcall), hi = lo + 1;
    const float w = __fdividef(xcall - s_xhii[lo], s_xhii[hi] - s_xhii[lo]);
    float heat = 0.f, ion = 0.f, lya = 0.f, star = 0.f;
    if (light) {
      const bool arrived = bulk::mbar_wait(&bars[k % STAGES], (unsigned)(k / STAGES) & 1u, full);
      if (__syncthreads_or(!arrived)) {
        if (threadIdx.x == 0) {
          atomicOr(a.err, bulk::ERR_PIPELINE_TIMEOUT);
          // copies of tiles k and k + 1 may still be in flight
          for (int j = k; j < my_tiles && j < k + STAGES; j++)
            bulk::mbar_drain(&bars[j % STAGES], (unsigned)(j / STAGES) & 1u);
        }
        return;
      }
      const float* st = stages + (size_t)(k % STAGES) * S * EV_TILE + threadIdx.x;
      const float4* Plo = s_P + lo * S;
      const float4* Phi = s_P + hi * S;
      // heat and ionisation, Ly-alpha and stars at the lower node, the same (stars
      // unused) at the upper one: a packed multiply-add for each pair
      float2 low_hi{}, low_ls{}, up_hi{}, up_ls{};
#pragma unroll 4
      for (int r = 0; r < S; r++) {
        const float sf = st[r * EV_TILE];
        const float4 pl = Plo[r], ph = Phi[r];
        low_hi = fma2(sf, make_float2(pl.x, pl.y), low_hi);
        low_ls = fma2(sf, make_float2(pl.z, pl.w), low_ls);
        up_hi = fma2(sf, make_float2(ph.x, ph.y), up_hi);
        up_ls = fma2(sf, make_float2(ph.z, ph.w), up_ls);
      }
      star = low_ls.y;
      heat = fmaf(w, up_hi.x - low_hi.x, low_hi.x);
      ion = fmaf(w, up_hi.y - low_hi.y, low_hi.y);
      lya = fmaf(w, up_ls.x - low_ls.x, low_ls.x);
      // every thread has read this tile's stage: refill it with tile k + STAGES
      __syncthreads();
      if (threadIdx.x == 0 && k + STAGES < my_tiles)
        ev_issue<STAGES>(bars, stages, a.shells, map, S, N, tile + (long long)STAGES * gridDim.x, k + STAGES);
    }
    if (!valid)
      continue;
    const float opd = 1.0f + delta;
    const float i1xe = __fdividef(1.0f, 1.0f + xe);
    const float dxheat_dzp = heat * i1xe;
    const float dxe_dzp = ion - c.fksink * alpha_A_f(T) * xe * xe * opd;
    float dadia = c.fadia0;
    // fdgrowth / (1/delta + fgrowth), as fdgrowth delta / (1 + fgrowth delta)
    if (fabsf(delta) > (float)FRACT_FLOAT_ERR)
      dadia += __fdividef(c.fdgrowth * delta, 1.0f + c.fgrowth * delta);
    dadia *= (2.0f / 3.0f) * T;
    const float dspec = -dxe_dzp * T * i1xe;
    const float dcomp = c.fccomp * __fdividef(xe, 1.0f + xe + c.ff_he) * (c.ftrad - T);
    const float d1 = dxheat_dzp + dcomp + dspec + dadia;
    const float Jalpha = lya * opd + star;

    xe = xe + dxe_dzp * c.fdzp;
    if (xe > 1.0f)
      xe = (float)(1 - FRACT_FLOAT_ERR);
    else if (xe < 0.0f)
      xe = 0.0f;
    if (T < MAX_TK)
      T = T + d1 * c.fdzp;
    if (T < 0.0f)
      T = c.ftk_floor;
    float TS, xalpha;
    const float lt = logf(T);
    if (!get_Ts_f(c, [&](int i) { return kappa_s(s_kappa, i, lt); }, delta, T, xe, Jalpha, &TS, &xalpha))
      TS = get_Ts_d(c, c.zp, delta, T, xe, Jalpha, &xalpha, a.err);
    a.x_e_prev[ip] = xe;
    a.Tk[ir] = T;
    a.TS[ir] = TS;
    sum[0].add(Jalpha);
    sum[1].add(xalpha);
    sum[2].add(dxheat_dzp);
    sum[3].add(ion);
  }
  double acc[4] = { sum[0].value(), sum[1].value(), sum[2].value(), sum[3].value() };
  block_sum_store<4>(acc, a.partials);
}

// Shared memory of the per-cell kernels, forward and adjoint, with S shells.  The
// function's limit is set to the size for MAX_SHELLS by every call: it belongs to
// the function in the device's context, and a call with fewer shells on another
// thread must not lower it between this call's set and its launch.
template <int STAGES>
static constexpr size_t ev_smem(int S)
{
  return sizeof(float) * (ev_ring_offset(S) + STAGES * (size_t)S * EV_TILE);
}
static constexpr size_t adjoint_smem(int S)
{
  return sizeof(float) * ((2 * ev_tables_floats(S) + 31) / 32 * 32 + 2 * (size_t)S * EV_TILE);
}

// Grid: every SM's resident blocks once (the blocks loop over their tiles),
// at most RED_BLOCKS (the partial-sum slots).
template <int STAGES>
static int launch_evolve_t(const EvolveArgs& a, const GridDims& gd, const bulk::TensorMap& map, int use_map,
                           cudaStream_t s)
{
  const size_t smem = ev_smem<STAGES>(a.n_shells);
  cudaFuncSetAttribute(k_evolve_f32<STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)ev_smem<STAGES>(MAX_SHELLS));
  int dev = 0, sms = 152, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_evolve_f32<STAGES>, RED_THREADS, smem);
  const int blocks = std::max(1, std::min(RED_BLOCKS, std::max(1, per_sm) * sms));
  k_evolve_f32<STAGES><<<blocks, RED_THREADS, smem, s>>>(a, gd.D, gd.H, gd.N, map, use_map);
  return blocks;
}

int launch_evolve(const EvolveArgs& a, const GridDims& gd, const void* shell_map, cudaStream_t s)
{
  bulk::TensorMap map{};
  if (shell_map)
    std::memcpy(&map, shell_map, sizeof(map));
  const int blocks = launch_evolve_t<2>(a, gd, map, shell_map ? 1 : 0, s);
  ts_launches++;
  return blocks;
}

// ======================================================================
// Adjoint of the spin-temperature update and of the 21cm box
// ======================================================================
namespace {

// Value and gradient (d/dTK, d/dxe, d/dJ) of get_Ts_f, by forward-mode
// differentiation of the same iteration (the number of iterations is that of
// the FP32 forward; its stopping test is not differentiated).
struct TsGrad
{
  float TS, dT, dxe, dJ;
};

__device__ TsGrad get_Ts_grad(const TsDevConst& c, const KappaTab& kt, float delta, float TK, float xe, float J)
{
  const float Trad = c.ftrad;
  const float opd = 1.0f + delta;
  float k[3], dk[3];
  const float lt = logf(TK);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    float dln;
    k[i] = kappa_s<true>(kt, i, lt, &dln);
    dk[i] = k[i] * dln / TK;  // d kappa / d TK
  }
  const float xc = c.fxc[0] * ((1.0f - xe) * opd) * k[0] + c.fxc[1] * (xe * opd) * k[1] + c.fxc[2] * (xe * opd) * k[2];
  const float xc_T = c.fxc[0] * ((1.0f - xe) * opd) * dk[0] + c.fxc[1] * (xe * opd) * dk[1] + c.fxc[2] * (xe * opd) * dk[2];
  const float xc_x = opd * (-c.fxc[0] * k[0] + c.fxc[1] * k[1] + c.fxc[2] * k[2]);
  const float iTK = __fdividef(1.0f, TK);
  const float iTrad = __fdividef(1.0f, Trad);
  TsGrad g;
  if (J > 1.0e-20f) {
    const float tgp = c.ftgp * opd * (1.0f - xe);
    const float q = 1.0e-7f * tgp * iTK * iTK;
    const float xi = cbrtf(q);
    // d xi: xi = q^(1/3); dq/dTK = -2 q / TK, dq/dxe = -1e-7 ftgp opd / TK^2
    const float xi_q = q > 0.0f ? xi / (3.0f * q) : 0.0f;
    const float xi_T = xi_q * (-2.0f * q / TK);
    const float xi_x = xi_q * (-1.0e-7f * c.ftgp * opd / TK / TK);
    const float den = 1.0f + 2.98394f * xi + 1.53583f * xi * xi + 3.85289f * xi * xi * xi;
    const float iden = __fdividef(1.0f, den);
    const float den_xi = 2.98394f + 2.0f * 1.53583f * xi + 3.0f * 3.85289f * xi * xi;
    const float den_T = den_xi * xi_T, den_x = den_xi * xi_x;
    const float iTK_T = -iTK * iTK;
    float TS = Trad, TSold = 0.0f;
    float TS_T = 0.f, TS_x = 0.f, TS_J = 0.f;  // d TS
    int it = 0;
    for (;;) {
      const float iTS = __fdividef(1.0f, TS);
      const float rel = fabsf(TS - TSold) * iTS;
      if (!(rel > 1.0e-3f) || ++it > TS_MAX_ITER)
        break;
      TSold = TS;
      const float iTS_T = -iTS * iTS * TS_T, iTS_x = -iTS * iTS * TS_x, iTS_J = -iTS * iTS * TS_J;
      const float num = 1.0f - 0.0631789f * iTK + 0.115995f * iTK * iTK - 0.401403f * iTS * iTK + 0.336463f * iTS * iTK * iTK;
      const float num_iTK = -0.0631789f + 2.0f * 0.115995f * iTK - 0.401403f * iTS + 2.0f * 0.336463f * iTS * iTK;
      const float num_iTS = -0.401403f * iTK + 0.336463f * iTK * iTK;
      const float num_T = num_iTK * iTK_T + num_iTS * iTS_T;
      const float num_x = num_iTS * iTS_x, num_J = num_iTS * iTS_J;
      const float St = num * iden;
      const float St_T = (num_T - St * den_T) * iden, St_x = (num_x - St * den_x) * iden, St_J = num_J * iden;
      const float xa = c.fxa * St * J;
      const float xa_T = c.fxa * St_T * J, xa_x = c.fxa * St_x * J, xa_J = c.fxa * (St_J * J + St);
      // 1 / Tceff = iTK + 0.405535 iTK (iTS - iTK)
      const float E = iTK + 0.405535f * iTK * (iTS - iTK);
      const float E_T = iTK_T + 0.405535f * (iTK_T * (iTS - iTK) + iTK * (iTS_T - iTK_T));
      const float E_x = 0.405535f * iTK * iTS_x, E_J = 0.405535f * iTK * iTS_J;
      const float A = iTrad + xa * E + xc * iTK;
      const float A_T = xa_T * E + xa * E_T + xc_T * iTK + xc * iTK_T;
      const float A_x = xa_x * E + xa * E_x + xc_x * iTK, A_J = xa_J * E + xa * E_J;
      const float B = 1.0f + xa + xc;
      const float B_T = xa_T + xc_T, B_x = xa_x + xc_x, B_J = xa_J;
      TS = __fdividef(B, A);
      const float iA = __fdividef(1.0f, A);
      TS_T = (B_T - TS * A_T) * iA;
      TS_x = (B_x - TS * A_x) * iA;
      TS_J = (B_J - TS * A_J) * iA;
    }
    g.TS = TS;
    g.dT = TS_T;
    g.dxe = TS_x;
    g.dJ = TS_J;
  } else {
    // TS = (1 + xc) / (1/Trad + xc/TK)
    const float A = iTrad + xc * iTK, B = 1.0f + xc;
    g.TS = __fdividef(B, A);
    const float A_T = xc_T * iTK - xc * iTK * iTK, A_x = xc_x * iTK;
    g.dT = (xc_T - g.TS * A_T) / A;
    g.dxe = (xc_x - g.TS * A_x) / A;
    g.dJ = 0.0f;
  }
  if (g.TS < 0.0f) {
    g.TS = -g.TS;
    g.dT = -g.dT;
    g.dxe = -g.dxe;
    g.dJ = -g.dJ;
  }
  return g;
}
}  // namespace

// One thread per cell, tiles of EV_TILE cells with the shell ring of
// k_evolve_f32.  From dL/d(delta_T) of the cell: the 21cm box adjoint
// (BrightnessTemperature.c:495-545) gives dL/dxH and dL/dT_S; dL/dxH reaches
// x_e and stars through the partial ionisation of the last (unfiltered) step
// (find_HII_bubbles.c:416-428) when 0 < xH < 1, the ionisation flags being
// held fixed; dL/dT_S goes back through get_Ts, the x_e / T_K update and the
// shell sums (ComputeTs.c:743-900).  The shell values are overwritten by
// dL/d(shell), zero where the shell was clamped at 0.  Per block: sums of
// heat_bar * heat + ion_bar * ion + lya_bar * lya (the L_X term) and of the
// E0 term with the dP/dE0 tables.
__global__ void __launch_bounds__(RED_THREADS) k_evolve_adjoint(AdjointArgs a, int D, int H, long long N,
                                                                 const __grid_constant__ bulk::TensorMap shell_map,
                                                                 int use_map)
{
  // the gradients of tile k are written in place while the tensor copies
  // read tiles k + 1 and k + 2: different cells
  const bulk::TensorMap* map = use_map ? &shell_map : nullptr;
  const TsDevConst& c = *a.cst;
  const int S = c.S;
  extern __shared__ __align__(128) float sm[];
  float4* s_P = reinterpret_cast<float4*>(sm);              // NXHII * S
  float4* s_dP = s_P + NXHII * S;                            // NXHII * S (d/dE0; w unused)
  float* stages = sm + (2 * ev_tables_floats(S) + 31) / 32 * 32;  // 2 * S * EV_TILE, 128-byte aligned
  __shared__ uint64_t bars[2];
  __shared__ KappaTab s_kappa;
  __shared__ float s_xhii[NXHII];
  fill_kappa(s_kappa, c);
  if (threadIdx.x < NXHII)
    s_xhii[threadIdx.x] = c.xhii[threadIdx.x];
  for (int i = threadIdx.x; i < NXHII * S; i += blockDim.x) {
    const int x = i / S, r = i % S;
    s_P[i] = make_float4(c.fKH[r] * c.ftab[0][x][r], c.fKI[r] * c.ftab[1][x][r], c.fKL[r] * c.ftab[2][x][r],
                         c.fKS[r]);
    s_dP[i] = a.dP_dE0[i];
  }
  const long long ntiles = (N + EV_TILE - 1) / EV_TILE;
  const int my_tiles = blockIdx.x < ntiles ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  const bool light = !c.no_light;
  const bool full = bulk::full_waits();
  if (threadIdx.x == 0 && light) {
    bulk::mbar_init(&bars[0], 1);
    bulk::mbar_init(&bars[1], 1);
    bulk::mbar_init_fence();
  }
  __syncthreads();
  if (threadIdx.x == 0 && light)
    for (int k = 0; k < 2 && k < my_tiles; k++)
      ev_issue(bars, stages, a.shells, map, S, N, blockIdx.x + (long long)k * gridDim.x, k);
  CSum sum[2];
  for (int k = 0; k < my_tiles; k++) {
    const long long tile = blockIdx.x + (long long)k * gridDim.x;
    const long long ir = tile * EV_TILE + threadIdx.x;
    const bool valid = ir < N;
    const long long ip = valid ? pad_index(ir, D, H) : 0;
    float delta = 0.f, xe = 0.f, T = 1.f, gT = 0.f, xH = 1.f, TSf = 1.f;
    if (valid) {
      delta = a.deltax[ip];
      xe = a.x_e_prev[ip];
      T = a.Tk[ir];
      gT = a.grad_dT[ir];
      xH = a.xH[ir];
      TSf = a.TS[ir];
    }
    // 21cm box: dT = cf * xH * (1 + delta) * (1 - Trad / TS)
    const float opd = 1.0f + delta;
    const float A1 = a.dT_factor * xH * opd;
    const float xH_bar = gT * a.dT_factor * opd * (1.0f - a.dT_trad / TSf);
    const float TS_bar = gT * A1 * a.dT_trad / (TSf * TSf);
    // partial ionisation of the last step: xH = (1 - x_e) - stars * kfc / (1 + dx)
    float xe_new_bar = 0.0f, stars_bar = 0.0f;
    if (valid && xH > 0.0f && xH < 1.0f) {
      const float xraw = a.x_e_new[ip];
      if (xraw >= 1e-8f && xraw < 0.999f)
        xe_new_bar = -xH_bar;
      const float sraw = a.stars[ip];
      if (sraw >= 1e-8f)
        stars_bar = -xH_bar * a.kfc_last / (1.0f + fmaxf(delta, -1.0f + 1e-5f));
    }
    if (valid)
      a.grad_stars[ip] = stars_bar;
    // x_HII bracket (ComputeTs.c:761-773)
    float xcall = xe;
    if (xcall > s_xhii[NXHII - 1] * 0.999f)
      xcall = s_xhii[NXHII - 1] * 0.999f;
    else if (xcall < s_xhii[0])
      xcall = 1.001f * s_xhii[0];
    const int lo = xhii_node(s_xhii, xcall), hi = lo + 1;
    const float w = __fdividef(xcall - s_xhii[lo], s_xhii[hi] - s_xhii[lo]);
    float heat = 0.f, ion = 0.f, lya = 0.f, star = 0.f, dheat = 0.f, dion = 0.f, dlya = 0.f;
    const float* st = nullptr;
    if (light) {
      const bool arrived = bulk::mbar_wait(&bars[k & 1], (unsigned)(k >> 1) & 1u, full);
      if (__syncthreads_or(!arrived)) {
        if (threadIdx.x == 0) {
          atomicOr(a.err, bulk::ERR_PIPELINE_TIMEOUT);
          for (int j = k; j < my_tiles && j < k + 2; j++)
            bulk::mbar_drain(&bars[j & 1], (unsigned)(j >> 1) & 1u);
        }
        return;
      }
      st = stages + (size_t)(k & 1) * S * EV_TILE + threadIdx.x;
      float hl = 0.f, il = 0.f, ll = 0.f, hh = 0.f, ih = 0.f, lh = 0.f;
      float dhl = 0.f, dil = 0.f, dll = 0.f, dhh = 0.f, dih = 0.f, dlh = 0.f;
      for (int r = 0; r < S; r++) {
        const float sf = st[r * EV_TILE];
        const float4 pl = s_P[lo * S + r], ph = s_P[hi * S + r];
        const float4 ql = s_dP[lo * S + r], qh = s_dP[hi * S + r];
        hl = fmaf(sf, pl.x, hl);
        il = fmaf(sf, pl.y, il);
        ll = fmaf(sf, pl.z, ll);
        star = fmaf(sf, pl.w, star);
        hh = fmaf(sf, ph.x, hh);
        ih = fmaf(sf, ph.y, ih);
        lh = fmaf(sf, ph.z, lh);
        dhl = fmaf(sf, ql.x, dhl);
        dil = fmaf(sf, ql.y, dil);
        dll = fmaf(sf, ql.z, dll);
        dhh = fmaf(sf, qh.x, dhh);
        dih = fmaf(sf, qh.y, dih);
        dlh = fmaf(sf, qh.z, dlh);
      }
      heat = fmaf(w, hh - hl, hl);
      ion = fmaf(w, ih - il, il);
      lya = fmaf(w, lh - ll, ll);
      dheat = fmaf(w, dhh - dhl, dhl);
      dion = fmaf(w, dih - dil, dil);
      dlya = fmaf(w, dlh - dll, dll);
    }
    // forward of the cell (k_evolve_f32, the same operations), keeping the
    // clamp states
    const float i1xe = __fdividef(1.0f, 1.0f + xe);
    const float dxe_dzp = ion - c.fksink * alpha_A_f(T) * xe * xe * opd;
    float dadia = c.fadia0;
    if (fabsf(delta) > (float)FRACT_FLOAT_ERR)
      dadia += __fdividef(c.fdgrowth * delta, 1.0f + c.fgrowth * delta);
    dadia *= (2.0f / 3.0f) * T;
    const float dspec = -dxe_dzp * T * i1xe;
    const float dcomp = c.fccomp * __fdividef(xe, 1.0f + xe + c.ff_he) * (c.ftrad - T);
    const float d1 = heat * i1xe + dcomp + dspec + dadia;
    const float Jalpha = lya * opd + star;
    float xn = xe + dxe_dzp * c.fdzp;
    bool xe_free = true;
    if (xn > 1.0f) {
      xn = (float)(1 - FRACT_FLOAT_ERR);
      xe_free = false;
    } else if (xn < 0.0f) {
      xn = 0.0f;
      xe_free = false;
    }
    float Tn = T;
    bool T_free = T < MAX_TK;
    if (T_free)
      Tn = T + d1 * c.fdzp;
    if (Tn < 0.0f) {
      Tn = c.ftk_floor;
      T_free = false;
    }
    const TsGrad tg = get_Ts_grad(c, s_kappa, delta, Tn, xn, Jalpha);
    // backward
    const float Tn_bar = TS_bar * tg.dT;
    xe_new_bar += TS_bar * tg.dxe;
    const float J_bar = TS_bar * tg.dJ;
    const float d1_bar = T_free ? Tn_bar * c.fdzp : 0.0f;
    const float dxe_bar = (xe_free ? xe_new_bar * c.fdzp : 0.0f) + d1_bar * (-T * i1xe);
    const float heat_bar = d1_bar * i1xe;
    const float ion_bar = dxe_bar;
    const float lya_bar = J_bar * opd;
    const float star_bar = J_bar;
    if (light) {
      // dL/d(shell r), zero where the shell was clamped at 0
      for (int r = 0; r < S; r++) {
        const float sf = st[r * EV_TILE];
        const float4 pl = s_P[lo * S + r], ph = s_P[hi * S + r];
        float u = heat_bar * fmaf(w, ph.x - pl.x, pl.x) + ion_bar * fmaf(w, ph.y - pl.y, pl.y) +
                  lya_bar * fmaf(w, ph.z - pl.z, pl.z) + star_bar * pl.w;
        if (!(sf > 0.0f) || !valid)
          u = 0.0f;
        if (valid)
          a.shells[(long long)r * N + ir] = u;
      }
      __syncthreads();
      if (threadIdx.x == 0 && k + 2 < my_tiles)
        ev_issue(bars, stages, a.shells, map, S, N, tile + 2LL * gridDim.x, k + 2);
    }
    if (valid) {
      sum[0].add(fmaf(heat_bar, heat, fmaf(ion_bar, ion, lya_bar * lya)));
      sum[1].add(fmaf(heat_bar, dheat, fmaf(ion_bar, dion, lya_bar * dlya)));
    }
  }
  double acc[2] = { sum[0].value(), sum[1].value() };
  block_sum_store<2>(acc, a.partials);
}

void launch_evolve_adjoint(const AdjointArgs& a, const GridDims& gd, const void* shell_map, cudaStream_t s)
{
  const size_t smem = adjoint_smem(a.n_shells);
  cudaFuncSetAttribute(k_evolve_adjoint, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adjoint_smem(MAX_SHELLS));
  bulk::TensorMap map{};
  if (shell_map)
    std::memcpy(&map, shell_map, sizeof(map));
  k_evolve_adjoint<<<RED_BLOCKS, RED_THREADS, smem, s>>>(a, gd.D, gd.H, gd.N, map, shell_map ? 1 : 0);
  ts_launches++;
}

int ts_kernel_launches() { return ts_launches; }

cudaError_t ts_set_wait_polls(long long polls) { return bulk::set_consumer_wait_polls(polls); }

// Homogeneous branch, ComputeTs.c:189-262: x_e and T_K from RECFAST, T_S with
// J_alpha = 0 (no iteration), and the collapse fraction.
__global__ void k_homog_f32(HomogArgs a, int D, int H, long long N)
{
  const TsDevConst& c = *a.cst;
  CSum sum;
  const float kcf = (float)((4.0 / 3.0) * 3.14159265358979323846 * a.R3 / a.pixel_volume / a.RtoM_h2);
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long ip = pad_index(ir, D, H);
    const float delta = a.deltax[ip];
    a.x_e_prev[ip] = a.xe0;
    a.Tk[ir] = a.tk0;
    float TS, xa;
    if (!get_Ts_f(c, [&](int i) { return kappa_f(c, i, a.tk0); }, delta, a.tk0, a.xe0, 0.0f, &TS, &xa))
      TS = get_Ts_d(c, c.zp, delta, a.tk0, a.xe0, 0.0f, &xa, a.err);
    a.TS[ir] = TS;
    const float cf = fminf(a.stars[ip] * kcf / (1.0f + delta), 1.0f);
    sum.add(cf);
  }
  double acc[1] = { sum.value() };
  block_sum_store<1>(acc, a.partials);
}

void launch_homog(const HomogArgs& a, const GridDims& gd, cudaStream_t s)
{
  k_homog_f32<<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, gd.D, gd.H, gd.N);
  ts_launches++;
}

}  // namespace mx
