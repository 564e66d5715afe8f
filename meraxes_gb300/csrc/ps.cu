// 21 cm power spectrum of delta_T: Compute_PS (ComputePowerSpectrum.c:44-255).
//
//   1. mean of delta_T (two-stage fixed-order FP64 sum);
//   2. the field delta_T - mean into the padded layout (its factor V / N is
//      applied to the sums);
//   3. R2C (cuFFT, in mx_reion.cu);
//   4. the binned sums over the half spectrum: every mode (kx, ky, kz <= D/2)
//      is counted once, |k| in float as the reference computes it, bins of
//      ratio 1.35 from delta_k (edges computed on the host in float by the
//      reference's recurrence), k^3 |X|^2 / (2 pi^2 V) and |k| summed in FP64.
//
// The binned sums are deterministic: a warp owns whole rows (kx, ky); lane l
// visits kz = l, l + 32, ... whose |k| increases, so its bin index never
// decreases along a row; it accumulates runs in registers and adds each run
// to its private histogram.  Histograms are reduced per block in a fixed
// order, then over blocks in a fixed order.
#include "ps.cuh"

namespace mx {

namespace {
// per host thread: a call counts its own launches when contexts run concurrently
thread_local int ps_launches = 0;

// SUM_BATCH cells of a thread's stride are read together
constexpr int SUM_BATCH = 8;
__global__ void k_ps_sum(const float* __restrict__ dT, long long N, double* partials)
{
  __shared__ double sh[RED_THREADS / 32];
  CSum sum;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < N; i0 += SUM_BATCH * stride) {
    float v[SUM_BATCH];
#pragma unroll
    for (int u = 0; u < SUM_BATCH; u++)
      v[u] = i0 + u * stride < N ? dT[i0 + u * stride] : 0.0f;
#pragma unroll
    for (int u = 0; u < SUM_BATCH; u++)
      sum.add(v[u]);
  }
  double acc = sum.value();
  for (int o = 16; o > 0; o >>= 1)
    acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0)
    sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < RED_THREADS / 32; w++)
      s += sh[w];
    partials[blockIdx.x] = s;
  }
}

// sums[v] = sum over blocks of partials[b * nvals + v], fixed order, a warp per
// value (see k_finalize, kernels.cu)
constexpr int FIN_WARPS = 4;
__global__ void __launch_bounds__(32 * FIN_WARPS) k_ps_finalize(const double* __restrict__ partials, int nblocks,
                                                                int nvals, double* __restrict__ sums)
{
  const int lane = threadIdx.x & 31, v = blockIdx.x * FIN_WARPS + (threadIdx.x >> 5);
  if (v >= nvals)
    return;
  double s = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblocks; b += 32)
    s += partials[(long long)b * nvals + v];
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0)
    sums[v] = s;
}

// The field of ComputePowerSpectrum.c:94-110, (dT / ave - 1) V / N ave, without
// its constant factor V / N (the binned sums take it squared, in FP64): dT less ave
// as a float.  What that leaves out of ave is the same in every cell and enters the
// k = 0 mode alone, whose power is k^3 = 0 times it; taken in, it would round in
// every ionised cell (dT = 0) to the same side.  A mean of 0 (a fully ionised box)
// makes every cell's quotient infinite or NaN and the field NaN, as written there.
// In FP64 as written, the quotient per cell bound the pass (507 us at 200^3).
__global__ void k_ps_field(const float* __restrict__ dT, const double* __restrict__ sum, double n_cells, int D, int H,
                           long long N, float* __restrict__ out)
{
  const double mean = sum[0] / n_cells;
  const float ave = mean == 0.0 ? __int_as_float(0x7fffffff) : (float)mean;
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    out[row * 2LL * H + (ir - row * D)] = __fsub_rn(dT[ir], ave);
  }
}

__device__ __forceinline__ float kcomp_ps(int n, int D, float delta_k)
{
  return (n > D / 2) ? __fmul_rn((float)(n - D), delta_k) : __fmul_rn((float)n, delta_k);
}

// ComputePowerSpectrum.c:160-215: sums of k^3 |X|^2, |k| and the modes of each
// bin; the constant 1 / (2 pi^2 V) is applied to the sums by the caller.  Bound
// by FP64 issue, now nine operations per mode (with that quotient, the count and
// the cube's square in FP64 per mode, 371 us at 200^3).
__global__ void __launch_bounds__(RED_THREADS) k_ps_bin(PsArgs a)
{
  double hp[PS_MAX_BINS], hk[PS_MAX_BINS];
  int hc[PS_MAX_BINS];
  for (int b = 0; b < a.nb; b++) {
    hp[b] = hk[b] = 0.0;
    hc[b] = 0;
  }
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (RED_THREADS / 32);
  const int D = a.D, H = D / 2 + 1;
  const long long rows = (long long)D * D;
  for (long long row = blockIdx.x * (RED_THREADS / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const int nx = (int)((unsigned)row / (unsigned)D), ny = (int)row - nx * D;
    const float kx = kcomp_ps(nx, D, a.delta_k), ky = kcomp_ps(ny, D, a.delta_k);
    // k_x*k_x + k_y*k_y + k_z*k_z in the reference's float operations (no
    // fused multiply-add)
    const float kxy = __fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky));
    const float2* __restrict__ spec = a.spec + row * H;
    int cur = 0, count = 0;  // |k| grows along a lane's modes, and so does its bin
    double sp = 0.0, sk = 0.0;
    auto flush = [&]() {
      if (count) {
        hp[cur] += sp;
        hk[cur] += sk;
        hc[cur] += count;
      }
      sp = sk = 0.0;
      count = 0;
    };
    for (int nz = lane; nz < H; nz += 32) {
      const float kz = __fmul_rn((float)nz, a.delta_k);
      // (float)sqrt((double)s) of the reference equals sqrtf(s): the double
      // square root of a float has enough bits that rounding it again to
      // float gives the correctly rounded float root
      const float kmag = sqrtf(__fadd_rn(kxy, __fmul_rn(kz, kz)));
      if (!(kmag < a.edges[a.nb]))
        break;
      if (!(kmag < a.edges[cur + 1])) {
        flush();
        do
          cur++;
        while (!(kmag < a.edges[cur + 1]));
      }
      const float2 X = spec[nz];
      const double k = (double)kmag, x = (double)X.x, y = (double)X.y;
      sp = fma(k * k * k, fma(x, x, y * y), sp);
      sk += k;
      count++;
    }
    flush();
  }
  // block reduction in a fixed order: the threads' values of one quantity
  // through shared memory, a warp per bin (eight values per lane, then a tree);
  // a tree over every warp's lanes took as many FP64 additions as the modes
  extern __shared__ double sh[];  // nb x RED_THREADS
  const int warp = threadIdx.x >> 5;
  for (int q = 0; q < 3; q++) {
    for (int b = 0; b < a.nb; b++)
      sh[b * RED_THREADS + threadIdx.x] = q == 0 ? hp[b] : (q == 1 ? hk[b] : (double)hc[b]);
    __syncthreads();
    for (int b = warp; b < a.nb; b += RED_THREADS / 32) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < RED_THREADS / 32; w++)
        v += sh[b * RED_THREADS + w * 32 + lane];
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0)
        a.partials[(long long)blockIdx.x * 3 * a.nb + q * a.nb + b] = v;
    }
    __syncthreads();
  }
}
// f = dT * scale into the padded layout (the power-spectrum loss field)
__global__ void k_ps_scale(const float* __restrict__ dT, float scale, int D, int H, long long N, float* __restrict__ out)
{
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    out[row * 2LL * H + (ir - row * D)] = dT[ir] * scale;
  }
}

// Gradient spectrum of the binned loss: Y_k = coef[b] k^3 X_k on the modes of
// bin b (the binning of k_ps_bin), times 2 on the kz = 0 and kz = D/2 planes,
// which a C2R counts once where it counts the others twice.  In place.
__global__ void k_ps_loss_grad(PsArgs a, const double* __restrict__ coef, float2* __restrict__ spec)
{
  const int D = a.D, H = D / 2 + 1;
  const long long n = (long long)D * D * H;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int nz = (int)(i % H);
    const long long row = i / H;
    const int nx = (int)(row / D), ny = (int)(row % D);
    const float kx = kcomp_ps(nx, D, a.delta_k), ky = kcomp_ps(ny, D, a.delta_k);
    const float kz = __fmul_rn((float)nz, a.delta_k);
    const float kmag = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky)), __fmul_rn(kz, kz)));
    float f = 0.0f;
    if (kmag < a.edges[a.nb]) {
      int b = 0;
      while (!(kmag < a.edges[b + 1]))
        b++;
      const double k = (double)kmag;
      f = (float)(coef[b] * k * k * k * ((nz == 0 || 2 * nz == D) ? 2.0 : 1.0));
    }
    float2 x = spec[i];
    spec[i] = make_float2(x.x * f, x.y * f);
  }
}

// REAL out = PADDED in * scale
__global__ void k_padded_to_real(const float* __restrict__ in, float scale, int D, int H, long long N,
                                 float* __restrict__ out)
{
  for (long long ir = blockIdx.x * (long long)blockDim.x + threadIdx.x; ir < N; ir += (long long)gridDim.x * blockDim.x) {
    const long long row = row_of(ir, D);
    out[ir] = in[row * 2LL * H + (ir - row * D)] * scale;
  }
}
}  // namespace

void launch_ps_mean(const float* dT, long long N, double* partials, double* sum, cudaStream_t s)
{
  k_ps_sum<<<RED_BLOCKS, RED_THREADS, 0, s>>>(dT, N, partials);
  k_ps_finalize<<<1, 32 * FIN_WARPS, 0, s>>>(partials, RED_BLOCKS, 1, sum);
  ps_launches += 2;
}

void launch_ps_field(const float* dT, const double* sum, const GridDims& gd, float* out, cudaStream_t s)
{
  k_ps_field<<<RED_BLOCKS, RED_THREADS, 0, s>>>(dT, sum, (double)gd.N, gd.D, gd.H, gd.N, out);
  ps_launches++;
}

cudaError_t launch_ps_bin(const PsArgs& a, double* sums, cudaStream_t s)
{
  const size_t smem = sizeof(double) * RED_THREADS * (size_t)a.nb;
  // the limit belongs to the function, not to the call: every caller sets the same
  // one, or a call on another thread with fewer bins could lower it before this
  // launch and make the launch fail
  constexpr size_t smem_max = sizeof(double) * RED_THREADS * (size_t)PS_MAX_BINS;
  const cudaError_t e =
    cudaFuncSetAttribute(k_ps_bin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
  if (e != cudaSuccess)
    return e;
  k_ps_bin<<<RED_BLOCKS, RED_THREADS, smem, s>>>(a);
  k_ps_finalize<<<(3 * a.nb + FIN_WARPS - 1) / FIN_WARPS, 32 * FIN_WARPS, 0, s>>>(a.partials, RED_BLOCKS, 3 * a.nb, sums);
  ps_launches += 2;
  return cudaSuccess;
}

void launch_ps_scale(const float* dT, float scale, const GridDims& gd, float* out, cudaStream_t s)
{
  k_ps_scale<<<RED_BLOCKS, RED_THREADS, 0, s>>>(dT, scale, gd.D, gd.H, gd.N, out);
  ps_launches++;
}

void launch_ps_loss_grad(const PsArgs& a, const double* coef, float2* spec, cudaStream_t s)
{
  k_ps_loss_grad<<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, coef, spec);
  ps_launches++;
}

void launch_padded_to_real(const float* in, float scale, const GridDims& gd, float* out, cudaStream_t s)
{
  k_padded_to_real<<<RED_BLOCKS, RED_THREADS, 0, s>>>(in, scale, gd.D, gd.H, gd.N, out);
  ps_launches++;
}

int ps_kernel_launches() { return ps_launches; }

}  // namespace mx
