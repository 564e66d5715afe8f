// Fused 3-D transforms for power-of-two grids and grids with a factor 3
// (see fft3d.cu).
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace mx {

// Band limits of a batch of filtered spectra.  The k-space top-hat is exactly
// zero beyond kR = 1 / 0.413566994, and the Gaussian underflows to zero; modes
// with kx^2 + ky^2 + kz^2 > m2[r] (in units of the fundamental) of radius r are
// zero.  The passes then leave out the tiles (16 kz columns from kz0 = 16 j)
// that hold no mode, and, with `compact`, store the spectra of radius r in rows
// of 16 nt[r] complex values instead of fft_pitch(D).  Without `compact` the
// y-pass fills the tiles that are left out with zeros.
constexpr int MAX_BANDED = MAX_SHELLS;
struct Bands
{
  int n = 0;  // radii; 0: no band limit
  int compact = 0;
  float m2[MAX_BANDED];
  unsigned short nt[MAX_BANDED];     // tiles with kz0^2 <= m2
  unsigned xstart[MAX_BANDED + 1];   // x-pass tiles (|ky|, kz0) before radius r
  unsigned ystart[MAX_BANDED + 1];   // y-pass tiles (field, x, kz0) before radius r
};
// Band limits of n radii R of a filter (none if the filter has no limit, n is
// above MAX_BANDED, or no tile can be left out); G fields per radius.
Bands filter_bands(int D, int filter_type, const float* R, int n, int G, float delta_k, bool compact);

// x-pass: filter + 1/N scale + inverse FFT along x for a batch of radii.
struct XPassArgs
{
  const float2* in[MAX_FIELDS];  // unfiltered, unnormalised half spectra, rows of fft_pitch(D)
  int G;                          // fields
  int n;                          // radii in the batch
  float2* out;                    // spectrum (r*G + g) at out + (r*G + g)*C
  long long C;                    // D * D * fft_pitch(D)
  float R[MAX_RADII];
  int apply[MAX_RADII];
  int filter_type;
  float delta_k;
  float scale;       // 1/N (exact for power-of-two N)
  float sharpk_max;  // set by launch_fft_x_filter
  Bands bands;
};

// Forward R2C of G padded real grids into spectra [kx][ky][kz] with rows of
// fft_pitch(D) complex values (the x-pass's input layout).
struct FwdArgs
{
  const float* src[MAX_FIELDS];  // PADDED real grids (8-byte aligned)
  int G;
  float2* out;  // spectrum g at out + g * C
  long long C;  // D * D * fft_pitch(D)
  // modes that are read of the spectra: kz < 16 nt, |ky| <= ny (0: all)
  int nt = 0, ny = 0;
};

// z-pass fused with the find_HII_bubbles per-cell test.
struct ZThresholdArgs
{
  const float2* spectra;  // batch spectra after the x and y passes
  long long C;
  int G, idx_xe, idx_nr;  // fields deltax, stars, weighted_sfr, [x_e if spin], [N_rec if recomb]
  int n_r;  // radii of the batch
  int n_f;  // of which filtered (spectra r*G + g for r < n_f); a last radius
            // with rp.last set reads the input grids directly
  const RadiusParams* rp;
  const float* direct[MAX_FIELDS];  // PADDED input grids for the unfiltered step
  float* xH;
  float* z_at_ion;
  float* r_bubble;
  float* J21;
  float* J21_at_ion;
  float* Gamma12;
  double pixel_volume, eff, redshift;
  float gamma_halo_bias;
  int uvb, recomb, spin;
  unsigned* err;  // bit 2: a pipeline wait timed out
  // row groups [group0, group0 + n_groups) of fft_z_row_groups(D) (n_groups
  // 0: all), so that a launch can cover a slab of rows
  int group0 = 0, n_groups = 0;
  // register budget of the launch: 2 or 3 resident blocks per SM
  int blocks_per_sm = 2;
};

bool fft3d_supported(int D);
// Row pitch (complex values) of the spectra between the fused passes: D/2 + 1
// rounded up to whole 128-byte lines.  A batch spectrum holds D * D * pitch.
int fft_pitch(int D);
// acc = (first ? 0 : acc) + W(|k| R) * scale * U on a half spectrum (any D);
// the filter of the x-pass
void launch_filter_accumulate(int D, float2* acc, const float2* U, float R, int filter_type, float delta_k,
                              float scale, bool first, cudaStream_t s);
// threads per tile of the passes of a power-of-two grid: 256 or 512, and for
// the x-pass at 64^3 and 128^3 also 128 (two tiles to a block of 256)
bool fft_x_threads_ok(int D, int threads);
bool launch_fft_x_filter(int D, const XPassArgs& a, int threads, cudaStream_t s);
bool launch_fft_y(int D, float2* data, long long C, int n_spectra, const Bands& bands, int threads, cudaStream_t s);
// three launches: z (real rows -> half spectrum), y, x; threads of the y and
// x passes 256 or 512
bool launch_fft_forward(int D, const FwdArgs& a, int threads, cudaStream_t s);
bool launch_fft_z_threshold(int D, const ZThresholdArgs& a, cudaStream_t s);
bool launch_fft_z_store(int D, const float2* spectra, long long C, int n, int r0, const Bands& bands, float* shells,
                        long long N, unsigned* err, cudaStream_t s);
// row groups of the threshold z-pass and rows (x * D + y) per group
int fft_z_row_groups(int D);
int fft_z_rows_per_group(int D);
int fft_kernel_launches();
// Sets the poll limit of this unit's pipeline waits (bulk.cuh).
cudaError_t fft_set_wait_polls(long long polls);

}  // namespace mx
