// Galaxy -> grid deposit and the Mvir_crit grid (see deposit.cu).
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace mx {

struct DepositArgs
{
  int n;                 // galaxies
  const float* pos;      // [n][3], Mpc/h
  const int* type;       // galaxies of type > 2 are skipped
  const double* fesc_gsm;
  const double* gross_sm;  // read only with the sfr grid
  const double* bhm;       // read only with BH feedback
  const double* ebhm;
  int flag_bh;
  double bh_limit;
  double alpha_uv_bh;
  double alpha_uv;
  double box_size;
  int spin;              // also deposit the sfr grid and its history slice 0
  double sfr_timescale;  // internal time units
  unsigned* keys_in;     // [n] REAL cell index, or the number of cells (skipped)
  unsigned* keys;        // [n] sorted
  int* idx_in;           // [n]
  int* idx;              // [n] sorted
  unsigned* err;         // bit 4: a galaxy below the box
  float* stars;          // PADDED outputs
  float* weighted_sfr;
  float* sfr;
  float* sfr_hist0;      // SFR history, newest slice first, or NULL
  int n_hist;            // its slices
  int shift_history;     // move them one snapshot back first
};

constexpr unsigned DEPOSIT_ERR_BELOW_BOX = 4u;

// CUB temporary storage for sorting n galaxies (bytes)
size_t deposit_sort_bytes(int n);
// Clears the padded grids and shifts the history on `side` (forked from and
// joined to s by the two events), sorts on s, sums and writes.
cudaError_t launch_deposit(const DepositArgs& a, void* sort_tmp, size_t sort_bytes, const GridDims& gd,
                           cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join);
// sm = {m0, a, b, c, d} of the Sobacchi & Mesinger (2013) fit
void launch_Mvir_crit(double redshift, const double sm[5], double hubble_h, const float* J21_at_ion,
                      const float* z_at_ion, float* out, const GridDims& gd, cudaStream_t s);
int deposit_kernel_launches();

}  // namespace mx
