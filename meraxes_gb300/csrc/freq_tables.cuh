// Frequency-integral tables of ComputeTs on the device (see freq_tables.cu).
#pragma once

#include <cuda_runtime.h>

#include "host_physics.h"
#include "kernels.cuh"

namespace mx {

constexpr int FREQ_SETS = 3;  // X-ray thresholds E0 of one call (the adjoint needs three)
constexpr int FREQ_INTERVALS = 128;  // intervals of one adaptive integral that the kernels hold
constexpr int FREQ_TAB = 3 * k::NXHII;  // rows of a set: tab[(flag * 14 + x) * S + r]

// Cross sections as polynomials: a sixteenth of an octave in nu / NU_HI per
// interval, XS_N coefficients in its local coordinate (-1 ... 1), from 1.5
// times the species' threshold (below, the formulas) to 2^17 NU_HI.
constexpr int XS_SUB = 16, XS_OCTAVES = 17, XS_INTERVALS = XS_SUB * XS_OCTAVES, XS_N = 10;

// The secondary-electron tables, the bin edges of their energy index, and the
// cross sections of HI, HeI and HeII (xs), and times (nu / NU_HI)^(-alpha - 1)
// (xs_spec).
struct FreqDevTables
{
  double xs[3][XS_INTERVALS][XS_N], xs_spec[3][XS_INTERVALS][XS_N];
  float4 bin[k::NENERGY];  // smallest energy of index n (loc_energy), of n + 1; energy n; unused
  float energy_cap, energy_top;  // energies above cap are looked up at top
  float xhii[k::NXHII];
  // value at an energy, slope to the next
  float2 fheat[k::NXHII][k::NENERGY], nlya[k::NXHII][k::NENERGY];
  float2 nion[3][k::NXHII][k::NENERGY];
};
void fill_freq_dev_tables(const HeatTables& ht, double alpha, FreqDevTables* t);

// What the kernels write: the frequency of unit optical depth of each shell,
// the tables (S entries per row), and whether an integral needed more
// intervals than the kernels hold (then the host builds the tables).
struct FreqDevResult
{
  double nu1[MAX_SHELLS];
  double tab[FREQ_SETS][FREQ_TAB * MAX_SHELLS];
  int fail;
};

struct FreqArgs
{
  const FreqDevTables* tables;  // device
  const double* sums;           // device: sum of f_coll and of x_e over the cells
  double total;                 // cells
  int S, n_sets;
  int intervals;  // at most FREQ_INTERVALS; fewer in a test of the host fallback
  double zp, zpp[MAX_SHELLS];
  double E0[FREQ_SETS];    // NuXrayGalThreshold [eV]
  double spec[FREQ_SETS];  // (NU_HI / E0)^(-alpha - 1)
  double alpha, numax, hubble;
  double om, ol, hubble_h, n_b0, f_h, f_he, eff;
  // collapse fraction over redshift (interpolate_fcoll): linear from fcoll0 at
  // z0 to this snapshot's at z1; constant for the first snapshot
  int first_snapshot;
  double fcoll0, z0, z1;
  FreqDevResult* out;  // device
};
FreqArgs make_freq_args(const mx_params& p, const Derived& d, const std::vector<double>& zz, const double* stored_fcoll,
                        int snapshot, const ShellPlan& sp);
void launch_freq_tables(const FreqArgs& a, cudaStream_t s);
int freq_kernel_launches();

}  // namespace mx
