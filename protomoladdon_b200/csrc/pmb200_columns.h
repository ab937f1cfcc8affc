// Host interface of the column kernels (pmb200_columns.cu).
#pragma once
#include "pmb200_columns.cuh"

namespace pmb200 {

// What a launch of the pair kernel needs beside the grid.
struct ColLaunch {
  int form, ntypes;
  bool full, mod;          // both switches end at the cutoff; modified pairs exist
  bool energy, virial, molvir;
  const float4 *lj32;      // unit-scaled tables
  const double2 *lj64;     // {A, B} of every type pair, then {A14, B14}
  const int *ctl;          // [0]: clusters in use
  int *count;              // column counts (cleared)
  int lsplit;              // log2 of the warps per cluster
  ColShare share;
  int clusters;            // upper bound of the clusters of the share
  double *partial;
};

cudaError_t col_launch_pair(const ColGrid &g, const MixedConsts &mc, const ColArrays &a,
                             const ColLaunch &l, cudaStream_t stream, bool pdl);

// The batch's pair kernel: launched on `grid` blocks, or (occ non-null) only
// its resident blocks per SM.
struct ColBatchLaunch {
  int form;
  bool full, mod, energy, virial;
  const ColBatchSys *sys;
  const int4 *tasks;
  int ntasks;
  int *counter;
  const short2 *st;
  const float4 *lj32;
  const double2 *lj64;
  const int *ctl;
  int *count;
  int ncol, lj_max, grid;
  double *partial;
};
cudaError_t col_launch_batch(const ColArrays &a, const ColBatchLaunch &l, cudaStream_t stream,
                             int *occ);

// The FP64 kernels (pmb200_columns64.cuh).
struct Col64Launch {
  int form, ntypes;
  bool full;               // cutoff form: both switches end at the cutoff, no modified pairs
  bool energy, pdl;
  const double4 *lj64;     // {A, B, A14, B14}
  unsigned long long *acc; // [8][n]
  const int *ctl;
  int *count;
  int lsplit, clusters;
  double *partial, *tpart;
};
cudaError_t col_launch_pair64(const ColGrid &g, const Fp64Consts &mc, const ColArrays &a,
                              const Col64Launch &l, cudaStream_t stream);
cudaError_t col_launch_deriv64(const ColGrid &g, const Fp64Consts &mc, const ColArrays &a,
                               const Col64Launch &l, int mode, bool params, cudaStream_t stream);

}  // namespace pmb200
