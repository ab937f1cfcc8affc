// Launches of the column pair kernels: the template instance for the form,
// the outputs and the topology.
#include "pmb200_columns.h"

namespace pmb200 {

namespace {

template <int F, bool E, bool V, bool M, bool FULL, bool MOD, bool G>
cudaError_t launch(const ColGrid &g, const MixedConsts &mc, const ColArrays &a, const ColLaunch &l,
                   cudaStream_t stream, bool pdl) {
  constexpr bool lj = F == FORM_CUTOFF || F == FORM_GENERIC, exact = E && F == FORM_CUTOFF;
  const size_t t2 = lj && !G ? (size_t)l.ntypes * l.ntypes : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.clusters << l.lsplit);
  cfg.blockDim = dim3(32);
  cfg.dynamicSmemBytes = ColLayout<exact, M>::bytes +
                         t2 * (sizeof(float4) + (exact ? (MOD ? 2 : 1) * sizeof(double2) : 0));
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (pdl && PMB200_PDL) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_col_pair<F, E, V, M, FULL, MOD, G>, g, mc, l.ntypes,
                            l.lj32, l.lj64, a, l.ctl, l.count, l.lsplit, l.share, l.partial);
}

template <int F, bool FULL, bool MOD, bool G>
cudaError_t flags(const ColGrid &g, const MixedConsts &mc, const ColArrays &a, const ColLaunch &l,
                  cudaStream_t stream, bool pdl) {
  if (l.molvir) return launch<F, true, true, true, FULL, MOD, G>(g, mc, a, l, stream, pdl);
  if (l.virial && l.energy)
    return launch<F, true, true, false, FULL, MOD, G>(g, mc, a, l, stream, pdl);
  if (l.virial) return launch<F, false, true, false, FULL, MOD, G>(g, mc, a, l, stream, pdl);
  if (l.energy) return launch<F, true, false, false, FULL, MOD, G>(g, mc, a, l, stream, pdl);
  return launch<F, false, false, false, FULL, MOD, G>(g, mc, a, l, stream, pdl);
}

}  // namespace

cudaError_t col_launch_pair(const ColGrid &g, const MixedConsts &mc, const ColArrays &a,
                            const ColLaunch &l, cudaStream_t stream, bool pdl) {
  const bool big = l.ntypes > kMaxTypes;
#define PMB_COL(F, FULL, MOD, G) return flags<F, FULL, MOD, G>(g, mc, a, l, stream, pdl)
  switch (l.form) {
    case FORM_CUTOFF:
      if (big) PMB_COL(FORM_CUTOFF, false, true, true);  // (tables read through L1)
      if (l.mod || !l.full) PMB_COL(FORM_CUTOFF, false, true, false);
      PMB_COL(FORM_CUTOFF, true, false, false);
    case FORM_GENERIC:
      if (big) PMB_COL(FORM_GENERIC, false, true, true);
      PMB_COL(FORM_GENERIC, false, true, false);
    case FORM_EWALD_POLY5: PMB_COL(FORM_EWALD_POLY5, true, true, false);
    default: PMB_COL(FORM_EWALD_EXACT, true, true, false);
  }
#undef PMB_COL
}

namespace {

template <int F, bool E, bool V, bool FULL, bool MOD>
cudaError_t launch_batch(const ColArrays &a, const ColBatchLaunch &l, cudaStream_t stream,
                         int *occ) {
  constexpr bool lj = F == FORM_CUTOFF || F == FORM_GENERIC, exact = E && F == FORM_CUTOFF;
  const size_t smem = ColLayout<exact, false>::bytes + (sizeof(ColBatchSys) + 15) / 16 * 16 +
                      (lj ? (size_t)l.lj_max : 0) *
                          (sizeof(float4) + (exact ? (MOD ? 2 : 1) * sizeof(double2) : 0));
  auto kernel = k_col_pair_batch<F, E, V, FULL, MOD>;
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kernel, 32, smem);
  kernel<<<l.grid, 32, smem, stream>>>(l.sys, l.tasks, l.ntasks, l.counter, l.st, l.lj32, l.lj64,
                                       a, l.ctl, l.count, l.ncol, l.lj_max, l.partial);
  return cudaGetLastError();
}

template <int F, bool FULL, bool MOD>
cudaError_t flags_batch(const ColArrays &a, const ColBatchLaunch &l, cudaStream_t stream,
                        int *occ) {
  if (l.energy && l.virial) return launch_batch<F, true, true, FULL, MOD>(a, l, stream, occ);
  if (l.energy) return launch_batch<F, true, false, FULL, MOD>(a, l, stream, occ);
  if (l.virial) return launch_batch<F, false, true, FULL, MOD>(a, l, stream, occ);
  return launch_batch<F, false, false, FULL, MOD>(a, l, stream, occ);
}

}  // namespace

cudaError_t col_launch_batch(const ColArrays &a, const ColBatchLaunch &l, cudaStream_t stream,
                             int *occ) {
  if (l.form == FORM_GENERIC) return flags_batch<FORM_GENERIC, false, true>(a, l, stream, occ);
  if (l.form == FORM_EWALD_POLY5)
    return flags_batch<FORM_EWALD_POLY5, true, true>(a, l, stream, occ);
  if (l.form == FORM_EWALD_EXACT)
    return flags_batch<FORM_EWALD_EXACT, true, true>(a, l, stream, occ);
  if (l.mod || !l.full) return flags_batch<FORM_CUTOFF, false, true>(a, l, stream, occ);
  return flags_batch<FORM_CUTOFF, true, false>(a, l, stream, occ);
}

}  // namespace pmb200
