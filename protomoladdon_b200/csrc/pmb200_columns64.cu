// Launches of the FP64 column kernels.
#include "pmb200_columns64.cuh"
#include "pmb200_columns.h"

namespace pmb200 {

namespace {

template <class K>
cudaError_t launch(K kernel, const Col64Launch &l, const ColGrid &g, const Fp64Consts &mc,
                   const ColArrays &a, size_t entries, cudaStream_t stream, double *out) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.clusters << l.lsplit);
  cfg.blockDim = dim3(32);
  cfg.dynamicSmemBytes =
      entries + (l.ntypes <= kCol64LjTypes ? sizeof(double4) * (size_t)l.ntypes * l.ntypes : 0);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (l.pdl && PMB200_PDL) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, g, mc, l.ntypes, l.lj64, a, l.acc, l.ctl, l.count,
                            l.lsplit, out);
}

template <int F, bool FULL>
cudaError_t pair(const Col64Launch &l, const ColGrid &g, const Fp64Consts &mc, const ColArrays &a,
                 cudaStream_t stream) {
  constexpr size_t entries = ColLayout64<false>::bytes;
  if (l.energy)
    return launch(k_col_pair64<F, true, FULL>, l, g, mc, a, entries, stream, l.partial);
  return launch(k_col_pair64<F, false, FULL>, l, g, mc, a, entries, stream, l.partial);
}

}  // namespace

cudaError_t col_launch_pair64(const ColGrid &g, const Fp64Consts &mc, const ColArrays &a,
                              const Col64Launch &l, cudaStream_t stream) {
  switch (l.form) {
    case FORM_CUTOFF:
      return l.full ? pair<FORM_CUTOFF, true>(l, g, mc, a, stream)
                    : pair<FORM_CUTOFF, false>(l, g, mc, a, stream);
    case FORM_GENERIC: return pair<FORM_GENERIC, false>(l, g, mc, a, stream);
    case FORM_EWALD_POLY5: return pair<FORM_EWALD_POLY5, false>(l, g, mc, a, stream);
    default: return pair<FORM_EWALD_EXACT, false>(l, g, mc, a, stream);
  }
}

cudaError_t col_launch_deriv64(const ColGrid &g, const Fp64Consts &mc, const ColArrays &a,
                               const Col64Launch &l, int mode, bool params,
                               cudaStream_t stream) {
  if (mode == DERIV_PARAMS)
    return launch(k_col_deriv64<DERIV_PARAMS, true>, l, g, mc, a, ColLayout64<false>::bytes,
                  stream, l.tpart);
  if (params)
    return launch(k_col_deriv64<DERIV_VJP, true>, l, g, mc, a, ColLayout64<true>::bytes, stream,
                  l.tpart);
  return launch(k_col_deriv64<DERIV_VJP, false>, l, g, mc, a, ColLayout64<true>::bytes, stream,
                l.tpart);
}

}  // namespace pmb200
