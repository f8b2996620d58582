// FP64-analytic two-lane kernel instantiations for metric kKerr.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* analytic_pair_kernel_kerr(bool positions) { return lean_kernel<AnalyticPairEngine<kKerr>, 2>(positions); }

}  // namespace foort
