// FP64-analytic two-lane kernel instantiations for metric kFlat.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* analytic_pair_kernel_flat(bool positions) { return lean_kernel<AnalyticPairEngine<kFlat>, 2>(positions); }

}  // namespace foort
