// FP64-analytic two-lane kernel instantiations for metric kJohannsen.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* analytic_pair_kernel_joh(bool positions) { return lean_kernel<AnalyticPairEngine<kJohannsen>, 2>(positions); }

}  // namespace foort
