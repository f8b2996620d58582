// Lean mixed-precision kernel instantiations for metric kJohannsen.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* mixed_lean_pair_kernel_joh(bool positions) { return lean_kernel<LeanCalledEngine<kJohannsen>, 2>(positions); }

}  // namespace foort
