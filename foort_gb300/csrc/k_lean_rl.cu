// Lean mixed-precision kernel instantiations for metric kRasheedLarsen.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* mixed_lean_pair_kernel_rl(bool positions) { return lean_kernel<LeanCalledEngine<kRasheedLarsen>, 2>(positions); }

}  // namespace foort
