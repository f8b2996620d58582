// Lean mixed-precision kernel instantiations for metric kRasheedLarsen.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

template <int MID>
__global__ void __launch_bounds__(128) integrate_lean_called_kernel(const __grid_constant__ LaunchArgs A,
                                                                    const __grid_constant__ RunConst R) {
    persistent_loop<LeanCalledEngine<MID>, 2>(A, R);
}

const void* mixed_lean_pair_kernel_rl() { return reinterpret_cast<const void*>(&integrate_lean_called_kernel<kRasheedLarsen>); }

}  // namespace foort
