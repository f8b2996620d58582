// Lean mixed-precision kernel instantiations for metric kFlat.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

template <int MID, bool RLOG>
__global__ void __launch_bounds__(128, 3) integrate_lean_kernel(const __grid_constant__ LaunchArgs A,
                                                             const __grid_constant__ RunConst R) {
    persistent_loop<LeanEngine<MID, RLOG>>(A, R);
}

template <int MID, bool RLOG>
__global__ void __launch_bounds__(128) integrate_lean_pair_kernel(const __grid_constant__ LaunchArgs A,
                                                                  const __grid_constant__ RunConst R) {
    persistent_loop<LeanEngine<MID, RLOG>, 2>(A, R);
}

const void* mixed_lean_kernel_flat() {
    return reinterpret_cast<const void*>(&integrate_lean_kernel<kFlat, false>);
}

const void* mixed_lean_pair_kernel_flat() {
    return reinterpret_cast<const void*>(&integrate_lean_pair_kernel<kFlat, false>);
}

}  // namespace foort
