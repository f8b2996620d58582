// Lean mixed-precision kernel instantiations for metric kJohannsen with alpha13 alone.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

// Two CTAs per SM: at three (168 registers) the packed body spills 592 bytes a step and 39,204
// rays in plain r take 344 ms instead of 255.
template <int MID, bool RLOG>
__global__ void __launch_bounds__(128, 2) integrate_lean_kernel(const __grid_constant__ LaunchArgs A,
                                                             const __grid_constant__ RunConst R) {
    persistent_loop<LeanEngine<MID, RLOG>>(A, R);
}

template <int MID, bool RLOG>
__global__ void __launch_bounds__(128) integrate_lean_pair_kernel(const __grid_constant__ LaunchArgs A,
                                                                  const __grid_constant__ RunConst R) {
    persistent_loop<LeanEngine<MID, RLOG>, 2>(A, R);
}

template <int MID, bool RLOG>
__global__ void __launch_bounds__(128, 3) integrate_lean_verlet_kernel(const __grid_constant__ LaunchArgs A,
                                                                       const __grid_constant__ RunConst R) {
    persistent_loop<LeanVerletEngine<MID, RLOG>>(A, R);
}

const void* mixed_lean_verlet_kernel_joh13(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_verlet_kernel<kJohannsen, true>)
                : reinterpret_cast<const void*>(&integrate_lean_verlet_kernel<kJohannsen, false>);
}

const void* mixed_lean_kernel_joh13(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_kernel<kJohannsen, true>)
                : reinterpret_cast<const void*>(&integrate_lean_kernel<kJohannsen, false>);
}

const void* mixed_lean_pair_kernel_joh13(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_pair_kernel<kJohannsen, true>)
                : reinterpret_cast<const void*>(&integrate_lean_pair_kernel<kJohannsen, false>);
}

}  // namespace foort
