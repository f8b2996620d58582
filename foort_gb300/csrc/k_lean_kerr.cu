// Lean mixed-precision kernel instantiations for metric kKerr.
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

template <int MID, bool RLOG>
__global__ void __launch_bounds__(128, 3) integrate_lean_verlet_kernel(const __grid_constant__ LaunchArgs A,
                                                                       const __grid_constant__ RunConst R) {
    persistent_loop<LeanVerletEngine<MID, RLOG>>(A, R);
}

const void* mixed_lean_verlet_kernel_kerr(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_verlet_kernel<kKerr, true>)
                : reinterpret_cast<const void*>(&integrate_lean_verlet_kernel<kKerr, false>);
}

const void* mixed_lean_kernel_kerr(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_kernel<kKerr, true>)
                : reinterpret_cast<const void*>(&integrate_lean_kernel<kKerr, false>);
}

const void* mixed_lean_pair_kernel_kerr(bool rlog) {
    return rlog ? reinterpret_cast<const void*>(&integrate_lean_pair_kernel<kKerr, true>)
                : reinterpret_cast<const void*>(&integrate_lean_pair_kernel<kKerr, false>);
}

}  // namespace foort
