// FP64-analytic two-lane kernel instantiation for metric kJohannsen.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

template <int MID>
__global__ void __launch_bounds__(128) integrate_analytic_pair_kernel(const __grid_constant__ LaunchArgs A,
                                                                      const __grid_constant__ RunConst R) {
    persistent_loop<AnalyticPairEngine<MID>, 2>(A, R);
}

const void* analytic_pair_kernel_joh() { return reinterpret_cast<const void*>(&integrate_analytic_pair_kernel<kJohannsen>); }

}  // namespace foort
