// FP64 kernel on four lanes per geodesic, metric kJohannsen.
#include "kernel_fp64_split.cuh"
#include "kernels.h"

namespace foort {

template <bool A13>
static const void* kernel(int integrator) {
    if (integrator == FOORT_INTEGRATOR_RK4)
        return reinterpret_cast<const void*>(&integrate_fp64_split_kernel<kJohannsen, A13, FOORT_INTEGRATOR_RK4>);
    return reinterpret_cast<const void*>(&integrate_fp64_split_kernel<kJohannsen, A13, FOORT_INTEGRATOR_VERLET>);
}

const void* fp64_split_kernel_joh(int integrator, bool only_alpha13) {
    return only_alpha13 ? kernel<true>(integrator) : kernel<false>(integrator);
}

}  // namespace foort
