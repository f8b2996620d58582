// FP64 kernel on four lanes per geodesic, metric kKerr.
#include "kernel_fp64_split.cuh"
#include "kernels.h"

namespace foort {

template <bool A13>
static const void* kernel(int integrator) {
    if (integrator == FOORT_INTEGRATOR_RK4)
        return reinterpret_cast<const void*>(&integrate_fp64_split_kernel<kKerr, A13, FOORT_INTEGRATOR_RK4>);
    return reinterpret_cast<const void*>(&integrate_fp64_split_kernel<kKerr, A13, FOORT_INTEGRATOR_VERLET>);
}

const void* fp64_split_kernel_kerr(int integrator) { return kernel<false>(integrator); }

}  // namespace foort
