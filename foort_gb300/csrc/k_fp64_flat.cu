// FP64 kernel instantiations for metric kFlat.
#include "kernel_fp64.cuh"
#include "kernels.h"

namespace foort {

const void* fp64_kernel_flat(int integrator) {
    if (integrator == FOORT_INTEGRATOR_RK4)
        return reinterpret_cast<const void*>(&integrate_fp64_kernel<kFlat, FOORT_INTEGRATOR_RK4>);
    return reinterpret_cast<const void*>(&integrate_fp64_kernel<kFlat, FOORT_INTEGRATOR_VERLET>);
}

const void* fp64_pair_kernel_flat() { return reinterpret_cast<const void*>(&integrate_fp64_pair_kernel<kFlat>); }

}  // namespace foort
