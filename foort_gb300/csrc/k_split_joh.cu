// FP64 kernels that end on four lanes per geodesic, metric kJohannsen.
#include "kernel_fp64_split.cuh"
#include "kernels.h"

namespace foort {

const void* fp64_split_kernel_joh(int integrator, bool only_alpha13, int start) {
    return only_alpha13 ? split_kernel<kJohannsen, true>(integrator, start)
                        : split_kernel<kJohannsen, false>(integrator, start);
}

}  // namespace foort
