// FP64 kernels whose lanes share a geodesic's step, metric kJohannsen.
#include "kernel_fp64_split.cuh"
#include "kernels.h"

namespace foort {

const void* fp64_split_kernel_joh(int integrator, bool only_alpha13, int start) {
    return only_alpha13 ? split_kernel<kJohannsen, true>(integrator, start)
                        : split_kernel<kJohannsen, false>(integrator, start);
}

}  // namespace foort
