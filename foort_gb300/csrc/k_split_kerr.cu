// FP64 kernels whose lanes share a geodesic's step, metric kKerr.
#include "kernel_fp64_split.cuh"
#include "kernels.h"

namespace foort {

const void* fp64_split_kernel_kerr(int integrator, int start) { return split_kernel<kKerr, false>(integrator, start); }

}  // namespace foort
