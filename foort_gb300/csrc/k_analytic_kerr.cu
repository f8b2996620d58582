// FP64-analytic two- and eight-lane kernel instantiations for metric kKerr.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* analytic_pair_kernel_kerr(bool positions) { return lean_kernel<AnalyticPairEngine<kKerr>, 2>(positions); }

const void* analytic_split_kernel_kerr(int start) {
    if (start == 8) return reinterpret_cast<const void*>(&integrate_lean_kernel<AnalyticSplitEngine<kKerr>, 8, 1>);
    return reinterpret_cast<const void*>(&integrate_lean_kernel<AnalyticPairEngine<kKerr>, 2, 1, AnalyticTail<kKerr>>);
}

}  // namespace foort
