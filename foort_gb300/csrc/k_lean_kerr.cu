// Lean mixed-precision kernel instantiations for metric kKerr.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* mixed_lean_kernel_kerr(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanEngine<kKerr, true>, 1, 3>(positions)
                : lean_kernel<LeanEngine<kKerr, false>, 1, 3>(positions);
}

const void* mixed_lean_pair_kernel_kerr(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanEngine<kKerr, true>, 2>(positions) : lean_kernel<LeanEngine<kKerr, false>, 2>(positions);
}

const void* mixed_lean_verlet_kernel_kerr(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanVerletEngine<kKerr, true>, 1, 3>(positions)
                : lean_kernel<LeanVerletEngine<kKerr, false>, 1, 3>(positions);
}

}  // namespace foort
