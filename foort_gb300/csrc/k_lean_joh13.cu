// Lean mixed-precision kernel instantiations for metric kJohannsen with alpha13 alone.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

// Two CTAs per SM: at three (168 registers) the packed body spills 592 bytes a step and 39,204
// rays in plain r take 344 ms instead of 255.
const void* mixed_lean_kernel_joh13(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanEngine<kJohannsen, true>, 1, 2>(positions)
                : lean_kernel<LeanEngine<kJohannsen, false>, 1, 2>(positions);
}

const void* mixed_lean_pair_kernel_joh13(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanEngine<kJohannsen, true>, 2>(positions) : lean_kernel<LeanEngine<kJohannsen, false>, 2>(positions);
}

const void* mixed_lean_verlet_kernel_joh13(bool rlog, bool positions) {
    return rlog ? lean_kernel<LeanVerletEngine<kJohannsen, true>, 1, 3>(positions)
                : lean_kernel<LeanVerletEngine<kJohannsen, false>, 1, 3>(positions);
}

}  // namespace foort
