// Lean mixed-precision kernel instantiations for metric kFlat.
#include "kernel_lean.cuh"
#include "kernels.h"

namespace foort {

const void* mixed_lean_kernel_flat(bool positions) { return lean_kernel<LeanEngine<kFlat, false>, 1, 3>(positions); }

const void* mixed_lean_verlet_kernel_flat(bool positions) {
    return lean_kernel<LeanVerletEngine<kFlat, false>, 1, 3>(positions);
}

const void* mixed_lean_pair_kernel_flat(bool positions) { return lean_kernel<LeanEngine<kFlat, false>, 2>(positions); }

}  // namespace foort
