// Kernel registry: every integration kernel is instantiated in its own translation unit
// (k_<precision>_<metric>.cu) and handed to the host library as a function pointer.
#pragma once

#include "engine.h"

namespace foort {

// Returns the __global__ function for (metric, integrator), or nullptr.
const void* fp64_kernel(int metric_id, int integrator);
// The kernel whose geodesics start on that many lanes (8, 4, 2 or 1) and end on four or eight; start
// 0: one lane to the end, Johannsen with alpha13 alone. nullptr where there is none.
const void* fp64_split_kernel(const RunConst& R, int start);
// Two lanes per geodesic throughout, or nullptr where that kernel does not exist.
const void* fp64_pair_kernel(int metric_id, int integrator);
const void* mixed_kernel(int metric_id, int integrator);
// decide64: terminations and diagnostics decided in FP64 (else in float-float)
const void* mixed_kernel_variant(int metric_id, int integrator, bool decide64);
// two lanes per geodesic, or nullptr where that kernel does not exist
const void* mixed_pair_kernel_variant(int metric_id, int integrator, bool decide64);

// The lean kernel (kernel_lean.cuh) of these options, with one or two lanes per geodesic,
// or nullptr where they need the general one.
const void* mixed_lean_kernel(const RunConst& R, bool pair, bool positions);

// FP64-analytic: eight lanes per geodesic, throughout (start 8) or for the last ones of a warp
// (start 2); nullptr where that kernel does not exist.
const void* analytic_split_kernel(const RunConst& R, int start);

// Host-side helpers of the mixed-precision kernels (per-image FP32 constants).
void fill_mixed_constants(int metric_id, ImageConst& ic, const RunConst& rc);
void fill_mixed_run(RunConst& rc);

}  // namespace foort
