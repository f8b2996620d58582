// What of a run's options, besides metric, integrator, precision and the FP64 steps, selects its
// kernels: used where kernels are chosen (mixed.cu, engine.cu) and where the tuning cache
// names them (tune.cpp).
#pragma once

#include "../../include/foort_gpu.h"

namespace foort {

// Johannsen's alpha22, alpha52 and epsilon3 are 0 in every image.
inline bool only_alpha13(const foort_run_desc& d) {
    for (uint32_t i = 0; d.images && i < d.n_images; ++i)
        for (int k = 2; k < 5; ++k)
            if (d.images[i].metric_params[k] != 0.0) return false;
    return true;
}

// Every termination and diagnostic in use updates at each step (the default). Flat space has
// no Horizon termination.
inline bool updates_each_step(const foort_run_desc& d) {
    auto each = [](bool used, uint64_t every) { return !used || every == 1; };
    return each((d.term_flags & FOORT_TERM_HORIZON) && d.metric_id != FOORT_METRIC_FLAT, d.horizon_every) &&
           each(d.term_flags & FOORT_TERM_BOUNDARY_SPHERE, d.boundary_every) &&
           each(d.term_flags & FOORT_TERM_TIMEOUT, d.timeout_every) &&
           each(d.term_flags & FOORT_TERM_THETA_SINGULARITY, d.theta_every) &&
           each(d.diag_flags & FOORT_DIAG_EQUATORIAL_PASSES, d.equat_freq.every_n) &&
           each(d.diag_flags & FOORT_DIAG_CLOSEST_RADIUS, d.closest_freq.every_n);
}

}  // namespace foort
