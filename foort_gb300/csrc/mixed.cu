// Host side of the mixed-precision kernels: kernel registry and per-image constants.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "kernel_mixed.cuh"
#include "kernels.h"

namespace foort {

const void* mixed_kernel_kerr(int integrator, bool decide64);
const void* mixed_kernel_joh(int integrator, bool decide64);
const void* mixed_kernel_flat(int integrator, bool decide64);
const void* mixed_kernel_rl(int integrator, bool decide64);
const void* mixed_kernel_mn(int integrator, bool decide64);

// Mixed kernels for every metric: analytic derivatives generated by gen_christoffel.py,
// and for Manko-Novikov by forward-mode differentiation (analytic_metric.cuh).
const void* mixed_kernel_variant(int metric_id, int integ, bool decide64) {
    switch (metric_id) {
    case kKerr: return mixed_kernel_kerr(integ, decide64);
    case kJohannsen: return mixed_kernel_joh(integ, decide64);
    case kFlat: return mixed_kernel_flat(integ, decide64);
    case kRasheedLarsen: return mixed_kernel_rl(integ, decide64);
    case kMankoNovikov: return mixed_kernel_mn(integ, decide64);
    default: return nullptr;
    }
}

const void* mixed_kernel(int metric_id, int integ) { return mixed_kernel_variant(metric_id, integ, true); }

const void* mixed_pair_kernel_kerr(bool decide64);
const void* mixed_pair_kernel_flat(bool decide64);

// Two-lane kernels: RK4 with the inlined plugins (Kerr, flat space).
const void* mixed_pair_kernel_variant(int metric_id, int integ, bool decide64) {
    if (integ != FOORT_INTEGRATOR_RK4) return nullptr;
    switch (metric_id) {
    case kKerr: return mixed_pair_kernel_kerr(decide64);
    case kFlat: return mixed_pair_kernel_flat(decide64);
    default: return nullptr;
    }
}

const void* mixed_lean_kernel_kerr(bool rlog, bool positions);
const void* mixed_lean_kernel_flat(bool positions);
const void* mixed_lean_pair_kernel_kerr(bool rlog, bool positions);
const void* mixed_lean_pair_kernel_flat(bool positions);
const void* mixed_lean_pair_kernel_joh(bool positions);
const void* mixed_lean_kernel_joh13(bool rlog, bool positions);
const void* mixed_lean_pair_kernel_joh13(bool rlog, bool positions);
const void* mixed_lean_verlet_kernel_kerr(bool rlog, bool positions);
const void* mixed_lean_verlet_kernel_joh13(bool rlog, bool positions);
const void* mixed_lean_verlet_kernel_flat(bool positions);
const void* mixed_lean_pair_kernel_rl(bool positions);
const void* analytic_pair_kernel_kerr(bool positions);
const void* analytic_split_kernel_kerr(int start);
const void* analytic_pair_kernel_flat(bool positions);

// Lean options: every termination and diagnostic in use updates at each step (the
// default), with decisions on the float-float state.
static bool lean_options(const RunConst& R) { return R.each_step && !(R.mixed_options & FOORT_MIXED_FP64_DECISIONS); }

// Whether some steps of a mixed launch are taken in FP64 (near the horizon, at turning points).
static bool fp64_regions(const RunConst& R) {
    return R.mixed_fp64_margin > 0.0 || (R.mixed_options & FOORT_MIXED_FP64_TURNING_POINTS);
}

const void* mixed_lean_kernel(const RunConst& R, bool pair, bool positions) {
    if (!lean_options(R)) return nullptr;
    if (R.integrator == FOORT_INTEGRATOR_VERLET) {
        if (pair || R.precision != FOORT_PREC_MIXED || fp64_regions(R)) return nullptr;
        if (R.metric_id == kFlat && !R.rlog) return mixed_lean_verlet_kernel_flat(positions);
        if (R.metric_id == kKerr) return mixed_lean_verlet_kernel_kerr(R.rlog != 0, positions);
        if (R.metric_id == kJohannsen && R.only_alpha13) return mixed_lean_verlet_kernel_joh13(R.rlog != 0, positions);
        return nullptr;
    }
    if (R.precision == FOORT_PREC_FP64_ANALYTIC) {
        if (!pair) return nullptr;
        switch (R.metric_id) {
        case kKerr: return analytic_pair_kernel_kerr(positions);
        case kFlat: return analytic_pair_kernel_flat(positions);
        default: return nullptr;
        }
    }
    if (R.precision != FOORT_PREC_MIXED || fp64_regions(R)) return nullptr;
    switch (R.metric_id) {
    case kKerr: return pair ? mixed_lean_pair_kernel_kerr(R.rlog != 0, positions) : mixed_lean_kernel_kerr(R.rlog != 0, positions);
    case kFlat: return R.rlog ? nullptr : pair ? mixed_lean_pair_kernel_flat(positions) : mixed_lean_kernel_flat(positions);
    case kJohannsen:
        if (R.only_alpha13)
            return pair ? mixed_lean_pair_kernel_joh13(R.rlog != 0, positions) : mixed_lean_kernel_joh13(R.rlog != 0, positions);
        return pair ? mixed_lean_pair_kernel_joh(positions) : nullptr;
    case kRasheedLarsen: return pair ? mixed_lean_pair_kernel_rl(positions) : nullptr;
    default: return nullptr;
    }
}

const void* analytic_split_kernel(const RunConst& R, int start) {
    if (R.precision != FOORT_PREC_FP64_ANALYTIC || R.integrator != FOORT_INTEGRATOR_RK4 || R.metric_id != kKerr ||
        !lean_options(R))
        return nullptr;
    return (start == 8 || start == 2) ? analytic_split_kernel_kerr(start) : nullptr;
}

void fill_mixed_run(RunConst& rc) {
    MixedRun& m = rc.mr;
    ff_split(rc.rlog ? std::log(rc.b_rad) : rc.b_rad, m.bthr[0], m.bthr[1]);
    ff_split(rc.th_eps, m.theps[0], m.theps[1]);
    ff_split(kRefPi, m.pi[0], m.pi[1]);
    ff_split(-(kRefPi / 2.0), m.mpio2[0], m.mpio2[1]);
    ff_split(kRefPi / 2.0 * rc.eq_thr, m.eqthr[0], m.eqthr[1]);
    ff_split(rc.eps, m.eps[0], m.eps[1]);
    m.hmin = static_cast<float>(rc.hmin);
    // a positive tolerance whose square is below FP32's range still iterates (as with 0)
    m.vtol2 = rc.vtol > 0.0 ? std::max(static_cast<float>(rc.vtol * rc.vtol), FLT_MIN) : 0.f;
    // theta's high part differs from theta by 6e-8 of it, so a distance from pi / 2 (or
    // from 0 and pi) this much above the threshold leaves no doubt
    m.eqfar = std::max(m.eqthr[0], 0.f) * 1.00001f + 4e-6f;
    m.thfar = std::max(m.theps[0], 0.f) * 1.00001f + 4e-6f;
}

void fill_mixed_constants(int metric_id, ImageConst& ic, const RunConst& rc) {
    MixedConst& mx = ic.mx;
    mixed_metric_constants(metric_id, ic.m, ic.qa);
    for (int i = 0; i < kMixedQ; ++i) mx.q[i] = static_cast<float>(ic.qa[i]);
    double rp, rm;
    mixed_horizons(metric_id, ic.m, rp, rm);
    mx.rpv = rp;
    mx.rmv = rm;
    ff_split(rp, mx.rp[0], mx.rp[1]);
    ff_split(rm, mx.rm[0], mx.rm[1]);
    ff_split(rp > 0 ? std::log(rp) : 0.0, mx.lrp[0], mx.lrp[1]);
    ff_split(rm > 0 ? std::log(rm) : 0.0, mx.lrm[0], mx.lrm[1]);
    const bool rlog = rc.rlog != 0;
    auto coord = [rlog](double r) { return rlog ? std::log(r) : r; };
    double r_fp64 = (rc.mixed_fp64_margin > 0.0 && rp > 0.0) ? rp + rc.mixed_fp64_margin : 0.0;
    // Manko-Novikov's exponents grow without bound toward the horizon and its metric
    // leaves FP32's range there: inside the radius where one exceeds 8 (e^8 ~ 3e3), the
    // right-hand side is always taken in FP64
    if (metric_id == kMankoNovikov) r_fp64 = std::max(r_fp64, mn_fp64_radius(ic.m, kMnMaxFp32Exponent));
    mx.r_fp64 = r_fp64 > 0.0 ? static_cast<float>(coord(r_fp64)) : 0.f;
    // FP64-analytic: every step in FP64 (x1 < +inf holds for every finite position)
    if (rc.precision == FOORT_PREC_FP64_ANALYTIC) mx.r_fp64 = HUGE_VALF;
    const double rh = ic.m.rh;
    ff_split(coord(rh * (1 + ic.h_eps)), mx.hthr[0], mx.hthr[1]);
    ff_split(ic.h_eps > 0 ? coord(ic.h_eps) : (rlog ? -HUGE_VAL : 0.0), mx.hthr0[0], mx.hthr0[1]);
    // the run's constants, also where the general kernels read them
    const MixedRun& m = rc.mr;
    for (int i = 0; i < 2; ++i) {
        mx.bthr[i] = m.bthr[i];
        mx.theps[i] = m.theps[i];
        mx.pi[i] = m.pi[i];
        mx.mpio2[i] = m.mpio2[i];
        mx.eqthr[i] = m.eqthr[i];
        mx.eps[i] = m.eps[i];
    }
    mx.hmin = m.hmin;
    mx.vtol2 = m.vtol2;
}

}  // namespace foort
