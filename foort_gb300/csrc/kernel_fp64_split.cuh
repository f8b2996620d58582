// The plain FP64 kernel on four (RK4 also: eight) lanes per geodesic for Kerr and Johannsen,
// throughout or for the last geodesics of each warp.
//
// An FP64 instruction occupies its scheduler's pipe for 64 cycles per warp on GB300, however
// many lanes are active: a launch that leaves lanes idle costs the instructions of one
// lane's step. Four lanes share a step here, or eight two stages of one (RK4):
// - finite differences: lane 0 evaluates the metric at r + h, lane 1 at r - h, lane 2 at
//   theta + h, lane 3 at theta - h (one exp, one sincos and one g_dd each instead of 3, 3
//   and 4);
// - lane i holds component i of position and velocity, divides out the inverse metric
//   components that a^i needs and sums the eight terms of a^i;
// - the step rule's three quotients are lanes 1 to 3's.
// A step takes 0.41 (RK4) to 0.44 (Verlet) of the one-lane kernel's time on four lanes and
// 0.30 on eight while the geodesics fit on the GPU (log r, 3,600 geodesics, on one, four and
// eight lanes: Kerr RK4 83, 35 and 24 ms, Johannsen 122, 48 and 34; Verlet 30 and 14, 35 and
// 16); still bound by the FP64 instructions in series.
// The values are the one-lane kernel's bit for bit: both have their roundings written out
// (fp64_rounded.cuh).
#pragma once

#include <type_traits>

#include "kernel_fp64.cuh"

namespace foort {

template <int MID, bool A13, int INTEG, int LANES = 4>
struct SplitEngine {
    using Metric = RoundedMetric<MID, A13>;
    static constexpr bool kSplit = true;
    static constexpr bool kCopyImage = false;

    struct Lane {
        double x, v;  // this lane's component
        double C[INTEG == FOORT_INTEGRATOR_VERLET ? 6 : 1];  // the lane's Christoffel symbols at the position
        double lam;
        uint64_t steps;
        TermState T;
        DiagState D;
        uint32_t err = 0;
        uint32_t img = 0;
        uint32_t rhs = 0;
        uint32_t fp64 = 0;
        int32_t term = 0;
    };

    static __device__ __forceinline__ double from(double a, int lane, unsigned m) { return __shfl_sync(m, a, lane, 4); }

    // The Christoffel symbols that a^i needs: for t and phi Gamma^i_01, _02, _13, _23 in
    // C[0..3], for r and theta Gamma^i_00, _03, _11, _12, _22, _33 in C[0..5].
    static __device__ __forceinline__ void symbols(const MetricConst& M, const RunConst& R, double x1, double th, int i,
                                                   unsigned m, double C[6], double& r0, double* kept = nullptr) {
        const bool rlog = R.rlog != 0;
        const double hr = (i == 0) ? R.hfd : (i == 1) ? -R.hfd : 0.0, ht = (i == 2) ? R.hfd : (i == 3) ? -R.hfd : 0.0;
        double r = (i < 2) ? d_add(x1, hr) : x1, s, c;
        if (rlog) r = exp(r);
        sincos((i < 2) ? th : d_add(th, ht), &s, &c);
        r0 = from(r, 2, m);
        const double s0 = from(s, 0, m), c0 = from(c, 0, m);
        const G5 g = Metric::dd(M.q, r, s, c, rlog, i < 2);
        double g1, g2;
        Metric::uu(M.q, r0, s0, c0, rlog, i, g1, g2);
        // central differences: lanes 0 and 1 form those in r, lanes 2 and 3 those in theta
        const double inv = 1 / (2 * R.hfd);
        const bool second = i & 1;
        auto diff = [&](double a) {
            const double b = __shfl_xor_sync(m, a, 1, 4);
            return d_mul(d_sub(second ? b : a, second ? a : b), inv);
        };
        G5 d = {diff(g.tt), diff(g.tp), diff(g.rr), diff(g.hh), diff(g.pp)};
        auto other = [&](double a) { return __shfl_xor_sync(m, a, 2, 4); };
        const G5 o = {other(d.tt), other(d.tp), other(d.rr), other(d.hh), other(d.pp)};
        const bool low = i < 2;
        const G5 dr = {low ? d.tt : o.tt, low ? d.tp : o.tp, low ? d.rr : o.rr, low ? d.hh : o.hh, low ? d.pp : o.pp};
        const G5 dh = {low ? o.tt : d.tt, low ? o.tp : d.tp, low ? o.rr : d.rr, low ? o.hh : d.hh, low ? o.pp : d.pp};
        rounded_symbols<MID>(dr, dh, g1, g2, i, C, kept);
    }
    static __device__ __forceinline__ void gather(double a, unsigned m, double v[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = from(a, k, m);
    }

    // Integrators::GetAdaptiveStep (Integrators.cpp:34-46): lanes 1 to 3 each divide for
    // their component (lane 0 follows lane 1).
    static __device__ __forceinline__ double adaptive_step(const RunConst& R, const Lane& L, int i, unsigned m) {
        const double pt = d_sub(kRefPi, L.x), mth = (pt < L.x) ? pt : L.x;
        const double num = (i == 2) ? d_mul(R.eps, mth) : R.eps;
        const double den = fabs(d_add((i == 3) ? L.v : fabs(L.v), 1e-20));
        const double w = 1 / fabs(num / den);
        const double h = 1 / d_add(d_add(from(w, 1, m), from(w, 2, m)), from(w, 3, m));
        return (h < R.hmin) ? R.hmin : h;
    }

    static __device__ __forceinline__ void init(Lane& L, const ImageConst& I, const RunConst& R, const foort_pixel& p,
                                                int sub, unsigned m) {
        const int i = sub & 3;
        double x[4], v[4];
        initial_conditions(I, p, x, v);
        L.x = (i == 0) ? x[0] : (i == 1) ? x[1] : (i == 2) ? x[2] : x[3];
        L.v = (i == 0) ? v[0] : (i == 1) ? v[1] : (i == 2) ? v[2] : v[3];
        if constexpr (INTEG == FOORT_INTEGRATOR_VERLET) {
            double r;
            symbols(I.m, R, x[1], x[2], i, m, L.C, r, L.C);
        }
        L.lam = 0.0;
        L.steps = 0;
        L.err = 0;
        L.term = FOORT_TERMCODE_CONTINUE;
        L.img = p.image;
        reset_lane_state(R, x, L.D, L.T);
    }

    // One Geodesic::Update (Geodesic.cpp:61-88). sub: this lane among the geodesic's, m: those
    // lanes; i: its component.
    static __device__ __forceinline__ bool step_split(Lane& L, const ImageConst& I, const RunConst& R, int sub,
                                                      unsigned m) {
        const int i = sub & 3;
        const MetricConst& M = I.m;
        const double h = adaptive_step(R, L, i, m);
        double va[4], nx, nv, r;
        gather(L.v, m, va);
        if constexpr (LANES == 8) {
            // The stage positions need only the velocities of earlier stages: lanes 0 to 3
            // evaluate the symbols of stages 1 and 3, lanes 4 to 7 those of 2 and 4, and both
            // contract them with both stages' velocities.
            const bool odd = sub & 4;
            const double hh = 0.5 * h, h6 = h / 6.0;
            double C[6], l[4], k, l2, l3, l4, t;
            t = odd ? d_fma(L.v, hh, L.x) : L.x;
            symbols(M, R, from(t, 1, m), from(t, 2, m), i, m, C, r);
            const double k1 = __shfl_sync(m, rounded_accel(C, va, i), i, 8);
            l2 = d_fma(k1, hh, L.v);
            gather(l2, m, l);
            const double k2 = __shfl_sync(m, rounded_accel(C, l, i), i + 4, 8);
            l3 = d_fma(k2, hh, L.v);
            t = d_fma(odd ? l3 : l2, odd ? h : hh, L.x);
            symbols(M, R, from(t, 1, m), from(t, 2, m), i, m, C, r);
            gather(l3, m, l);
            const double k3 = __shfl_sync(m, rounded_accel(C, l, i), i, 8);
            l4 = d_fma(k3, h, L.v);
            gather(l4, m, l);
            const double k4 = __shfl_sync(m, rounded_accel(C, l, i), i + 4, 8);
            nv = d_fma(d_add(d_fma(k3, 2.0, d_fma(k2, 2.0, k1)), k4), h6, L.v);
            nx = d_fma(d_add(d_fma(l3, 2.0, d_fma(l2, 2.0, L.v)), l4), h6, L.x);
            L.rhs += (sub == 0) ? 4 : 0;
        } else if constexpr (INTEG == FOORT_INTEGRATOR_RK4) {  // Integrators.cpp:51-94
            const double hh = 0.5 * h, h6 = h / 6.0;
            double C[6], l[4], k1, k2, k3, k4, l2, l3, l4, t;
            symbols(M, R, from(L.x, 1, m), from(L.x, 2, m), i, m, C, r);
            k1 = rounded_accel(C, va, i);
            t = d_fma(L.v, hh, L.x);
            l2 = d_fma(k1, hh, L.v);
            gather(l2, m, l);
            symbols(M, R, from(t, 1, m), from(t, 2, m), i, m, C, r);
            k2 = rounded_accel(C, l, i);
            t = d_fma(l2, hh, L.x);
            l3 = d_fma(k2, hh, L.v);
            gather(l3, m, l);
            symbols(M, R, from(t, 1, m), from(t, 2, m), i, m, C, r);
            k3 = rounded_accel(C, l, i);
            t = d_fma(l3, h, L.x);
            l4 = d_fma(k3, h, L.v);
            gather(l4, m, l);
            symbols(M, R, from(t, 1, m), from(t, 2, m), i, m, C, r);
            k4 = rounded_accel(C, l, i);
            nv = d_fma(d_add(d_fma(k3, 2.0, d_fma(k2, 2.0, k1)), k4), h6, L.v);
            nx = d_fma(d_add(d_fma(l3, 2.0, d_fma(l2, 2.0, L.v)), l4), h6, L.x);
            L.rhs += (i == 0) ? 4 : 0;
        } else {  // Integrators.cpp:99-152
            const double a0 = rounded_accel(L.C, va, i), hh2 = h * h / 2.0, h2 = h / 2.0;
            double C[6], via[4], nva[4];
            nx = d_fma(a0, hh2, d_fma(L.v, h, L.x));
            const double vi = d_fma(a0, h, L.v);
            gather(vi, m, via);
            symbols(M, R, from(nx, 1, m), from(nx, 2, m), i, m, C, r, L.C);
#pragma unroll
            for (int k = (MID == kKerr) ? 2 : 0; k < 6; ++k) L.C[k] = C[k];
            double a1 = rounded_accel(C, via, i);
            nv = d_fma(d_add(a0, a1), h2, L.v);
            L.rhs += (i == 0) ? 2 : 0;
            if (R.vtol > 0.0) {
                const double tol2 = R.vtol * R.vtol;
                for (int it = 0;; ++it) {
                    gather(nv, m, nva);
                    double num = 0.0, den = 0.0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const double d = d_sub(nva[k], via[k]);
                        num = k ? d_fma(d, d, num) : d_mul(d, d);
                        den = k ? d_fma(nva[k], nva[k], den) : d_mul(nva[k], nva[k]);
                    }
                    if (!(num / den > tol2)) break;
                    if (it >= R.verlet_cap) {
                        L.err |= FOORT_ERR_VERLET_ITER;
                        break;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) via[k] = nva[k];
                    a1 = rounded_accel(C, via, i);
                    nv = d_fma(d_add(a0, a1), h2, L.v);
                    L.rhs += (i == 0) ? 1 : 0;
                }
            }
        }
        L.lam += h;
        L.x = nx;
        L.v = nv;
        ++L.steps;
        const double x1 = from(nx, 1, m), th = from(nx, 2, m), ph = from(nx, 3, m);
        if (INTEG == FOORT_INTEGRATOR_RK4) r = radius_of(R, x1);  // Verlet's symbols have it
        L.term = check_terms(R, M.rh, I.h_eps, r, th, L.T);
        update_diags(R, r, th, ph, L.lam, L.term, L.D);
        const bool bad = (__ballot_sync(m, !(isfinite(nx) && isfinite(nv))) & m) != 0;
        if (bad) {
            L.err |= FOORT_ERR_NONFINITE;
            if (L.term == FOORT_TERMCODE_CONTINUE && !(R.term_flags & FOORT_TERM_TIMEOUT)) return false;
        }
        return L.term == FOORT_TERMCODE_CONTINUE;
    }

    // Every lane writes its component, lane 0 the rest of the record.
    static __device__ __forceinline__ void write(const Lane& L, foort_result* o, int term, uint32_t err, int i) {
        if (i >= 4) return;
        o->pos[i] = L.x;
        o->vel[i] = L.v;
        if (i) return;
        o->term = term;
        o->err = err;
        o->steps = L.steps;
        o->lambda = L.lam;
        o->quadrant = L.D.quad;
        o->equat_passes = L.D.passes;
        o->closest_r = L.D.rmin;
    }
    static __device__ __forceinline__ void finish(const Lane& L, const RunConst&, foort_result* o, int i) {
        write(L, o, L.term, L.err, i);
    }
    static __device__ __forceinline__ void stop(const Lane& L, const RunConst&, foort_result* o, uint32_t err, int i) {
        write(L, o, FOORT_TERMCODE_CONTINUE, L.err | err, i);
    }
};

// RK4: at most 4 geodesics of a warp on four lanes each continue on eight.
template <int MID, bool A13>
struct OctTail {
    using S = SplitEngine<MID, A13, FOORT_INTEGRATOR_RK4, 8>;
    static constexpr unsigned kLeft = 4;

    static __device__ __forceinline__ void run(const LaunchArgs& A, const RunConst& R,
                                               const typename SplitEngine<MID, A13, FOORT_INTEGRATOR_RK4>::Lane& L,
                                               unsigned left, uint64_t idx) {
        const int lane = threadIdx.x & 31;
        unsigned rest = left;
        for (int k = 0; k < (lane >> 3); ++k) rest &= rest - 1;
        const bool active = rest != 0;
        const int src = __ffs(active ? rest : left) - 1 + (lane & 3);  // the same component's lane
        typename S::Lane T;
        T.x = from_lane(L.x, src);
        T.v = from_lane(L.v, src);
        T.lam = from_lane(L.lam, src);
        T.steps = from_lane(L.steps, src);
        T.T = from_lane(L.T, src);
        T.D = from_lane(L.D, src);
        T.err = from_lane(L.err, src);
        T.img = from_lane(L.img, src);
        T.term = from_lane(L.term, src);
        work_loop<S, 8, NoTail>(A, R, T, active, from_lane(idx, src), true);
    }
};

// The tail of a launch of Fp64Engine (one or two lanes per geodesic): at most 8 geodesics of
// a warp continue on four lanes each, from the state between two steps. A warp's step takes
// the same time with one geodesic left as with all its lanes busy, and the longest rays end a
// launch alone: 62,500 Johannsen rays in FP64 Verlet 122 ms on one lane throughout, 111 on
// four, 98 on one and then four; 15,625 Kerr rays in RK4 107 on one lane, 67 from two.
template <int MID, bool A13, int INTEG, class Engine>
struct SplitTail {
    using S = SplitEngine<MID, A13, INTEG>;
    static constexpr unsigned kLeft = 8;

    static __device__ __forceinline__ double component(const double a[4], int i, int lane) {
        const double a0 = from_lane(a[0], lane), a1 = from_lane(a[1], lane), a2 = from_lane(a[2], lane), a3 = from_lane(a[3], lane);
        return (i == 0) ? a0 : (i == 1) ? a1 : (i == 2) ? a2 : a3;
    }

    // left: the lanes that hold the geodesics; every lane of the warp calls it.
    static __device__ __forceinline__ void run(const LaunchArgs& A, const RunConst& R,
                                               const typename Engine::Lane& L, unsigned left,
                                               uint64_t idx) {
        const int lane = threadIdx.x & 31, i = lane & 3, group = lane >> 2;
        unsigned rest = left;
        for (int k = 0; k < group; ++k) rest &= rest - 1;  // drops the groups before this one
        const bool active = rest != 0;
        const int src = __ffs(active ? rest : left) - 1;
        typename S::Lane T;
        T.x = component(L.x, i, src);
        T.v = component(L.v, i, src);
        T.lam = from_lane(L.lam, src);
        T.steps = from_lane(L.steps, src);
        T.T = from_lane(L.T, src);
        T.D = from_lane(L.D, src);
        T.err = from_lane(L.err, src);
        T.img = from_lane(L.img, src);
        T.term = from_lane(L.term, src);
        if constexpr (INTEG == FOORT_INTEGRATOR_VERLET) {
            const G5 dr = from_lane(L.P.dr, src), dh = from_lane(L.P.dh, src), gu = from_lane(L.P.gu, src);
            const double g1 = (i == 0) ? gu.tt : (i == 1) ? gu.rr : (i == 2) ? gu.hh : gu.pp;
            rounded_symbols<MID>(dr, dh, g1, gu.tp, i, T.C, T.C);
        }
        using Next = std::conditional_t<INTEG == FOORT_INTEGRATOR_RK4, OctTail<MID, A13>, NoTail>;
        work_loop<S, 4, Next>(A, R, T, active, from_lane(idx, src), true);
    }
};

// START: lanes per geodesic, from 1 and 2 until a warp has eight geodesics left; 0: one lane
// to the end (A13).
// Without the zero terms Johannsen's right-hand side saves nine divisions of 34: one-lane
// Verlet, 176,400 rays in log r 200 to 157 ms, RK4 653 to 475; 62,500 rays of the reference's
// debug view with the tail 98 to 79.
template <int MID, bool A13, int INTEG, int START>
__global__ void __launch_bounds__(128) integrate_fp64_split_kernel(const __grid_constant__ LaunchArgs A,
                                                                   const __grid_constant__ RunConst R) {
    if constexpr (START == 4) {
        persistent_loop<SplitEngine<MID, A13, INTEG>, 4>(A, R);
    } else if constexpr (START == 8) {
        persistent_loop<SplitEngine<MID, A13, INTEG, 8>, 8>(A, R);
    } else {
        using E = Fp64Engine<MID, INTEG, RoundedMetric<MID, A13>>;
        if constexpr (START == 0) {
            persistent_loop<E, 1>(A, R);
        } else {
            persistent_loop<E, START, SplitTail<MID, A13, INTEG, E>>(A, R);
        }
    }
}

template <int MID, bool A13, int INTEG, int START>
const void* split_instance() {
    return reinterpret_cast<const void*>(&integrate_fp64_split_kernel<MID, A13, INTEG, START>);
}

template <int MID, bool A13, int INTEG>
const void* split_kernel(int start) {
    constexpr bool kRk4 = INTEG == FOORT_INTEGRATOR_RK4;
    if constexpr (A13) {
        if (start == 0) return split_instance<MID, A13, INTEG, 0>();
    }
    if (start == 1) return split_instance<MID, A13, INTEG, 1>();
    if constexpr (kRk4) {
        if (start == 2) return split_instance<MID, A13, INTEG, 2>();
        if (start == 8) return split_instance<MID, A13, INTEG, 8>();
    } else {
        if (start == 4) return split_instance<MID, A13, INTEG, 4>();
    }
    return nullptr;
}

template <int MID, bool A13>
const void* split_kernel(int integrator, int start) {
    return integrator == FOORT_INTEGRATOR_RK4 ? split_kernel<MID, A13, FOORT_INTEGRATOR_RK4>(start)
                                              : split_kernel<MID, A13, FOORT_INTEGRATOR_VERLET>(start);
}

}  // namespace foort
