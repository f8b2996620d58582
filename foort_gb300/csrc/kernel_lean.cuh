// Lean mixed-precision kernels: the mixed kernel's arithmetic (kernel_mixed.cuh) for the
// options nearly every run has, with packed FP32 instructions (packed.cuh).
//
// Lean options (lean_options, mixed.cu): every termination and diagnostic in use updates
// at each step, decisions on the float-float state, no FP64 steps. A lane then carries no
// update counters and no copy of the options' constants (they sit in the kernel's parameters,
// RunConst::mr); positions are recorded by a variant of each kernel (Recording). Results are
// the general kernel's bit for bit, also where a state overflows: each rounding is written out
// as the compiler contracts the scalar code (gen_packed.py), and the shortcuts below only
// skip work whose outcome is known.
//
// RK4, one lane per geodesic: the metric parts of stages 1 and 2 need only the step's
// start, those of stages 3 and 4 only k1 and k2, so each of the two pairs is evaluated
// packed, one stage per half. On two lanes per geodesic each lane evaluates one stage of a
// pair, and only the contraction's last sums and the state's update are packed.
//
// What bounds it: a warp alone on its scheduler waits for fixed latencies (0.93 of 2.42
// cycles per issue; 799 instructions a step, 0.97 us; on two lanes 692 each, 0.86 us; the
// general kernels take 1.66 us on one lane and 1.17 us on two). Three warps per scheduler take 1,338
// cycles per warp and step, near the FP32 pipe (377 packed and 244 scalar instructions, 998
// cycles) with what mixing scalar and packed ones costs it. Kerr views from r = 1000, GB300 at
// 2,070 MHz: 9,728 geodesics 61 ms on two lanes and 69 on one, 16,384 64 ms on one (general
// kernels: 82 to 94), 93,000 278 ms.
#pragma once

#include "kernel_mixed.cuh"
#include "packed.cuh"
#include "gen_packed.inc"

namespace foort {

template <int MID>
struct PackedMetric;

#define FOORT_DEFINE_PACKED_METRIC(ID, NAME)                                                              \
    template <>                                                                                           \
    struct PackedMetric<ID> {                                                                             \
        static constexpr int kSlots = FOORT_PACKED_SLOTS_##NAME;                                          \
        static __device__ __forceinline__ void constants(const float* q, float* k) {                      \
            using T = float;                                                                              \
            (void)q; (void)k;                                                                             \
            FOORT_PACKED_CONST_##NAME                                                                     \
        }                                                                                                 \
        template <typename T>                                                                             \
        static __device__ __forceinline__ void eval(const float* k, T r, T dp, T dm, T s, T c, G5T<T>& dr, \
                                                    G5T<T>& dh, G5T<T>& gu) {                             \
            (void)k; (void)dp; (void)dm;                                                                  \
            FOORT_PACKED_BODY_##NAME                                                                      \
        }                                                                                                 \
    };
#define MUL p_mul
#define ADD p_add
#define FMA p_fma
#define RCP p_rcp
#define K p_all<T>
#define B(i) p_all<T>(k[i])
FOORT_DEFINE_PACKED_METRIC(kKerr, KERR)
FOORT_DEFINE_PACKED_METRIC(kFlat, FLAT)
// Johannsen with alpha13 alone (RunConst::only_alpha13): the compiled body's roundings with
// the terms of the deviation parameters that are 0 left out, exactly (x + 0 y = x, x / 1 = x):
// 386 operations of 857. A screen of 6,561 rays in log r takes 2.55 ms on two lanes, 9.0 with
// the called body on one.
FOORT_DEFINE_PACKED_METRIC(kJohannsen, JOHANNSEN13)
#undef MUL
#undef ADD
#undef FMA
#undef RCP
#undef K
#undef B

// accel_part (kernel_mixed.cuh) with the compiler's contraction written out. Where a sum has
// two products, it depends on the code around which of them joins as a fused multiply-add:
// FORM 0 is the step with an inlined plugin, 1 and 2 the called right-hand side of
// Johannsen and of Rasheed-Larsen. m.gu.rr and m.gu.hh come multiplied by -1/2. The other
// factors of 2 and -1/2 change no rounding, but are multiplied out as the general kernel does:
// where a sum is within a factor of 2 of the type's largest value its double overflows, and
// the ray would end otherwise without them (steps that diverge next to the axis or inside a
// horizon). Taken two at a time they cost next to nothing: 200,000 Kerr rays cut at 1,000 steps 7.20 ms
// without them, 7.28 one by one, 7.19 so (two lanes, 9,000 cut at 20,000: 18.9, 19.1 and
// 17.8; Johannsen in Verlet, 147,456 cut at 900: 3.82, 3.89 and 3.81). Flat space takes them
// one by one (58,368 cut at 3,000: 3.71 without, 3.78 and 3.87).
// a[2] is the product of m.gu.hh and *f2 (where asked for).
constexpr int kFlatForm = 3;  // FORM 0 of flat space
template <int FORM, typename T>
__device__ __forceinline__ void accel_lean(const MetricAt<T>& m, const T u[4], T a[4], T* f2 = nullptr) {
    // x y + z w with the first or the second product fused
    auto first = [](T x, T y, T z, T w) { return p_fma(x, y, p_mul(z, w)); };
    auto second = [](T x, T y, T z, T w) { return p_fma(z, w, p_mul(x, y)); };
    const T w1t = first(m.d1.tt, u[0], m.d1.tp, u[3]), w1p = first(m.d1.tp, u[0], m.d1.pp, u[3]);
    const T w2t = first(m.d2.tt, u[0], m.d2.tp, u[3]);
    constexpr bool kSecond = FORM == 1 || FORM == 2, kPairs = sizeof(T) == sizeof(float) && FORM != kFlatForm;
    const T w2p = (FORM == 1) ? second(m.d2.tp, u[0], m.d2.pp, u[3]) : first(m.d2.tp, u[0], m.d2.pp, u[3]);
    const T w1r = p_mul(m.d1.rr, u[1]), w1h = p_mul(m.d1.hh, u[2]);
    const T w2r = p_mul(m.d2.rr, u[1]), w2h = p_mul(m.d2.hh, u[2]);
    const T q1 = p_fma(u[3], w1p, p_fma(u[2], w1h, first(u[0], w1t, u[1], w1r)));
    const T q2a = first(u[0], w2t, u[1], w2r);
    const T q2b = kSecond ? p_fma(u[2], w2h, q2a) : p_add(q2a, p_mul(u[2], w2h));
    const T q2 = p_fma(u[3], w2p, q2b);
    const T St = kSecond ? second(u[1], w1t, u[2], w2t) : first(u[1], w1t, u[2], w2t);
    const T Sp = kSecond ? second(u[1], w1p, u[2], w2p) : first(u[1], w1p, u[2], w2p);
    const T Sr = first(u[1], w1r, u[2], w2r);
    const T Sh = kSecond ? second(u[1], w1h, u[2], w2h) : first(u[1], w1h, u[2], w2h);
    T Ft, Fp, Fr, Fh;
    if constexpr (kPairs) {
        const foort::f2 tp = pack2(St, Sp), rh = pack2(Sr, Sh);
        const foort::f2 F = p_add(tp, tp), G = p_sub(p_add(rh, rh), pack2(q1, q2));
        Ft = lo2(F), Fp = hi2(F), Fr = lo2(G), Fh = hi2(G);
    } else {
        Ft = p_mul(T(2), St), Fp = p_mul(T(2), Sp);
        Fr = p_sub(p_mul(T(2), Sr), q1), Fh = p_sub(p_mul(T(2), Sh), q2);
    }
    const T xt = first(m.gu.tt, Ft, m.gu.tp, Fp), xp = first(m.gu.tp, Ft, m.gu.pp, Fp);
    if constexpr (kPairs) {
        const foort::f2 x = p_mul(p_all<foort::f2>(-0.5f), pack2(xt, xp));
        a[0] = lo2(x), a[3] = hi2(x);
    } else {
        a[0] = p_mul(T(-0.5), xt), a[3] = p_mul(T(-0.5), xp);
    }
    a[1] = p_mul(m.gu.rr, Fr);
    a[2] = p_mul(m.gu.hh, Fh);
    if (f2) *f2 = Fh;
}
// The form of each metric's FP32 right-hand side.
constexpr int accel_form(int mid) {
    return mid == kJohannsen ? 1 : mid == kRasheedLarsen ? 2 : mid == kFlat ? kFlatForm : 0;
}
// In log-r mode the coordinate term -(u^1)^2 joins a^1 (accel_log_r).
template <int FORM, typename T>
__device__ __forceinline__ void accel_lean(const MetricAt<T>& m, bool rlog, const T u[4], T a[4], T* f2 = nullptr) {
    accel_lean<FORM, T>(m, u, a, f2);
    if (rlog) a[1] = p_fma(-u[1], u[1], a[1]);
}

// Image constants a lane of a packed plugin keeps.
template <int MID>
struct LeanConst {
    float k[PackedMetric<MID>::kSlots ? PackedMetric<MID>::kSlots : 1];
    float rp[2], rm[2];
    float lrp[2];  // log-r only

    __device__ __forceinline__ void load(const ImageConst& I) {
        PackedMetric<MID>::constants(I.mx.q, k);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            rp[i] = I.mx.rp[i];
            rm[i] = I.mx.rm[i];
            lrp[i] = I.mx.lrp[i];
        }
    }
};

// metric_part (kernel_mixed.cuh) with a plugin of PackedMetric, on every half.
template <int MID, bool RLOG, typename T>
__device__ __forceinline__ MetricAt<T> metric_lean(const LeanConst<MID>& C, T x1h, T x1l, T thh, T thl) {
    T r, dp, dm;
    if (!RLOG) {
        r = p_add(x1h, x1l);
        dp = p_add(p_sub(x1h, p_all<T>(C.rp[0])), p_sub(x1l, p_all<T>(C.rp[1])));
        dm = p_add(p_sub(x1h, p_all<T>(C.rm[0])), p_sub(x1l, p_all<T>(C.rm[1])));
    } else {
        const T e = p_each([](float x) { return expf(x); }, x1h);
        r = p_fma(e, x1l, e);
        const T yp = p_add(p_sub(x1h, p_all<T>(C.lrp[0])), p_sub(x1l, p_all<T>(C.lrp[1])));
        const float rp = C.rp[0];
        dp = p_each([rp](float y, float rr) { return (y > 1.f) ? __fsub_rn(rr, rp) : __fmul_rn(rp, expm1f(y)); }, yp, r);
        dm = p_sub(r, p_all<T>(C.rm[0]));
    }
    T s, c;
    p_sincos(thh, thl, s, c);
    MetricAt<T> m;
    PackedMetric<MID>::template eval<T>(C.k, r, dp, dm, s, c, m.d1, m.d2, m.gu);
    if (RLOG) {  // scale_log_r
        const T r2 = p_mul(r, r);
        m.d1.tt = p_mul(m.d1.tt, r);
        m.d1.tp = p_mul(m.d1.tp, r);
        m.d1.hh = p_mul(m.d1.hh, r);
        m.d1.pp = p_mul(m.d1.pp, r);
        m.d1.rr = p_mul(m.d1.rr, p_mul(r2, r));
        m.d2.rr = p_mul(m.d2.rr, r2);
        m.gu.rr = p_each([](float a, float b) { return __fdiv_rn(a, b); }, m.gu.rr, r2);
    }
    m.gu.rr = p_mul(p_all<T>(-0.5f), m.gu.rr);
    m.gu.hh = p_mul(p_all<T>(-0.5f), m.gu.hh);
    return m;
}

// One half of a packed metric part.
__device__ __forceinline__ G5T<float> half_of(const G5T<f2>& g, bool hi) {
    auto h = [hi](f2 a) { return hi ? hi2(a) : lo2(a); };
    return {h(g.tt), h(g.tp), h(g.rr), h(g.hh), h(g.pp)};
}
__device__ __forceinline__ MetricAt<float> half_of(const MetricAt<f2>& m, bool hi) {
    return {half_of(m.d1, hi), half_of(m.d2, hi), half_of(m.gu, hi)};
}

// adaptive_step_f32 (kernel_mixed.cuh) with the run's constants.
__device__ __forceinline__ float adaptive_step_lean(const MixedRun& G, float thh, float thl, float v1, float v2, float v3) {
    const float t = __fadd_rn(thh, thl), pt = __fadd_rn(__fsub_rn(G.pi[0], thh), __fsub_rn(G.pi[1], thl));
    const float m = fabsf((pt < t) ? pt : t);
    const float s1 = __fadd_rn(fabsf(v1), 1e-20f);
    const float s2 = __fadd_rn(fabsf(v2), 1e-20f);
    const float s3 = fabsf(__fadd_rn(v3, 1e-20f));
    const float den = __fmaf_rn(m, __fadd_rn(s1, s3), s2);
    const float inv = rcp(den);
    const float num = __fmul_rn(G.eps[0], m);
    const float q0 = __fmul_rn(num, inv);
    const float res = __fmaf_rn(-q0, den, num);
    const float h = __fmaf_rn(__fmaf_rn(G.eps[1], m, res), inv, q0);
    return (h < G.hmin) ? G.hmin : h;
}

// A lane's state and everything of a step but its right-hand sides. C: the image constants
// that those need.
template <class C>
struct LeanState {
    static constexpr bool kLean = true;
    static constexpr bool kCopyImage = false;

    // x and v: [0] holds components 0 (t) and 3 (phi), [1] components 1 (r or ln r) and 2
    // (theta), high and low parts.
    struct Lane {
        f2 xh[2], xl[2], vh[2], vl[2];
        ff lam;
        ff rmin;
        float hthr[2];
        C c;
        uint64_t steps;
        uint32_t err;
        int32_t term;
        int32_t passes;
        int32_t side;  // EquatorialPasses' last sample: 0 none (or theta <= 0), 1 below, 2 above pi/2
    };

    static __device__ __forceinline__ void init(Lane& L, const ImageConst& I, const RunConst& R, const foort_pixel& p) {
        double x[4], v[4];
        initial_conditions(I, p, x, v);
        ff fx[4], fv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ff_split(x[i], fx[i].hi, fx[i].lo);
            ff_split(v[i], fv[i].hi, fv[i].lo);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int a = i, b = 3 - i;
            L.xh[i] = pack2(fx[a].hi, fx[b].hi);
            L.xl[i] = pack2(fx[a].lo, fx[b].lo);
            L.vh[i] = pack2(fv[a].hi, fv[b].hi);
            L.vl[i] = pack2(fv[a].lo, fv[b].lo);
        }
        L.c.load(I);
        L.hthr[0] = I.mx.hthr[0];
        L.hthr[1] = I.mx.hthr[1];
        // without a horizon (r_h = 0) either threshold ends the ray: the larger one decides
        if (I.m.rh == 0.0 && ff_lt(ff_of(I.mx.hthr), ff_of(I.mx.hthr0))) {
            L.hthr[0] = I.mx.hthr0[0];
            L.hthr[1] = I.mx.hthr0[1];
        }
        L.lam = {0.f, 0.f};
        L.steps = 0;
        L.err = 0;
        L.term = FOORT_TERMCODE_CONTINUE;
        L.passes = 0;
        L.side = 0;
        L.rmin = fx[1];  // Geodesic::Reset's start sample
        diags(L, R);
    }

    // EquatorialPasses and ClosestRadius (MixedEngine::diags) on the new state.
    static __device__ __forceinline__ void diags(Lane& L, const RunConst& R) {
        if (R.diag_flags & FOORT_DIAG_EQUATORIAL_PASSES) {
            const MixedRun& G = R.mr;
            const float thh = hi2(L.xh[1]);
            // (with the low part, which is NaN where theta has overflowed: no sample then)
            const float d0 = __fadd_rn(thh, __fadd_rn(G.mpio2[0], hi2(L.xl[1])));
            bool upd = true, neg = d0 < 0.f;
            if (!(fabsf(d0) > G.eqfar)) {  // near the equator: the float-float difference decides
                const ff dt = ff_add(ff{thh, hi2(L.xl[1])}, ff_of(G.mpio2));
                upd = ff_lt(ff_of(G.eqthr), ff_abs(dt));
                neg = ff_neg_sign(dt);
            }
            const int32_t side = neg ? 1 : 2;
            L.passes += (upd & (L.side + side == 3)) ? 1 : 0;
            L.side = upd ? (thh > 0.f ? side : 0) : L.side;
        }
        if (R.diag_flags & FOORT_DIAG_CLOSEST_RADIUS) {
            const ff x1 = {lo2(L.xh[1]), lo2(L.xl[1])};
            const bool upd = ff_lt(x1, L.rmin);
            L.rmin.hi = upd ? x1.hi : L.rmin.hi;
            L.rmin.lo = upd ? x1.lo : L.rmin.lo;
        }
    }

    // MixedEngine::terms with every termination checked at each step; L.steps counts the
    // steps before this one, as TimeOut's counter does.
    static __device__ __forceinline__ int terms(const Lane& L, const RunConst& R) {
        const MixedRun& G = R.mr;
        int code = FOORT_TERMCODE_CONTINUE;
        if (R.term_flags & FOORT_TERM_THETA_SINGULARITY) {
            // within theps of 0 or pi; well away from both, the high part alone says no
            const float thh = hi2(L.xh[1]);
            if (!(fminf(fabsf(thh), fabsf(__fadd_rn(thh, -G.pi[0]))) > G.thfar)) {
                const ff th = {thh, hi2(L.xl[1])}, e = ff_of(G.theps);
                const bool hit = ff_lt(ff_abs(th), e) | ff_lt(ff_abs(ff_add(ff_of(G.pi), ff_neg(th))), e);
                code = hit ? FOORT_TERMCODE_THETA_SINGULARITY : code;
            }
        }
        if (R.term_flags & FOORT_TERM_TIMEOUT)
            code = (static_cast<uint32_t>(L.steps) >= R.t_max) ? FOORT_TERMCODE_TIMEOUT : code;
        const ff x1 = {lo2(L.xh[1]), lo2(L.xl[1])};
        if (R.term_flags & FOORT_TERM_BOUNDARY_SPHERE)
            code = ff_lt(ff_of(G.bthr), x1) ? FOORT_TERMCODE_BOUNDARY_SPHERE : code;
        if (R.term_flags & FOORT_TERM_HORIZON) code = ff_lt(x1, ff_of(L.hthr)) ? FOORT_TERMCODE_HORIZON : code;
        return code;
    }

    // us = u + t k
    static __device__ __forceinline__ void stage(f2 t, f2 uf03, f2 uf12, const float k[4], float us[4]) {
        const f2 a = p_fma(t, pack2(k[0], k[3]), uf03), b = p_fma(t, pack2(k[1], k[2]), uf12);
        us[0] = lo2(a);
        us[3] = hi2(a);
        us[1] = lo2(b);
        us[2] = hi2(b);
    }

    // MixedEngine::rk4_combine and advance.
    static __device__ __forceinline__ bool advance(Lane& L, const RunConst& R, float h, const float k1[4],
                                                   const float k2[4], const float k3[4], const float k4[4]) {
        const float q0 = __fmul_rn(h, 0.166666672f);
        const float h6 = __fmaf_rn(__fmaf_rn(-6.f, q0, h), 0.166666672f, q0), hh6 = __fmul_rn(h, h6);
        const f2 two = p_all<f2>(2.f), ph = p_all<f2>(h), ph6 = p_all<f2>(h6), phh6 = p_all<f2>(hh6);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const f2 a1 = pack2(k1[i], k1[3 - i]), a2 = pack2(k2[i], k2[3 - i]);
            const f2 a3 = pack2(k3[i], k3[3 - i]), a4 = pack2(k4[i], k4[3 - i]);
            const f2 du = p_mul(ph6, p_add(p_fma(two, a3, p_fma(two, a2, a1)), a4));
            const f2 dxc = p_mul(phh6, p_add(p_add(a1, a2), a3));
            const f2 th = p_mul(ph, L.vh[i]), tl = p_fma(ph, L.vh[i], -th);
            const f2 bl = p_add(tl, p_fma(ph, L.vl[i], dxc));
            f2 s, e;
            p_two_sum(L.xh[i], th, s, e);
            p_fast_two_sum(s, p_add(e, p_add(L.xl[i], bl)), L.xh[i], L.xl[i]);
            p_ff_add_f(L.vh[i], L.vl[i], du, L.vh[i], L.vl[i]);
        }
        return after_step(L, R, ff_add_f(L.lam, h));
    }

    // MixedEngine::after_step
    static __device__ __forceinline__ bool after_step(Lane& L, const RunConst& R, ff lam) {
        L.lam = lam;
        L.term = terms(L, R);
        ++L.steps;
        diags(L, R);
        const bool bad = !(isfinite(lo2(L.xh[1])) & isfinite(lo2(L.vh[1])));
        L.err |= bad ? FOORT_ERR_NONFINITE : 0u;
        return (L.term == FOORT_TERMCODE_CONTINUE) & !(bad & !(R.term_flags & FOORT_TERM_TIMEOUT));
    }

    // Component i of the state as a double.
    static __device__ __forceinline__ double component(const f2 h[2], const f2 l[2], int i) {
        const int k = (i == 1 || i == 2) ? 1 : 0;
        return (i < 2) ? ff_d({lo2(h[k]), lo2(l[k])}) : ff_d({hi2(h[k]), hi2(l[k])});
    }

    static __device__ __forceinline__ void write(const Lane& L, const RunConst& R, foort_result* o, int term,
                                                 uint32_t err) {
        double x[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[i] = component(L.xh, L.xl, i);
            v[i] = component(L.vh, L.vl, i);
        }
        if (!(finite4(x) && finite4(v))) err |= FOORT_ERR_NONFINITE;
        DiagState D;
        D.quad = 0;
        if ((R.diag_flags & FOORT_DIAG_FOUR_COLOR_SCREEN) && term == FOORT_TERMCODE_BOUNDARY_SPHERE)
            D.quad = four_color_quadrant(x[2], x[3]);
        D.passes = (term == FOORT_TERMCODE_HORIZON) ? -L.passes : L.passes;
        D.rmin = -1.0;
        if (R.diag_flags & FOORT_DIAG_CLOSEST_RADIUS) {
            D.rmin = R.rlog ? exp(ff_d(L.rmin)) : ff_d(L.rmin);
            if (term == FOORT_TERMCODE_HORIZON) D.rmin = 0.0;
        }
        write_result(o, term, err, L.steps, ff_d(L.lam), x, v, D);
    }
    static __device__ __forceinline__ void finish(const Lane& L, const RunConst& R, foort_result* o) {
        write(L, R, o, L.term, L.err);
    }
    static __device__ __forceinline__ void stop(const Lane& L, const RunConst& R, foort_result* o, uint32_t err) {
        write(L, R, o, FOORT_TERMCODE_CONTINUE, L.err | err);
    }
};

// RK4 with a packed plugin.
template <int MID, bool RLOG>
struct LeanEngine : LeanState<LeanConst<MID>> {
    using Base = LeanState<LeanConst<MID>>;
    using Lane = typename Base::Lane;
    using Base::advance;
    using Base::stage;
    static constexpr unsigned kRhsPerStep = 4;

    static __device__ __forceinline__ bool step(Lane& L, const RunConst& R) {
        const f2 uf03 = p_add(L.vh[0], L.vl[0]), uf12 = p_add(L.vh[1], L.vl[1]);
        const float uf[4] = {lo2(uf03), lo2(uf12), hi2(uf12), hi2(uf03)};
        const float x1h = lo2(L.xh[1]), x1l = lo2(L.xl[1]), thh = hi2(L.xh[1]), thl = hi2(L.xl[1]);
        const float h = adaptive_step_lean(R.mr, thh, thl, uf[1], uf[2], uf[3]);
        const float hh = 0.5f * h;
        const f2 hh2 = pack2(hh, hh), h2 = pack2(h, h);
        float k1[4], k2[4], k3[4], k4[4], us[4];
        // stages 1 (low half) and 2 (high half)
        f2 ph, pl;
        p_ff_add_f(L.xh[1], L.xl[1], p_mul(hh2, uf12), ph, pl);
        MetricAt<f2> m = metric_lean<MID, RLOG, f2>(L.c, pack2(x1h, lo2(ph)), pack2(x1l, lo2(pl)), pack2(thh, hi2(ph)),
                                                    pack2(thl, hi2(pl)));
        accel_lean<accel_form(MID)>(half_of(m, false), RLOG, uf, k1);
        stage(hh2, uf03, uf12, k1, us);
        accel_lean<accel_form(MID)>(half_of(m, true), RLOG, us, k2);
        // stages 3 and 4: x + h/2 (u + h/2 k1), x + h (u + h/2 k2)
        const f2 hs = pack2(hh, h);
        f2 rh, rl, qh, ql;
        p_ff_add_f(pack2(x1h, x1h), pack2(x1l, x1l),
                   p_mul(hs, p_fma(hh2, pack2(k1[1], k2[1]), pack2(uf[1], uf[1]))), rh, rl);
        p_ff_add_f(pack2(thh, thh), pack2(thl, thl),
                   p_mul(hs, p_fma(hh2, pack2(k1[2], k2[2]), pack2(uf[2], uf[2]))), qh, ql);
        m = metric_lean<MID, RLOG, f2>(L.c, rh, rl, qh, ql);
        stage(hh2, uf03, uf12, k2, us);
        accel_lean<accel_form(MID)>(half_of(m, false), RLOG, us, k3);
        stage(h2, uf03, uf12, k3, us);
        accel_lean<accel_form(MID)>(half_of(m, true), RLOG, us, k4);
        return advance(L, R, h, k1, k2, k3, k4);
    }

    // The step on two lanes (MixedEngine::step_pair): in each of two rounds the even lane
    // evaluates stage 1 (then 3) and the odd lane stage 2 (then 4).
    static __device__ __forceinline__ bool step_pair(Lane& L, const RunConst& R, bool odd, unsigned pmask) {
        const f2 uf03 = p_add(L.vh[0], L.vl[0]), uf12 = p_add(L.vh[1], L.vl[1]);
        const float uf[4] = {lo2(uf03), lo2(uf12), hi2(uf12), hi2(uf03)};
        const f2 x12h = L.xh[1], x12l = L.xl[1];
        const float h = adaptive_step_lean(R.mr, hi2(x12h), hi2(x12l), uf[1], uf[2], uf[3]);
        const float hh = 0.5f * h;
        const f2 hh2 = pack2(hh, hh), h2 = pack2(h, h);
        float k1[4], k2[4], k3[4], k4[4], us[4], ka[4];
        auto share = [&](float k[4], int from) {
#pragma unroll
            for (int i = 0; i < 4; ++i) k[i] = __shfl_sync(pmask, ka[i], from, 2);
        };
        f2 ph, pl;
        p_ff_add_f(x12h, x12l, p_mul(hh2, uf12), ph, pl);
        MetricAt<float> m = metric_lean<MID, RLOG, float>(L.c, odd ? lo2(ph) : lo2(x12h), odd ? lo2(pl) : lo2(x12l),
                                                          odd ? hi2(ph) : hi2(x12h), odd ? hi2(pl) : hi2(x12l));
        accel_lean<accel_form(MID)>(m, RLOG, uf, ka);
        share(k1, 0);
        stage(hh2, uf03, uf12, k1, us);
        accel_lean<accel_form(MID)>(m, RLOG, us, ka);
        share(k2, 1);
        const float hs = odd ? h : hh;
        const f2 k12 = odd ? pack2(k2[1], k2[2]) : pack2(k1[1], k1[2]);
        p_ff_add_f(x12h, x12l, p_mul(pack2(hs, hs), p_fma(hh2, k12, uf12)), ph, pl);
        m = metric_lean<MID, RLOG, float>(L.c, lo2(ph), lo2(pl), hi2(ph), hi2(pl));
        stage(hh2, uf03, uf12, k2, us);
        accel_lean<accel_form(MID)>(m, RLOG, us, ka);
        share(k3, 0);
        stage(h2, uf03, uf12, k3, us);
        accel_lean<accel_form(MID)>(m, RLOG, us, ka);
        share(k4, 1);
        return advance(L, R, h, k1, k2, k3, k4);
    }
};

// Velocity Verlet with its metric part kept from step to step (MixedEngine::
// step_verlet_cached): one metric part per step, so nothing of it to pack but the state's
// update. What it gains over the general kernel are the lean checks and state (for Kerr 67.6
// -> 45.5 ms, 1,600 rays in plain r) and, for Johannsen with alpha13 alone, the body without
// zero terms and with it the registers that held three CTAs to 168 with 1,142 bytes of spills
// (4,096 rays 141 -> 59.5 ms, 147,456 rays 599 -> 281 ms; two CTAs 304, four 275).
template <int MID, bool RLOG>
struct LeanVerletEngine : LeanState<LeanConst<MID>> {
    using Base = LeanState<LeanConst<MID>>;
    static constexpr bool kCountsRhs = true;
    static constexpr int kForm = (MID == kFlat) ? kFlatForm : 0;  // Johannsen's is inlined here

    struct Lane : Base::Lane {
        MetricAt<float> m;  // at (x1, theta)
        uint32_t rhs = 0;
    };

    static __device__ __forceinline__ void init(Lane& L, const ImageConst& I, const RunConst& R, const foort_pixel& p) {
        Base::init(L, I, R, p);
        L.m = metric_lean<MID, RLOG, float>(L.c, lo2(L.xh[1]), lo2(L.xl[1]), hi2(L.xh[1]), hi2(L.xl[1]));
    }

    static __device__ __forceinline__ bool step(Lane& L, const RunConst& R) {
        const MixedRun& G = R.mr;
        const f2 uf03 = p_add(L.vh[0], L.vl[0]), uf12 = p_add(L.vh[1], L.vl[1]);
        const float uf[4] = {lo2(uf03), lo2(uf12), hi2(uf12), hi2(uf03)};
        const float h = adaptive_step_lean(G, hi2(L.xh[1]), hi2(L.xl[1]), uf[1], uf[2], uf[3]);
        float a0[4], a1[4], vi[4];
        accel_lean<kForm>(L.m, RLOG, uf, a0);
        const float h2 = 0.5f * h, hh2 = __fmul_rn(h2, h);
        const f2 ph = p_all<f2>(h), ph2 = p_all<f2>(h2), phh2 = p_all<f2>(hh2);
        const f2 a03 = pack2(a0[0], a0[3]), a12 = pack2(a0[1], a0[2]);
        Base::stage(ph, uf03, uf12, a0, vi);
        // x += h u + h^2/2 a0: x1 and theta as the metric part sees them, then t and phi
        f2 th = p_mul(ph, L.vh[1]), tl = p_fma(ph, L.vh[1], -th), s, e, f, g;
        p_two_sum(L.xh[1], th, s, e);  // ff_add
        p_two_sum(L.xl[1], tl, f, g);
        p_fast_two_sum(s, p_add(e, f), s, e);
        p_fast_two_sum(s, p_add(e, g), s, e);
        p_ff_add_f(s, e, p_fma(ph, L.vl[1], p_mul(phh2, a12)), L.xh[1], L.xl[1]);
        th = p_mul(ph, L.vh[0]);
        tl = p_add(p_fma(ph, L.vh[0], -th), p_fma(ph, L.vl[0], p_mul(phh2, a03)));
        p_two_sum(L.xh[0], th, s, e);
        p_fast_two_sum(s, p_add(e, p_add(L.xl[0], tl)), L.xh[0], L.xl[0]);
        L.m = metric_lean<MID, RLOG, float>(L.c, lo2(L.xh[1]), lo2(L.xl[1]), hi2(L.xh[1]), hi2(L.xl[1]));
        accel_lean<kForm>(L.m, RLOG, vi, a1);
        L.rhs += 2;
        f2 b03 = pack2(a1[0], a1[3]), b12 = pack2(a1[1], a1[2]);
        f2 du03 = p_mul(ph2, p_add(a03, b03)), du12 = p_mul(ph2, p_add(a12, b12));
        if (G.vtol2 > 0.f) {
            f2 dv03 = p_mul(ph2, p_sub(b03, a03)), dv12 = p_mul(ph2, p_sub(b12, a12));
            for (int it = 0;; ++it) {
                const f2 n03 = p_add(uf03, du03), n12 = p_add(uf12, du12);
                const float nv[4] = {lo2(n03), lo2(n12), hi2(n12), hi2(n03)};
                const float dv[4] = {lo2(dv03), lo2(dv12), hi2(dv12), hi2(dv03)};
                float num = __fmul_rn(dv[0], dv[0]), den = __fmul_rn(nv[0], nv[0]);
#pragma unroll
                for (int i = 1; i < 4; ++i) {
                    num = __fmaf_rn(dv[i], dv[i], num);
                    den = __fmaf_rn(nv[i], nv[i], den);
                }
                if (!(num > __fmul_rn(G.vtol2, den))) break;  // num / den > tol^2 with den = |v|^2 > 0
                if (it >= R.verlet_cap) {
                    L.err |= FOORT_ERR_VERLET_ITER;
                    break;
                }
                // (in log-r mode the compiled loop rounds (u^1)^2 before it subtracts it)
                accel_lean<kForm>(L.m, false, nv, a1);
                if (RLOG) a1[1] = __fsub_rn(a1[1], __fmul_rn(nv[1], nv[1]));
                const f2 c03 = pack2(a1[0], a1[3]), c12 = pack2(a1[1], a1[2]);
                dv03 = p_mul(ph2, p_sub(c03, b03));
                dv12 = p_mul(ph2, p_sub(c12, b12));
                b03 = c03;
                b12 = c12;
                du03 = p_mul(ph2, p_add(a03, b03));
                du12 = p_mul(ph2, p_add(a12, b12));
                L.rhs += 1;
            }
        }
        p_ff_add_f(L.vh[0], L.vl[0], du03, L.vh[0], L.vl[0]);
        p_ff_add_f(L.vh[1], L.vl[1], du12, L.vh[1], L.vl[1]);
        return Base::after_step(L, R, ff_add_f(L.lam, h));
    }
};

// RK4 on two lanes with a plugin too large to pack or to inline (Johannsen,
// Rasheed-Larsen): the compiler's scalar body, in one function that both rounds of a step
// call. Its ~900 and ~1,800 instructions set the pace; on one lane the general kernel calls
// it four times in sequence. GB300, log r, the general kernel's one lane and two lanes:
// Johannsen 3,721 geodesics 7.4 and 3.6 ms, 90,000 14.2 and 10.6 ms; Rasheed-Larsen 14.9 and
// 6.9, 38 and 23.5 ms (larger launches: pair_limit, engine.cu). Without a register cap (230
// and 255, Rasheed-Larsen with 124 bytes of spills): capped to three CTAs per SM 90,000 take
// 11.5 and 29.4 ms.
struct ImageRef {
    const MixedConst* mx;
    const double* qa;
    __device__ __forceinline__ void load(const ImageConst& I) {
        mx = &I.mx;
        qa = I.qa;
    }
};

struct TwoK {
    F4 a, b;
};

// One round: the metric part at this lane's stage, contracted with the velocity u (the even
// lane's acceleration counts, k_a) and then with uf + t k_a (the odd lane's, k_b).
template <int MID>
__device__ __noinline__ TwoK round_called(const MixedConst& mc, bool rlog, ff x1, ff th, F4 uf, F4 u, float t,
                                          unsigned pmask) {
    MetricAt<float> m = metric_part<MID, float>(mc.q, mc, rlog, x1, th);
    m.gu.rr = __fmul_rn(-0.5f, m.gu.rr);
    m.gu.hh = __fmul_rn(-0.5f, m.gu.hh);
    auto contract = [&](const float v[4], int from) {
        float a[4];
        accel_lean<accel_form(MID)>(m, rlog, v, a);
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = __shfl_sync(pmask, a[i], from, 2);
        return F4{a[0], a[1], a[2], a[3]};
    };
    const float ua[4] = {u.x, u.y, u.z, u.w};
    TwoK k;
    k.a = contract(ua, 0);
    const float ub[4] = {__fmaf_rn(t, k.a.x, uf.x), __fmaf_rn(t, k.a.y, uf.y), __fmaf_rn(t, k.a.z, uf.z),
                         __fmaf_rn(t, k.a.w, uf.w)};
    k.b = contract(ub, 1);
    return k;
}

template <int MID>
struct LeanCalledEngine : LeanState<ImageRef> {
    static constexpr unsigned kRhsPerStep = 4;

    static __device__ __forceinline__ bool step_pair(Lane& L, const RunConst& R, bool odd, unsigned pmask) {
        const bool rlog = R.rlog != 0;
        const f2 uf03 = p_add(L.vh[0], L.vl[0]), uf12 = p_add(L.vh[1], L.vl[1]);
        const F4 uf = {lo2(uf03), lo2(uf12), hi2(uf12), hi2(uf03)};
        const f2 x12h = L.xh[1], x12l = L.xl[1];
        const float h = adaptive_step_lean(R.mr, hi2(x12h), hi2(x12l), uf.y, uf.z, uf.w);
        const float hh = 0.5f * h;
        const f2 hh2 = pack2(hh, hh);
        f2 ph, pl;
        p_ff_add_f(x12h, x12l, p_mul(hh2, uf12), ph, pl);
        const ff r12 = odd ? ff{lo2(ph), lo2(pl)} : ff{lo2(x12h), lo2(x12l)};
        const ff t12 = odd ? ff{hi2(ph), hi2(pl)} : ff{hi2(x12h), hi2(x12l)};
        const TwoK k12 = round_called<MID>(*L.c.mx, rlog, r12, t12, uf, uf, hh, pmask);
        const float hs = odd ? h : hh;
        const f2 kp = odd ? pack2(k12.b.y, k12.b.z) : pack2(k12.a.y, k12.a.z);
        p_ff_add_f(x12h, x12l, p_mul(pack2(hs, hs), p_fma(hh2, kp, uf12)), ph, pl);
        const f2 us03 = p_fma(hh2, pack2(k12.b.x, k12.b.w), uf03), us12 = p_fma(hh2, pack2(k12.b.y, k12.b.z), uf12);
        const TwoK k34 = round_called<MID>(*L.c.mx, rlog, ff{lo2(ph), lo2(pl)}, ff{hi2(ph), hi2(pl)}, uf,
                                           F4{lo2(us03), lo2(us12), hi2(us12), hi2(us03)}, h, pmask);
        const float k1[4] = {k12.a.x, k12.a.y, k12.a.z, k12.a.w}, k2[4] = {k12.b.x, k12.b.y, k12.b.z, k12.b.w};
        const float k3[4] = {k34.a.x, k34.a.y, k34.a.z, k34.a.w}, k4[4] = {k34.b.x, k34.b.y, k34.b.z, k34.b.w};
        return advance(L, R, h, k1, k2, k3, k4);
    }
};

// FOORT_PREC_FP64_ANALYTIC with RK4 on two lanes per geodesic: step_fp64 (kernel_mixed.cuh)
// with the metric parts of stages 1 and 2, and of 3 and 4, side by side. GB300 takes 64
// cycles per warp for an FP64 instruction however many lanes are active, so a step costs
// its FP64 instructions: about 1,400 on one lane, 850 here.
struct D4 {
    double x, y, z, w;
};
struct TwoKD {
    D4 a, b;
    double bg, bf;  // b.z unrounded: the product of these
};
template <int MID>
__device__ __noinline__ TwoKD round_fp64(const double* q, const MixedConst& mc, bool rlog, double x1, double th, D4 uf,
                                         D4 u, double t, unsigned pmask) {
    MetricAt<double> m = metric_part_d<MID>(q, mc, rlog, x1, th);
    m.gu.rr = __dmul_rn(-0.5, m.gu.rr);
    m.gu.hh = __dmul_rn(-0.5, m.gu.hh);
    double f;
    auto contract = [&](const double v[4], int from) {
        double a[4];
        accel_lean<0>(m, rlog, v, a, &f);
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = __shfl_sync(pmask, a[i], from, 2);
        return D4{a[0], a[1], a[2], a[3]};
    };
    const double ua[4] = {u.x, u.y, u.z, u.w};
    TwoKD k;
    k.a = contract(ua, 0);
    const double ub[4] = {__fma_rn(t, k.a.x, uf.x), __fma_rn(t, k.a.y, uf.y), __fma_rn(t, k.a.z, uf.z),
                          __fma_rn(t, k.a.w, uf.w)};
    k.b = contract(ub, 1);
    k.bg = __shfl_sync(pmask, m.gu.hh, 1, 2);
    k.bf = __shfl_sync(pmask, f, 1, 2);
    return k;
}

template <int MID>
struct AnalyticPairEngine : LeanState<ImageRef> {
    static constexpr unsigned kRhsPerStep = 4;
    static constexpr bool kFp64Steps = true;

    static __device__ __forceinline__ bool step_pair(Lane& L, const RunConst& R, bool odd, unsigned pmask) {
        const bool rlog = R.rlog != 0;
        double x[4], u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[i] = component(L.xh, L.xl, i);
            u[i] = component(L.vh, L.vl, i);
        }
        const double h = adaptive_step_fp64(R, x, u), hh = 0.5 * h;
        const D4 uf = {u[0], u[1], u[2], u[3]};
        auto ahead = [](double a, double t, double b) { return __fma_rn(t, b, a); };  // a + t b
        const TwoKD k12 = round_fp64<MID>(L.c.qa, *L.c.mx, rlog, odd ? ahead(x[1], hh, u[1]) : x[1],
                                          odd ? ahead(x[2], hh, u[2]) : x[2], uf, uf, hh, pmask);
        const double ts = odd ? h : hh, ky = odd ? k12.b.y : k12.a.y, kz = odd ? k12.b.z : k12.a.z;
        const D4 us = {ahead(u[0], hh, k12.b.x), ahead(u[1], hh, k12.b.y), ahead(u[2], hh, k12.b.z),
                       ahead(u[3], hh, k12.b.w)};
        const TwoKD k34 = round_fp64<MID>(L.c.qa, *L.c.mx, rlog, ahead(x[1], ts, ahead(u[1], hh, ky)),
                                          ahead(x[2], ts, ahead(u[2], hh, kz)), uf, us, h, pmask);
        const double k1[4] = {k12.a.x, k12.a.y, k12.a.z, k12.a.w}, k2[4] = {k12.b.x, k12.b.y, k12.b.z, k12.b.w};
        const double k3[4] = {k34.a.x, k34.a.y, k34.a.z, k34.a.w}, k4[4] = {k34.b.x, k34.b.y, k34.b.z, k34.b.w};
        const double h6 = h / 6.0, hh6 = __dmul_rn(h, h6);
        ff nx[4], nv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double s3 = __fma_rn(k3[i], 2.0, __fma_rn(k2[i], 2.0, k1[i]));
            // step_fp64's sum takes k4[2], a product used only here, unrounded
            const double dv = __dmul_rn(i == 2 ? __fma_rn(k34.bg, k34.bf, s3) : __dadd_rn(s3, k4[i]), h6);
            const double dx = __fma_rn(u[i], h, __dmul_rn(__dadd_rn(__dadd_rn(k1[i], k2[i]), k3[i]), hh6));
            nx[i] = ff_from_d(__dadd_rn(x[i], dx));
            nv[i] = ff_from_d(__dadd_rn(u[i], dv));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            L.xh[i] = pack2(nx[i].hi, nx[3 - i].hi);
            L.xl[i] = pack2(nx[i].lo, nx[3 - i].lo);
            L.vh[i] = pack2(nv[i].hi, nv[3 - i].hi);
            L.vl[i] = pack2(nv[i].lo, nv[3 - i].lo);
        }
        return after_step(L, R, ff_add(L.lam, ff_from_d(h)));
    }
};

// The same on eight lanes: lanes 0 to 3 hold stages 1 and 3, lanes 4 to 7 stages 2 and 4. Each
// evaluates its stage's metric part; lane i of four contracts, sums and rounds component i.
// accel_lean<0>'s roundings, with a product alone as fma(x, y, -0): the pair's values. The
// metric part, over half of a step, is the same on all four lanes; the rest is a quarter:
// 4,096 Kerr rays in log r 40 ms on two lanes, 33 on eight.
struct SplitK {
    double k, F;  // a^i, and the sum it is the inverse metric's product with
};
struct SplitTwoK {
    double a, b, bg, bf;
};
static __device__ __forceinline__ double lane4(double a, int lane, unsigned m) { return __shfl_sync(m, a, lane, 4); }

static __device__ __forceinline__ SplitK contract_split(const MetricAt<double>& m, bool rlog, double u, int i,
                                                        unsigned pmask) {
    const bool ends = i == 0 || i == 3;
    double v[4], w1s[4], w2s[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = lane4(u, k, pmask);
    const double ua = ends ? v[0] : u;
    auto lower = [&](const G5T<double>& d) {
        const double A = (i == 0) ? d.tt : (i == 1) ? d.rr : (i == 2) ? d.hh : d.tp, B = (i == 0) ? d.tp : d.pp;
        const double p = __dmul_rn(B, v[3]);
        return __fma_rn(A, ua, ends ? p : -0.0);
    };
    const double w1 = lower(m.d1), w2 = lower(m.d2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        w1s[k] = lane4(w1, k, pmask);
        w2s[k] = lane4(w2, k, pmask);
    }
    auto of = [&](int k) { return (i == 2) ? w2s[k] : w1s[k]; };
    const double qa = __fma_rn(v[0], of(0), __dmul_rn(v[1], of(1))), qh = __dmul_rn(v[2], of(2));
    const double qb = __fma_rn((i == 2) ? 1.0 : v[2], (i == 2) ? qh : of(2), qa);  // q2's product is rounded
    const double q = __fma_rn(v[3], of(3), qb);
    const double s = __fma_rn(v[1], w1, __dmul_rn(v[2], w2));
    SplitK k;
    k.F = __dsub_rn(__dmul_rn(2.0, s), ends ? 0.0 : q);
    const double Ft = lane4(k.F, 0, pmask), Fp = lane4(k.F, 3, pmask);
    const double c1 = (i == 0) ? m.gu.tt : (i == 1) ? m.gu.rr : (i == 2) ? m.gu.hh : m.gu.tp;
    const double p = __dmul_rn((i == 0) ? m.gu.tp : m.gu.pp, Fp);
    k.k = __fma_rn(c1, ends ? Ft : k.F, ends ? p : -0.0);
    k.k = __dmul_rn(ends ? -0.5 : 1.0, k.k);
    if (rlog) {
        const double al = __fma_rn(-u, u, k.k);
        k.k = (i == 1) ? al : k.k;
    }
    return k;
}

// As round_fp64: a of lanes 0 to 3, b of lanes 4 to 7.
template <int MID>
__device__ __noinline__ SplitTwoK round_split(const double* q, const MixedConst& mc, bool rlog, double x, double uf,
                                              double u, double t, int i, unsigned pmask) {
    MetricAt<double> m = metric_part_d<MID>(q, mc, rlog, lane4(x, 1, pmask), lane4(x, 2, pmask));
    m.gu.rr = __dmul_rn(-0.5, m.gu.rr);
    m.gu.hh = __dmul_rn(-0.5, m.gu.hh);
    SplitTwoK k;
    k.a = __shfl_sync(pmask, contract_split(m, rlog, u, i, pmask).k, i, 8);
    const SplitK b = contract_split(m, rlog, __fma_rn(t, k.a, uf), i, pmask);
    k.b = __shfl_sync(pmask, b.k, i + 4, 8);
    k.bg = __shfl_sync(pmask, m.gu.hh, i + 4, 8);
    k.bf = __shfl_sync(pmask, b.F, i + 4, 8);
    return k;
}

template <int MID>
struct AnalyticSplitEngine : LeanState<ImageRef> {
    static constexpr unsigned kRhsPerStep = 4;
    static constexpr bool kFp64Steps = true;

    static __device__ __forceinline__ double own(const f2 h[2], const f2 l[2], int i) {
        const f2 a = (i == 0 || i == 3) ? h[0] : h[1], b = (i == 0 || i == 3) ? l[0] : l[1];
        return (i < 2) ? ff_d({lo2(a), lo2(b)}) : ff_d({hi2(a), hi2(b)});
    }
    // Every lane gets the four components, in parts.
    static __device__ __forceinline__ void share(double a, unsigned pmask, f2 h[2], f2 l[2]) {
        const ff f = ff_from_d(a);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            h[k] = pack2(__shfl_sync(pmask, f.hi, k, 4), __shfl_sync(pmask, f.hi, 3 - k, 4));
            l[k] = pack2(__shfl_sync(pmask, f.lo, k, 4), __shfl_sync(pmask, f.lo, 3 - k, 4));
        }
    }
    // adaptive_step_fp64: lanes 1 to 3 each divide for their component.
    static __device__ __forceinline__ double step_size(const RunConst& R, double x, double u, int i, unsigned pmask) {
        const double pt = __dsub_rn(kRefPi, x), mth = (pt < x) ? pt : x;
        const double num = (i == 2) ? __dmul_rn(R.eps, mth) : R.eps;
        const double w = 1 / fabs(num / fabs(__dadd_rn((i == 3) ? u : fabs(u), 1e-20)));
        const double h = 1 / __dadd_rn(__dadd_rn(lane4(w, 1, pmask), lane4(w, 2, pmask)), lane4(w, 3, pmask));
        return (h < R.hmin) ? R.hmin : h;
    }

    static __device__ __forceinline__ void init(Lane& L, const ImageConst& I, const RunConst& R, const foort_pixel& p,
                                                int, unsigned) {
        LeanState<ImageRef>::init(L, I, R, p);
    }
    static __device__ __forceinline__ bool step_split(Lane& L, const RunConst& R, int sub, unsigned pmask) {
        const bool rlog = R.rlog != 0, odd = sub & 4;
        const int i = sub & 3;
        const double x = own(L.xh, L.xl, i), u = own(L.vh, L.vl, i);
        const double h = step_size(R, x, u, i, pmask), hh = 0.5 * h;
        auto ahead = [](double a, double t, double b) { return __fma_rn(t, b, a); };  // a + t b
        const SplitTwoK k12 =
            round_split<MID>(L.c.qa, *L.c.mx, rlog, odd ? ahead(x, hh, u) : x, u, u, hh, i, pmask);
        const SplitTwoK k34 =
            round_split<MID>(L.c.qa, *L.c.mx, rlog, ahead(x, odd ? h : hh, ahead(u, hh, odd ? k12.b : k12.a)), u,
                             ahead(u, hh, k12.b), h, i, pmask);
        const double h6 = h / 6.0, hh6 = __dmul_rn(h, h6);
        const double s3 = __fma_rn(k34.a, 2.0, __fma_rn(k12.b, 2.0, k12.a));
        // as the pair's: k4 of theta joins unrounded
        const double dv = __dmul_rn(__fma_rn((i == 2) ? k34.bg : 1.0, (i == 2) ? k34.bf : k34.b, s3), h6);
        const double dx = __fma_rn(u, h, __dmul_rn(__dadd_rn(__dadd_rn(k12.a, k12.b), k34.a), hh6));
        share(__dadd_rn(x, dx), pmask, L.xh, L.xl);
        share(__dadd_rn(u, dv), pmask, L.vh, L.vl);
        return after_step(L, R, ff_add(L.lam, ff_from_d(h)));
    }
    static __device__ __forceinline__ void finish(const Lane& L, const RunConst& R, foort_result* o, int sub) {
        if (sub == 0) LeanState<ImageRef>::finish(L, R, o);
    }
    static __device__ __forceinline__ void stop(const Lane& L, const RunConst& R, foort_result* o, uint32_t err,
                                                int sub) {
        if (sub == 0) LeanState<ImageRef>::stop(L, R, o, err);
    }
};

// The tail of a launch of AnalyticPairEngine: a warp's last four geodesics, eight lanes each.
template <int MID>
struct AnalyticTail {
    using S = AnalyticSplitEngine<MID>;
    static constexpr unsigned kLeft = 4;

    static __device__ __forceinline__ void run(const LaunchArgs& A, const RunConst& R, const typename S::Lane& L,
                                               unsigned left, uint64_t idx) {
        unsigned rest = left;
        for (unsigned k = 0; k < (threadIdx.x & 31) >> 3; ++k) rest &= rest - 1;
        const bool active = rest != 0;
        const int src = __ffs(active ? rest : left) - 1;
        typename S::Lane T = from_lane(L, src);
        work_loop<S, 8, NoTail>(A, R, T, active, from_lane(idx, src), true);
    }
};

// A lean engine that records positions (Fp64Engine's and MixedEngine's samples): the second
// pass of foort_gpu_positions takes the first one's steps. 3,600 Kerr rays in Verlet, ln r, 25
// positions kept of each: 2.06 ms with the general kernel, 1.25 with this (1.09 without
// recording).
template <class E>
struct Recording : E {
    static constexpr bool kRecords = true;

    struct Lane : E::Lane {
        GeoposRec gp;  // set by the loop before init (dst null: not recording)
    };

    static __device__ __forceinline__ void sample(Lane& L, const RunConst& R, double lam) {
        if (!L.gp.dst) return;
        if (double* d = geopos_slot(L.gp, R, lam, L.term)) {  // as MixedEngine::geopos
            float4* f = reinterpret_cast<float4*>(d);
            f[0] = make_float4(lo2(L.xh[0]), lo2(L.xl[0]), lo2(L.xh[1]), lo2(L.xl[1]));
            f[1] = make_float4(hi2(L.xh[1]), hi2(L.xl[1]), hi2(L.xh[0]), hi2(L.xl[0]));
        }
    }
    static __device__ __forceinline__ void init(Lane& L, const ImageConst& I, const RunConst& R, const foort_pixel& p) {
        E::init(L, I, R, p);
        sample(L, R, 0.0);
    }
    static __device__ __forceinline__ bool step(Lane& L, const RunConst& R) {
        const bool more = E::step(L, R);
        sample(L, R, 1.0);  // lambda > 0 after a step; only compared with 0
        return more;
    }
    static __device__ __forceinline__ bool step_pair(Lane& L, const RunConst& R, bool odd, unsigned pmask) {
        const bool more = E::step_pair(L, R, odd, pmask);
        sample(L, R, 1.0);
        return more;
    }
};

template <class E, int LANES, int CTAS, class Tail = NoTail>
__global__ void __launch_bounds__(128, CTAS) integrate_lean_kernel(const __grid_constant__ LaunchArgs A,
                                                                   const __grid_constant__ RunConst R) {
    persistent_loop<E, LANES, Tail>(A, R);
}

template <class E, int LANES, int CTAS = 1>
const void* lean_kernel(bool positions) {
    return positions ? reinterpret_cast<const void*>(&integrate_lean_kernel<Recording<E>, LANES, CTAS>)
                     : reinterpret_cast<const void*>(&integrate_lean_kernel<E, LANES, CTAS>);
}

}  // namespace foort
