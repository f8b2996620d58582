// The FP64 right-hand side of Kerr and Johannsen with every rounding written out, as the
// compiler contracts Fp64Engine's expressions (found by comparing evaluations). The kernels
// that take a geodesic on one lane, on two, or share its step between four or eight
// (kernel_fp64.cuh, kernel_fp64_split.cuh) use these, so that their results are the same bit
// for bit whatever a compiler would contract: foort_gpu_positions retraces a launch that may
// have run on another of them.
#pragma once

#include "kernel_common.cuh"

namespace foort {

__device__ __forceinline__ double d_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double d_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double d_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double d_sub(double a, double b) { return __dsub_rn(a, b); }

// p q - t s, the difference of g_phiphi's numerator: the compiler fuses the first product
// where it belongs to this point alone (r + h and r - h), the second where several points
// share the first.
__device__ __forceinline__ double product_difference(double p, double t, double s, bool own) {
    const double a = own ? p : -t, b = own ? p : s;  // the fused product
    const double c = own ? -t : p, d = own ? s : p;  // the rounded one
    return d_fma(a, b, d_mul(c, d));
}

// Metrics: dd(M, r, s, c, rlog, own) = g_dd; uu(M, r, s, c, rlog, i, g1, g2) = the inverse
// components of lane i: g1 = g^tt, g^rr, g^thth or g^phiphi, g2 = g^tphi.
template <int MID, bool A13>
struct RoundedMetric;

template <>
struct RoundedMetric<kKerr, false> {
    static constexpr bool kOwnR = true;

    static __device__ __forceinline__ G5 dd(const double* q, double r, double s, double c, bool rlog, bool own) {
        const double a = q[0], aa = d_mul(a, a), rr = d_mul(r, r), r2 = d_mul(2.0, r);
        const double sig = d_fma(d_mul(aa, c), c, rr), x = d_add(rr, aa), del = d_sub(x, r2);
        const double A = product_difference(x, d_mul(d_mul(d_mul(del, a), a), s), s, own);
        G5 g;
        g.tt = -d_sub(1.0, r2 / sig);
        g.rr = sig / del;
        g.hh = sig;
        g.pp = d_mul(d_mul(A / sig, s), s);
        g.tp = -(d_mul(d_mul(d_mul(d_mul(2.0, a), r), s), s) / sig);
        if (rlog) g.rr = d_mul(g.rr, rr);
        return g;
    }
    static __device__ __forceinline__ void uu(const double* q, double r, double s, double c, bool rlog, int i,
                                              double& g1, double& g2) {
        const double a = q[0], aa = d_mul(a, a), rr = d_mul(r, r), r2 = d_mul(2.0, r);
        const double sig = d_fma(d_mul(aa, c), c, rr), x = d_add(rr, aa), del = d_sub(x, r2);
        const double A = product_difference(x, d_mul(d_mul(d_mul(del, a), a), s), s, false);
        const double sd = d_mul(sig, del);
        const double num = (i == 0) ? -A : (i == 1) ? del : (i == 2) ? 1.0 : d_fma(-d_mul(aa, s), s, del);
        const double den = (i == 0) ? sd : (i == 3) ? d_mul(d_mul(sd, s), s) : sig;
        g1 = num / den;
        g2 = -(d_mul(d_mul(2.0, a), r) / sd);
        if (rlog && i == 1) g1 = d_mul(g1, 1.0 / rr);
    }
};

// Johannsen. A13: alpha22, alpha52 and epsilon3 are 0, whose terms vanish exactly.
template <bool A13>
struct RoundedMetric<kJohannsen, A13> {
    static constexpr bool kOwnR = true;

    struct Parts {
        double A1, A2, A5, rho2, del, ra, aa, rr;
    };
    static __device__ __forceinline__ Parts parts(const double* q, double r, double c) {
        const double a = q[0];
        Parts p;
        p.aa = d_mul(a, a);
        p.rr = d_mul(r, r);
        p.A1 = d_add(1.0, q[1] / d_mul(p.rr, r));
        p.rho2 = d_fma(d_mul(p.aa, c), c, p.rr);
        if (!A13) {
            p.A2 = d_add(1.0, q[2] / p.rr);
            p.A5 = d_add(1.0, q[3] / p.rr);
            p.rho2 = d_add(p.rho2, q[4] / r);
        }
        const double x = d_add(p.rr, p.aa);
        p.del = d_sub(x, d_mul(2.0, r));
        p.ra = d_mul(x, p.A1);
        return p;
    }
    static __device__ __forceinline__ double times(double x, double A) { return A13 ? x : d_mul(x, A); }

    static __device__ __forceinline__ G5 dd(const double* q, double r, double s, double c, bool rlog, bool own) {
        const double a = q[0];
        const Parts p = parts(q, r, c);
        const double a2 = times(p.aa, p.A2);
        const double den = d_fma(-d_mul(a2, s), s, p.ra), den2 = d_mul(den, den);
        G5 g;
        g.tt = -(d_mul(p.rho2, d_fma(-d_mul(times(a2, p.A2), s), s, p.del)) / den2);
        g.rr = p.rho2 / times(p.del, p.A5);
        g.hh = p.rho2;
        const double n = product_difference(p.ra, d_mul(d_mul(p.aa, p.del), s), s, own);
        g.pp = d_mul(d_mul(d_mul(p.rho2, s), s), n) / den2;
        const double w = A13 ? d_sub(p.ra, p.del) : d_fma(p.ra, p.A2, -p.del);
        g.tp = -(d_mul(d_mul(d_mul(d_mul(a, w), p.rho2), s), s) / den2);
        if (rlog) g.rr = d_mul(g.rr, p.rr);
        return g;
    }
    static __device__ __forceinline__ void uu(const double* q, double r, double s, double c, bool rlog, int i,
                                              double& g1, double& g2) {
        const double a = q[0];
        const Parts p = parts(q, r, c);
        const double a2 = times(times(p.aa, p.A2), p.A2);
        const double n = d_fma(d_mul(d_mul(p.aa, p.del), s), s, -d_mul(p.ra, p.ra));
        const double dr = d_mul(p.del, p.rho2);
        const double num = (i == 0)   ? n
                           : (i == 1) ? times(p.del, p.A5)
                           : (i == 2) ? 1.0
                                      : d_fma(-d_mul(a2, s), s, p.del);
        const double den = (i == 0) ? dr : (i == 3) ? d_mul(d_mul(dr, s), s) : p.rho2;
        g1 = num / den;
        const double x = d_add(p.rr, p.aa);
        const double w = d_fma(A13 ? p.A1 : d_mul(p.A2, p.A1), x, -p.del);
        g2 = -(d_mul(a, w) / dr);
        if (rlog && i == 1) g1 = d_mul(g1, 1.0 / p.rr);
    }
};

// Every inverse component.
template <class Metric>
__device__ __forceinline__ G5 rounded_inverse(const MetricConst& M, double r, double s, double c, bool rlog) {
    G5 g;
    Metric::uu(M.q, r, s, c, rlog, 0, g.tt, g.tp);
    Metric::uu(M.q, r, s, c, rlog, 1, g.rr, g.tp);
    Metric::uu(M.q, r, s, c, rlog, 2, g.hh, g.tp);
    Metric::uu(M.q, r, s, c, rlog, 3, g.pp, g.tp);
    return g;
}

// (x + x) - x of the symbols with three like indices (gen_fd_christoffel.inc): x, but NaN or
// infinite where the sum is.
__device__ __forceinline__ double twice_less_once(double x) {
    return ((__double2hiint(x) & 0x7fffffff) < 0x7fe00000) ? x : d_sub(d_add(x, x), x);
}
__device__ __forceinline__ double two_products(double a, double x, double b, double y) {
    return d_fma(a, x, d_mul(b, y));
}

// The Christoffel symbols that a^i needs, from the central differences of g_dd and the inverse
// metric's g1 (g^tt, g^rr, g^thth or g^phiphi) and g2 = g^tphi: for t and phi Gamma^i_01, _02,
// _13, _23 in C[0..3], for r and theta Gamma^i_00, _03, _11, _12, _22, _33 in C[0..5].
template <int MID>
__device__ __forceinline__ void rounded_symbols(const G5& dr, const G5& dh, double g1, double g2, int i, double C[6],
                                                double* kept) {
    const double h1 = d_mul(0.5, g1), h2 = d_mul(0.5, g2);
    const bool ends = i == 0 || i == 3;
    // t: 0.5 g^tt d_. g_t. + 0.5 g^tphi d_. g_phi.; phi: 0.5 g^tphi d_. g_t. + 0.5 g^phiphi d_. g_phi.
    // (r and theta have no second product: 1 times -0, which adds nothing; g^tphi may be infinite)
    const double own = (i == 1) ? dr.rr : dh.hh, self = twice_less_once(own);
    const double ha = (i == 3) ? h2 : h1, hb = (i == 3) ? h1 : (i == 0) ? h2 : 1.0;
    const double a0 = ends ? dr.tt : (i == 1) ? -dr.tt : -dh.tt, b0 = ends ? dr.tp : -0.0;
    const double a1 = ends ? dh.tt : (i == 1) ? -dr.tp : -dh.tp, b1 = ends ? dh.tp : -0.0;
    const double a2 = ends ? dr.tp : (i == 1) ? self : -dh.rr, b2 = ends ? dr.pp : -0.0;
    const double a3 = ends ? dh.tp : (i == 1) ? dh.rr : dr.hh, b3 = ends ? dh.pp : -0.0;
    const double a4 = (i == 1) ? -dr.hh : self, a5 = (i == 1) ? -dr.pp : -dh.pp;
    // The compiler fuses the first product of a sum, but the second in Kerr's Gamma^t_01 and
    // Gamma^t_02; not so in Verlet's symbols of the position it starts from, kept for it.
    const bool swap = MID == kKerr && i == 0;
    C[0] = two_products(swap ? hb : ha, swap ? b0 : a0, swap ? ha : hb, swap ? a0 : b0);
    C[1] = two_products(swap ? hb : ha, swap ? b1 : a1, swap ? ha : hb, swap ? a1 : b1);
    if (MID == kKerr && kept) {
        kept[0] = two_products(ha, a0, hb, b0);
        kept[1] = two_products(ha, a1, hb, b1);
    }
    C[2] = two_products(ha, a2, hb, b2);
    C[3] = two_products(ha, a3, hb, b3);
    C[4] = d_mul(ha, a4);
    C[5] = d_mul(ha, a5);
}

// a^i = -Gamma^i_jk v^j v^k in the reference's order of terms.
__device__ __forceinline__ double rounded_accel(const double C[6], const double v[4], int i) {
    const bool ends = i == 0 || i == 3;
    const double q0 = ends ? v[1] : v[0], q1 = ends ? v[2] : v[3], q2 = ends ? v[0] : v[1], q3 = ends ? v[3] : v[2];
    const double q4 = ends ? v[0] : v[1], q5 = ends ? v[3] : v[2], q6 = ends ? v[1] : v[0], q7 = ends ? v[2] : v[3];
    const double c2 = ends ? C[0] : C[2], c3 = ends ? C[2] : C[3], c4 = ends ? C[1] : C[3];
    const double c5 = ends ? C[3] : C[4], c6 = ends ? C[2] : C[1], c7 = ends ? C[3] : C[5];
    const double t0 = d_mul(C[0], v[0]), t1 = d_mul(C[1], v[0]);
    double acc = -d_fma(t0, q0, d_mul(t1, q1));
    acc = d_fma(-d_mul(c2, v[1]), q2, acc);
    acc = d_fma(-d_mul(c3, v[1]), q3, acc);
    acc = d_fma(-d_mul(c4, v[2]), q4, acc);
    acc = d_fma(-d_mul(c5, v[2]), q5, acc);
    acc = d_fma(-d_mul(c6, v[3]), q6, acc);
    return d_fma(-d_mul(c7, v[3]), q7, acc);
}

}  // namespace foort
