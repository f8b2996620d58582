// Packed FP32 arithmetic (two floats per instruction) for the lean mixed kernels.
//
// sm_103a's fma / add / sub / mul .f32x2 take one issue slot and two cycles of the FP32
// pipe for two operations (measured: 2.0 cycles per warp and sub-partition, dependent
// latency 4.1 cycles, both as two scalar ones), so they do not raise the FP32 peak. They
// free issue slots and register-file bandwidth: 2.5 cycles for one packed FMA beside a
// LOP3 against 4.4 for two scalar FMAs beside a LOP3. Negating operands, exchanging halves and
// moving halves in and out cost nothing measurable.
// The same operations exist for one float (p_mul ...), so that one body serves both.
// Every one rounds to nearest and flushes denormals, as the scalar code of the mixed
// kernels does (-ftz=true).
#pragma once

#include <cuda_runtime.h>

namespace foort {

struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d.v) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(f2 a) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(a.v));
    return d;
}
__device__ __forceinline__ float lo2(f2 a) { return unpack2(a).x; }
__device__ __forceinline__ float hi2(f2 a) { return unpack2(a).y; }
__device__ __forceinline__ f2 operator-(f2 a) {
    const float2 x = unpack2(a);
    return pack2(-x.x, -x.y);
}

__device__ __forceinline__ f2 p_fma(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
// A product is a b + (-0), which rounds the same (and keeps a zero's sign): ptxas merges
// mul.rn.f32x2 with an add.rn.f32x2 or sub.rn.f32x2 of its result into one rounding (seen in
// results; its -fmad=false changes nothing), and a literal -0 is folded away first. From
// constant memory it is a value that ptxas does not know.
static __constant__ unsigned long long kNegZero2 = 0x8000000080000000ull;
__device__ __forceinline__ f2 p_mul(f2 a, f2 b) { return p_fma(a, b, f2{kNegZero2}); }
__device__ __forceinline__ f2 p_add(f2 a, f2 b) {
    f2 d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ f2 p_sub(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ float p_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float p_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float p_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float p_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double p_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double p_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double p_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double p_sub(double a, double b) { return __dsub_rn(a, b); }

// A float in every half, and a function of a float on every half.
template <typename T>
__device__ __forceinline__ T p_all(float a);
template <>
__device__ __forceinline__ float p_all<float>(float a) { return a; }
template <>
__device__ __forceinline__ f2 p_all<f2>(float a) { return pack2(a, a); }

template <class F>
__device__ __forceinline__ float p_each(F f, float a) { return f(a); }
template <class F>
__device__ __forceinline__ f2 p_each(F f, f2 a) {
    const float2 x = unpack2(a);
    return pack2(f(x.x), f(x.y));
}
template <class F>
__device__ __forceinline__ float p_each(F f, float a, float b) { return f(a, b); }
template <class F>
__device__ __forceinline__ f2 p_each(F f, f2 a, f2 b) {
    const float2 x = unpack2(a), y = unpack2(b);
    return pack2(f(x.x, y.x), f(x.y, y.y));
}
template <class F>
__device__ __forceinline__ float p_each(F f, float a, float b, float c) { return f(a, b, c); }
template <class F>
__device__ __forceinline__ f2 p_each(F f, f2 a, f2 b, f2 c) {
    const float2 x = unpack2(a), y = unpack2(b), z = unpack2(c);
    return pack2(f(x.x, y.x, z.x), f(x.y, y.y, z.y));
}
__device__ __forceinline__ bool p_any_above(float a, float bound) { return fabsf(a) > bound; }
__device__ __forceinline__ bool p_any_above(f2 a, float bound) {
    const float2 x = unpack2(a);
    return fmaxf(fabsf(x.x), fabsf(x.y)) > bound;
}

// rcp() of analytic_metric.cuh on every half.
__device__ __forceinline__ float p_rcp(float x) { return rcp(x); }
__device__ __forceinline__ f2 p_rcp(f2 x) {
    const f2 r0 = p_each(
        [](float a) {
            float b;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(a));
            return b;
        },
        x);
    return p_fma(r0, p_fma(-x, r0, p_all<f2>(1.0f)), r0);
}

// Float-float sums on every half (two_sum, fast_two_sum, ff_add_f of kernel_mixed.cuh).
template <typename T>
__device__ __forceinline__ void p_two_sum(T a, T b, T& s, T& e) {
    s = p_add(a, b);
    const T bb = p_sub(s, a);
    e = p_add(p_sub(a, p_sub(s, bb)), p_sub(b, bb));
}
template <typename T>
__device__ __forceinline__ void p_fast_two_sum(T a, T b, T& s, T& e) {
    const T t = p_add(a, b);
    e = p_sub(b, p_sub(t, a));
    s = t;
}
template <typename T>
__device__ __forceinline__ void p_ff_add_f(T ah, T al, T b, T& h, T& l) {
    T s, e;
    p_two_sum(ah, b, s, e);
    p_fast_two_sum(s, p_add(e, al), h, l);
}

// ff_sincos (analytic_metric.cuh) on every half, with the same operations. The quadrant
// k = rint(x) comes from adding 1.5 * 2^23, whose sum holds k in its low bits: two adds
// instead of a rounding and a conversion of 8 issue cycles each per warp. That needs
// |x| < 2^22; angles beyond 10^6 (states on their way to infinity) take ff_sincos itself.
static __device__ __noinline__ float4 sincos_far(float ah, float al, float bh, float bl) {
    float4 r;
    ff_sincos(ah, al, r.x, r.y);
    ff_sincos(bh, bl, r.z, r.w);
    return r;
}
__device__ __forceinline__ void p_sincos_far(float th, float tl, float& s, float& c) {
    const float4 r = sincos_far(th, tl, 0.f, 0.f);
    s = r.x;
    c = r.y;
}
__device__ __forceinline__ void p_sincos_far(f2 th, f2 tl, f2& s, f2& c) {
    const float2 h = unpack2(th), l = unpack2(tl);
    const float4 r = sincos_far(h.x, l.x, h.y, l.y);
    s = pack2(r.x, r.z);
    c = pack2(r.y, r.w);
}
template <typename T>
__device__ __forceinline__ void p_sincos(T th, T tl, T& s, T& c) {
    if (p_any_above(th, 1e6f)) {
        p_sincos_far(th, tl, s, c);
        return;
    }
    auto K = [](float v) { return p_all<T>(v); };
    const T sum = p_add(p_mul(th, K(0.636619772f)), K(12582912.0f));
    const T k = p_sub(sum, K(12582912.0f));
    T d = p_add(p_fma(-k, K(0x1.921fb6p+0f), th), p_fma(-k, K(-0x1.777a5cp-25f), tl));
    d = p_fma(-k, K(-0x1.ee59dap-50f), d);
    const T d2 = p_mul(d, d);
    T sp = p_fma(d2, K(2.75573192e-6f), K(-1.98412698e-4f));
    sp = p_fma(d2, sp, K(8.33333333e-3f));
    sp = p_fma(d2, sp, K(-1.66666667e-1f));
    const T sd = p_fma(p_mul(d, d2), sp, d);
    T cp = p_fma(d2, K(-2.75573192e-7f), K(2.48015873e-5f));
    cp = p_fma(d2, cp, K(-1.38888889e-3f));
    cp = p_fma(d2, cp, K(4.16666667e-2f));
    cp = p_fma(d2, cp, K(-0.5f));
    const T cd = p_fma(d2, cp, K(1.0f));
    // quadrant q: sin = sd, cd, -sd, -cd; cos = cd, -sd, -cd, sd
    s = p_each(
        [](float m, float a, float b) {
            const int q = __float_as_int(m);
            return __int_as_float(__float_as_int((q & 1) ? b : a) ^ ((q << 30) & 0x80000000));
        },
        sum, sd, cd);
    c = p_each(
        [](float m, float a, float b) {
            const int q = __float_as_int(m);
            return __int_as_float(__float_as_int((q & 1) ? a : b) ^ (((q + 1) << 30) & 0x80000000));
        },
        sum, sd, cd);
}

}  // namespace foort
