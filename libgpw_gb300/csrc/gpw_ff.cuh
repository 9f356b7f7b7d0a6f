// Float-float ("double-single") arithmetic on the FP32 pipe.  GB300 runs FP64 at
// about 1/64 of its FP32 rate, so the mixed path keeps ~44-bit intermediates as
// unevaluated sums hi + lo of two floats.  All operations use round-to-nearest
// intrinsics so that the compiler cannot contract or reorder them.
#pragma once

#include <cuda_runtime.h>

namespace gpw {

// 8-byte aligned, so that shared-memory arrays of ff load and store as one
// 64-bit access per element
struct alignas(8) ff {
    float hi, lo;
};

__device__ __forceinline__ ff ff_make(float a) { return {a, 0.0f}; }

__device__ __forceinline__ ff ff_from_double(double d) {
    const float h = __double2float_rn(d);
    return {h, __double2float_rn(d - (double)h)};
}

__device__ __forceinline__ double ff_to_double(ff a) { return (double)a.hi + (double)a.lo; }

// s + e == a + b exactly (Knuth)
__device__ __forceinline__ ff two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return {s, e};
}

// requires |a| >= |b|
__device__ __forceinline__ ff fast_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ ff ff_add(ff a, ff b) {
    ff s = two_sum(a.hi, b.hi);
    s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ ff ff_mul(ff a, ff b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ ff ff_mul_f(ff a, float b) {
    const float p = __fmul_rn(a.hi, b);
    float e = __fmaf_rn(a.hi, b, -p);
    e = __fmaf_rn(a.lo, b, e);
    return fast_two_sum(p, e);
}

// a*b + c in one pass: exact product error by FMA, exact sum with c.hi, one renormalisation
__device__ __forceinline__ ff ff_fma(ff a, ff b, ff c) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    const ff s = two_sum(p, c.hi);
    const float t = __fadd_rn(s.lo, __fadd_rn(e, c.lo));
    return fast_two_sum(s.hi, t);
}

// s += a*b with the sum kept unnormalised: s.hi takes the rounded sum of the
// leading products (exact error by two-sum), s.lo gathers the errors and the
// cross terms.  |s.lo| stays a few ulps of s.hi over short sums; normalise with
// ff_add / fast_two_sum before the value is used elsewhere.
__device__ __forceinline__ void ff_acc_lazy(ff &s, ff a, ff b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    const ff t = two_sum(s.hi, p);
    s.hi = t.hi;
    s.lo = __fadd_rn(s.lo, __fadd_rn(t.lo, e));
}

// Two independent floats per instruction (FFMA2 / FADD2 / FMUL2): the same
// round-to-nearest results as the scalar operations, half the instructions.  A packed
// instruction takes two cycles of the FP32 pipe (measured: 1.88 a cycle and SM against
// 3.62 FFMA), so it adds no peak rate; what it saves is issue slots, instruction fetch
// and the length of dependent chains, which bound the tiled kernels.  With the slicing
// and the readout packed, then stages 1 and 2, collocate went from 87.6 to 78.8 to
// 70.7 ms (100k pairs, 256^3; 7270 to 6220 warp instructions per item).
// a - b is formed as fma(b, -1, a), which rounds once as the subtraction does.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.0f), a); }
// round to integers, |a| < 2^22: adding and subtracting 1.5 * 2^23 rounds to nearest
// even as rintf does, on the FP32 pipe instead of the conversion pipe's quarter rate
__device__ __forceinline__ float2 f2_rint(float2 a) { return f2_add(f2_add(a, f2(12582912.0f)), f2(-12582912.0f)); }

__device__ __forceinline__ float2 f2_neg(float2 a) { return make_float2(-a.x, -a.y); }
// two independent float-float values, operation by operation as the scalar forms above
struct ff2 {
    float2 hi, lo;
};
__device__ __forceinline__ ff2 ff2_dup(ff a) { return {f2(a.hi), f2(a.lo)}; }
__device__ __forceinline__ ff2 ff2_pair(ff a, ff b) { return {make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)}; }
__device__ __forceinline__ ff2 two_sum2(float2 a, float2 b) {
    const float2 s = f2_add(a, b), bb = f2_sub(s, a);
    return {s, f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb))};
}
__device__ __forceinline__ ff2 fast_two_sum2(float2 a, float2 b) {
    const float2 s = f2_add(a, b);
    return {s, f2_sub(b, f2_sub(s, a))};
}
__device__ __forceinline__ ff2 ff2_add(ff2 a, ff2 b) {
    const ff2 s = two_sum2(a.hi, b.hi);
    return fast_two_sum2(s.hi, f2_add(s.lo, f2_add(a.lo, b.lo)));
}
// A factor with its negatives at hand: the product's error needs a b and -(a b), and a
// table that many products read keeps both signs instead of turning one each time.
struct ff2n {
    float2 hi, nhi, nlo;  // b.hi, -b.hi, -b.lo
};
__device__ __forceinline__ ff2n ff2n_dup(ff a) { return {f2(a.hi), f2(-a.hi), f2(-a.lo)}; }
// the leading product and its error terms: a b = p - n
__device__ __forceinline__ ff2 ff2_prodn(ff2 a, ff2n b) {
    const float2 p = f2_mul(a.hi, b.hi);
    float2 n = f2_fma(a.hi, b.nhi, p);
    n = f2_fma(a.hi, b.nlo, n);
    n = f2_fma(a.lo, b.nhi, n);
    return {p, n};
}
__device__ __forceinline__ ff2 ff2_mul(ff2 a, ff2n b) {
    const ff2 q = ff2_prodn(a, b);
    return fast_two_sum2(q.hi, f2_neg(q.lo));
}
__device__ __forceinline__ ff2 ff2_fma(ff2 a, ff2n b, ff2 c) {
    const ff2 q = ff2_prodn(a, b), s = two_sum2(q.hi, c.hi);
    return fast_two_sum2(s.hi, f2_add(s.lo, f2_sub(c.lo, q.lo)));
}
__device__ __forceinline__ void ff2_acc_lazy(ff2 &s, ff2 a, ff2n b) {
    const ff2 q = ff2_prodn(a, b), t = two_sum2(s.hi, q.hi);
    s.hi = t.hi;
    s.lo = f2_add(s.lo, f2_sub(t.lo, q.lo));
}

// 2^(j/32), j = 0..31, as float-float (hi = the float nearest, lo = the rest)
__constant__ float2 c_exp2_32[32] = {
    {1.0f, 0.0f},
    {1.0218971967697144f, -4.811559861650494e-08f},
    {1.0442737340927124f, 4.8334701574503924e-08f},
    {1.0671404600143433f, -5.9337519786595294e-08f},
    {1.0905077457427979f, -1.3077539939843064e-08f},
    {1.114386796951294f, -5.435540018083884e-08f},
    {1.1387885808944702f, 5.386222312608879e-08f},
    {1.1637248992919922f, -4.051441493402308e-08f},
    {1.1892070770263672f, 3.797635272917432e-08f},
    {1.215247392654419f, -3.267394887984665e-08f},
    {1.2418577671051025f, 4.496838101886169e-08f},
    {1.2690509557724f, 1.419333317542737e-09f},
    {1.2968395948410034f, -4.018999533172973e-08f},
    {1.3252366781234741f, -3.496373324196611e-08f},
    {1.3542555570602417f, -1.0123349269974824e-08f},
    {1.3839099407196045f, -5.875577357983275e-08f},
    {1.4142135381698608f, 2.4203234971764687e-08f},
    {1.4451807737350464f, 3.324199937537742e-08f},
    {1.4768261909484863f, -4.500898853621038e-08f},
    {1.5091644525527954f, -2.4959373234878512e-08f},
    {1.5422108173370361f, 8.070904833346049e-09f},
    {1.5759809017181396f, -5.661025426206834e-08f},
    {1.610490322113037f, 9.836217174097328e-09f},
    {1.6457555294036865f, -5.124972091152813e-08f},
    {1.6817928552627563f, -2.4755326677450284e-08f},
    {1.7186193466186523f, -4.8496175963919086e-08f},
    {1.7562521696090698f, -9.235770370707996e-09f},
    {1.7947090864181519f, -1.141504490931311e-08f},
    {1.8340080976486206f, -1.1239277952768134e-08f},
    {1.8741676807403564f, -4.663005626071026e-08f},
    {1.9152065515518188f, 9.845328108326612e-09f},
    {1.9571441411972046f, -1.7021804410433106e-08f}};

// exp(a) in float-float, table-driven (Tang's method): a = (32 m + j) ln2/32 + r
// with k = 32 m + j = round(a 32/ln2), |r| <= ln2/64, so exp(a) = 2^m 2^(j/32) exp(r).
// ln2/32 is split Cody-Waite style as C1 (11 significant bits: k C1 and a - k C1
// are exact for |k| < 2^13) plus the float-float C2 + C3.  exp(r) = 1 + r + r^2 h
// with h = 1/2 + r/6 + r^2/24 + r^3/120 (the tail after r^2/2 is below 2^-20 and
// needs only float precision; truncation r^6/720 < 2^-48).  Relative error about
// 2^-45 while the result is a normal float with a normal low part (a > -60);
// below, the low part underflows gradually; a.hi < -103 returns 0.  Valid for
// a.hi < 88.
__device__ __forceinline__ ff ff_exp(ff a) {
    if (a.hi < -103.0f) return {0.0f, 0.0f};
    const float kf = rintf(__fmul_rn(a.hi, 46.16624069213867f));
    const int k = (int)kf;
    ff r = two_sum(__fmaf_rn(-kf, 0.02166748046875f, a.hi), a.lo);
    r = ff_add(r, ff_mul_f(ff{-6.631076303165173e-06f, 5.14560928046269e-14f}, -kf));
    const float s = r.hi;
    const float t = __fmul_rn(s, __fmaf_rn(s, __fmaf_rn(s, 0.008333333767950535f, 0.0416666679084301f),
                                           0.1666666716337204f));
    const ff h = fast_two_sum(0.5f, t);
    ff p = ff_add(ff_add(ff{1.0f, 0.0f}, r), ff_mul(ff_mul(r, r), h));
    const float2 tj = c_exp2_32[k & 31];
    p = ff_mul(p, ff{tj.x, tj.y});
    // 2^m in two normal-range factors (m >= -149 here)
    const int m = k >> 5, m1 = m >> 1, m2 = m - m1;
    const float s1 = __int_as_float((127 + m1) << 23), s2 = __int_as_float((127 + m2) << 23);
    return {__fmul_rn(__fmul_rn(p.hi, s1), s2), __fmul_rn(__fmul_rn(p.lo, s1), s2)};
}

}  // namespace gpw
