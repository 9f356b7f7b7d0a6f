// Float-float ("double-single") arithmetic on the FP32 pipe.  GB300 runs FP64 at
// about 1/64 of its FP32 rate, so the mixed path keeps ~44-bit intermediates as
// unevaluated sums hi + lo of two floats.  All operations use round-to-nearest
// intrinsics so that the compiler cannot contract or reorder them.
#pragma once

#include <cuda_runtime.h>

#include "gpw_common.cuh"

namespace gpw {

// 8-byte aligned, so that shared-memory arrays of ff load and store as one
// 64-bit access per element
struct alignas(8) ff {
    float hi, lo;
};


// The same split on the integer pipe (a conversion costs as much as an FP64 multiply-add
// here, 17 cycles a warp and SM): the 23 leading mantissa bits rounded to nearest, then
// the signed 29-bit rest.  Values whose low part would leave the normal range of float
// (below 2^-70, zero among them; above 2^126; infinities, NaN) take ff_from_double.
__device__ __forceinline__ ff ff_from_double_bits(double d) {
    const int hw = __double2hiint(d);
    const unsigned lw = (unsigned)__double2loint(d);
    const int e = (hw >> 20) & 0x7ff;  // biased by 1023
    if ((unsigned)(e - (1023 - 70)) > 196u) return {__double2float_rn(d), __double2float_rn(d - (double)__double2float_rn(d))};
    const int up = (int)(lw >> 28) & 1;                   // the rest is half a unit or more
    const int rest = (int)(lw & 0x1fffffffu) - (up << 29);
    const int fb = ((e - 896) << 23 | (hw & 0xfffff) << 3 | (int)(lw >> 29)) + up;
    const float sg = __int_as_float((hw & 0x80000000) | (e - 1023 - 52 + 127) << 23);  // +- 2^(e - 52)
    return {__int_as_float((hw & 0x80000000) | fb), __fmul_rn((float)rest, sg)};
}
// hi + lo (|lo| <= ulp(hi) / 2) as a double, rounded to nearest (ties to even of the low
// part's scale), on the integer pipe; hi below 2^-70 or beyond float's range takes the
// FP64 addition.
__device__ __forceinline__ double ff_to_double_bits(ff a) {
    const int h = __float_as_int(a.hi), e = (h >> 23) & 0xff;  // biased by 127
    if ((unsigned)(e - (127 - 70)) > 196u) return (double)a.hi + (double)a.lo;
    // the low part in units of hi's 2^-52, away from hi's sign: |r| <= 2^28; one binade
    // down where hi is a power of two and the low part takes away from it
    const float u = __int_as_float((h & 0x80000000) | (52 + 127 - (e - 127)) << 23);  // +- 2^(52 - e)
    float r = __fmul_rn(a.lo, u);
    if ((h & 0x7fffff) == 0 && r < 0.0f) r = __fadd_rn(r, r);
    const long long bits = ((long long)(e - 127 + 1023) << 52 | (long long)(h & 0x7fffff) << 29) + (long long)__float2int_rn(r);
    return __hiloint2double((int)(bits >> 32) | (h & 0x80000000), (int)bits);
}

__device__ __forceinline__ ff ff_from_double(double d) {
    const float h = __double2float_rn(d);
    return {h, __double2float_rn(d - (double)h)};
}


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
// s += a b with the sums kept unnormalised: s.hi takes the rounded sum of the leading
// products (exact error by two-sum), s.lo gathers the errors and the cross terms.
// |s.lo| stays a few ulps of s.hi over short sums; normalise before other use.
__device__ __forceinline__ void ff2_acc_lazy(ff2 &s, ff2 a, ff2n b) {
    const ff2 q = ff2_prodn(a, b), t = two_sum2(s.hi, q.hi);
    s.hi = t.hi;
    s.lo = f2_add(s.lo, f2_sub(t.lo, q.lo));
}

__device__ __forceinline__ ff2n ff2n_of(ff2 b) {
    return {b.hi, f2_mul(b.hi, f2(-1.0f)), f2_mul(b.lo, f2(-1.0f))};
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
__device__ __forceinline__ ff ff_exp(ff a, const float2 *tab) {  // tab: c_exp2_32, or its copy in shared memory
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
    const float2 tj = tab[k & 31];
    p = ff_mul(p, ff{tj.x, tj.y});
    // 2^m in two normal-range factors (m >= -149 here)
    const int m = k >> 5, m1 = m >> 1, m2 = m - m1;
    const float s1 = __int_as_float((127 + m1) << 23), s2 = __int_as_float((127 + m2) << 23);
    return {__fmul_rn(__fmul_rn(p.hi, s1), s2), __fmul_rn(__fmul_rn(p.lo, s1), s2)};
}

__device__ __forceinline__ ff ff_exp(ff a) { return ff_exp(a, c_exp2_32); }

// Two exponentials at once, ff_exp operation by operation.  tab: c_exp2_32 in shared
// memory (the lanes' indices differ: a constant-bank read would be replayed per value).
__device__ __forceinline__ ff2 ff2_exp(ff2 a, const float2 *tab) {
    const float2 ah = make_float2(fmaxf(a.hi.x, -104.0f), fmaxf(a.hi.y, -104.0f));
    const float2 km = f2_add(f2_mul(ah, f2(46.16624069213867f)), f2(12582912.0f));  // 1.5 * 2^23 + k
    const float2 nk = f2_sub(f2(12582912.0f), km);                                  // -k
    const int k0 = __float_as_int(km.x) - 0x4b400000, k1 = __float_as_int(km.y) - 0x4b400000;
    ff2 r = two_sum2(f2_fma(nk, f2(0.02166748046875f), ah), a.lo);
    const ff2n c = ff2n_dup(ff{-6.631076303165173e-06f, 5.14560928046269e-14f});
    const float2 cp = f2_mul(nk, c.hi);
    const float2 cn = f2_fma(nk, c.nlo, f2_fma(nk, c.nhi, cp));  // the product's error terms, negated
    r = ff2_add(r, fast_two_sum2(cp, f2_mul(cn, f2(-1.0f))));
    const float2 q = r.hi;
    const float2 t = f2_mul(q, f2_fma(q, f2_fma(q, f2(0.008333333767950535f), f2(0.0416666679084301f)), f2(0.1666666716337204f)));
    const ff2 h = fast_two_sum2(f2(0.5f), t);
    const ff2n rn = ff2n_of(r);
    ff2 p = ff2_add(ff2_add(ff2{f2(1.0f), f2(0.0f)}, r), ff2_mul(h, ff2n_of(ff2_mul(r, rn))));
    const float2 t0 = tab[k0 & 31], t1 = tab[k1 & 31];
    p = ff2_mul(p, ff2n_of(ff2{make_float2(t0.x, t1.x), make_float2(t0.y, t1.y)}));
    auto pw = [](int m) { return __int_as_float((127 + m) << 23); };
    const int m0 = k0 >> 5, m1 = k1 >> 5, u0 = m0 >> 1, u1 = m1 >> 1;
    const float2 s1 = make_float2(a.hi.x < -103.0f ? 0.0f : pw(u0), a.hi.y < -103.0f ? 0.0f : pw(u1));
    const float2 s2 = make_float2(pw(m0 - u0), pw(m1 - u1));
    return {f2_mul(f2_mul(p.hi, s1), s2), f2_mul(f2_mul(p.lo, s1), s2)};
}

// ---------------------------------------------------------------------------
// Where general_row_fast32 is unsure (0.6 % of the rows near a sphere at steps of 0.12,
// so one warp in six): the same quadratic in float-float with its error bound; only
// where that is unsure too the FP64 rule, some 150 instructions of the FP64 pipe.  (9.3e7
// random rows, exact ties among them: no row differs from the FP64 rule.  1500 pairs,
// 128^3, float-float kernel: 7.86 -> 7.65 ms; 8000 pairs, tiled: 17.6 -> 16.9 ms.)
struct GeneralRowFF {
    ff dh[3][3];   // lattice steps
    ff a4, inv2a;  // 4 |v0|^2 and 1 / (2 |v0|^2)
    float hmax;    // largest |dh|
};
__host__ __device__ inline ff ff_split(double d) {
    const float h = (float)d;
    return {h, (float)(d - (double)h)};
}
__host__ __device__ inline void general_row_constants(const double dh[3][3], GeneralRow32 &r, GeneralRowFF &f) {
    const double a = dh[0][0] * dh[0][0] + dh[0][1] * dh[0][1] + dh[0][2] * dh[0][2];
    f.hmax = 0.0f;
    for (int i = 0; i < 3; i++)
        for (int k = 0; k < 3; k++) {
            r.dh[i][k] = (float)dh[i][k];
            f.dh[i][k] = ff_split(dh[i][k]);
            f.hmax = fmaxf(f.hmax, fabsf((float)dh[i][k]));
        }
    r.a = (float)a;
    r.inv2a = (float)(0.5 / a);
    f.a4 = ff_split(4.0 * a);
    f.inv2a = ff_split(0.5 / a);
}
#if defined(__CUDACC__)
// The row (jj, kk) of a box at cc: its i-range, decided by float-float where the bound
// allows, else by FP64.
__device__ __noinline__ inline bool general_row_unsure(const GeneralRowFF *G, const double dh[3][3], const double gp[3],
                                                       int cc0, int jj, int kk, double radius, int &ismin, int &ismax) {
    const ff g0 = ff_from_double_bits(gp[0]), g1 = ff_from_double_bits(gp[1]), g2 = ff_from_double_bits(gp[2]);
    const ff mgi = ff_add(ff{(float)cc0, 0.0f}, ff{-g0.hi, -g0.lo});  // -(gp_0 - cc_0): i' = i - cc_0
    const ff dj = ff_add(ff{(float)jj, 0.0f}, ff{-g1.hi, -g1.lo}), dk = ff_add(ff{(float)kk, 0.0f}, ff{-g2.hi, -g2.lo});
    const ff rad = ff_from_double_bits(radius), r2 = ff_mul(rad, rad);
    ff hb = {0.0f, 0.0f}, c = {0.0f, 0.0f};  // b / 2 and c
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
        const ff v = ff_add(ff_add(ff_mul(G->dh[2][i], dk), ff_mul(G->dh[1][i], dj)), ff_mul(mgi, G->dh[0][i]));
        hb = ff_add(hb, ff_mul(v, G->dh[0][i]));
        c = ff_add(c, ff_mul(v, v));
    }
    const ff b = {2.0f * hb.hi, 2.0f * hb.lo};
    const ff d = ff_add(ff_mul(b, b), ff_mul(ff{-G->a4.hi, -G->a4.lo}, ff_add(c, ff{-r2.hi, -r2.lo})));
    // every operation to 2^-44 of its operands; the largest are bounded by V
    const float eps = 2.3e-13f;  // 2^-42
    const float V = 3.0f * G->hmax * (fabsf(mgi.hi) + fabsf(dj.hi) + fabsf(dk.hi) +
                                      fabsf(g0.hi) + fabsf(g1.hi) + fabsf(g2.hi) + 3.0f);
    const float eb = 6.0f * eps * V * G->hmax;
    const float ed = 2.0f * fabsf(b.hi) * eb + eb * eb + eps * (b.hi * b.hi + G->a4.hi * (6.0f * V * V + r2.hi));
    bool unsure = fabsf(d.hi) <= 4.0f * ed || fabsf((float)jj) > 4.0e6f || fabsf((float)kk) > 4.0e6f || fabsf((float)cc0) > 4.0e6f;
    if (!unsure && d.hi < 0.0f) return false;
    if (!unsure) {
        const float s0 = sqrtf(d.hi);
        const float res = __fadd_rn(__fmaf_rn(-s0, s0, d.hi), d.lo);
        const ff sd = fast_two_sum(s0, res / (2.0f * s0));
        const ff lo = ff_mul(ff_add(ff{-b.hi, -b.lo}, ff{-sd.hi, -sd.lo}), G->inv2a);
        const ff hi = ff_mul(ff_add(ff{-b.hi, -b.lo}, sd), G->inv2a);
        const float er = 2.0f * (eb + ed / s0 + eps * (fabsf(b.hi) + s0)) * G->inv2a.hi + 1e-10f;
        const float l0 = rintf(lo.hi), h0 = rintf(hi.hi);
        const float lf = __fadd_rn(__fsub_rn(lo.hi, l0), lo.lo), hf = __fadd_rn(__fsub_rn(hi.hi, h0), hi.lo);  // from the nearest integer
        unsure = fabsf(lf) <= er || fabsf(hf) <= er;
        ismin = cc0 + (int)l0 + (lf > 0.0f ? 1 : 0);
        ismax = cc0 + (int)h0 - (hf < 0.0f ? 1 : 0);
    }
    if (unsure) return general_row(dh, gp, rsub((double)jj, gp[1]), rsub((double)kk, gp[2]), radius, ismin, ismax);
    return true;
}
#endif

}  // namespace gpw
