// sph_df64.cuh — double-float arithmetic: a value is the unevaluated sum
// hi + lo of two FP32 numbers (|lo| <= ulp(hi)/2), about 48 significant
// bits, computed on the FP32 pipes.
//
// The operations are the error-free transformations of Knuth (two-sum) and
// Dekker (two-product, here with a fused multiply-add), with the
// renormalisation of the double-double literature (Hida, Li and Bailey,
// "Library for double-double and quad-double arithmetic", 2007; Thall,
// "Extended-precision floating-point numbers for GPU computation", 2006).
// Relative error of add/mul about 2^-44 to 2^-46 per operation; the exponent
// range is FP32's.
#pragma once

#include <cuda_runtime.h>

namespace sph {

struct DF {
    float hi, lo;
};

__device__ __forceinline__ DF df(float a) { return DF{a, 0.0f}; }

// FP64 -> double-float (two conversions) and back.
__device__ __forceinline__ DF df_from(double a) {
    const float h = __double2float_rn(a);
    return DF{h, __double2float_rn(a - (double)h)};
}
__device__ __forceinline__ double df_to(const DF& a) { return (double)a.hi + (double)a.lo; }

// s + e = a + b exactly (Knuth); no precondition on |a|, |b|.
__device__ __forceinline__ DF two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return DF{s, e};
}
// s + e = a + b exactly when |a| >= |b| (Dekker).
__device__ __forceinline__ DF quick_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
// p + e = a b exactly.
__device__ __forceinline__ DF two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return DF{p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ DF df_add(const DF& a, const DF& b) {
    DF s = two_sum(a.hi, b.hi);
    const float e = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
    return quick_two_sum(s.hi, e);
}
__device__ __forceinline__ DF df_neg(const DF& a) { return DF{-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_sub(const DF& a, const DF& b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ DF df_add_f(const DF& a, float b) {
    DF s = two_sum(a.hi, b);
    return quick_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}

__device__ __forceinline__ DF df_mul(const DF& a, const DF& b) {
    DF p = two_prod(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.lo, p.lo);
    e = __fmaf_rn(a.lo, b.hi, e);
    return quick_two_sum(p.hi, e);
}
__device__ __forceinline__ DF df_mul_f(const DF& a, float b) {
    DF p = two_prod(a.hi, b);
    return quick_two_sum(p.hi, __fmaf_rn(a.lo, b, p.lo));
}
// a b + c
__device__ __forceinline__ DF df_fma(const DF& a, const DF& b, const DF& c) { return df_add(df_mul(a, b), c); }

// 1 / a and 1 / sqrt(a) (a > 0): an FP32 estimate y0 and the residual of
// y0, which fused multiply-adds give to FP32 accuracy (its leading part is
// exact), so the correction y0 (r + r^2) resp. y0 (r / 2 + 3/8 r^2) adds the low
// half: error about 2^-46, in 8 and 11 FP32 operations (a Newton step in
// double-float arithmetic took 30 and 38).
__device__ __forceinline__ DF df_rcp(const DF& a) {
    const float y0 = __frcp_rn(a.hi);
    const float r = __fmaf_rn(-a.lo, y0, __fmaf_rn(-a.hi, y0, 1.0f));   // 1 - a y0
    return quick_two_sum(y0, __fmul_rn(y0, __fmaf_rn(r, r, r)));
}
__device__ __forceinline__ DF df_rsqrt(const DF& a) {
    const float y0 = rsqrtf(a.hi);
    // 1 - (a y0) y0: a y0 is about sqrt(a), so it and its low half stay normal
    // over FP32's whole range, which y0^2 does not
    const float z = __fmul_rn(a.hi, y0);
    const float zl = __fmaf_rn(a.lo, y0, __fmaf_rn(a.hi, y0, -z));
    const float r = __fmaf_rn(-zl, y0, __fmaf_rn(-z, y0, 1.0f));
    return quick_two_sum(y0, __fmul_rn(y0, __fmaf_rn(__fmul_rn(0.375f, r), r, 0.5f * r)));
}

// Two double-floats advanced together by the packed FP32 instructions (FADD2 /
// FMUL2 / FFMA2): per component the operations of the scalar forms above,
// with subtractions as fused multiply-adds by -1 (which round alike).
struct DF2 {
    float2 hi, lo;
};
__device__ __forceinline__ DF2 df2(const DF& a, const DF& b) {
    return DF2{make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)};
}
__device__ __forceinline__ DF df2_x(const DF2& a) { return DF{a.hi.x, a.lo.x}; }
__device__ __forceinline__ DF df2_y(const DF2& a) { return DF{a.hi.y, a.lo.y}; }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ DF2 two_sum2(float2 a, float2 b) {
    const float2 s = __fadd2_rn(a, b);
    const float2 bb = sub2(s, a);
    return DF2{s, __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ DF2 df2_add(const DF2& a, const DF2& b) {
    const DF2 s = two_sum2(a.hi, b.hi);
    const float2 e = __fadd2_rn(s.lo, __fadd2_rn(a.lo, b.lo));
    const float2 h = __fadd2_rn(s.hi, e);
    return DF2{h, sub2(e, sub2(h, s.hi))};
}
// a - b
__device__ __forceinline__ DF2 df2_sub(const DF2& a, const DF2& b) {
    const float2 m1 = make_float2(-1.0f, -1.0f);
    return df2_add(a, DF2{__fmul2_rn(b.hi, m1), __fmul2_rn(b.lo, m1)});
}
__device__ __forceinline__ DF2 df2_mul(const DF2& a, const DF2& b) {
    const float2 p = __fmul2_rn(a.hi, b.hi);
    const float2 np = __fmul2_rn(p, make_float2(-1.0f, -1.0f));
    float2 e = __ffma2_rn(a.hi, b.hi, np);
    e = __ffma2_rn(a.hi, b.lo, e);
    e = __ffma2_rn(a.lo, b.hi, e);
    const float2 h = __fadd2_rn(p, e);
    return DF2{h, sub2(e, __fadd2_rn(h, np))};
}

// A compensated accumulator of products and sums (the Dot2 scheme of
// Ogita, Rump and Oishi, "Accurate sum and dot product", SIAM J. Sci.
// Comput. 26, 2005, extended to double-float inputs): s collects the
// rounded terms, c their exact rounding errors (two-product, two-sum) and
// the low-order cross terms; the pair is normalised once, at the end.
struct DFAcc {
    float s = 0.0f, c = 0.0f;
    // += a b
    __device__ __forceinline__ void add_prod(const DF& a, const DF& b) {
        const float p = __fmul_rn(a.hi, b.hi);
        float e = __fmaf_rn(a.hi, b.hi, -p);
        e = __fmaf_rn(a.hi, b.lo, e);
        e = __fmaf_rn(a.lo, b.hi, e);
        const DF t = two_sum(s, p);
        s = t.hi;
        c = __fadd_rn(c, __fadd_rn(t.lo, e));
    }
    // += a
    __device__ __forceinline__ void add(const DF& a) {
        const DF t = two_sum(s, a.hi);
        s = t.hi;
        c = __fadd_rn(c, __fadd_rn(t.lo, a.lo));
    }
    __device__ __forceinline__ DF value() const { return two_sum(s, c); }
    __device__ __forceinline__ double to_double() const { return (double)s + (double)c; }
};

// Two of them advanced together.
struct DFAcc2 {
    float2 s = make_float2(0.0f, 0.0f), c = make_float2(0.0f, 0.0f);
    __device__ __forceinline__ void add_prod(const DF2& a, const DF2& b) {
        const float2 p = __fmul2_rn(a.hi, b.hi);
        float2 e = __ffma2_rn(a.hi, b.hi, __fmul2_rn(p, make_float2(-1.0f, -1.0f)));
        e = __ffma2_rn(a.hi, b.lo, e);
        e = __ffma2_rn(a.lo, b.hi, e);
        const DF2 t = two_sum2(s, p);
        s = t.hi;
        c = __fadd2_rn(c, __fadd2_rn(t.lo, e));
    }
    __device__ __forceinline__ void add(const DF2& a) {
        const DF2 t = two_sum2(s, a.hi);
        s = t.hi;
        c = __fadd2_rn(c, __fadd2_rn(t.lo, a.lo));
    }
    __device__ __forceinline__ double x() const { return (double)s.x + (double)c.x; }
    __device__ __forceinline__ double y() const { return (double)s.y + (double)c.y; }
};

}  // namespace sph
