// mph_twofloat.cuh - two-float arithmetic (an unevaluated sum h + l of two
// FP32 numbers, about 47 bits).
#pragma once

namespace mph {

// two-float arithmetic (D. E. Knuth's two-sum; T. J. Dekker)
struct F2 { float h, l; };
__device__ __forceinline__ F2 f2_fast(float h, float l)   // |h| >= |l|
{
    const float s = __fadd_rn(h, l);
    return {s, __fadd_rn(l, -__fadd_rn(s, -h))};
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b)
{
    const float s = __fadd_rn(a.h, b.h), t = __fadd_rn(s, -a.h);
    const float e = __fadd_rn(__fadd_rn(a.h, -__fadd_rn(s, -t)), __fadd_rn(b.h, -t));
    return f2_fast(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b)
{
    const float p = __fmul_rn(a.h, b.h);
    return f2_fast(p, __fadd_rn(__fmaf_rn(a.h, b.h, -p), __fmaf_rn(a.h, b.l, __fmul_rn(a.l, b.h))));
}
// a / b: a first quotient by the approximate reciprocal and two residual
// corrections (Newton's method), without the FP32 division's own chain
__device__ __forceinline__ F2 f2_div(F2 a, F2 b)
{
    const float m = fabsf(b.h);
    if (!(m > 1e-30f && m < 1e30f)) {   // the reciprocal would leave FP32's normal range
        const float q = __fdiv_rn(a.h, b.h);
        const float r = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
        return f2_fast(q, __fdiv_rn(r, b.h));
    }
    const float y = __fdividef(1.f, b.h);
    const float q0 = __fmul_rn(a.h, y);
    const float q = __fmaf_rn(__fmaf_rn(-q0, b.h, a.h), y, q0);
    const float r = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
    return f2_fast(q, __fmul_rn(r, y));
}
__device__ __forceinline__ F2 f2_of(double v)
{
    const float h = (float)v;
    return {h, (float)(v - (double)h)};
}
__device__ __forceinline__ F2 f2_warp_sum(F2 v, int from)
{
    for (int o = from; o > 0; o >>= 1)
        v = f2_add(v, F2{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)});
    return v;
}

// (s, e) with s + e = a + b exactly
__device__ __forceinline__ float f2_two_sum(float a, float b, float& e)
{
    const float s = __fadd_rn(a, b), t = __fadd_rn(s, -a);
    e = __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -t)), __fadd_rn(b, -t));
    return s;
}

}  // namespace mph
