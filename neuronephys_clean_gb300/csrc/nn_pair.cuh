// Unevaluated sums of two floats (about 48 bits), for the few operations that
// need more than FP32 on a chip whose FP64 pipe is narrow.  Sums and products
// by the error-free transformations of Knuth and Dekker (T. J. Dekker, "A
// floating-point technique for extending the available precision", Numer.
// Math. 18, 1971); every operation is explicitly rounded.  h is the nearest
// float to h + l.
#pragma once

struct Pair {
    float h, l;
};

__device__ __forceinline__ Pair pair_norm(float h, float l)
{
    const float s = __fadd_rn(h, l);
    return {s, __fsub_rn(l, __fsub_rn(s, h))};
}
__device__ __forceinline__ Pair pair_add(const Pair& x, const Pair& y)
{
    const float s = __fadd_rn(x.h, y.h), t = __fsub_rn(s, x.h);
    const float e = __fadd_rn(__fsub_rn(x.h, __fsub_rn(s, t)), __fsub_rn(y.h, t));
    return pair_norm(s, __fadd_rn(e, __fadd_rn(x.l, y.l)));
}
__device__ __forceinline__ Pair pair_mul(const Pair& x, const Pair& y)
{
    const float p = __fmul_rn(x.h, y.h);
    return pair_norm(p, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.h, y.h, -p))));
}
__device__ __forceinline__ Pair pair_div(const Pair& x, const Pair& y)
{
    const float q = __fdividef(x.h, y.h);
    const float r = __fadd_rn(__fmaf_rn(-q, y.h, x.h), __fmaf_rn(-q, y.l, x.l));
    return pair_norm(q, __fdividef(r, y.h));
}
__device__ __forceinline__ Pair pair_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Pair pair_mulf(const Pair& x, float y)
{
    const float p = __fmul_rn(x.h, y);
    return pair_norm(p, __fmaf_rn(x.l, y, __fmaf_rn(x.h, y, -p)));
}
