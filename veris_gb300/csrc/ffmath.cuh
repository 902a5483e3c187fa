// Double-float arithmetic: a value as the unevaluated sum of two floats, h the
// nearest float of it, about 2^-47 of it precise (T. J. Dekker, Numer. Math.
// 18 (1971) 224; D. E. Knuth's two-sum).  GB300 runs float32 at 64 times its
// float64 rate, so a dozen float32 operations cost a fifth of one float64
// operation.  The intrinsics keep the compiler from contracting a product
// whose rounding error is formed separately.
#pragma once

#include "f64math.cuh"

namespace veris {

struct Ff {
    float h, l;
};

// h + l for |a| >= |b|
__device__ __forceinline__ Ff ff_fast_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Ff ff_sum(float a, float b) {
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Ff ff_add(Ff a, Ff b) {
    const Ff s = ff_sum(a.h, b.h);
    return ff_fast_sum(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ Ff ff_add(Ff a, float b) {
    const Ff s = ff_sum(a.h, b);
    return ff_fast_sum(s.h, s.l + a.l);
}
__device__ __forceinline__ Ff ff_mul(Ff a, Ff b) {
    const float p = __fmul_rn(a.h, b.h);
    return ff_fast_sum(p, fmaf(a.h, b.h, -p) + fmaf(a.h, b.l, __fmul_rn(a.l, b.h)));
}
__device__ __forceinline__ Ff ff_mul(Ff a, float b) {
    const float p = __fmul_rn(a.h, b);
    return ff_fast_sum(p, fmaf(a.h, b, -p) + __fmul_rn(a.l, b));
}
__device__ __forceinline__ Ff ff_neg(Ff a) { return {-a.h, -a.l}; }

// one float64 operation each way; outside the float range infinite or NaN
__device__ __forceinline__ Ff ff_of(double x) {
    const float h = narrow(x);
    return {h, narrow(x - widen(h))};
}
__device__ __forceinline__ double ff_value(Ff a) { return widen(a.h) + widen(a.l); }

}  // namespace veris
