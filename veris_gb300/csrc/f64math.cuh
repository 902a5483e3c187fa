// Float64 arithmetic off the float64 pipe, for kernels that it bounds: GB300
// has 2 float64 lanes per SM and cycle, 1/64 of its float32 rate.  Division and
// square root in integer and float32 instructions, comparisons and conversions
// on the integer pipe, a table-driven exponential and psi functions; the
// reciprocal square root from the hardware's seed and the series of the exact
// correction.  No slow paths inside: a lane or warp whose operands leave a safe
// exponent range takes IEEE division or square root instead.
#pragma once
#include <cuda_runtime.h>

#include "f64tables.cuh"

namespace veris {

__device__ __forceinline__ double rsqrt_seed(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// positive, normal, and at least 2^64 away from both ends of the exponent
// range (so neither a seed nor its square flushes or overflows)
__device__ __forceinline__ bool seed_range(double b) {
    const int hi = __double2hiint(b);
    return hi >= (64 << 20) && hi < (1984 << 20);
}

// the bits of x through a move the compiler cannot fold back into a float
// comparison (which would run on the float64 pipe)
__device__ __forceinline__ unsigned long long bits_of(double x) {
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}

__device__ __forceinline__ bool is_zero(double x) { return (bits_of(x) << 1) == 0; }

// Division and square root without the float64 pipe: it takes a warp's
// instruction every 64 cycles per scheduler, in which the scheduler issues as
// many integer and float32 instructions.  With the significands as 53-bit
// integers, a double-float quotient (root) is good to 2^-45, so an integer Q
// within 2^9 of the scaled result; the remainder, exact modulo 2^64 by three
// 32-bit products (its size is below 2^63), divided in float32 gives the
// integer correction.  The result is within 0.51 units in the last place.
// About fifty instructions each, against four and five on the float64 pipe
// (reciprocal and reciprocal square root seeds and their series).

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// the significand of a normal value: its leading 24 bits as a float in [1, 2),
// the other 29 as a float in units of 2^-52
__device__ __forceinline__ float lead24(unsigned hi, unsigned lo) {
    return __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffffu) | 0x3f800000u);
}
__device__ __forceinline__ float rest29(unsigned lo) { return (float)(int)(lo & 0x1fffffffu); }

// a / b, b in seed_range, a 0 or of such a magnitude, the quotient's exponent
// in the normal range (div_range)
__device__ __forceinline__ bool div_range(double a, double b) {
    const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = __double2hiint(b) >> 20;
    return eb >= 64 && eb < 1984 && (is_zero(a) || ((unsigned)(ea - 64) < 1920u && (unsigned)(ea - eb + 1020) < 2040u));
}
__device__ __forceinline__ double div_int(double a, double b) {
    const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
    const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
    const float fa = lead24(ah, al), fb = lead24(bh, bl);
    float r = rcp_approx(fb);
    r = fmaf(r, fmaf(-fb, r, 1.f), r);
    const float q0 = __fmul_rn(fa, r);
    const float rm = fmaf(fmaf(-q0, rest29(bl), rest29(al)), 0x1p-52f, fmaf(-q0, fb, fa));
    const unsigned long long ma = ((unsigned long long)(ah & 0xfffffu) << 32) | al,
                             mb = ((unsigned long long)(bh & 0xfffffu) << 32) | bl;
    const int lt = ma < mb ? 1 : 0;   // quotient below 1
    const int i0 = __float2int_rn(q0 * 0x1p24f), i1 = __float2int_rn(rm * (r * 0x1p52f));
    const unsigned long long Q = (unsigned long long)(((long long)i0 << 28) + i1) << lt;
    const unsigned Ql = (unsigned)Q, Qh = (unsigned)(Q >> 32);
    const unsigned P = __umulhi(Ql, bl) + Ql * ((bh & 0xfffffu) | 0x100000u) + Qh * bl;
    const int rem = (int)((al << (20 + lt)) - P);   // high word of (ma << (52 + lt)) - Q mb
    const int d = __float2int_rn((float)rem * (r * 0x1p-20f));
    const int e = (int)((ah >> 20) & 0x7ffu) - (int)(bh >> 20) + 1022 - lt;
    const unsigned long long z = Q + (long long)d + ((unsigned long long)(unsigned)e << 52);
    const double q = __longlong_as_double((long long)(z | ((unsigned long long)(ah & 0x80000000u) << 32)));
    return (((ah << 1) | al) == 0) ? a : q;
}

// sqrt(x) for x in seed_range
__device__ __forceinline__ double sqrt_int(double x) {
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const int odd = ((xh >> 20) & 1) ^ 1;   // the unbiased exponent's parity
    const float fx = odd ? 2.f * lead24(xh, xl) : lead24(xh, xl);
    float y = rsqrt_approx(fx);
    float s0 = __fmul_rn(fx, y);
    y = fmaf(0.5f * y, fmaf(-s0, y, 1.f), y);
    s0 = __fmul_rn(fx, y);
    const float rm = fmaf(rest29(xl), odd ? 0x1p-51f : 0x1p-52f, fmaf(-s0, s0, fx));
    const int i0 = __float2int_rn(s0 * 0x1p24f), i1 = __float2int_rn(rm * (y * 0x1p51f));
    const unsigned long long S = (unsigned long long)(((long long)i0 << 28) + i1);
    const unsigned Sl = (unsigned)S, Sh = (unsigned)(S >> 32);
    const unsigned P = __umulhi(Sl, Sl) + Sl * (Sh << 1);
    const int rem = (int)((xl << (20 + odd)) - P);   // high word of (m << (52 + odd)) - S^2
    const int d = __float2int_rn((float)rem * (y * 0x1p-21f));
    const int e = (((int)(xh >> 20) - 1023) >> 1) + 1022;
    return __longlong_as_double((long long)(S + (long long)d + ((unsigned long long)(unsigned)e << 52)));
}

// a / b on the lanes of `m` (all of which call it); IEEE division for the
// whole warp when any operand or quotient leaves the safe range (b zero,
// denormal, negative, huge or NaN; a denormal, huge or NaN)
__device__ __forceinline__ double div64(double a, double b, unsigned m) {
    if (__all_sync(m, div_range(a, b))) return div_int(a, b);
    return a / b;
}

// sqrt(x), x >= 0 or -0, on the lanes of `m`
__device__ __forceinline__ double sqrt64(double x, unsigned m) {
    const bool z = is_zero(x);
    if (__all_sync(m, z || seed_range(x))) {
        const double s = sqrt_int(z ? 1.0 : x);
        return z ? 0.0 : s;
    }
    return sqrt(x);
}

// x > y for x, y >= 0 (or -0); false when x is NaN, as the float comparison
__device__ __forceinline__ bool gt_nonneg(double x, double y) {
    const long long a = (long long)bits_of(x), b = (long long)bits_of(y);
    return a > b && a <= 0x7ff0000000000000LL;
}

// 1/b for b in seed_range
__device__ __forceinline__ double rcp_int(double b) { return div_int(1.0, b); }

// 1/sqrt(x) for x in seed_range: y ~ x^(-1/2) (20 bits), r = 1 - x*y^2,
// x^(-1/2) = y*(1 - r)^(-1/2) = y*(1 + r/2 + 3r^2/8 + O(r^3)) (Newton-Raphson
// taken to second order in series form, P. Markstein, IBM J. Res. Dev. 34
// (1990) 111)
__device__ __forceinline__ double rsqrt_series(double x) {
    const double y = rsqrt_seed(x);
    const double r = fma(-(x * y), y, 1.0);
    return fma(y, r * fma(0.375, r, 0.5), y);
}

// 1/b on the lanes of `m`; IEEE division for the whole warp when any b
// leaves the seed range
__device__ __forceinline__ double rcp64(double b, unsigned m) {
    if (__all_sync(m, seed_range(b))) return rcp_int(b);
    return 1.0 / b;
}

// 1/sqrt(x), x > 0, on the lanes of `m`
__device__ __forceinline__ double rsqrt64(double x, unsigned m) {
    if (__all_sync(m, seed_range(x))) return rsqrt_series(x);
    return 1.0 / sqrt(x);
}

// The same per lane, for code where the lanes that reach the call are not
// known (data-dependent branches): the series where the operand is in the
// seed range, IEEE otherwise (a warp whose lanes disagree runs both).
__device__ __forceinline__ double div_lane(double a, double b) {
    return div_range(a, b) ? div_int(a, b) : a / b;
}
__device__ __forceinline__ double rcp_lane(double b) { return seed_range(b) ? rcp_int(b) : 1.0 / b; }
__device__ __forceinline__ double sqrt_lane(double x) {
    if (is_zero(x)) return x;
    return seed_range(x) ? sqrt_int(x) : sqrt(x);
}
__device__ __forceinline__ double rsqrt_lane(double x) { return seed_range(x) ? rsqrt_series(x) : 1.0 / sqrt(x); }

// ------------------------------------------------ tests on the integer pipe
// Comparisons of float64 values cost a slot of the float64 pipe each; on the
// bits they run on the integer pipe.  As the float comparisons, they are
// false where an operand is NaN.
__device__ __forceinline__ bool is_nan64(double x) { return (bits_of(x) << 1) > 0xffe0000000000000ULL; }
__device__ __forceinline__ bool finite64(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
// the bits as a signed integer in the order of the values (-0 just below +0)
__device__ __forceinline__ long long order64(double x) {
    const long long b = (long long)bits_of(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool is_pos(double x) {   // x > 0
    const long long b = (long long)bits_of(x);
    return b > 0 && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool is_neg(double x) {   // x < 0
    const unsigned long long b = bits_of(x);
    return b > 0x8000000000000000ULL && b <= 0xfff0000000000000ULL;
}
__device__ __forceinline__ bool gt64(double a, double b) {   // a > b
    return order64(a) > order64(b) && !is_nan64(a) && !is_nan64(b) && !(is_zero(a) && is_zero(b));
}

__device__ __forceinline__ bool ne64(double a, double b) {   // a != b (true on NaN)
    return (bits_of(a) != bits_of(b) && !(is_zero(a) && is_zero(b))) || is_nan64(a);
}
__device__ __forceinline__ bool ge64(double a, double b) {   // a >= b
    return !gt64(b, a) && !is_nan64(a) && !is_nan64(b);
}

// ------------------------------- float32 <-> float64 on the integer pipe
// a normal float, exactly (0 gives 2^-127 with its sign, for correction terms)
__device__ __forceinline__ double widen(float x) {
    const unsigned b = __float_as_uint(x);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
// truncated to float; magnitudes below 2^-126 become about 2^-126, those
// above the float range infinite or NaN: for approximations and tails
__device__ __forceinline__ float narrow(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = min(max(hi & 0x7fffffffu, 0x38100000u), 0x47f00000u) - 0x38000000u;
    return __uint_as_float((hi & 0x80000000u) | (e << 3) | (lo >> 29));
}

// rounded to the nearest float, as a conversion, which takes a slot of the
// float64 pipe; results outside the normal floats (but zeros) are converted
__device__ __forceinline__ float to_float(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned mag = hi & 0x7fffffffu, sign = hi & 0x80000000u;
    if (mag - 0x38100000u >= 0x0fe00000u && (mag | lo) != 0) return __double2float_rn(x);
    unsigned f = ((mag - 0x38000000u) << 3) | (lo >> 29);
    const unsigned rest = lo & 0x1fffffffu;
    f += rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
    return __uint_as_float(sign | ((mag | lo) != 0 ? f : 0u));
}

// ------------------------------------------- exponential, logarithm, arctangent
// Table-driven (P. T. P. Tang, ACM Trans. Math. Softw. 15 (1989) 144 and 16
// (1990) 378): the tables of f64tables.cuh leave a remainder so small that
// the last terms of its series, below 2^-30 of the result, are evaluated in
// float32, and the float64 pipe sees eight, seven and eleven operations.

// e^x for |x| <= 700: x = (512 n + k) ln2/512 + r, |r| <= ln2/1024; e^x = 2^n
// 2^(k/512) (1 + r + r^2 (1/2 + r/6 + r^2/24))
__device__ __forceinline__ double exp_core(double x) {
    const double magic = 6755399441055744.0;   // 1.5 * 2^52: the sum's low word is the rounded integer
    const double s = fma(x, 0x1.71547652b82fep+9, magic);
    const int n = __double2loint(s);
    const double k = s - magic;
    const double r = fma(k, -0x1.473de6af278edp-43, fma(k, -0x1.62e42fef00000p-10, x));
    const float f = narrow(r);
    const double q = 0.5 + widen(f * fmaf(f, 1.f / 24.f, 1.f / 6.f));
    const double p = fma(r * r, q, r);
    const double T = __ldg(EXP2_512 + (n & 511));
    const double e = fma(T, p, T);
    return __hiloint2double(__double2hiint(e) + ((n >> 9) << 20), __double2loint(e));
}
// any x: beyond the core's range the square of e^(x/2), up to overflow and to the subnormals
static __device__ __noinline__ double exp_far(double x) {
    if (is_nan64(x)) return x;
    if (gt64(x, 1400.0)) return __hiloint2double(0x7ff00000, 0);
    if (gt64(-1400.0, x)) return 0.0;
    const double e = exp_core(0.5 * x);
    return e * e;
}
__device__ __forceinline__ double exp_table(double x) {
    return (unsigned)(__double2hiint(x) & 0x7fffffff) < 0x4085e000u ? exp_core(x) : exp_far(x);
}

// The bulk formula's psi_m and psi_h at s = 1 - 16 huol in [1, 161]
//   psi_m = 2 ln((1 + x)/2) + 2 ln((1 + x^2)/2) - 2 atan x + pi/2,
//   psi_h = 2 ln((1 + x^2)/2), x = s^(1/4)
// from their series about the nearest of 32 points an octave (|t| <= 2^-6: the
// float32 part, from t^5 on, is below 2^-34 of 1), 12 float64 operations for
// both.  Absolute error at most 9e-16 and 5e-16 (4000 points against 200-bit
// values; with the float64 square roots, logarithms and arctangent 1.5e-15).
// The tables are read by random index: in shared memory, one plane per coefficient.
struct PsiTables {
    double head[10 * PSI_POINTS];
    float tail[8 * PSI_POINTS], r[32];
    __device__ __forceinline__ void load(int threads) {
        for (int q = threadIdx.x; q < 10 * PSI_POINTS; q += threads) head[q] = PSI_HEAD[q];
        for (int q = threadIdx.x; q < 8 * PSI_POINTS; q += threads) tail[q] = PSI_TAIL[q];
        if (threadIdx.x < 32) r[threadIdx.x] = PSI_R[threadIdx.x];
    }
    // a NaN's or larger s takes the last point: NaN, or no value of use
    __device__ __forceinline__ void eval(double s, double &psim, double &psih) const {
        const unsigned at = (unsigned)(__double2hiint(s) - 0x3ff00000) >> 15;
        const int n = at < PSI_POINTS ? (int)at : PSI_POINTS - 1;
        const double c = widen(r[n & 31]);
        const double t = fma(s, __hiloint2double(__double2hiint(c) - ((n >> 5) << 20), __double2loint(c)), -1.0);
        const float f = narrow(t);
        auto series = [&](const double *h, const float *l) {
            const float e = f * fmaf(f, fmaf(f, fmaf(f, l[3 * PSI_POINTS], l[2 * PSI_POINTS]), l[PSI_POINTS]), l[0]);
            double p = h[4 * PSI_POINTS] + widen(e);
            p = fma(p, t, h[3 * PSI_POINTS]);
            p = fma(p, t, h[2 * PSI_POINTS]);
            p = fma(p, t, h[PSI_POINTS]);
            return fma(p, t, h[0]);
        };
        psim = series(head + n, tail + n);
        psih = series(head + 5 * PSI_POINTS + n, tail + 4 * PSI_POINTS + n);
    }
};

}  // namespace veris
