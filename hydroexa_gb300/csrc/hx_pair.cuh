// Pairs of floats (h + l, |l| at most about an ulp of h): ~48 significant
// bits on the FP32 pipe.
//
// GB300 issues FP64 at 2 lanes per clock and SM and FP32 at 128, so one FP64
// instruction costs a warp 64 issue cycles, and a pair product (7 FP32
// instructions) or sum (11) a small part of that.  The FP64 fast form takes
// velocities, their slopes and the Roe dissipation in pairs and keeps in
// doubles what the balance of a step hangs on: free surfaces, depths, their
// differences, the hydrostatic pressure and the update itself.
//
// Error-free sums and products: Knuth's and Dekker's (T. J. Dekker, Numer.
// Math. 18, 1971); products by fma.  Every operation is an explicit
// round-to-nearest intrinsic, so no contraction can differ between the kernels
// that share this code.  Relative error of a normalised sum (of its larger
// operand) or product: a few 2^-48; quotients and roots take one correction
// of a 2^-22.4 seed, so a few 2^-47.
#pragma once

#include <cuda_runtime.h>

namespace hx {

struct F2 {
    float h, l;
};

// A double kept in a pair's place, and back.
__device__ __forceinline__ F2 f2_bits(double x) {
    return {__int_as_float(__double2hiint(x)), __int_as_float(__double2loint(x))};
}
__device__ __forceinline__ double bits_f2(F2 a) { return __hiloint2double(__float_as_int(a.h), __float_as_int(a.l)); }

__device__ __forceinline__ float f_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float f_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// a + b exactly, |a| >= |b| (or a == 0)
__device__ __forceinline__ F2 f2_norm(float a, float b) {
    const float s = __fadd_rn(a, b);
    return {s, __fadd_rn(b, -__fadd_rn(s, -a))};
}
// a + b exactly
__device__ __forceinline__ F2 f2_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b), t = __fadd_rn(s, -a);
    return {s, __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -t)), __fadd_rn(b, -t))};
}
__device__ __forceinline__ F2 f2_neg(F2 a) { return {-a.h, -a.l}; }
__device__ __forceinline__ F2 f2_half(F2 a) { return {__fmul_rn(0.5f, a.h), __fmul_rn(0.5f, a.l)}; }
// |a| by the sign of its high part
__device__ __forceinline__ F2 f2_abs(F2 a) {
    const int s = __float_as_int(a.h) & (int)0x80000000;
    return {__int_as_float(__float_as_int(a.h) ^ s), __int_as_float(__float_as_int(a.l) ^ s)};
}
__device__ __forceinline__ F2 f2_sel(bool c, F2 a) { return {c ? a.h : 0.f, c ? a.l : 0.f}; }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    const F2 s = f2_two_sum(a.h, b.h);
    return f2_norm(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_add(a, f2_neg(b)); }
// a b with the low part not yet normalised (|l| a few ulps of h): for sums
__device__ __forceinline__ F2 f2_mul_raw(F2 a, F2 b) {
    const float p = __fmul_rn(a.h, b.h);
    return {p, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -p)))};
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    const F2 p = f2_mul_raw(a, b);
    return f2_norm(p.h, p.l);
}
// a / d, y an estimate of 1 / d.h
__device__ __forceinline__ F2 f2_div(F2 a, F2 d, float y) {
    const float q = __fmul_rn(a.h, y);
    const float r = __fmaf_rn(-q, d.l, __fadd_rn(__fmaf_rn(-q, d.h, a.h), a.l));
    return f2_norm(q, __fmul_rn(r, y));
}
// 1 / d
__device__ __forceinline__ F2 f2_rcp(F2 d) {
    const float y = f_rcp(d.h);
    const float e = __fmaf_rn(-d.l, y, __fmaf_rn(-d.h, y, 1.f));
    return f2_norm(y, __fmul_rn(y, e));
}
// sqrt(a), a >= 0 (0 gives 0); r receives the seed of 1 / sqrt(a)
__device__ __forceinline__ F2 f2_sqrt(F2 a, float& r) {
    r = f_rsqrt(fmaxf(a.h, 1e-37f));
    const float s = __fmul_rn(a.h, r);
    const float d = __fadd_rn(__fmaf_rn(-s, s, a.h), a.l);
    return f2_norm(s, __fmul_rn(d, __fmul_rn(0.5f, r)));
}

// h^(-1/3), 0 < h in the float range: the float seed rcbrtf (within ~2^-22) and one third-order step,
// r + r e (1/3 + 2 e / 9) with e = 1 - h r^3 in pairs
__device__ __forceinline__ F2 f2_rcbrt(F2 h) {
    const float r = rcbrtf(h.h);
    const F2 r1{r, 0.f}, r3 = f2_mul(f2_mul(r1, r1), r1);
    const F2 e = f2_add(F2{1.f, 0.f}, f2_neg(f2_mul_raw(h, r3)));
    return f2_norm(r, __fmul_rn(__fmul_rn(r, e.h), __fmaf_rn(0.22222222f, e.h, 0.33333334f)));
}

// The leading ~48 bits of a double, made on the integer pipe (a double to
// float conversion issues on the FP64 pipe): h the leading 24 significand bits
// (truncated), l the other 29 rounded to a float.  Below 2^-71 l is 0, below
// 2^-126 the pair is; beyond the float range, and for infinities and NaNs, h
// is NaN.
__device__ __forceinline__ F2 f2_of(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned m = hi & 0x7FFFFFFFu;
    // the float exponent is the double's low eight exponent bits with the top one flipped (897 <= e <= 1150)
    const unsigned f = ((__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7FFFFFFFu) | (hi & 0x80000000u);
    const float lf = __uint2float_rn(lo << 3);
    const float sc = __uint_as_float((f & 0xFF800000u) - (55u << 23));
    F2 r;
    r.l = m >= (952u << 20) ? __fmul_rn(lf, sc) : 0.f;
    r.h = __uint_as_float(f);
    if (m - (897u << 20) >= (254u << 20)) {  // outside the normal float range
        r.h = m >= (1151u << 20) ? __uint_as_float(0x7FFFFFFFu) : 0.f;
        r.l = 0.f;
    }
    return r;
}
// The same rounded: h the nearest float, so that l is at most half a place of h and the pair within 2^-50.6 of x
// (root mean square; f2_of 2^-49.6), for a few more integer instructions.
__device__ __forceinline__ F2 f2_of_rn(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned m = hi & 0x7FFFFFFFu;
    const unsigned long long b = (((unsigned long long)hi << 32) | lo) + 0x10000000ull;  // half a float place
    const unsigned bh = (unsigned)(b >> 32), bl = (unsigned)b;
    const unsigned f = ((__funnelshift_l(bl, bh, 3) ^ 0x40000000u) & 0x7FFFFFFFu) | (hi & 0x80000000u);
    // the 29 bits left, signed, in units of the double's own last place (its exponent, before any carry)
    const float lf = __int2float_rn((int)(lo << 3));
    const float sc = __uint_as_float(((((hi << 3) ^ 0x40000000u) & 0x7F800000u) | (hi & 0x80000000u)) - (55u << 23));
    F2 r;
    r.l = m >= (952u << 20) ? __fmul_rn(lf, sc) : 0.f;
    r.h = __uint_as_float(f);
    if (m - (897u << 20) >= (252u << 20)) {  // below 2^-126, from 2^126 on (whose reciprocal is no normal float)
        r.h = m >= (1149u << 20) ? __uint_as_float(0x7FFFFFFFu) : 0.f;
        r.l = 0.f;
    }
    return r;
}
// Doubles past the float range in a pair's place (velocities, fluxes): a quiet NaN that holds the double's sign,
// exponent and leading 43 bits of significand, so arithmetic on it gives NaN, and who meets a NaN takes FP64.  A NaN
// keeps its sign, which comparisons of bit patterns go by; one that arithmetic made (0x7FFFFFFF) reads as a NaN too.
__device__ __forceinline__ F2 f2_box(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
    const unsigned long long p = (b > 0x7FF0000000000000ull ? 0x7FFFFFFFFFFFFFFFull : b + 0x100ull) >> 9;
    return {__uint_as_float(((unsigned)__double2hiint(x) & 0x80000000u) | 0x7FC00000u | (unsigned)(p >> 32)),
            __uint_as_float((unsigned)p)};
}
__device__ __forceinline__ F2 f2_any(double x) {
    return ((unsigned)__double2hiint(x) & 0x7FFFFFFFu) < ((1023u + 126u) << 20) ? f2_of_rn(x) : f2_box(x);
}
// a / d for rounded pairs, y within 2^-24 of 1 / d.h: every rounding falls on the low parts (of two doubles' quotient,
// conversions included, 2^-48.6 root mean square and 2^-45.5 at most over 10^6 random pairs).
__device__ __forceinline__ F2 f2_div_rn(F2 a, F2 d, float y) {
    const float q = __fmul_rn(a.h, y);
    const F2 r = f2_two_sum(__fmaf_rn(-q, d.h, a.h), __fmaf_rn(-q, d.l, a.l));
    const float l = __fmul_rn(r.h, y);
    return f2_norm(q, __fmaf_rn(__fadd_rn(__fmaf_rn(-l, d.h, r.h), r.l), y, l));
}

// h + l as a double, rounded to nearest, on the integer pipe: l in units of the high part's last place is
// added to the bits of h (an FP64 addition costs a warp 64 issue cycles, this ~35).  0 where h is 0 or
// subnormal, h alone below 2^-75, NaN where h is not finite.  THIRD: with a third part e, below 2^-28 of h.
template <bool THIRD = false> __device__ __forceinline__ double f64_of(F2 a, float e = 0.f) {
    const int b = __float_as_int(a.h);
    const unsigned m = (unsigned)b & 0x7FFFFFFFu, sg = (unsigned)b & 0x80000000u;
    // l 2^(52 - e) for a high part of exponent e (biased E = e + 127): 306 - E is that factor's biased exponent
    const float sc = __uint_as_float((306u << 23) - (m & 0x7F800000u));
    int li = __float2int_rn(__fmul_rn(__int_as_float(__float_as_int(a.l) ^ (int)sg), sc));
    if constexpr (THIRD) li += __float2int_rn(__fmul_rn(__int_as_float(__float_as_int(e) ^ (int)sg), sc));
    if (li < 0 && (m & 0x7FFFFFu) == 0) li += li;  // below a power of two the last place is half as large
    li = m >= (52u << 23) ? li : 0;
    const unsigned long long v =
        (((unsigned long long)((m >> 3) + 0x38000000u) << 32) | (unsigned)(b << 29)) + (unsigned long long)(long long)li;
    unsigned hi = (unsigned)(v >> 32) | sg, lo = (unsigned)v;
    if (m - 0x00800000u >= 0x7F000000u) {  // zero and subnormal, or not finite
        hi = m >= 0x7F800000u ? 0x7FF80000u : sg;
        lo = 0u;
    }
    return __hiloint2double((int)hi, (int)lo);
}
// The double that f2_any put in a pair's place.
__device__ __forceinline__ double f64_any(F2 a) {
    if (a.h == a.h) return f64_of(a);
    const unsigned h = __float_as_uint(a.h);
    const unsigned long long p = ((unsigned long long)(h & 0x3FFFFFu) << 32) | __float_as_uint(a.l);
    return __longlong_as_double((long long)(((unsigned long long)(h & 0x80000000u) << 32) | (p << 9)));
}

}  // namespace hx
