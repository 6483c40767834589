// IEEE double division and square root, correctly rounded to nearest even, on
// the integer and FP32 pipes.
//
// GB300 issues FP64 at 2 lanes per clock and SM; a division or square root
// takes the FP64 pipe for about ten instructions, 64 issue cycles of the warp
// each, and the exact form's update has some 40 of them per cell.  Here the
// quotient of the 53-bit significands comes from integer long division with
// two digits: the leading 21 bits from a float product with the reciprocal
// seed, the next from the float remainder (together within 2^-43), then one
// exact 64-bit integer remainder gives the correction and decides the
// rounding.  Ties do not occur: a quotient or root of two 53-bit significands
// is never halfway between two 53-bit numbers.  Operands or results outside
// the normal range (with a margin), infinities and NaNs go to the hardware
// operation.
#pragma once

#include <cuda_runtime.h>

#include "hx_pair.cuh"

namespace hx {

static __device__ __noinline__ double ieee_div_slow(double a, double b) { return a / b; }
static __device__ __noinline__ double ieee_sqrt_slow(double x) { return sqrt(x); }

// A divisor, unpacked once for the quotients that share it.
struct IeeeDivisor {
    double b;
    unsigned mhi, mlo;  // significand, 53 bits
    float bh, bl, y;    // significand in [1, 2) as a pair, estimate of 1 / bh
    unsigned e;         // biased exponent << 20, sign cleared; 0 where the fast path does not apply
};
__device__ __forceinline__ IeeeDivisor ieee_divisor(double b) {
    IeeeDivisor d;
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    d.b = b;
    d.mhi = (hi & 0xFFFFFu) | 0x100000u;
    d.mlo = lo;
    d.bh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7FFFFFu) | 0x3F800000u);
    d.bl = __fmul_rn(__uint2float_rn(lo << 3), 0x1p-55f);
    const float y = f_rcp(d.bh);
    d.y = __fmaf_rn(y, __fmaf_rn(-d.bh, y, 1.f), y);  // within ~2^-23.5: keeps the remainder in range
    d.e = hi & 0x7FF00000u;
    return d;
}
// a / d.b.  CHECKED == false: the caller knows that a is zero or normal, d.b is normal and the quotient's
// exponent stays within +-1000, so nothing here branches.
template <bool CHECKED = true> __device__ __forceinline__ double ieee_div(double a, const IeeeDivisor& d) {
    const unsigned ahi = (unsigned)__double2hiint(a), alo = (unsigned)__double2loint(a);
    const unsigned sg = (ahi ^ (unsigned)__double2hiint(d.b)) & 0x80000000u;
    const unsigned ae = ahi & 0x7FF00000u;
    unsigned mhi = (ahi & 0xFFFFFu) | 0x100000u, mlo = alo;
    float ah = __uint_as_float((__funnelshift_l(alo, ahi, 3) & 0x7FFFFFu) | 0x3F800000u);
    float al = __fmul_rn(__uint2float_rn(alo << 3), 0x1p-55f);
    // the quotient of the significands brought into [1, 2)
    const unsigned long long mb = ((unsigned long long)d.mhi << 32) | d.mlo;
    const bool less = (((unsigned long long)mhi << 32) | mlo) < mb;
    if (less) {
        mhi = __funnelshift_l(mlo, mhi, 1);
        mlo <<= 1;
        ah = __fadd_rn(ah, ah);
        al = __fadd_rn(al, al);
    }
    // leading digit in units of 2^-21, the last place of 4 + q; second one to 2^-51 (below 2^30:
    // the seed and the first digit are each within 2^-22)
    const float t = __fmaf_rn(ah, d.y, 4.0f), q = __fadd_rn(t, -4.0f);
    const float r = __fmaf_rn(-q, d.bl, __fadd_rn(__fmaf_rn(-q, d.bh, ah), al));
    const int q2 = __float2int_rn(__fmul_rn(r, __fmul_rn(d.y, 0x1p51f)));
    const unsigned qi = (unsigned)__float_as_int(t) & 0x7FFFFFu;
    unsigned long long Q = ((unsigned long long)qi << 31) + ((unsigned long long)(long long)q2 << 1);
    // remainder ma 2^52 - Q mb, modulo 2^64 (its magnitude stays below 2^62)
    unsigned long long R = ((unsigned long long)(mlo << 20) << 32) - Q * mb;
    const int Rh = (int)(R >> 32);
    const int c = __float_as_int(__fmaf_rn(__int2float_rn(Rh), __fmul_rn(d.y, 0x1p-20f), 12582912.0f)) - 0x4B400000;
    Q += (unsigned long long)(long long)c;
    R -= (unsigned long long)(long long)c * mb;
    // |R| is at most a little over half of mb: the nearest quotient is Q or a neighbour
    const long long R2 = (long long)(R + R);
    if (R2 > (long long)mb) Q += 1;
    if (R2 < -(long long)mb) Q -= 1;
    // exponent of the quotient, less one (Q's leading bit adds it back)
    const unsigned e = ae - d.e + (1022u << 20) - (less ? 0x100000u : 0u);
    const unsigned vh = (((unsigned)(Q >> 32)) + e) | sg, vl = (unsigned)Q;
    if constexpr (!CHECKED) {
        return __hiloint2double((int)(ae != 0u ? vh : sg), (int)(ae != 0u ? vl : 0u));
    } else {
        const bool dok = d.e - 0x00100000u < 0x7FE00000u, zero = (ae | (ahi & 0xFFFFFu) | alo) == 0u;
        const bool ok = dok & (zero | ((ae - 0x00100000u < 0x7FE00000u) & (ae - d.e + (1000u << 20) < (2000u << 20))));
        double v = __hiloint2double((int)(zero ? sg : vh), (int)(zero ? 0u : vl));
        if (!ok) v = ieee_div_slow(a, d.b);
        return v;
    }
}
template <bool CHECKED = true> __device__ __forceinline__ double ieee_div(double a, double b) {
    return ieee_div<CHECKED>(a, ieee_divisor(b));
}

// sqrt(x).  CHECKED == false: the caller knows that x is +0 or positive and normal.
template <bool CHECKED = true> __device__ __forceinline__ double ieee_sqrt(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    // x = m 4^k with m in [1, 4): an odd unbiased exponent leaves a factor of two in m
    const bool odd = (hi & 0x00100000u) == 0u;  // biased exponents are odd where the unbiased ones are even
    unsigned mhi = (hi & 0xFFFFFu) | 0x100000u, mlo = lo;
    float mh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7FFFFFu) | 0x3F800000u);
    float ml = __fmul_rn(__uint2float_rn(lo << 3), 0x1p-55f);
    if (odd) {
        mhi = __funnelshift_l(mlo, mhi, 1);
        mlo <<= 1;
        mh = __fadd_rn(mh, mh);
        ml = __fadd_rn(ml, ml);
    }
    float y = f_rsqrt(mh);
    y = __fmaf_rn(y, __fmaf_rn(__fmul_rn(-0.5f, __fmul_rn(mh, y)), y, 0.5f), y);  // within ~2^-23.5: keeps R in range
    const float hy = __fmul_rn(0.5f, y);
    const float t = __fmaf_rn(mh, y, 4.0f), s = __fadd_rn(t, -4.0f);
    const float r = __fadd_rn(__fmaf_rn(-s, s, mh), ml);
    const float g = __fmul_rn(r, hy);  // sqrt(m) - s up to g^2 / (2 sqrt(m)), added here
    const int s2 = __float2int_rn(__fmul_rn(__fmaf_rn(__fmul_rn(g, hy), g, g), 0x1p51f));
    const unsigned si = (unsigned)__float_as_int(t) & 0x7FFFFFu;
    unsigned long long S = ((unsigned long long)si << 31) + ((unsigned long long)(long long)s2 << 1);
    unsigned long long R = ((unsigned long long)(mlo << 20) << 32) - S * S;  // m 2^104 - S^2, below 2^62
    const int Rh = (int)(R >> 32);
    const int c = __float_as_int(__fmaf_rn(__int2float_rn(Rh), __fmul_rn(hy, 0x1p-20f), 12582912.0f)) - 0x4B400000;
    R -= (unsigned long long)(long long)c * (S + S + (unsigned long long)(long long)c);
    S += (unsigned long long)(long long)c;
    if ((long long)R > (long long)S) S += 1;
    else if ((long long)R <= -(long long)S) S -= 1;
    // exponent of the root, less one: (biased + 1023) / 2 for even unbiased exponents
    const unsigned e = (((hi >> 20) + 1023u - (odd ? 1u : 0u)) >> 1) - 1u;
    const unsigned vh = (unsigned)(S >> 32) + (e << 20), vl = (unsigned)S;
    if constexpr (!CHECKED) {
        return __hiloint2double((int)(hi != 0u ? vh : 0u), (int)(hi != 0u ? vl : 0u));
    } else {
        const bool zero = (hi | lo) == 0u;
        double v = __hiloint2double((int)(zero ? 0u : vh), (int)(zero ? 0u : vl));
        if (!(zero | (hi - 0x00100000u < 0x7FE00000u))) v = ieee_sqrt_slow(x);
        return v;
    }
}

}  // namespace hx
