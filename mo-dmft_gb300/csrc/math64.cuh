// math64.cuh -- FP64 device arithmetic shared by the kernels.
//
// GB300 issues an FP64 warp instruction every 64 cycles per sub-partition, so
// these helpers count FP64 instructions and use the integer and FP32 pipes
// where that is exact.
#pragma once

#include <cuda_runtime.h>

namespace moed {

// 1/d for d > 0 from an FP32 seed y0 = rcp.approx(d) refined by one
// third-order step of the Newton-Raphson family for the reciprocal,
//   y1 = y0 + y0 (e + e^2),  e = 1 - d y0,
// the truncated series y0 / (1 - e) = y0 (1 + e + e^2 + ...).  d is narrowed
// to FP32 by truncating its significand (relative error < 2^-23) and the seed
// widened back exactly, both with integer operations, so the FP64 pipe sees
// only the three FMAs.  The seed's relative error |e| is below 2^-21, the
// truncation error |e|^3 < 2^-63, and y1 is within one ulp of 1/d.  Outside
// [2^-125, 2^126) (and for d <= 0, non-finite d) it is the IEEE division.
__device__ __forceinline__ double rcp_pos(double d)
{
    const long long b = __double_as_longlong(d);
    const int ex = (int)(b >> 52);                          // biased exponent (sign bit 0)
    if ((unsigned)(ex - 898) > 250u) return 1.0 / d;        // FP32 exponent ex - 896 outside [2, 252]
    const float df = __int_as_float(((ex - 896) << 23) | (int)((b >> 29) & 0x7fffff));
    float yf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(df));
    const int fb = __float_as_int(yf);                      // a normal float: 1/df in (2^-126, 2^125]
    const double y0 = __longlong_as_double(((long long)(((fb >> 23) & 0xff) + 896) << 52) |
                                           ((long long)(fb & 0x7fffff) << 29));
    const double e = fma(-d, y0, 1.0);
    return fma(y0, fma(e, e, e), y0);
}

// N of them with one look at the ranges, so that their chains of instructions
// overlap; the same results.
template <int N>
__device__ __forceinline__ void rcp_pos_n(const double (&d)[N], double (&y)[N])
{
    bool odd = false;
    float yf[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const long long b = __double_as_longlong(d[i]);
        const int ex = (int)(b >> 52);
        odd = odd || (unsigned)(ex - 898) > 250u;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf[i]) : "f"(__int_as_float(((ex - 896) << 23) | (int)((b >> 29) & 0x7fffff))));
    }
    if (odd) {
#pragma unroll 1
        for (int i = 0; i < N; ++i) y[i] = rcp_pos(d[i]);
        return;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int fb = __float_as_int(yf[i]);
        const double y0 = __longlong_as_double(((long long)(((fb >> 23) & 0xff) + 896) << 52) |
                                               ((long long)(fb & 0x7fffff) << 29));
        const double e = fma(-d[i], y0, 1.0);
        y[i] = fma(y0, fma(e, e, e), y0);
    }
}

// s / d for d whose reciprocal r is known to an ulp: q = s r and one correction,
// three dependent instructions.  Half an ulp and little more; correctly rounded
// (Markstein, IBM J. Res. Dev. 34, 1990) where r = RN(1 / d) and q is within an
// ulp, as for d of up to 24 significant bits.  Outside the range of s where
// nothing under- or overflows it is the division.
__device__ __forceinline__ double div_by(double s, double d, double r)
{
    if ((unsigned)(((__double2hiint(s) >> 20) & 0x7ff) - 523) > 1000u) return s / d;   // |s| in [2^-500, 2^500]
    const double q = s * r;
    return fma(fma(-q, d, s), r, q);
}

__device__ __forceinline__ double widen(float f);

// 1/sqrt(d) for d > 0: an FP32 seed y0 of rsqrt.approx refined by one step of
// the binomial series
//   (1 - e)^(-1/2) = 1 + e (1/2 + 3/8 e) + O(e^3),  e = 1 - d y0^2, |e| < 2^-20,
// five dependent FP64 instructions where a square root and a division take
// tens, within an ulp (d y0 goes into e with its rounding error).  Outside
// [2^-100, 2^100] (and for d <= 0, non-finite d) it is those.
__device__ __forceinline__ double rsqrt_pos(double d)
{
    if ((unsigned)((int)(__double_as_longlong(d) >> 52) - 923) > 200u) return 1.0 / sqrt(d);
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"((float)d));
    const double y0 = widen(yf), e = fma(-(d * y0), y0, 1.0);
    return fma(y0 * e, fma(e, 0.375, 0.5), y0);
}

// sqrt(d) and 1/sqrt(d) to half an ulp and little more from y = rsqrt_pos(d):
// one correction each with an exact residual, for d where nothing under- or
// overflows ([2^-500, 2^500])
__device__ __forceinline__ double sqrt_by(double d, double y)
{
    const double h = d * y;
    return fma(fma(-h, h, d), 0.5 * y, h);
}
__device__ __forceinline__ double rsqrt_by(double d, double y)
{
    const double p = d * y, e = fma(-fma(d, y, -p), y, fma(-p, y, 1.0));
    return fma(0.5 * y, e, y);
}

// (double)f by integer operations: a conversion instruction takes a slot of
// the FP64 pipe, even one that is predicated off, so the rare cases have none
// either.  Infinities and NaN need the exponent 2047 instead of 255 + 896; a
// denormal is scaled by 2^24 in FP32 first.
__device__ __forceinline__ double widen(float f)
{
    const unsigned b = __float_as_uint(f);
    unsigned m = b & 0x7fffffffu, e = 0x38000000u;   // 896 more in the exponent
    if (m >= 0x7f800000u) e = 0x70000000u;
    if (m < 0x00800000u) {
        m = __float_as_uint(f * 16777216.0f) & 0x7fffffffu;
        e = m ? 0x38000000u - (24u << 20) : 0u;
    }
    return __hiloint2double((int)(((m >> 3) + e) | (b & 0x80000000u)), (int)(m << 29));
}
__device__ __forceinline__ double widen(double f) { return f; }

}  // namespace moed
