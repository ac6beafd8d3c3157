// Reciprocals, quotients of a shared divisor and square roots rounded to
// nearest, without branches, so that the chains of one update overlap.  For
// normal operands and results well inside the exponent range.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace sa {

// a / b rounded to nearest from rh = RN(1/b) and rl = recip_lo(b, rh), about
// 1/b - rh: RN(a rh + a rl) lies within an ulp of a / b, its remainder is
// exact, and one correction by rh rounds correctly (Markstein, IBM J. Res.
// Dev. 34(1) 1990); for |a| above 2^-900 or 0.  Four operations where
// several quotients share a divisor, against about ten of a division.
__device__ __forceinline__ double recip_lo(double b, double rh) { return fma(-rh, b, 1.0) * rh; }
__device__ __forceinline__ double quot(double a, double b, double rh, double rl) {
    const double q = fma(a, rh, a * rl);
    return fma(fma(-q, b, a), rh, q);
}

// Whether the last 32 bits of b are ones: rcp_rn rounds correctly otherwise.
__device__ __forceinline__ bool low_ones(double b) {
#if defined(__CUDA_ARCH__)
    return __double2loint(b) == -1;
#else
    uint64_t u;
    memcpy(&u, &b, 8);
    return (uint32_t)u == 0xffffffffu;
#endif
}

// 1 / b: Newton's iteration y + y (1 - b y), the residual rounded once, which
// squares the relative error of y.  From the hardware's start value (2^-18 or
// better) two steps leave 2^-72 and a rounding, so that y lies within an ulp of
// 1 / b, 1 - b y is exact, and a step from there rounds 1 / b correctly unless
// the mantissa of b is all ones (Markstein 1990).
__device__ __forceinline__ double rcp_rn(double b) {
    double y;
#if defined(__CUDA_ARCH__)
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#else
    y = (double)(1.0f / (float)b);
#endif
#pragma unroll
    for (int i = 0; i < 3; i++) y = fma(y, fma(-b, y, 1.0), y);
    return y;
}

// sqrt x: Goldschmidt's coupled iteration, g to sqrt x and h to 1 / (2 sqrt x),
// squares the start value's relative error (2^-18 or better) twice; then g
// plus its residual's correction (x - g^2) h, whose own error is below 2^-44 of
// it.  *sure is false where that error could change the rounding, one case in
// 2^40 or so.
__device__ __forceinline__ double sqrt_rn(double x, bool* sure) {
    double y;
#if defined(__CUDA_ARCH__)
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#else
    y = (double)(1.0f / sqrtf((float)x));
#endif
    double g = x * y, h = 0.5 * y;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const double r = fma(-g, h, 0.5);
        g = fma(g, r, g);
        h = fma(h, r, h);
    }
    const double d = fma(-g, g, x);
    const double up = fma(d, fma(h, 0x1p-44, h), g), dn = fma(d, fma(h, -0x1p-44, h), g);
    *sure = up == dn;
    return up;
}

}  // namespace sa
