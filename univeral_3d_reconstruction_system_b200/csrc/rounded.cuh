// rounded.cuh - quotients and roots rounded to nearest like the operators, by fused steps that share or
// approximate the reciprocal: Markstein's sequences (IBM Journal of Research and Development 34, 1990), a
// quotient or root corrected by its exact remainder. Each names the operands it is for; the operands between
// them were compared with the operators by tests/test_rounding.py, which runs these functions.
#pragma once

#include <cstdint>

#include "paired.cuh"

namespace u3dg {

// 2^lo <= |t| < 2^hi
__device__ __forceinline__ bool withinPowers(float t, int lo, int hi)
{
    return (__float_as_uint(t) & 0x7fffffffu) - (uint32_t(lo + 127) << 23) < (uint32_t(hi - lo) << 23);
}

__device__ __forceinline__ float rcpApprox(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rsqrtApprox(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The operands that a group of divisions met: dividends in size, zeros apart, and whether a divisor was out of
// Divisor's range.
struct Operands {
    uint32_t least = ~0u, most = 0; // bits, `least` less one
    bool divisors = true;
    __device__ __forceinline__ void dividend(float a)
    {
        const uint32_t m = __float_as_uint(a) & 0x7fffffffu;
        least = min(least, m - 1u); // a zero's is the largest
        most = max(most, m);
    }
    // Dividends of 0 or from 2^-83 to 2^97, divisors from 2^-30 to 2^42.
    __device__ __forceinline__ bool usual() const
    {
        return divisors && least >= (uint32_t(127 - 83) << 23) - 1u && most < uint32_t(127 + 97) << 23;
    }
};

// Several divisions by one divisor, by fused steps that are right for the usual operands: there the quotient is
// normal and its remainder exact (a zero quotient has its sign already). Where the operands were not, the caller
// does the same again with Division. The operator at each quotient instead takes its slow path for every zero.
struct Divisor {
    float b, y;
    __device__ __forceinline__ Divisor(float d, Operands &ops) : b(d), y(1.0f / d)
    {
        ops.divisors = ops.divisors && withinPowers(d, -30, 42);
    }
    __device__ __forceinline__ float under(float a, Operands &ops) const
    {
        ops.dividend(a);
        const float q = __fmul_rn(a, y);
        return a == 0.0f ? q : __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    }
};

// The operator in Divisor's place.
struct Division {
    float b;
    __device__ __forceinline__ Division(float d, Operands &) : b(d) {}
    __device__ __forceinline__ float under(float a, Operands &) const { return __fdiv_rn(a, b); }
};

// The square root of 0 and of values from 2^-100 to 2^100.
__device__ __forceinline__ float roundedRoot(float v)
{
    const float r = rsqrtApprox(v), s = __fmul_rn(v, r);
    return v == 0.0f ? 0.0f : __fmaf_rn(__fmaf_rn(-s, s, v), __fmul_rn(0.5f, r), s);
}

// a / b for a = 0 or |a| from 2^-90 to 2^60, b from 2^-50 to 2^55 (a subnormal quotient is right too: the remainder
// is exact and the last step rounds once).
__device__ __forceinline__ float roundedQuotient(float a, float b)
{
    float y = rcpApprox(b);
    y = __fmaf_rn(y, __fmaf_rn(-b, y, 1.0f), y);
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// Whether Adam's quotient a / (root(v) inv + 1e-15), inv from 1 to 32, is one of roundedRoot and roundedQuotient:
// a is 0 or from 2^-90 to 2^60, v 0 or from 2^-100 to 2^100.
__device__ __forceinline__ bool adamUsual(float a, float v)
{
    return (v == 0.0f || (v > 0.0f && withinPowers(v, -100, 100))) && (a == 0.0f || withinPowers(a, -90, 60));
}

// T / d per lane for divisors d = -nd that are multiples of 2^-24 from 0.01 to 1 (one less an alpha) and T from
// 2^-90 to 2; y becomes the reciprocals of d.
__device__ __forceinline__ float2 roundedQuotient2(float2 T, float2 nd, float2 &y)
{
    y = make_float2(rcpApprox(-nd.x), rcpApprox(-nd.y));
    y = fma2rn(y, fma2rn(nd, y, both(1.0f)), y);
    const float2 q = mul2rn(T, y);
    return fma2rn(fma2rn(nd, q, T), y, q);
}

} // namespace u3dg
