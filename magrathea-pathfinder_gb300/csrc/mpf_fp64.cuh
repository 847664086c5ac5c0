// float64 operations on the integer bits.  An SM sub-partition's FP64 pipe
// takes a warp's add, multiply, fused multiply-add, compare or conversion 64
// cycles, however many of its lanes are active (measured; the integer and FP32
// pipes take 1 to 2); the functions below give the bits of the hardware's
// conversions, products with powers of two and compares in 4 to 10 integer
// instructions, and leave zeros, subnormals, infinities and NaN to it.  They
// pay where that pipe is the bound: the float64 kernel, the deposit, the
// compares of the FP32-gather kernel's CIC and velocity instantiations.  That
// kernel's conversions overlap its other latencies (on integer bits they
// measured 3 to 10 % slower).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "mpf_keys.cuh"

namespace mpf {

// (double)v
__device__ __forceinline__ double wide(float v)
{
    const unsigned b = __float_as_uint(v), a = b & 0x7fffffffu;
    if (a - 0x00800000u < 0x7f000000u)
        return __hiloint2double((int)(((a >> 3) + 0x38000000u) | (b & 0x80000000u)), (int)(b << 29));
    return (double)v;
}

// Range of the high word's magnitude whose value rounds to a normal float
// below 2^127: exponents -126 to 126.
__device__ __forceinline__ bool normal_float_range(unsigned hi) { return (hi & 0x7fffffffu) - 0x38100000u < 0x47e00000u - 0x38100000u; }

// (double)(float)d: round to nearest even at bit 29
__device__ __forceinline__ double round32(double d)
{
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    if (normal_float_range(hi)) {
        const unsigned l2 = lo + 0x0fffffffu + ((lo >> 29) & 1u);
        return __hiloint2double((int)(hi + (l2 < lo ? 1u : 0u)), (int)(l2 & 0xe0000000u));
    }
    return (double)__double2float_rn(d);
}

// d * 2^e (|e| < 512)
__device__ __forceinline__ double times_pow2(double d, int e)
{
    const unsigned hi = (unsigned)__double2hiint(d);
    if ((hi & 0x7fffffffu) - 0x20000000u < 0x3fe00000u) return __hiloint2double((int)(hi + ((unsigned)e << 20)), __double2loint(d));
    return d * __longlong_as_double((long long)(1023 + e) << 52);
}

// a < b for numbers (of two zeros the negative one is the smaller; a NaN is
// beyond the infinity of its sign)
__device__ __forceinline__ bool less64(double a, double b)
{
    long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    x ^= (long long)((unsigned long long)(x >> 63) >> 1);
    y ^= (long long)((unsigned long long)(y >> 63) >> 1);
    return x < y;
}

// a < 0: the bits of the negative numbers up to -infinity (neither -0 nor a NaN)
__device__ __forceinline__ bool negative(double a)
{
    return (unsigned long long)__double_as_longlong(a) - 0x8000000000000001ull < 0x7ff0000000000000ull;
}

// axis_coord(L, x), its product with the power of two and its truncation on
// the integer bits where x lies in the domain
__device__ __forceinline__ uint64_t axis_coord_bits(int L, double x)
{
    const double u = __dadd_rn(x, (double)kExtent / 2.0);
    const unsigned hi = (unsigned)__double2hiint(u);
    // 2^-512 <= u < 4
    if (hi - 0x1ff00000u < 0x40100000u - 0x1ff00000u) {
        const int drop = 52 - ((int)(hi >> 20) - 1023) - (L - kLevelShift);
        const uint64_t m = ((uint64_t)__double_as_longlong(u) & 0xfffffffffffffull) | 0x10000000000000ull;
        return (drop < 53) ? m >> drop : 0ull;
    }
    return axis_coord(L, x);
}

// coord_center(L, c) for c < 2^32: c + 1/2 from the bits of 2^52 + c, the rest
// exact as there
__device__ __forceinline__ double coord_center_bits(int L, uint64_t c)
{
    const double v = __dsub_rn(__hiloint2double(0x43300000, (int)(uint32_t)c), 4503599627370495.5);
    return __dadd_rn(times_pow2(v, kLevelShift - L), -(double)kExtent / 2.0);
}

// a / b for a divisor with y = 1 / b rounded to nearest, correctly rounded
// where nothing over- or underflows (Markstein, IBM J. Res. Dev. 34, 1990: a
// quotient within one ulp and the residual of a fused multiply-add)
__device__ __forceinline__ double divide_by(double a, double b, double y)
{
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

}  // namespace mpf
