// split.cuh — FP64 values to and from FP32 words by integer operations.
//
// GB300 converts between FP32 and FP64 on its FP64 pipe, at two lanes per clock
// and SM; an integer instruction takes a thirty-second of that.  These give
// the values of the conversions (round to nearest, ties to even) for
// magnitudes in [2^-70, 2^127) and leave the others, zero included, to the
// conversion itself (tests/test_gpu_exact_helpers.py).
#pragma once

#include <cuda_runtime.h>

namespace b2d {

// The conversions themselves, as calls: inlined, the compiler runs them ahead
// of the test that decides whether they are wanted.
static __device__ __noinline__ float narrow_any(double v) { return (float)v; }
static __device__ __noinline__ double widen_any(float v) { return (double)v; }
static __device__ __noinline__ double halve_any(double v) { return 0.5 * v; }
static __device__ __noinline__ float2 split_any(double v)
{
    const float hi = (float)v;
    return make_float2(hi, (float)(v - (double)hi));
}

__device__ __forceinline__ bool split_range(double v)
{
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - 0x3b900000u < 0x47e00000u - 0x3b900000u;
}

// v = hi + lo to 2^-49 of v, v in split_range.
__device__ __forceinline__ void split_bits(double v, float& hi, float& lo)
{
    const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v), s = h & 0x80000000u;
    const unsigned m = h & 0x7fffffffu;
    unsigned f = __funnelshift_l(l, m - 0x38000000u, 3);       // exponent rebased, mantissa cut to 23 bits
    const unsigned rest = l & 0x1fffffffu;
    const unsigned up = (rest + 0x0fffffffu + (f & 1u)) >> 29;
    f += up;
    hi = __uint_as_float(f | s);
    // what was cut, in units of the FP64 mantissa's last place
    const float r = __int2float_rn((int)rest - (int)(up << 29));
    lo = __fmul_rn(r, __uint_as_float((((m >> 20) - 948u) << 23) | s));
}

__device__ __forceinline__ void split_double(double v, float& hi, float& lo)
{
    if (split_range(v)) split_bits(v, hi, lo);
    else {
        const float2 w = split_any(v);
        hi = w.x;
        lo = w.y;
    }
}

// (float)v, v in split_range.
__device__ __forceinline__ float narrow_bits(double v)
{
    const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
    unsigned f = __funnelshift_l(l, (h & 0x7fffffffu) - 0x38000000u, 3);
    f += ((l & 0x1fffffffu) + 0x0fffffffu + (f & 1u)) >> 29;
    return __uint_as_float(f | (h & 0x80000000u));
}

__device__ __forceinline__ float narrow(double v) { return split_range(v) ? narrow_bits(v) : narrow_any(v); }

// v / 2: one off the exponent.
__device__ __forceinline__ double halve(double v)
{
    const unsigned h = (unsigned)__double2hiint(v);
    if ((h & 0x7fffffffu) - 0x00200000u >= 0x7fd00000u) return halve_any(v);   // zero, next to subnormal, infinite, NaN
    return __hiloint2double((int)(h - 0x00100000u), __double2loint(v));
}

// Exact for zero, normal and (flushed to zero) subnormal v.
__device__ __forceinline__ double widen(float v)
{
    const unsigned f = __float_as_uint(v), m = f & 0x7fffffffu;
    if (m - 0x00800000u >= 0x7f000000u) return widen_any(v);       // zero, subnormal, infinite, NaN
    return __hiloint2double((int)((f & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(f << 29));
}

}  // namespace b2d
