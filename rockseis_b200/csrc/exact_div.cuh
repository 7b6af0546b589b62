// Correctly rounded division by a spacing known before the launch (the exact float modes).
// Host compilers can include it too: the same operations, checked there against the host's
// own division.
#pragma once
#include <cmath>
#include <cstring>
#include <cuda_runtime.h>
#include "rsgpu_internal.h"

namespace rsgpu {

// Operations with one rounding (a host program that uses them is compiled without contraction).
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float to_float(double a) { return __double2float_rn(a); }
__device__ __forceinline__ unsigned bits_of(float a) { return __float_as_uint(a); }
#else
inline float mul_rn(float a, float b) { return a * b; }
inline float fma_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline double mul_rn(double a, double b) { return a * b; }
inline double fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline double div_rn(double a, double b) { return a / b; }
inline float to_float(double a) { return (float)a; }
inline unsigned bits_of(float a)
{
    unsigned u;
    std::memcpy(&u, &a, sizeof u);
    return u;
}
#endif

// 2*bits - 1 of x: above r.lo for the operands the formula serves (zero wraps to the top, above
// infinities and NaN)
__host__ __device__ __forceinline__ unsigned div_key(float x) { return 2u * bits_of(x) - 1u; }
// Operands that the Rcp formula does not serve (tiny ones, whose error terms underflow;
// all of them when the divisor failed its check), in double: the quotient is corrected
// once, so it is exact where x/d is a double (ties of subnormal results among these) and
// within 2^-52 elsewhere, where x/d is at least 2^-49 from any tie between floats; zeros
// (neighbours of a tiny operand) and infinities are returned as they are.  A travelling
// wave is preceded by a fringe of such values: dividing them with __fdiv_rn took a 32 x 32
// tile 23,000 cycles instead of 3,700 (its scaled path, lane by lane).
static __host__ __device__ __attribute__((noinline)) float div_slow(float x, float d, double rd)
{
    double q = mul_rn((double)x, rd);
    q = fma_rn(fma_rn(-q, (double)d, (double)x), rd, q);
    return div_key(x) >= div_key(INFINITY) ? x : to_float(q);
}
static __host__ __device__ __attribute__((noinline)) float4 div_slow4(float4 x, float d, double rd)
{
    return make_float4(div_slow(x.x, d, rd), div_slow(x.y, d, rd), div_slow(x.z, d, rd), div_slow(x.w, d, rd));
}
__host__ __device__ __forceinline__ float div_by(float x, float d, const Rcp<float> &r)
{
    float q = fma_rn(x, r.h, mul_rn(x, r.l));
    if (div_key(x) < r.lo) q = div_slow(x, d, r.rd);
    return q;
}
__host__ __device__ __forceinline__ double div_by(double x, double d, const Rcp<double> &) { return div_rn(x, d); }
// Four quotients with one test between them.
__host__ __device__ __forceinline__ void div_by4(float (&x)[4], float d, const Rcp<float> &r)
{
    const float4 v = make_float4(x[0], x[1], x[2], x[3]);
#pragma unroll
    for (int j = 0; j < 4; j++) x[j] = fma_rn(x[j], r.h, mul_rn(x[j], r.l));
    const unsigned k0 = div_key(v.x), k1 = div_key(v.y), k2 = div_key(v.z), k3 = div_key(v.w);
    const unsigned ka = k0 < k1 ? k0 : k1, kb = k2 < k3 ? k2 : k3;
    if ((ka < kb ? ka : kb) < r.lo) {
        const float4 s = div_slow4(v, d, r.rd);
        x[0] = s.x; x[1] = s.y; x[2] = s.z; x[3] = s.w;
    }
}
__host__ __device__ __forceinline__ void div_by4(double (&x)[4], double d, const Rcp<double> &)
{
#pragma unroll
    for (int j = 0; j < 4; j++) x[j] = div_rn(x[j], d);
}

}  // namespace rsgpu
