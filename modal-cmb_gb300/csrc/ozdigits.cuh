// ozdigits.cuh -- balanced 7-bit digits of scaled FP64 numbers, two at a time, as FP16
// (ozgemm.cu has the layout, gamma_split.cu slices its rows with the same digits).
//
// F = x 2^sh rounded to an integer, |F| < 2^55, is sum_p d_p 128^(s-1-p) with d_p in
// [-64, 64).  Adding 64 to every digit but the first leaves plain base-128 fields, so no
// digit waits for the one below it: a shift and a mask give d + 64, which is placed in
// the significand of the FP16 number 1024 (unit 1) and freed of its 1024 + 64 by one
// packed addition for two elements.  Digit by digit with carries and conversions, that
// was 8 integer instructions and a conversion (quarter rate) per digit and element.
#pragma once
#include <cuda_fp16.h>
#include <cmath>
#include "dfbits.cuh"

namespace modal {
namespace ozd {

// x 2^sh rounded where the bit patterns do not reach.  A call of its own: inlined, its FP64
// instructions are executed for every element and thrown away.
static __device__ __noinline__ long long far_int(double x, int sh)
{
    const double y = ldexp(x, sh);
    return isfinite(y) ? __double2ll_rn(y) : 0ll;
}

__device__ __forceinline__ long long to_int(double x, int sh)
{
    long long F;
    if (!dfb::near_int(x, sh, &F)) F = far_int(x, sh);
    return F;
}

// Digits of the elements x0, x1 (neighbours in K) to o[p * plane], p = 0 .. s - 1; s <= 8.
__device__ __forceinline__ void store2(double x0, double x1, int sh, int s, __half2 *o, size_t plane)
{
    long long bias = 0;  // 64 in every digit but the first
#pragma unroll
    for (int j = 0; j < 7; j++)
        if (j < s - 1) bias |= 64ll << (7 * j);
    const unsigned long long f0 = (unsigned long long)(to_int(x0, sh) + bias), f1 = (unsigned long long)(to_int(x1, sh) + bias);
    const uint32_t k1088 = 0x64406440u;
    const __half2 sub = *reinterpret_cast<const __half2 *>(&k1088);
#pragma unroll
    for (int j = 0; j < 7; j++)  // digit s - 1 - j
        if (j < s - 1) {
            const uint32_t w = 0x64006400u | ((uint32_t)(f0 >> (7 * j)) & 127u) | (((uint32_t)(f1 >> (7 * j)) & 127u) << 16);
            o[(size_t)(s - 1 - j) * plane] = __hsub2(*reinterpret_cast<const __half2 *>(&w), sub);
        }
    // the first digit, in [-64, 64], is signed
    const uint32_t t0 = (uint32_t)((long long)f0 >> (7 * (s - 1))) + 64u, t1 = (uint32_t)((long long)f1 >> (7 * (s - 1))) + 64u;
    const uint32_t w = 0x64006400u + t0 + (t1 << 16);
    o[0] = __hsub2(*reinterpret_cast<const __half2 *>(&w), sub);
}

}  // namespace ozd
}  // namespace modal
