// divsmall.cuh -- quotients by integers without a division, for the CPU and the GPU.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define DIVSMALL_HD __host__ __device__ __forceinline__
#else
#define DIVSMALL_HD inline
#endif

namespace modal {

// n / c for an integer 1 <= c < 2^49 and r = 1 / c rounded: Markstein's correction of n r (P. W.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Develop. 34 (1990)).  Three dependent operations instead of a division's dozen, and the same
// value wherever n, n r and the residual are normal numbers or zero (a zero comes out as +0):
// q = n r rounded is within two units of n / c, the residual n - q c is an integer number of units below
// 2^53 and so exact, and the last operation rounds n / c + d with |d| <= 2^-51 units, while a quotient by c is
// never nearer than 1 / (2c) units to a midpoint, nor on one (n would need 54 bits).
DIVSMALL_HD double div_small(double n, double c, double r)
{
    const double q = n * r;
#ifdef __CUDA_ARCH__
    return fma(fma(-q, c, n), r, q);
#else
    return std::fma(std::fma(-q, c, n), r, q);
#endif
}

}  // namespace modal
