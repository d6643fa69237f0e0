// Correctly rounded division by a spline pivot.  The back substitution of a line solve divides by
// a pivot d whose reciprocal r = RN(1/d) the Thomas tables hold already (the multiplier of the
// next row), and the quotient of each point enters the next, so the division's latency is the
// solve's.  With r known, q = RN(a r) and q' = RN(q + r (a - q d)) is RN(a/d) as long as nothing
// underflows or overflows (P. Markstein, IBM J. Res. Dev. 34 (1990) 111; N. Brisebarre,
// J.-M. Muller, S. K. Raina, IEEE Trans. Comput. 53 (2004) 1069): three dependent operations
// in place of a library division.  Outside pivot_in_range (zeros, tiny, huge and non-finite
// numerators) the caller divides.
#pragma once

#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define GKM_PIVOT_HD __host__ __device__ __forceinline__
#else
#define GKM_PIVOT_HD inline
#endif

namespace gkm {

// 2^-895 <= |a| < 2^897: q, q d and the remainder, 2^-106 of a at the least, are normal numbers
GKM_PIVOT_HD bool pivot_in_range(double a)
{
#ifdef __CUDA_ARCH__
    const unsigned hi = (unsigned)__double2hiint(a);
#else
    unsigned long long b;
    memcpy(&b, &a, sizeof(b));
    const unsigned hi = (unsigned)(b >> 32);
#endif
    return (hi & 0x7fffffffu) - 0x08000000u < 0x70000000u;
}

// a / d, r = RN(1/d), for a in range
GKM_PIVOT_HD double pivot_quotient(double a, double d, double r)
{
#ifdef __CUDA_ARCH__
    const double q = __dmul_rn(a, r);
    return __fma_rn(__fma_rn(-q, d, a), r, q);
#else
    const double q = a * r;
    return fma(fma(-q, d, a), r, q);
#endif
}

}  // namespace gkm
