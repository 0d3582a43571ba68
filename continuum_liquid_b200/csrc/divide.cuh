// x / d for one d and many x, as the red-black updates divide by a cell's diagonal. Plain C++ as well, so that it can be
// checked against the division on the host.
#pragma once
#include <cmath>

namespace clb {

#ifdef __CUDACC__
#define CLB_DIVIDE __device__ __forceinline__
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
#else
#define CLB_DIVIDE inline
inline float fma_rn(float a, float b, float c) { return std::fma(a, b, c); }
#endif

// x / d for a positive integer-valued d up to 32768 (every diagonal: a sum of small weights) with r = 1 / d correctly
// rounded: Markstein's correction (P. Markstein, IBM J. Res. Dev. 34, 1990) of the product q = x r by its exact
// remainder x - q d. Four dependent operations after x, without a branch, instead of the general division's dozen.
// The IEEE quotient for every x whose quotient is normal, and where it is subnormal too, except that one half way between
// two neighbours may go to the odd one: the remainder is exact there (a multiple of 2^-149), r is not. (To find those and
// give them the even one costs 10 % of the solves that this serves.) Zeros, infinities and NaN are x r: the correction
// would lose the sign of a zero (0.6 % of a solve).
CLB_DIVIDE float divide_by(float x, float d, float r) {
    const float q = x * r;
    const float y = fma_rn(fma_rn(-q, d, x), r, q);
    return fabsf(x) < INFINITY && x != 0.0f ? y : q;
}

}  // namespace clb
