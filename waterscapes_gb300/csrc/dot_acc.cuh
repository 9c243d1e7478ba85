// Sums of products in which the error stays below that of an FP64 sum.  Plain C++ apart from the
// two qualifiers, so that a host compiler (without contraction of products and sums) can check it.
#pragma once

#ifndef __CUDACC__
#include <cmath>
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace mpet {

// FP32 products and sums without the FP64 pipe: a sum in FP64 of the 7.5e6 products of x . A x costs
// 40 us at 64^3 (two FP64 operations per clock and SM).  Compensated dot product in threefold
// working precision (Ogita, Rump and Oishi, Accurate sum and dot product, SIAM J. Sci. Comput. 26,
// 2005, algorithm DotK with K = 3): TwoProduct by a fused multiply-add, TwoSum (Knuth; Moller)
// for the running sum and for the sum of its errors, whose own errors are added up last.  About 70
// bits are kept, against 53 of an FP64 sum; products below 1e-38 lose their low bits.
struct DotAcc {
    float hi = 0.f, lo = 0.f, rest = 0.f;

    // a += b; returns the rounding error
    static __host__ __device__ __forceinline__ float two_sum(float& a, float b) {
#ifdef __CUDA_ARCH__
        const float s = __fadd_rn(a, b), z = __fsub_rn(s, a);
        const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
#else
        const float s = a + b, z = s - a;
        const float e = (a - (s - z)) + (b - z);
#endif
        a = s;
        return e;
    }
    __host__ __device__ __forceinline__ void add(float a, float b) {
#ifdef __CUDA_ARCH__
        const float p = __fmul_rn(a, b), e = __fmaf_rn(a, b, -p);
#else
        const float p = a * b, e = std::fma(a, b, -p);
#endif
        const float t = two_sum(hi, p);
        const float u = two_sum(lo, t);
        rest += u + two_sum(lo, e);
    }
    __host__ __device__ __forceinline__ double value() const { return (double)hi + ((double)lo + (double)rest); }
};

// the same for FP64 products: an FP64 sum
struct DotAcc64 {
    double s = 0.0;
    __host__ __device__ __forceinline__ void add(double a, double b) { s += a * b; }
    __host__ __device__ __forceinline__ double value() const { return s; }
};

template <typename T>
struct DotOf {
    typedef DotAcc64 type;
};
template <>
struct DotOf<float> {
    typedef DotAcc type;
};

}  // namespace mpet
