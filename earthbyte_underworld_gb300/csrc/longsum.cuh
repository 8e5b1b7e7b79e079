// Sums of many products.
//
// The Krylov vectors of the mixed form are FP32, and FP64 additions take 64 cycles per warp instruction on this part,
// so a thread adds up its products without FP64.  A plain FP32 chain loses a bit with every few products, though: 59
// equal ones are off by 1e-6.  So the FP32 form keeps an unevaluated pair of FP32 values (TwoSum: Knuth, The Art of
// Computer Programming vol. 2, 4.2.2): each product is rounded once and the sum is exact to 2^-46 or so, for seven
// additions a product.  FP64 products are added as they come.
#pragma once

#include <cmath>

#ifndef __CUDACC__   // (a C++ compiler on the host)
#define __host__
#define __device__
#define __forceinline__ inline
using std::isfinite;
#endif

namespace uwg {

template <typename T>
struct LongSum;

template <>
struct LongSum<double> {
    double v = 0.0;
    __host__ __device__ __forceinline__ void add(double a, double b) { v = fma(a, b, v); }
    __host__ __device__ __forceinline__ void merge(const LongSum& o) { v += o.v; }
    __host__ __device__ __forceinline__ double value() const { return v; }
};

template <>
struct LongSum<float> {
    float h = 0.f, l = 0.f;   // the sum is h + l
    // additions and products that no compiler fuses
    static __host__ __device__ __forceinline__ float plus(float a, float b) {
#ifdef __CUDA_ARCH__
        return __fadd_rn(a, b);
#else
        volatile float s = a + b;
        return s;
#endif
    }
    static __host__ __device__ __forceinline__ float times(float a, float b) {
#ifdef __CUDA_ARCH__
        return __fmul_rn(a, b);
#else
        volatile float p = a * b;
        return p;
#endif
    }
    __host__ __device__ __forceinline__ void join(float bh, float bl) {
        const float s = plus(h, bh), t = plus(s, -h);
        const float e = plus(plus(h, -plus(s, -t)), plus(bh, -t));
        h = s;
        l = plus(plus(l, bl), e);
    }
    __host__ __device__ __forceinline__ void add(float a, float b) { join(times(a, b), 0.f); }
    // symmetric in its operands, so all lanes of an xor tree end with the same bits
    __host__ __device__ __forceinline__ void merge(const LongSum& o) { join(o.h, o.l); }
    // (of an infinite sum the low part is not a number)
    __host__ __device__ __forceinline__ double value() const { return isfinite(l) ? (double)h + (double)l : (double)h; }
};

#ifdef __CUDACC__
// the sum over a warp's lanes, in every lane
__device__ __forceinline__ void warp_merge(LongSum<double>& s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        LongSum<double> other;
        other.v = __shfl_xor_sync(0xffffffffu, s.v, o);
        s.merge(other);
    }
}
__device__ __forceinline__ void warp_merge(LongSum<float>& s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        LongSum<float> other;
        other.h = __shfl_xor_sync(0xffffffffu, s.h, o);
        other.l = __shfl_xor_sync(0xffffffffu, s.l, o);
        s.merge(other);
    }
}
#endif

}  // namespace uwg
