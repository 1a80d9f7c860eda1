// hcore-gb300: small device helpers shared by the recompression kernels
// (warp reductions, exact scaling by powers of two, the SVD's deflation bound).
#pragma once
#include <cuda_runtime.h>

#include "hc_internal.h"

namespace hc {

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// binary exponent (floor(log2|x|), subnormals included), per precision
__device__ __forceinline__ int binary_exponent(double x) { return ilogb(x); }
__device__ __forceinline__ int binary_exponent(float x) { return ilogbf(x); }
// 2^n built from its bits, n within the normal exponent range
template <typename T>
__device__ __forceinline__ T exp2i(int n);
template <>
__device__ __forceinline__ double exp2i<double>(int n) {
    return __longlong_as_double((long long)(n + 1023) << 52);
}
template <>
__device__ __forceinline__ float exp2i<float>(int n) {
    return __int_as_float((n + 127) << 23);
}
// x * 2^n for |n| up to twice the normal exponent range: two exact multiplies
template <typename T>
__device__ __forceinline__ T mul_exp2(T x, int n) {
    return (x * exp2i<T>(n / 2)) * exp2i<T>(n - n / 2);
}

// Squared deflation bound of the SVD kernel's QR (described there): delta^2
// for an FP64 update ranked by accuracy, -1 (no deflation) otherwise.  f2 is
// ||T||_F^2 of T scaled by 2^-sexp.
template <typename T>
__device__ __forceinline__ T deflation_bound2(T f2, int k, int M, int rk, int rule, double acc, int sexp) {
    if constexpr (sizeof(T) != sizeof(double)) {
        return T(-1);
    } else {
        const T fro = sqrt(f2);
        if (rule & kRuleRange) {
            const T dl = kCoreShare * range_delta(
                fro, M, rule & kRuleRelative, (rule & kRuleRelative) ? acc : mul_exp2(acc, -sexp));
            return isfinite(dl) ? dl * dl : T(-1);
        }
        if (rk != 0 || !(acc > 0.0)) return T(-1);
        const T thr = (rule & kRuleRelative) ? (T)acc * fro * rsqrt(T(k)) : mul_exp2((T)acc, -sexp);
        const T dl = min(T(1e-13) * thr, T(1e-16) * fro);
        return isfinite(dl) ? dl * dl : T(-1);
    }
}

// odd leading dimension of a k x k matrix in shared memory
__host__ __device__ inline int svd_ld(int k) { return k | 1; }

}  // namespace hc
