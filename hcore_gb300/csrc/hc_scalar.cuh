// hcore-gb300: small device helpers shared by the recompression kernels
// (warp reductions, exact scaling by powers of two, reciprocals and square roots
// from FP32 seeds, the SVD's deflation bound).
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

// ---- numbers from their bits -------------------------------------------------
// x = m 2^(e - 1023), m in [1, 2) as FP32 (truncated); e = 0 for zero and
// subnormals (their m is meaningless and not used)
__device__ __forceinline__ void split(double x, float &m, int &e) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    e = (int)((hi >> 20) & 0x7FFu);
    m = __uint_as_float(0x3F800000u | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
}
// q 2^d as FP64 for a positive normal FP32 q; 0 when the result is not normal
__device__ __forceinline__ double widen(float q, int d) {
    const unsigned b = __float_as_uint(q);
    const int e = (int)(b >> 23) + (1023 - 127) + d;
    if (e <= 0) return 0.0;
    return __hiloint2double((int)(((unsigned)e << 20) | ((b & 0x7FFFFFu) >> 3)), (int)(b << 29));
}
__device__ __forceinline__ float fsqrt_fast(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float frsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1 / sqrt(x), x normal and positive: y (1 + e/2 + 3 e^2/8), e = 1 - x y^2
__device__ __forceinline__ double inv_sqrt(double x) {
    float m;
    int e;
    split(x, m, e);
    const int ex = e - 1023, odd = ex & 1, half = (ex - odd) >> 1;
    const double y = widen(frsqrt_fast(odd ? 2.f * m : m), -half);
    const double r = fma(-x * y, y, 1.0);
    return fma(y * r, fma(0.375, r, 0.5), y);
}
__device__ __forceinline__ float inv_sqrt(float x) {   // one Newton step
    const float y = frsqrt_fast(x), h = 0.5f * y;
    return fmaf(h, fmaf(-x * y, y, 1.f), y);
}
// 1 / x, x normal and positive: y (1 + e + e^2), e = 1 - x y
__device__ __forceinline__ double inv(double x) {
    float m;
    int e;
    split(x, m, e);
    const double y = widen(__fdividef(1.f, m), 1023 - e);
    const double r = fma(-x, y, 1.0);
    return fma(y, fma(r, r, r), y);
}
__device__ __forceinline__ float inv(float x) {   // one Newton step
    const float y = __fdividef(1.f, x);
    return fmaf(y, fmaf(-x, y, 1.f), y);
}

// ---- Jacobi rotations ----------------------------------------------------------
// t = v / (|w| + sqrt(w^2 + v^2)) with the sign of w v (w = 0: of v), the
// tangent of the rotation that makes the pair orthogonal, w = a_qq - a_pp,
// v = 2 a_pq
__device__ __forceinline__ double tangent(double app, double aqq, double apq) {
    const double w = aqq - app;
    float mw, mv;
    int ew, ev;
    split(w, mw, ew);
    split(apq, mv, ev);
    ev += 1;
    if (ew == 0) {   // equal norms: 45 degrees
        mw = 0.f;
        ew = ev;
    }
    const int em = max(ew, ev), dv = ev - em;
    const float fw = mw * __int_as_float((max(ew - em, -60) + 127) << 23);
    const float fv = mv * __int_as_float((max(dv, -60) + 127) << 23);
    const float q = __fdividef(mv, fw + fsqrt_fast(fmaf(fw, fw, fv * fv)));
    const double t = widen(q, dv);
    const int sgn = ((ew == ev && mw == 0.f ? 0 : __double2hiint(w)) ^ __double2hiint(apq)) & (int)0x80000000;
    return __hiloint2double(__double2hiint(t) | sgn, __double2loint(t));
}
__device__ __forceinline__ float tangent(float app, float aqq, float apq) {
    const float w = aqq - app, v = 2.f * apq;
    const float h = fsqrt_fast(fmaf(w, w, v * v));
    const float t = __fdividef(fabsf(v), fabsf(w) + h);
    return (w < 0.f) != (v < 0.f) ? -t : t;
}

// ---- a cluster of CTAs on one update -------------------------------------------
// (.aligned wants the whole warp at the barrier together, and callers come from loops
// and branches that lanes leave at different times)
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// what to add to a shared-memory address here for the same place in CTA `to`
__device__ __forceinline__ unsigned peer_delta(const void *any, int to) {
    const unsigned here = (unsigned)__cvta_generic_to_shared(any);
    unsigned there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(to));
    return there - here;
}
__device__ __forceinline__ void peer_store(double *p, unsigned delta, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p) + delta), "d"(v)
                 : "memory");
}
__device__ __forceinline__ void peer_store(float *p, unsigned delta, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p) + delta), "f"(v)
                 : "memory");
}
__device__ __forceinline__ void peer_store(int *p, unsigned delta, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p) + delta), "r"(v)
                 : "memory");
}

// odd leading dimension of a k x k matrix in shared memory
__host__ __device__ inline int svd_ld(int k) { return k | 1; }

}  // namespace hc
