// hcore-gb300 — batched low-rank recompression kernels for sm_103a.
//
// One Schur update C <- beta*C + alpha*A*B^T (A, B, C in U*V^T form) follows
// the reference HCORE_dgemm (src/compute/hcore_dgemm.c:703-1012) as four
// batched phases, each a grid over the updates of the batch:
//
//   1. stack  (hcore_dgemm.c:79-225)  UA = [beta*CU | alpha*AU],
//              F = AV^T BV, G = BU F^T, VB = [CV | G]            -> workspace
//   2. geqrf  (hcore_dgemm.c:123, :216) Householder QR of UA and VB
//              (blockIdx.y selects the side), LAPACK dlarfg conventions
//   3. gesvd  (hcore_dgemm.c:296-503) T = R_A R_B^T, pivoted QR (in FP64
//              deflated below 1e-13 of the threshold), one-sided Jacobi SVD,
//              singular values sorted, rank rule, U_r and V_r S_r
//   4. apply  (hcore_dgemm.c:508-696) CU = Q_A [U_r; 0], CV = Q_B [V_r S_r; 0]
//              written straight into the caller's output factors
//
// In FP64 plans the QR runs blocked, its trailing updates on the tensor cores
// (hc_qr_tc.cu); the rebuild of updates with a + c <= 64 runs there too
// (hc_rebuild_tc.cu).  The SVD is in hc_svd.cu; this file keeps the stack, the
// QR's panels, the rebuild in every other case, and the launches.
//
// The scalar type T is double (HCORE_dgemm) or float (HCORE_sgemm); every
// step computes in T, like the reference's two copies.  With the plan flag
// HCORE_GPU_MIXED_FACTORS an FP64 plan computes the factor products (stack)
// and the Q.U rebuild in FP32 (compute type Tc = float, FP32 accumulation,
// FP64 storage) while the QRs, the SVD and the truncation stay FP64.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <mutex>
#include <set>
#include <utility>

#include "hc_internal.h"
#include "hc_scalar.cuh"

namespace hc {

// -x by its sign bit (integer pipe; exact, NaN payloads kept)
__device__ __forceinline__ double flip_sign(double x) {
    return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ULL);
}
__device__ __forceinline__ float flip_sign(float x) {
    return __int_as_float(__float_as_int(x) ^ (int)0x80000000u);
}

// ---------------------------------------------------------------------------
// phase 1: stack the factors
// ---------------------------------------------------------------------------
// Two kernels: the copies [beta CU | alpha AU], [CV | .] and F = AV^T BV, then
// G = BU F^T (or B AV for a dense B).  Both are bound by FP64 issue, so a warp
// takes four entries of F at a time (one load of BV's column for four FMAs, six
// shuffled additions for the four sums instead of twenty), and an update's
// columns and rows are split over CTAs until the GPU is full.  On one CTA each,
// and now: one update of M = 512 and ranks 32 405, 74 us; 384 of M = 1024,
// ranks 6-34, 1648, 720 us; 24 of M = 1000, ranks 40-110, 6.7, 0.83 ms.
// tc_products: the products F and G of updates that stack_tc_eligible accepts
// are left to the tensor-core kernel (hc_stack_tc.cu).
template <typename T, typename Tc>
__global__ void __launch_bounds__(kThreads) stack_inner_kernel(const Desc *__restrict__ descs,
                                                               T *__restrict__ ws, bool tc_products) {
    const Desc d = descs[blockIdx.x];
    if (d.status0) return;
    const int M = d.M, a = d.a, b = d.b, c = d.c;
    const WsLayout L = ws_layout(d);
    T *UA = ws + d.ws + L.UA, *VB = ws + d.ws + L.VB, *F = ws + d.ws + L.F;
    const T alpha = (T)d.alpha, beta = (T)d.beta;
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.y * kWarps + (threadIdx.x >> 5), nwarps = gridDim.y * kWarps;

    // [beta*CU | alpha*AU] and [CV | .] (hcore_dgemm.c:106-114, :199-205), a
    // warp per column.  The Schur update's coefficients 1 and -1 are applied
    // without an FP64 instruction (a copy, a sign-bit flip on the integer
    // pipe): same bits.
    const bool beta_one = beta == T(1), alpha_minus_one = alpha == T(-1);
    for (int q = warp; q < 2 * c + a; q += nwarps) {
        const T *src;
        T *dst;
        if (q < c) {
            src = (const T *)d.CU + (size_t)q * d.ldc;
            dst = UA + (size_t)q * M;
        } else if (q < 2 * c) {
            src = (const T *)d.CV + (size_t)(q - c) * d.ldc;
            dst = VB + (size_t)(q - c) * M;
        } else {
            src = (const T *)d.AU + (size_t)(q - 2 * c) * d.lda;
            dst = UA + (size_t)(q - c) * M;
        }
        if (q >= c && q < 2 * c) {
#pragma unroll 4
            for (int i = lane; i < M; i += 32) dst[i] = src[i];
        } else if (q < c) {
#pragma unroll 4
            for (int i = lane; i < M; i += 32) dst[i] = beta_one ? src[i] : beta * src[i];
        } else {
#pragma unroll 4
            for (int i = lane; i < M; i += 32) dst[i] = alpha_minus_one ? flip_sign(src[i]) : alpha * src[i];
        }
    }
    if (a == 0 || d.Bd || (tc_products && stack_tc_eligible(d))) return;
    // F = AV^T BV, a x b (hcore_dgemm.c:175-178)
    const T *AV = (const T *)d.AV, *BV = (const T *)d.BV;
    const int quads = (a + 3) / 4;
    for (int e = warp; e < quads * b; e += nwarps) {
        const int p0 = e % quads * 4, q = e / quads;
        const T *y = BV + (size_t)q * d.ldb;
        const T *x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = AV + (size_t)min(p0 + u, a - 1) * d.lda;
        Tc s[4] = {};
#pragma unroll 2
        for (int l = lane; l < M; l += 32) {
            const Tc yv = (Tc)y[l];
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += (Tc)x[u][l] * yv;
        }
        // lanes 8 u .. 8 u + 7 end with sum u
        const bool h16 = lane & 16, h8 = lane & 8;
        const Tc s0 = (h16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, h16 ? s[0] : s[2], 16);
        const Tc s1 = (h16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, h16 ? s[1] : s[3], 16);
        Tc r = (h8 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, h8 ? s0 : s1, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        const int p = p0 + (lane >> 3);
        if ((lane & 7) == 0 && p < a) F[(size_t)q * a + p] = (T)r;
    }
}

// G (M x a): a thread per row, four columns at a time
template <typename T, typename Tc>
__global__ void __launch_bounds__(128) stack_outer_kernel(const Desc *__restrict__ descs,
                                                          T *__restrict__ ws, bool tc_products) {
    const Desc d = descs[blockIdx.x];
    if (d.status0) return;
    const int M = d.M, a = d.a, b = d.b, i = blockIdx.y * 128 + threadIdx.x;
    if (i >= M || a == 0 || (tc_products && stack_tc_eligible(d))) return;
    const WsLayout L = ws_layout(d);
    const T *F = ws + d.ws + L.F;
    T *G = ws + d.ws + L.VB + (size_t)d.c * M;
    for (int p0 = 0; p0 < a; p0 += 4) {
        Tc s[4] = {};
        if (d.Bd) {   // dense B: G = B * AV (hcore_dgemm.c:262-271)
            const T *B = (const T *)d.Bd + i, *AV = (const T *)d.AV;
#pragma unroll 4
            for (int l = 0; l < M; ++l) {
                const Tc x = (Tc)B[(size_t)l * d.ldb];
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] += x * (Tc)AV[(size_t)min(p0 + u, a - 1) * d.lda + l];
            }
        } else {      // G = BU F^T (hcore_dgemm.c:199-205)
            const T *BU = (const T *)d.BU + i;
#pragma unroll 4
            for (int q = 0; q < b; ++q) {
                const Tc x = (Tc)BU[(size_t)q * d.ldb];
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] += x * (Tc)F[(size_t)q * a + min(p0 + u, a - 1)];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (p0 + u < a) G[(size_t)(p0 + u) * M + i] = (T)s[u];
    }
}

template <typename T, typename Tc>
static void launch_stack(const Desc *d_desc, int n, T *ws, bool tc_products, int updates, int maxM,
                         cudaStream_t s) {
    // eight CTAs an SM's worth over the updates that share the GPU
    const int split = std::max(1, std::min(32, 1216 / std::max(updates, 1)));
    stack_inner_kernel<T, Tc><<<dim3(n, split), kThreads, 0, s>>>(d_desc, ws, tc_products);
    stack_outer_kernel<T, Tc><<<dim3(n, (maxM + 127) / 128), 128, 0, s>>>(d_desc, ws, tc_products);
}

// ---------------------------------------------------------------------------
// phase 2: Householder QR of UA (blockIdx.y = 0) or VB (blockIdx.y = 1)
// ---------------------------------------------------------------------------
// Reflector j is H_j = I - tau_j v v^T with v(j) = 1, v(i<j) = 0 and v(i>j)
// stored below the diagonal, beta = -sign(alpha)*||x||, tau = (beta-alpha)/beta
// (LAPACK dlarfg); ||x|| = 0 gives tau = 0.  R ends up on and above the
// diagonal, as dgeqrf leaves it.
//
// FP64 issue slots are the scarce resource on this GPU, so a warp keeps the
// column it updates in registers (RPL rows per lane, row = lane + 32 t): one
// load, one dot, one axpy, one store per column and reflector.  The reflector
// vector is published in shared memory, zero outside rows j..M-1, so the dot
// and the axpy need no predicates.  Look-ahead: warp 0 updates column j+1
// first and turns it into reflector j+1 while the other warps finish step j,
// so there is a single barrier per column.
// lo/hi: range in which a plain sum of squares neither under- nor overflows;
// safmin = (smallest normal) / eps, the LAPACK dlamch('S')/dlamch('E')
// threshold below which 1/beta is not safe (a power of two).
template <typename T>
struct NormLim;
template <>
struct NormLim<double> {
    static constexpr double lo = 1e-280, hi = 1e280;
    static constexpr double safmin = DBL_MIN / DBL_EPSILON;
    static constexpr int max_shift = 1000;   // 2^(+-max_shift) is a normal double
};
template <>
struct NormLim<float> {
    static constexpr float lo = 1e-30f, hi = 1e30f;
    static constexpr float safmin = FLT_MIN / FLT_EPSILON;
    static constexpr int max_shift = 120;
};

// dlarfg's rescaling for a column whose beta is below safmin (subnormal
// entries; warp-uniform and rare, so kept out of line to spare the
// registers of the common path).  With alpha and ||x|| scaled by 2^s
// (|beta| -> ~1) tau follows, and v = x 2^s / (as - bs) is applied in two
// exact factors to the x that make_reflector published; beta stays
// unscaled.  Each lane rescales the rows it stored.  Returns tau.
template <typename T>
__device__ __noinline__ T rescale_reflector(T alpha, T xnorm, T beta, int j, int M, int lane,
                                            T *Aj, T *sv) {
    const int sh = -binary_exponent(beta);
    const T as = mul_exp2(alpha, sh);
    const T xs = mul_exp2(xnorm, sh);   // as, xs <= ~1: no overflow below
    const T bs = -copysign(sqrt(as * as + xs * xs), as);
    const T sc = exp2i<T>(sh - sh / 2) / (as - bs), post = exp2i<T>(sh / 2);
    for (int i = lane; i < M; i += 32) {
        if (i <= j) continue;
        const T v = (sv[i] * sc) * post;
        sv[i] = v;
        Aj[i] = v;
    }
    return (bs - as) / bs;
}

// Build reflector j from the register column x (already updated by all
// earlier reflectors); store the column back and publish v and tau.
// Tiny columns (subnormal entries, e.g. far-field interactions in FP32)
// take a scaled norm (dnrm2) and dlarfg's rescaling, so that no reciprocal
// overflows; both scale by powers of two only (exact, no division).
template <typename T, int RPL>
__device__ __forceinline__ void make_reflector(T (&x)[RPL], int j, int M, int lane, T *Aj,
                                               T *sv, T *s_tau, T *tau_out) {
    T alpha_l = 0, ss = 0;
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
        const int i = lane + 32 * t;
        if (i == j) alpha_l = x[t];
        if (i > j && i < M) ss += x[t] * x[t];
    }
    const T alpha = __shfl_sync(0xffffffffu, alpha_l, j & 31);
    ss = warp_sum(ss);
    T xnorm = 0, tj = 0, beta = alpha, scal = 1;
    bool rescale = false;
    const T n2 = fma(alpha, alpha, ss);
    const bool plain = sizeof(T) == sizeof(double) && ss > NormLim<T>::lo && n2 < NormLim<T>::hi;
    if (plain) {
        // the short square root and reciprocals (hc_scalar.cuh): hypot, a square root
        // and two divisions take about 100 FP64 instructions of 65 cycles in the
        // chain of every column (QR panels of one update of order 512, k = 64: 432 us
        // with them, 388 so)
        const T rs = inv_sqrt(n2);
        T nb = n2 * rs;
        nb = fma(fma(-nb, nb, n2) * T(0.5), rs, nb);
        beta = -copysign(nb, alpha);
        tj = fma(abs(alpha), rs, T(1));   // (beta - alpha) / beta; 2 where x is small
        scal = copysign(inv(abs(alpha - beta)), alpha);
    } else if (ss > NormLim<T>::lo && ss < NormLim<T>::hi) {
        xnorm = sqrt(ss);
    } else {  // scaled recomputation (dnrm2's guard against under/overflow)
        T amax = 0;
#pragma unroll
        for (int t = 0; t < RPL; ++t) {
            const int i = lane + 32 * t;
            if (i > j && i < M) amax = max(amax, abs(x[t]));
        }
        amax = warp_max(amax);
        T s2 = 0;
        int sc = 0;
        if (amax > T(0)) {
            // y = x 2^sc with |y| < 2 (sc clamped to a representable power)
            sc = min(max(-binary_exponent(amax), -NormLim<T>::max_shift), NormLim<T>::max_shift);
            const T f = exp2i<T>(sc);
#pragma unroll
            for (int t = 0; t < RPL; ++t) {
                const int i = lane + 32 * t;
                if (i > j && i < M) {
                    const T y = x[t] * f;
                    s2 += y * y;
                }
            }
        }
        xnorm = mul_exp2(sqrt(warp_sum(s2)), -sc);
    }
    if (!plain && xnorm > T(0)) {
        beta = -copysign(hypot(alpha, xnorm), alpha);
        if (abs(beta) >= NormLim<T>::safmin) {
            tj = (beta - alpha) / beta;
            scal = T(1) / (alpha - beta);
        } else if (beta == beta) {
            rescale = true;   // 1/(alpha - beta) would overflow: x is published as is
        }
    }
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
        const int i = lane + 32 * t;
        T v = 0;
        if (i > j && i < M) {
            v = x[t] * scal;
            Aj[i] = v;
        } else if (i == j) {
            v = T(1);
            Aj[i] = beta;
        } else if (i < j) {
            Aj[i] = x[t];  // R entries above the diagonal
        }
        sv[i] = v;
    }
    if (rescale) tj = rescale_reflector(alpha, xnorm, beta, j, M, lane, Aj, sv);
    if (lane == 0) {
        *s_tau = tj;
        tau_out[j] = tj;
    }
}

// NW warps per CTA (a tuning choice): 8 gives the shortest path per update;
// 4 or 2 keep the same warps per SM in two or four times as many CTAs, so
// that one CTA's per-column barrier stall is covered by the others.
// panel < 0: all k columns; panel p >= 0: the columns [c0, c1) of the blocked
// QR's panel p (qr_panel_bounds), whose earlier columns are already factored
// and whose own columns already hold the earlier panels' updates.
template <typename T, int RPL, int NW>
__global__ void __launch_bounds__(NW * 32, (RPL <= 32 ? 2 : 1) * (8 / NW))
    geqrf_kernel(const Desc *__restrict__ descs, T *__restrict__ ws, int panel) {
    __shared__ T sv[2][32 * RPL];
    __shared__ T s_tau[2];
    const Desc d = descs[blockIdx.x];
    if (d.status0) return;
    const int M = d.M, k = d.k;
    int c0 = 0, c1 = k;
    if (panel >= 0 && !qr_panel_bounds(k, panel, c0, c1)) return;
    const WsLayout L = ws_layout(d);
    const int side = blockIdx.y;
    T *A = ws + d.ws + (side ? L.VB : L.UA);
    T *tau = ws + d.ws + (side ? L.tauB : L.tauA);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x[RPL];

    if (warp == 0) {
        const T *A0 = A + (size_t)c0 * M;
#pragma unroll
        for (int t = 0; t < RPL; ++t) {
            const int i = lane + 32 * t;
            x[t] = i < M ? A0[i] : T(0);
        }
        make_reflector<T, RPL>(x, c0, M, lane, A + (size_t)c0 * M, sv[0], &s_tau[0], tau);
    }
    __syncthreads();
    for (int j = c0; j + 1 < c1; ++j) {
        const int cur = (j - c0) & 1;
        const T *v = sv[cur];
        const T tj = s_tau[cur];
        for (int col = j + 1 + warp; col < c1; col += NW) {
            T *Ac = A + (size_t)col * M;
#pragma unroll
            for (int t = 0; t < RPL; ++t) {
                const int i = lane + 32 * t;
                x[t] = i < M ? Ac[i] : T(0);
            }
            if (tj != T(0)) {
                // two chains: four measured slower here (register pressure at
                // four CTAs per SM; other CTAs already hide the chain's latency)
                T d0 = 0, d1 = 0;
#pragma unroll
                for (int t = 0; t < RPL; t += 2) {
                    d0 += v[lane + 32 * t] * x[t];
                    if (t + 1 < RPL) d1 += v[lane + 32 * (t + 1)] * x[t + 1];
                }
                const T sc = tj * warp_sum(d0 + d1);
                // re-read v from shared memory instead of holding RPL values in registers
                const volatile T *vv = v;
#pragma unroll
                for (int t = 0; t < RPL; ++t) x[t] -= sc * vv[lane + 32 * t];
            }
            if (col == j + 1) {
                make_reflector<T, RPL>(x, j + 1, M, lane, Ac, sv[cur ^ 1], &s_tau[cur ^ 1], tau);
            } else {
#pragma unroll
                for (int t = 0; t < RPL; ++t) {
                    const int i = lane + 32 * t;
                    if (i >= j && i < M) Ac[i] = x[t];
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// phase 3: T = R_A R_B^T, SVD, rank rule (hc_svd.cu)
// ---------------------------------------------------------------------------
// Lanes per column pair of the shared-memory SVD (hc_svd.cu), by the plan's
// tuning for buckets of up to 24, up to 64 and more pairs.  A tuning value of
// 0 takes as many lanes (a power of two) as fit in the warps that one lane
// per pair needs.  Without a tuning (-1): eight lanes while every update has
// an SM of its own and they fit in eight warps (two a sub-partition), else
// four.  More lanes shorten a round's rows, but each warp repeats the
// rotation parameters, which counts once the FP64 pipes are shared.  SVD
// phase with 2, 4 and 8 lanes (us): 16 updates of k 8-24 410, 287, 250; one
// of k = 64 2839, 1753, 1453; 24 of k 80-116 8262, 5794, 6099; 384 of k
// 12-68 4120, 3220, 3205 (whole plan 10787, 9669, 10455); 1900 of the same
// 6216, 5747, 6881.  FP32 (no pipe to wait for, so eight lanes up to two updates an
// SM and 16 warps), the whole plan with 4 and 8 lanes: 256 of k 10-48 570, 535; 1000
// of the same 933, 991; 20 of k 60-120 2611, 2276.
template <typename T>
static int svd_smem_lanes(int K, const int *lanes, int updates) {
    const int np = (K + 1) / 2;
    int g = np <= 24 ? lanes[0] : (np <= 64 ? lanes[1] : lanes[2]);
    if (g < 0 && sizeof(T) == 4) g = updates <= 304 && 8 * np <= 512 ? 8 : 4;
    if (g < 0) g = updates <= 152 && 8 * np <= 256 ? 8 : 4;
    if (g == 0) {
        const int w = (np + 31) / 32;
        g = 1;
        while (g < 32 && 2 * g * np <= 32 * w) g *= 2;
    }
    return g;
}

// CTAs per update of the shared-memory SVD, the same bits whatever their number:
// as many as leave each eight column pairs (one warp a sub-partition at 16 lanes a
// pair) and as run at once for all of the plan's updates (a cluster's CTAs share a
// GPC: 48 clusters of three fill 152 SMs, and the two left over of 50 ran alone
// after them, 7.2 ms with one CTA, 7.7 so).  One where the update has at most 24
// pairs, or where that gives too few, since an exchange costs 0.8 us of a round,
// about as much as it saves there.  FP32 rounds wait for latency, not for a pipe.
// SVD phase, one CTA and a cluster, us: one update of k = 40 550, 589; 64 1403,
// 1175; 116 6241, 3556; 24 of k 80-116 5725, 4680 (six); 36 of k 16-56 913, 841
// (four); 40 of k 80-116 5780, 4182, 48 of k 60-80 2801, 2168, of k 32-64 1355, 1389
// (three).
template <typename T>
static int svd_spread(int K, const int *lanes, int updates) {
    const int np = (K + 1) / 2;
    if (sizeof(T) != sizeof(double) || np <= 24 || (np <= 64 ? lanes[1] : lanes[2]) >= 0) return 1;
    for (int cs = std::min({8, (np + 7) / 8, 152 / std::max(1, updates)}); cs >= (np > 32 ? 3 : 4); --cs)
        if (svd_spread_fit<T>(K, cs) >= updates) return cs;
    return 1;
}

// ---------------------------------------------------------------------------
// phase 4: CU = Q_A [U_r; 0], CV = Q_B [V_r S_r; 0]   (dormqr 'L','N')
// ---------------------------------------------------------------------------
// A CTA owns up to kWarps output columns of one (update, side), one per warp,
// each kept in registers (RPL rows per lane, row = lane + 32 t) for the whole
// product.  The k reflectors are applied last to first, staged through
// shared memory kApplyChunk at a time (one coalesced load per CTA, zero
// outside rows j..M-1 so that the dot and the axpy need no predicates); the
// column is stored once, coalesced, into the caller's factor.  blockIdx.z
// selects the group of columns; groups past the new rank exit at once.
constexpr int kApplyChunk = 8;

template <typename T, int RPL, typename Tc>
__global__ void __launch_bounds__(kThreads, RPL <= 32 ? 2 : 1) apply_kernel(const Desc *__restrict__ descs,
                                                         const T *__restrict__ ws,
                                                         const int *__restrict__ rank,
                                                         const int *__restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    Tc *sv = reinterpret_cast<Tc *>(smem_raw);   // kApplyChunk x (32 RPL)
    __shared__ Tc s_tau[kApplyChunk];
    const Desc d = descs[blockIdx.x];
    if (d.status0 || status[d.idx] != HCORE_GPU_S_OK) return;
    const int r = rank[d.idx];
    const int col0 = blockIdx.z * kWarps;
    if (col0 >= r) return;
    const int side = blockIdx.y;
    const int M = d.M, k = d.k;
    const WsLayout L = ws_layout(d);
    const T *base = ws + d.ws;
    const T *Y = base + (side ? L.VB : L.UA);
    const T *tau = base + (side ? L.tauB : L.tauA);
    const T *X0 = base + (side ? L.Vo : L.Uo);
    T *out = (T *)(side ? d.CVo : d.CUo);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = col0 + warp;
    const bool active = col < r;
    constexpr int ROWS = 32 * RPL;

    Tc x[RPL];
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
        const int i = lane + 32 * t;
        x[t] = (active && i < k) ? (Tc)X0[(size_t)col * k + i] : Tc(0);
    }
    const int nch = (k + kApplyChunk - 1) / kApplyChunk;
    for (int ch = nch - 1; ch >= 0; --ch) {
        const int j0 = ch * kApplyChunk;
        const int nj = min(kApplyChunk, k - j0);
        __syncthreads();  // the previous chunk is no longer read
        for (int e = tid; e < nj * ROWS; e += kThreads) {
            const int c = e / ROWS, i = e % ROWS;
            const int j = j0 + c;
            Tc v = Tc(0);
            if (i > j && i < M) v = (Tc)Y[(size_t)j * M + i];
            else if (i == j) v = Tc(1);
            sv[c * ROWS + i] = v;
        }
        if (tid < nj) s_tau[tid] = (Tc)tau[j0 + tid];
        __syncthreads();
        if (!active) continue;
        for (int c = nj - 1; c >= 0; --c) {
            const Tc tj = s_tau[c];
            if (tj == Tc(0)) continue;
            const Tc *v = sv + c * ROWS;
            Tc d0 = 0, d1 = 0;
#pragma unroll
            for (int t = 0; t < RPL; t += 2) {
                d0 += v[lane + 32 * t] * x[t];
                if (t + 1 < RPL) d1 += v[lane + 32 * (t + 1)] * x[t + 1];
            }
            const Tc s = tj * warp_sum(d0 + d1);
            const volatile Tc *vv = v;  // re-read rather than hold RPL values in registers
#pragma unroll
            for (int t = 0; t < RPL; ++t) x[t] -= s * vv[lane + 32 * t];
        }
    }
    if (active) {
#pragma unroll
        for (int t = 0; t < RPL; ++t) {
            const int i = lane + 32 * t;
            if (i < M) out[(size_t)col * d.ldco + i] = (T)x[t];
        }
    }
}

// ---------------------------------------------------------------------------
template <typename T, int RPL, typename Tc>
static void launch_apply(const Desc *d_desc, int n, const T *ws, const int *d_rank,
                         const int *d_status, int maxK, cudaStream_t s) {
    const int groups = (maxK + kWarps - 1) / kWarps;   // the new rank is at most k
    const size_t smem = (size_t)kApplyChunk * 32 * RPL * sizeof(Tc);
    apply_kernel<T, RPL, Tc><<<dim3(n, 2, groups), kThreads, smem, s>>>(d_desc, ws, d_rank,
                                                                       d_status);
}

template <typename T, typename Tc>
static void launch_apply_all(const Desc *d_desc, int n, const T *ws, const int *d_rank,
                             const int *d_status, int maxK, int rpl, cudaStream_t s) {
    if (rpl <= 4) launch_apply<T, 4, Tc>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else if (rpl <= 8) launch_apply<T, 8, Tc>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else if (rpl <= 16) launch_apply<T, 16, Tc>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else if (rpl <= 32) launch_apply<T, 32, Tc>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else launch_apply<T, 64, Tc>(d_desc, n, ws, d_rank, d_status, maxK, s);
}

template <typename T, typename Tc>
static cudaError_t set_apply_smem() {
    const int s64 = kApplyChunk * 32 * 64 * (int)sizeof(Tc);
    cudaError_t e = cudaFuncSetAttribute(apply_kernel<T, 64, Tc>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, s64);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(apply_kernel<T, 32, Tc>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, s64 / 2);
    return e;
}

template <typename T, int RPL>
static void launch_geqrf(const Desc *d_desc, int n, T *ws, int warps, int panel, cudaStream_t s) {
    if (n <= 0) return;
    if (warps == 2) geqrf_kernel<T, RPL, 2><<<dim3(n, 2), 64, 0, s>>>(d_desc, ws, panel);
    else if (warps == 4) geqrf_kernel<T, RPL, 4><<<dim3(n, 2), 128, 0, s>>>(d_desc, ws, panel);
    else geqrf_kernel<T, RPL, 8><<<dim3(n, 2), 256, 0, s>>>(d_desc, ws, panel);
}

template <typename T>
static void launch_geqrf_all(const Desc *d_desc, int n, T *ws, int warps, int rpl, int panel,
                             cudaStream_t s) {
    if (rpl <= 4) launch_geqrf<T, 4>(d_desc, n, ws, warps, panel, s);
    else if (rpl <= 8) launch_geqrf<T, 8>(d_desc, n, ws, warps, panel, s);
    else if (rpl <= 16) launch_geqrf<T, 16>(d_desc, n, ws, warps, panel, s);
    else if (rpl <= 32) launch_geqrf<T, 32>(d_desc, n, ws, warps, panel, s);
    else launch_geqrf<T, 64>(d_desc, n, ws, warps, panel, s);
}

// Launch plan of the blocked QR over a shape's k-sorted buckets: panel p runs
// over every descriptor that has one, and the trailing update after panel p
// once per update-size class.  fn(kind, start, count, panel, class, groups):
// kind 1 panel, 2 trailing update.
//
// Every rank sum takes it: a column's update by one reflector is 2 M FP64 FMAs
// on the register kernel, while the update by a panel of 16 is a sixteenth of
// one pass over the column on the tensor cores.  QR phase of 24 updates of M =
// 1000 and k 80-220 25.5 ms unblocked, 5.4 blocked; of 384 of M = 1024 and k
// 12-68 5.06 ms with k > 64 unblocked, 3.17 (one GB300, graph replay).
template <typename F>
static void qr_plan(const LaunchShape &shape, int n, F &&fn) {
    if (n <= 0 || shape.nbuckets <= 0) return;
    const int kmax = shape.buckets[0].K;
    for (int p = 0;; ++p) {
        int c0, c1;
        if (!qr_panel_bounds(kmax, p, c0, c1)) break;
        // descriptors below the buckets that have this panel exit at once
        int count = 0;
        for (int b = 0; b < shape.nbuckets && qr_panel_bounds(shape.buckets[b].K, p, c0, c1); ++b)
            count += shape.buckets[b].count;
        fn(1, 0, count, p, 0, 1);
        // trailing updates: descriptors whose panel p is not their last
        int bb = 0, start = 0;
        while (bb < shape.nbuckets) {
            const int K = shape.buckets[bb].K;
            if (!qr_panel_bounds(K, p, c0, c1) || c1 >= K) break;  // sorted: none below
            const int cls = qr_update_class(K - 16 * p), groups = (K - c1 + kQrGroup - 1) / kQrGroup;
            count = 0;
            while (bb < shape.nbuckets && qr_panel_bounds(shape.buckets[bb].K, p, c0, c1) &&
                   c1 < shape.buckets[bb].K && qr_update_class(shape.buckets[bb].K - 16 * p) == cls)
                count += shape.buckets[bb++].count;
            if (count > 0) fn(2, start, count, p, cls, groups);
            start += count;
        }
    }
}

int qr_launches(const LaunchShape &shape, bool fp64) {
    if (!fp64 || !shape.tc_qr || shape.nbuckets <= 0) return 1;
    int c = 0;
    int n = 0;
    for (int b = 0; b < shape.nbuckets; ++b) n += shape.buckets[b].count;
    qr_plan(shape, n, [&](int, int, int count, int, int, int) { c += count > 0; });
    return c;
}

cudaError_t allow_smem(const void *kernel) {
    static std::mutex mu;
    static std::set<std::pair<int, const void *>> done;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({dev, kernel})) return cudaSuccess;
    cudaFuncAttributes fa;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e == cudaSuccess) done.insert({dev, kernel});
    return e;
}

template <typename T>
static cudaError_t configure_recompress_once(int dev, int *svd_smem_kmax);

// The kernel attributes are per device and do not depend on the plan, so
// they are set once per device and scalar type; later calls (every drop-in
// call, every plan) only read the cached limits.
template <typename T>
cudaError_t configure_recompress(int maxK, int *svd_smem_kmax) {
    (void)maxK;
    constexpr int kDevices = 64;
    static std::mutex mu;
    static int done[kDevices], kmax_c[kDevices];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kDevices) return configure_recompress_once<T>(dev, svd_smem_kmax);
    std::lock_guard<std::mutex> lk(mu);
    if (!done[dev]) {
        e = configure_recompress_once<T>(dev, &kmax_c[dev]);
        if (e != cudaSuccess) return e;
        done[dev] = 1;
    }
    *svd_smem_kmax = kmax_c[dev];
    return cudaSuccess;
}

template <typename T>
static cudaError_t configure_recompress_once(int dev, int *svd_smem_kmax) {
    // the Jacobi matrices live in shared memory when they fit (k <= 119 in FP64,
    // 168 in FP32, with 227 KB per CTA)
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    e = configure_svd_smem<T>(optin, svd_smem_kmax);
    if (e != cudaSuccess) return e;
    e = set_apply_smem<T, T>();
    if (e == cudaSuccess) e = set_apply_smem<T, float>();
    if (e == cudaSuccess && sizeof(T) == sizeof(double)) e = configure_rebuild_tc();
    if (e == cudaSuccess && sizeof(T) == sizeof(double)) e = configure_qr_tc();
    if (e == cudaSuccess && sizeof(T) == sizeof(double)) e = configure_stack_tc();
    if (e != cudaSuccess) return e;
    return cudaSuccess;
}

int bucket_edge(int k, int width) {
    static const int fine[] = {8, 16, 24, 32, 40, 48, 56, 64, 80, 96, 112, 128,
                               160, 192, 224, 256, 320, 384, 448, 512};
    static const int coarse[] = {16, 32, 48, 64, 96, 128, 192, 256, 384, 512};
    if (width >= 16) {
        for (int e : coarse)
            if (k <= e) return e;
    } else {
        for (int e : fine)
            if (k <= e) return e;
    }
    return kMaxK;
}

template <typename T>
cudaError_t launch_recompress(const Desc *d_desc, int n, T *ws, int *d_rank, int *d_status,
                              int *d_info, const LaunchShape &shape, cudaStream_t s,
                              unsigned phases) {
    if (n <= 0) return cudaSuccess;
    const int maxM = shape.maxM;
    if (shape.maxK > kMaxK || maxM > 32 * kMaxRowsPerLane) return cudaErrorInvalidValue;
    const int rpl = (maxM + 31) / 32;
    const bool mixed = shape.mixed && sizeof(T) == sizeof(double);
    if (phases & kPhaseStack) {
        if (mixed) {
            launch_stack<T, float>(d_desc, n, ws, false, shape.updates, maxM, s);
        } else {
            const bool tcs = sizeof(T) == sizeof(double) && shape.tc_stack;
            launch_stack<T, T>(d_desc, n, ws, tcs, shape.updates, maxM, s);
            if (tcs) launch_stack_tc(d_desc, n, (double *)ws, d_status, s);
        }
    }
    if (phases & kPhaseQR) {
        const int qw = shape.qr_warps;
        if (sizeof(T) == sizeof(double) && shape.tc_qr && shape.nbuckets > 0) {
            qr_plan(shape, n, [&](int kind, int start, int count, int p, int cls, int groups) {
                if (count <= 0) return;
                if (kind == 2)
                    launch_qr_update_tc(d_desc + start, count, (double *)ws, p, d_status, cls, groups, s);
                else
                    launch_geqrf_all<T>(d_desc + start, count, ws, qw, rpl, p, s);
            });
        } else {
            launch_geqrf_all<T>(d_desc, n, ws, qw, rpl, -1, s);
        }
    }
    if (phases & kPhaseSVD) {
        // buckets run concurrently (largest k first) when the plan provides
        // side streams; otherwise back to back on s
        const bool forked = shape.fork != nullptr && shape.nbuckets > 1;
        if (forked) cudaEventRecord(shape.fork, s);
        for (int b = 0; b < shape.nbuckets; ++b) {
            const Bucket &bk = shape.buckets[b];
            if (bk.count <= 0) continue;
            const int K = bk.K;
            cudaStream_t sb = forked ? shape.side[b] : s;
            if (forked) cudaStreamWaitEvent(sb, shape.fork, 0);
            const int cs = K <= shape.svd_smem_kmax ? svd_spread<T>(K, shape.svd_lanes, shape.updates) : 1;
            if (cs > 1) {
                const cudaError_t e =
                    launch_svd_spread<T>(d_desc + bk.start, bk.count, ws, d_rank, d_status, d_info, K, cs, sb);
                if (e != cudaSuccess) return e;
            } else if (K <= shape.svd_smem_kmax) {
                launch_svd_smem<T>(d_desc + bk.start, bk.count, ws, d_rank, d_status, d_info, K,
                                   svd_smem_lanes<T>(K, shape.svd_lanes, shape.updates), sb);
            } else {
                const cudaError_t e = launch_svd_cluster<T>(d_desc + bk.start, bk.count, ws, d_rank, d_status,
                                                            d_info, K, shape.big_updates, sb);
                if (e != cudaSuccess) return e;
            }
            if (forked) {
                cudaEventRecord(shape.join[b], sb);
                cudaStreamWaitEvent(s, shape.join[b], 0);
            }
        }
    }
    if (phases & kPhaseApply) {
        const int ncols = shape.maxR > 0 ? std::min(shape.maxR, shape.maxK) : shape.maxK;
        if (mixed) {
            launch_apply_all<T, float>(d_desc, n, ws, d_rank, d_status, ncols, rpl, s);
        } else if (sizeof(T) == sizeof(double) && shape.tc_rebuild && shape.nbuckets > 0) {
            // descriptors are sorted by decreasing k: the buckets above
            // kTcMaxK take the DFMA kernel, the rest one tensor-core launch
            // per padded-k class
            int b = 0;
            while (b < shape.nbuckets) {
                const int cls = tc_rebuild_class(shape.buckets[b].K);
                const int start = shape.buckets[b].start;
                int count = 0;
                while (b < shape.nbuckets && tc_rebuild_class(shape.buckets[b].K) == cls)
                    count += shape.buckets[b++].count;
                if (count <= 0) continue;
                if (cls == 0)
                    launch_apply_all<T, T>(d_desc + start, count, ws, d_rank, d_status, ncols,
                                           rpl, s);
                else
                    launch_rebuild_tc(d_desc + start, count, (const double *)ws, d_rank,
                                      d_status, cls, s);
            }
        } else {
            launch_apply_all<T, T>(d_desc, n, ws, d_rank, d_status, ncols, rpl, s);
        }
    }
    return cudaGetLastError();
}

int rebuild_launches(const LaunchShape &shape, bool fp64) {
    if (!fp64 || shape.mixed || !shape.tc_rebuild || shape.nbuckets <= 0) return 1;
    int launches = 0, b = 0;
    while (b < shape.nbuckets) {
        const int cls = tc_rebuild_class(shape.buckets[b].K);
        int count = 0;
        while (b < shape.nbuckets && tc_rebuild_class(shape.buckets[b].K) == cls)
            count += shape.buckets[b++].count;
        launches += count > 0;
    }
    return launches;
}

// Rebuild of updates that ended with HCORE_GPU_S_STORAGE: their U_r and
// V_r S_r are still in the workspace, so only the rebuild phase runs again,
// over descriptors that point at the new output storage.
// cap[q] > 0 keeps the leading cap[q] singular triplets only (the fixed-rank
// truncation of HCORE_dgemm's rk argument, applied after the fact).
__global__ void storage_to_ok_kernel(const int *__restrict__ idx, const int *__restrict__ cap,
                                     int n, int *__restrict__ status, int *__restrict__ rank) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n || status[idx[q]] != HCORE_GPU_S_STORAGE) return;
    status[idx[q]] = HCORE_GPU_S_OK;
    if (cap && cap[q] > 0 && rank[idx[q]] > cap[q]) rank[idx[q]] = cap[q];
}

template <typename T>
cudaError_t launch_rebuild(const Desc *d_desc, const int *d_idx, const int *d_cap, int n, T *ws,
                           int *d_rank, int *d_status, int maxM, int maxK, bool mixed,
                           bool tc_rebuild, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (maxK > kMaxK || maxM > 32 * kMaxRowsPerLane) return cudaErrorInvalidValue;
    storage_to_ok_kernel<<<(n + 255) / 256, 256, 0, s>>>(d_idx, d_cap, n, d_status, d_rank);
    const int rpl = (maxM + 31) / 32;
    if (mixed && sizeof(T) == sizeof(double))
        launch_apply_all<T, float>(d_desc, n, ws, d_rank, d_status, maxK, rpl, s);
    else if (sizeof(T) == sizeof(double) && tc_rebuild && tc_rebuild_class(maxK) > 0)
        launch_rebuild_tc(d_desc, n, (const double *)ws, d_rank, d_status,
                          tc_rebuild_class(maxK), s);
    else
        launch_apply_all<T, T>(d_desc, n, ws, d_rank, d_status, maxK, rpl, s);
    return cudaGetLastError();
}
template cudaError_t launch_rebuild<double>(const Desc *, const int *, const int *, int, double *,
                                            int *, int *, int, int, bool, bool, cudaStream_t);
template cudaError_t launch_rebuild<float>(const Desc *, const int *, const int *, int, float *,
                                           int *, int *, int, int, bool, bool, cudaStream_t);

template cudaError_t configure_recompress<double>(int, int *);
template cudaError_t configure_recompress<float>(int, int *);
template cudaError_t launch_recompress<double>(const Desc *, int, double *, int *, int *, int *,
                                               const LaunchShape &, cudaStream_t, unsigned);
template cudaError_t launch_recompress<float>(const Desc *, int, float *, int *, int *, int *,
                                              const LaunchShape &, cudaStream_t, unsigned);

}  // namespace hc
