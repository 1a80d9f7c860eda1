// hcore-gb300 — native complex (FP64) low-rank recompression kernels.
//
// The complex update of HCORE_zgemm (src/compute/hcore_zgemm.c:663-976):
// C <- beta*C + alpha*A*B^T with X = XU*XV^T (plain transposes), then
// recompression by QR of [beta*CU | alpha*AU] and of [CV | BU*(AV^T BV)^T]
// (zgeqrf, :115), the SVD of T = R_A R_B^T (zgesvd, :327), truncation at the
// first sigma_i < acc, and the rebuild CU = Q_A [U_r; 0], CV = Q_B [conj(W_r)
// S_r; 0] (zunmqr, :483), where T = U S W^H.  (C = Q_A T Q_B^T, so the plain
// transpose puts conj(W) next to Q_B.)  Four phases, one grid each, as the
// real kernels (hc_kernels.cu):
//
//   zstack kernels  UA = [beta CU | alpha AU], F = AV^T BV, G = BU F^T, VB = [CV | G]
//   zgeqrf_kernel   Householder QR of UA and VB, rows over a cluster (zlarfg conventions: beta real,
//                   tau complex, H = I - tau v v^H, Q^H applied to the trailing columns)
//   zgesvd_kernel   T = R_A R_B^T, QR with column pivoting T P = Q R (deflated
//                   as the real kernel's), one-sided Jacobi on B = R^H with
//                   real column scales, rank rule;
//                   U_r = Q V_J, conj(W_r S_r) = conj(P (rotated B))
//   zapply_kernel   CU = Q_A [U_r; 0], CV = Q_B [conj(W_r S_r); 0]
//
// Complex arithmetic costs four real multiply-adds per product, so this is
// half the FP64 work of the order-2M real embedding, and a rank sum of 64
// keeps both Jacobi matrices in shared memory (the embedding's 128 does not).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "hc_scalar.cuh"
#include "hc_zinternal.h"

namespace hc {

__device__ __forceinline__ zd zmk(double re, double im) { return zd{re, im}; }
__device__ __forceinline__ zd zadd(zd a, zd b) { return zd{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ zd zsub(zd a, zd b) { return zd{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ zd zmul(zd a, zd b) {
    return zd{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
// conj(a) * b
__device__ __forceinline__ zd zcmul(zd a, zd b) {
    return zd{a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re};
}
__device__ __forceinline__ zd zconj(zd a) { return zd{a.re, -a.im}; }
__device__ __forceinline__ zd zscal(double s, zd a) { return zd{s * a.re, s * a.im}; }
__device__ __forceinline__ double zabs2(zd a) { return a.re * a.re + a.im * a.im; }
// acc + a * b
__device__ __forceinline__ zd zfma(zd a, zd b, zd acc) {
    return zd{fma(a.re, b.re, fma(-a.im, b.im, acc.re)), fma(a.re, b.im, fma(a.im, b.re, acc.im))};
}
// acc + conj(a) * b
__device__ __forceinline__ zd zcfma(zd a, zd b, zd acc) {
    return zd{fma(a.re, b.re, fma(a.im, b.im, acc.re)), fma(a.re, b.im, fma(-a.im, b.re, acc.im))};
}
// acc - a * b (four FMAs)
__device__ __forceinline__ zd zfms(zd a, zd b, zd acc) {
    return zd{fma(-a.re, b.re, fma(a.im, b.im, acc.re)), fma(-a.re, b.im, fma(-a.im, b.re, acc.im))};
}
// 1 / a
__device__ __forceinline__ zd zinv(zd a) {
    const double d = 1.0 / zabs2(a);
    return zd{a.re * d, -a.im * d};
}
__device__ __forceinline__ double zwarp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ zd zwarp_sum(zd v) { return zd{zwarp_sum(v.re), zwarp_sum(v.im)}; }
// ---------------------------------------------------------------------------
// phase 1: stack (hcore_zgemm.c:79-225 in complex arithmetic)
// ---------------------------------------------------------------------------
// Two launches: F = AV^T BV, a warp for one column of F and a group of its rows
// (the column of BV read once for kZf columns of AV), then row blocks of UA and
// VB.  FP64 work, 4 M b (a + 1) multiply-adds an update: with one CTA per update
// the whole phase took 1.10 ms for 48 updates of order 512, ranks 16-32, 0.44 now.
constexpr int kZf = 4, kZsRows = 64;

__global__ void __launch_bounds__(256) zstack_inner_kernel(const ZDesc *__restrict__ descs, zd *__restrict__ ws) {
    const ZDesc d = descs[blockIdx.x];
    if (d.status0) return;
    const int lane = threadIdx.x & 31, M = d.M, a = d.a;
    zd *F = ws + d.ws + zlayout(M, a, d.b, d.k).F;
    for (int q = blockIdx.y * 8 + (threadIdx.x >> 5); q < d.b; q += gridDim.y * 8) {
        const zd *y = d.BV + (size_t)q * d.ldbv;
        for (int p0 = blockIdx.z * kZf; p0 < a; p0 += gridDim.z * kZf) {
            const zd *x[kZf];
            zd s[kZf];
#pragma unroll
            for (int h = 0; h < kZf; ++h) {
                x[h] = d.AV + (size_t)min(p0 + h, a - 1) * d.ldav;
                s[h] = zmk(0, 0);
            }
            for (int l = lane; l < M; l += 32) {
                const zd v = y[l];
#pragma unroll
                for (int h = 0; h < kZf; ++h) s[h] = zfma(x[h][l], v, s[h]);
            }
#pragma unroll
            for (int h = 0; h < kZf; ++h) {
                s[h] = zwarp_sum(s[h]);
                if (lane == 0 && p0 + h < a) F[(size_t)q * a + p0 + h] = s[h];
            }
        }
    }
}

__global__ void __launch_bounds__(256) zstack_outer_kernel(const ZDesc *__restrict__ descs, zd *__restrict__ ws) {
    const ZDesc d = descs[blockIdx.x];
    const int i = blockIdx.y * kZsRows + threadIdx.x % kZsRows, grp = threadIdx.x / kZsRows;
    constexpr int NG = 256 / kZsRows;
    if (d.status0 || i >= d.M) return;
    const int M = d.M, a = d.a, b = d.b, c = d.c;
    const ZLayout L = zlayout(M, a, b, d.k);
    zd *UA = ws + d.ws + L.UA, *VB = ws + d.ws + L.VB;
    const zd *F = ws + d.ws + L.F;
    for (int j = grp; j < c; j += NG) {
        UA[(size_t)j * M + i] = zmul(d.beta, d.CU[(size_t)j * d.ldcu + i]);
        VB[(size_t)j * M + i] = d.CV[(size_t)j * d.ldcv + i];
    }
    UA += (size_t)c * M;
    VB += (size_t)c * M;   // G = BU F^T (M x a) after CV
    for (int j = grp; j < a; j += NG) UA[(size_t)j * M + i] = zmul(d.alpha, d.AU[(size_t)j * d.ldau + i]);
    for (int p0 = grp * kZf; p0 < a; p0 += NG * kZf) {
        zd s[kZf];
#pragma unroll
        for (int h = 0; h < kZf; ++h) s[h] = zmk(0, 0);
        for (int q = 0; q < b; ++q) {
            const zd u = d.BU[(size_t)q * d.ldbu + i];
#pragma unroll
            for (int h = 0; h < kZf; ++h) s[h] = zfma(u, F[(size_t)q * a + min(p0 + h, a - 1)], s[h]);
        }
#pragma unroll
        for (int h = 0; h < kZf; ++h)
            if (p0 + h < a) VB[(size_t)(p0 + h) * M + i] = s[h];
    }
}

// ---------------------------------------------------------------------------
// phase 2: Householder QR, a cluster of CTAs per (update, side)
// ---------------------------------------------------------------------------
// zlarfg on (alpha, ||x||^2): beta = -sign(Re alpha) sqrt(|alpha|^2 + ||x||^2),
// tau = (beta - alpha) / beta, x scaled by 1 / (alpha - beta); tau = 0 when
// x = 0 and alpha is real
__device__ __forceinline__ void zlarfg(zd alpha, double xn2, double &beta, zd &tau, zd &scal) {
    if (xn2 == 0.0 && alpha.im == 0.0) {
        beta = alpha.re;
        tau = zmk(0, 0);
        scal = zmk(1, 0);
        return;
    }
    const double n2 = zabs2(alpha) + xn2;
    if (n2 > 1e-280 && n2 < 1e280) {   // the short square root and reciprocal (hc_scalar.cuh)
        const double rs = inv_sqrt(n2);
        double nb = n2 * rs;
        nb = fma(fma(-nb, nb, n2) * 0.5, rs, nb);
        beta = -copysign(nb, alpha.re);
        const double ib = -copysign(rs, alpha.re), dr = alpha.re - beta;
        tau = zmk(fma(fabs(alpha.re), rs, 1.0), -alpha.im * ib);
        const double id = inv(fma(dr, dr, alpha.im * alpha.im));
        scal = zmk(dr * id, -alpha.im * id);
        return;
    }
    beta = -copysign(sqrt(n2), alpha.re);
    tau = zmk((beta - alpha.re) / beta, -alpha.im / beta);
    scal = zinv(zmk(alpha.re - beta, alpha.im));
}

// The rows are split over the CTAs of a cluster (R each, a multiple of 32), which
// keep them in shared memory from the first column to the last.  A step has one
// exchange: every CTA sends its part of x^H y for x, the rows below j of column j
// (not yet scaled), and every remaining column y, and the owner of row j that row,
// to all CTAs; then each of them forms the reflector and its coefficients and
// updates its rows.  Bound by FP64 issue (8 k^2 M / 2 multiply-adds a side), which
// one SM per side made 2.95 ms for 48 updates of order 512, ranks 16-32; 1.71 now.
// A warp takes four columns at a time, so that x is read once for them and their
// eight sums share the shuffles (9 additions instead of 40).
constexpr int kZqThreads = 256, kZqMaxCluster = 8;

// shared memory of a CTA: slab k x R | partial sums 2 x 8 x k | row j 2 x k |
// coefficients k | scales k | diagonal k
__host__ __device__ inline size_t zqr_smem_bytes(int K, int R) {
    return ((size_t)K * R + (size_t)(2 * kZqMaxCluster + 5) * K) * sizeof(zd);
}

__device__ __forceinline__ void zq_send(zd *local, int cta, int word, double v) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(local) + 8u * word), "r"(cta));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

__global__ void __launch_bounds__(kZqThreads) zgeqrf_kernel(const ZDesc *__restrict__ descs, zd *__restrict__ ws,
                                                            int cs, int R, int K) {
    extern __shared__ __align__(16) unsigned char zsm[];
    const ZDesc d = descs[blockIdx.x / cs];
    if (d.status0) return;   // (the whole cluster)
    const int M = d.M, k = d.k, side = blockIdx.y, cta = blockIdx.x % cs, r0 = cta * R;
    const ZLayout L = zlayout(M, d.a, d.b, k);
    zd *A = ws + d.ws + (side ? L.VB : L.UA);
    zd *tau = ws + d.ws + (side ? L.tauB : L.tauA);
    zd *Y = reinterpret_cast<zd *>(zsm);                 // column c, row i: Y[c R + i]
    zd *part = Y + (size_t)K * R;                        // [parity][source CTA][column]
    zd *rowj = part + (size_t)2 * kZqMaxCluster * K;     // [parity][column]
    zd *coef = rowj + 2 * (size_t)K, *scale = coef + K, *diag = scale + K;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nr = R / 32;
    for (int c = warp; c < k; c += kZqThreads / 32)
        for (int i = lane; i < R; i += 32) Y[(size_t)c * R + i] = r0 + i < M ? A[(size_t)c * M + r0 + i] : zmk(0, 0);
    cluster_sync();   // (every CTA has started before the first remote store)
    for (int j = 0; j < k; ++j) {
        const int par = j & 1, jl = j - r0;   // row j here if 0 <= jl < R
        const bool owner = jl >= 0 && jl < R;
        const int t0 = max(0, jl + 1) >> 5;   // 32-row pieces above are done
        const zd *x = Y + (size_t)j * R;
        zd *pt = part + (size_t)(par * kZqMaxCluster + cta) * K, *rj = rowj + par * K;
        for (int g = j + 4 * warp; g < k; g += kZqThreads / 8) {
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            const zd *y[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) y[h] = Y + (size_t)min(g + h, k - 1) * R;
            for (int t = t0; t < nr; ++t) {
                const int i = lane + 32 * t;
                const zd xi = i > jl ? x[i] : zmk(0, 0);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const zd s = zcfma(xi, y[h][i], zmk(v[2 * h], v[2 * h + 1]));
                    v[2 * h] = s.re;
                    v[2 * h + 1] = s.im;
                }
            }
            // lane l comes to hold sum l >> 2
#pragma unroll
            for (int n = 4, o = 16; n >= 1; n /= 2, o /= 2) {
                const bool up = lane & o;
#pragma unroll
                for (int e = 0; e < n; ++e) {
                    const double keep = up ? v[e + n] : v[e], send = up ? v[e] : v[e + n];
                    v[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            const int c = g + (lane >> 3);
            if (c < k)
                for (int to = lane & 3; to < cs; to += 4) zq_send(pt + c, to, (lane >> 2) & 1, v[0]);
        }
        if (owner)
            for (int e = tid; e < (k - j) * cs; e += kZqThreads) {
                const int c = j + e / cs, to = e % cs;
                const zd y = Y[(size_t)c * R + jl];
                zq_send(rj + c, to, 0, y.re);
                zq_send(rj + c, to, 1, y.im);
            }
        cluster_sync();
        // two lanes a column (real and imaginary part); every warp with columns forms
        // the reflector itself
        const double *ps = reinterpret_cast<const double *>(part + (size_t)par * kZqMaxCluster * K);
        for (int c0 = j + 16 * warp; c0 < k; c0 += kZqThreads / 2) {
            double ss = lane < cs ? ps[((size_t)lane * K + j) * 2] : 0.0;
#pragma unroll
            for (int o = kZqMaxCluster / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            ss = __shfl_sync(0xffffffffu, ss, 0);
            const int c = min(c0 + (lane >> 1), k - 1), im = lane & 1;
            double w = 0;
            for (int q = 0; q < cs; ++q) w += ps[((size_t)q * K + c) * 2 + im];
            const double ow = __shfl_xor_sync(0xffffffffu, w, 1);
            double beta;
            zd tj, scal;
            zlarfg(rj[j], ss, beta, tj, scal);
            if (im == 0 && c0 + (lane >> 1) < k) {
                if (c == j) {
                    scale[j] = scal;
                    diag[j] = zmk(beta, 0);
                    if (cta == 0) tau[j] = tj;
                } else {
                    // conj(tau) v^H y, v = (1, scal x); then y -= that times v
                    const zd s = zmul(zconj(tj), zadd(rj[c], zcmul(scal, zmk(w, ow))));
                    coef[c] = zmul(s, scal);
                    if (owner) Y[(size_t)c * R + jl] = zsub(rj[c], s);
                }
            }
        }
        __syncthreads();
        for (int g = j + 1 + 4 * warp; g < k; g += kZqThreads / 8) {
            zd *y[4], s[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                y[h] = Y + (size_t)min(g + h, k - 1) * R;
                s[h] = coef[min(g + h, k - 1)];
            }
            for (int t = t0; t < nr; ++t) {
                const int i = lane + 32 * t;
                if (i <= jl) continue;
                const zd xi = x[i];
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    if (g + h < k) y[h][i] = zfms(s[h], xi, y[h][i]);
            }
        }
        __syncthreads();
    }
    for (int c = warp; c < k; c += kZqThreads / 32) {
        const zd sc = scale[c];
        for (int i = lane; i < R && r0 + i < M; i += 32) {
            const zd y = Y[(size_t)c * R + i];
            A[(size_t)c * M + r0 + i] = r0 + i > c ? zmul(y, sc) : (r0 + i == c ? diag[c] : y);
        }
    }
}

// ---------------------------------------------------------------------------
// phase 3: SVD of T = R_A R_B^T, both Jacobi matrices in shared memory
// ---------------------------------------------------------------------------
// Written as the real kernel (hc_svd.cu): the same pivoted QR, deflation, tournament
// of column pairs, FP32 tangents and short reciprocals.  Bound by the FP64 FMAs of
// the rotations' rows (16 a pair of rows and matrix column, four times the real
// kernel's), so few updates take a cluster of CTAs each (CL), which share a round's
// pairs and pass columns on as there.
//
// Rotations: column j is sqrt(w_j) x_j in B = R^H and in V_J, w_j real (a common
// phase of a column of both cancels in U_r conj(W_r S_r)^T, so none is kept).  With
// s = x_p^H x_q, m = |a_pq| = sqrt(w_p w_q) |s| and t the real Jacobi tangent of
// (a_pp, a_qq, m): x_p -= (t / m) w_q conj(s) x_q, x_q += (t / m) w_p s x_p, w_p and
// w_q divided by 1 + t^2: no square root but 1 / m, no complex scale.  (A pair whose
// |a_pq|^2 is subnormal, |a_pq| < 2^-511 of T's largest entry, counts as orthogonal.)
// SVD phase of 48 updates of order 512, ranks 16-32 (k 32-64): 4.87 ms with one CTA
// an update, four lanes a pair, complex scales, a thread per column in the QR and in
// U_r; 2.77 now.
constexpr int kZvThreads = 384, kZvRows = 3;   // (k <= 96)

// sum over a group of G lanes: real and imaginary part take half of the lanes each
template <int G>
__device__ __forceinline__ zd zgroup_add(zd v, int lig) {
    const bool up = lig & (G / 2);
    double r = up ? v.im : v.re;
    r += __shfl_xor_sync(0xffffffffu, up ? v.re : v.im, G / 2);
#pragma unroll
    for (int o = G / 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    const double other = __shfl_xor_sync(0xffffffffu, r, G / 2);
    return up ? zmk(other, r) : zmk(r, other);
}
// sum of conj(x_i) y_i, start <= i < k, by a group of G lanes
template <int G>
__device__ __forceinline__ zd zgroup_dot(bool act, const zd *x, const zd *y, int start, int k, int lig) {
    zd v = zmk(0, 0);
    if (act)
        for (int i = start + ((lig - start) & (G - 1)); i < k; i += G) v = zcfma(x[i], y[i], v);
    return zgroup_add<G>(v, lig);
}
// sum of |x_i|^2, start <= i < k, by a group of G lanes
template <int G>
__device__ __forceinline__ double zgroup_norm(bool act, const zd *x, int start, int k, int lig) {
    double v = 0, w = 0;
    if (act)
        for (int i = start + ((lig - start) & (G - 1)); i < k; i += G) {
            v = fma(x[i].re, x[i].re, v);
            w = fma(x[i].im, x[i].im, w);
        }
    v += w;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// is the pair to be rotated, m2 > tol^2 app aqq, and above the stopping level (big)?
__device__ __forceinline__ bool zpair_test(double app, double aqq, double m2, float tol, bool &big) {
    float mp, mq, mm;
    int ep, eq, em;
    split(app, mp, ep);
    split(aqq, mq, eq);
    split(m2, mm, em);
    const int ex = em - ep - eq + 1023;
    if (em == 0 || ex < -110) return false;
    const float x = mm * __int_as_float((min(ex, 60) + 127) << 23), y = mp * mq;
    big = x > tol * y;
    return x > tol * tol * y;
}
__device__ __forceinline__ long long zkey(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ bool zbelow_pow2(double x, double y, int n) {   // x < y 2^-n, y >= 0
    return __double2hiint(x) < __double2hiint(y) - (n << 20);
}

template <int G, bool CL>
__global__ void __launch_bounds__(kZvThreads, 1)
    zgesvd_kernel(const ZDesc *__restrict__ descs, zd *__restrict__ ws, int *__restrict__ rank,
                  int *__restrict__ status, int maxK, int cs) {
    extern __shared__ __align__(16) unsigned char zsm[];
    __shared__ double s_wmax[kZvThreads / 32];
    __shared__ zd s_vj;
    __shared__ int s_big[2][8], s_rank;
    __shared__ short s_own[128];
    const ZDesc d = descs[CL ? blockIdx.x / cs : blockIdx.x];
    const int cr = CL ? blockIdx.x % cs : 0;
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
    if (d.status0) {
        if (tid == 0 && cr == 0) {
            status[d.idx] = d.status0;
            rank[d.idx] = 0;
        }
        return;
    }
    const int M = d.M, k = d.k, ld = zsvd_ld(k);
    const ZLayout L = zlayout(M, d.a, d.b, k);
    zd *base = ws + d.ws;
    const zd *UA = base + L.UA, *VB = base + L.VB;
    const size_t mat = (size_t)maxK * zsvd_ld(maxK);
    zd *A = reinterpret_cast<zd *>(zsm);   // R_A, T, its QR, then V_J
    zd *B = A + mat;                       // R_B, then R^H; at the end Q's reflectors
    zd *s_tau = B + mat, *s_rd = s_tau + (maxK + 1);   // reflector j's conj(tau) |scale|^2, R's diagonal
    double *X0 = reinterpret_cast<double *>(s_rd + (maxK + 1)), *X1 = X0 + (maxK + 1);
    double *s_w = X1 + (maxK + 1);
    short *s_perm = reinterpret_cast<short *>(s_w + (maxK + 1)), *s_pcol = s_perm + (maxK + 1);
    zd *Yg = base + L.Y;   // reflectors of Q (k x k, ld k)
    const int grp = tid / G, lig = tid & (G - 1), ngrp = nthr / G;
    constexpr int D = G < 8 ? G : 8;   // lanes per column in the QR
    const int qgrp = tid / D, qlig = tid & (D - 1), nqgrp = nthr / D;

    // ---- T = triu(R_A) triu(R_B)^T: a warp per row, the row of T replaces the row
    // of R_A that only it reads
    for (int l = warp; l < k; l += nw)
        for (int i = lane; i < k; i += 32) {
            A[(size_t)l * ld + i] = i <= l ? UA[(size_t)l * M + i] : zmk(0, 0);
            B[(size_t)l * ld + i] = i <= l ? VB[(size_t)l * M + i] : zmk(0, 0);
        }
    __syncthreads();
    double amax = 0;
    bool bad = false;
    for (int i = warp; i < k; i += nw) {
        zd acc[kZvRows];
#pragma unroll
        for (int c = 0; c < kZvRows; ++c) {
            acc[c] = zmk(0, 0);
            if (32 * c < k) {
                const zd *b = B + min(lane + 32 * c, k - 1);
                for (int l = max(i, 32 * c); l < k; ++l)
                    acc[c] = zfma(A[(size_t)l * ld + i], b[(size_t)l * ld], acc[c]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kZvRows; ++c) {
            const int j = lane + 32 * c;
            if (j < k) {
                A[(size_t)j * ld + i] = acc[c];
                amax = max(amax, max(fabs(acc[c].re), fabs(acc[c].im)));
                bad = bad || !isfinite(acc[c].re) || !isfinite(acc[c].im);
            }
        }
    }
    amax = warp_max(amax);
    if (lane == 0) s_wmax[warp] = amax;
    if (__syncthreads_or(bad)) {   // a NaN or infinity: the update is not written
        if (cr != 0) return;
        for (int t = tid; t < k; t += nthr) base[L.sig + t] = zmk(NAN, 0);
        if (tid == 0) {
            rank[d.idx] = d.rk != 0 && d.rk < k ? d.rk : k;
            status[d.idx] = HCORE_GPU_S_NOCONV;
        }
        return;
    }
    amax = 0;
    for (int w = 0; w < nw; ++w) amax = max(amax, s_wmax[w]);
    const int sexp = amax > 0 ? binary_exponent(amax) : 0;
    for (int c0 = 0; c0 < k; c0 += nqgrp) {
        const int c = c0 + qgrp;
        zd *ac = A + (size_t)c * ld;
        if (c < k && sexp != 0)
            for (int i = qlig; i < k; i += D) ac[i] = zmk(mul_exp2(ac[i].re, -sexp), mul_exp2(ac[i].im, -sexp));
        const double s = zgroup_norm<D>(c < k, ac, 0, k, qlig);
        if (c < k && qlig == 0) {
            X0[c] = s;    // norms of rows j.. of column c, squared; -1: pivoted already
            s_w[c] = s;   // the same at the last exact computation
        }
    }
    __syncthreads();
    double f2 = 0;
    for (int c = lane; c < k; c += 32) f2 += X0[c];
    const double defl2 = deflation_bound2(warp_sum(f2), k, M, d.rk, 0, d.acc, sexp);

    // ---- QR with column pivoting, T P = Q R (columns stay in place) -----------------
    int kk = k;
    for (int j = 0; j < k; ++j) {
        const double *nr = (j & 1) ? X1 : X0;
        double *nr2 = (j & 1) ? X0 : X1;
        long long best = zkey(-1.0);
        int pv = 0;
        for (int c = lane; c < k; c += 32) {
            const long long x = zkey(nr[c]);
            if (x > best) {
                best = x;
                pv = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, pv, o);
            if (ob > best || (ob == best && oi < pv)) {
                best = ob;
                pv = oi;
            }
        }
        if (j >= 1 && defl2 >= 0.0 && best <= zkey(defl2)) {
            double tail = 0;
            for (int c = lane; c < k; c += 32) tail += max(nr[c], 0.0);
            if (warp_sum(tail) <= defl2) {
                kk = j;
                break;
            }
        }
        // reflector of column pv, rows j.., unscaled: v = (alpha - beta, x), H^H y =
        // y - g (v^H y) v, g = 1 / (beta (beta - alpha)), by warp 0 while the others
        // form x^H y for the remaining columns y
        const zd *ap = A + (size_t)pv * ld;
        if (warp == 0) {
            const zd alpha = ap[j];
            double ss = 0;
            for (int i = j + 1 + lane; i < k; i += 32) ss += zabs2(ap[i]);
            ss = warp_sum(ss);
            zd beta = alpha, vj = zmk(0, 0), g = zmk(0, 0);
            if (ss > DBL_MIN / DBL_EPSILON) {
                const double n2 = zabs2(alpha) + ss, rs = inv_sqrt(n2);
                double nb = n2 * rs;
                nb = fma(fma(-nb, nb, n2) * 0.5, rs, nb);
                beta = zmk(-copysign(nb, alpha.re), 0);
                vj = zsub(alpha, beta);
                const double ib = -copysign(rs, alpha.re), iv = inv(zabs2(vj)) * ib;
                g = zmk(-vj.re * iv, vj.im * iv);   // -1 / (beta vj)
            }
            if (lane == 0) {
                s_pcol[j] = (short)pv;
                s_rd[j] = beta;
                s_tau[j] = g;
                s_vj = vj;
            }
        }
        zd *dots = B;   // (free until R^H is formed)
        for (int c0 = 0; c0 < k; c0 += nqgrp) {
            const int c = c0 + qgrp;
            const bool act = c < k && c != pv && zkey(nr[c]) >= 0;
            const zd w = zgroup_dot<D>(act, ap, A + (size_t)c * ld, j + 1, k, qlig);
            if (act && qlig == 0) dots[c] = w;
        }
        __syncthreads();
        const zd g = s_tau[j], vj = s_vj;
        const bool none = g.re == 0.0 && g.im == 0.0;
        for (int c0 = 0; c0 < k; c0 += nqgrp) {
            const int c = c0 + qgrp;
            const double nc = c < k ? nr[c] : -1.0;
            const bool act = c < k && c != pv && zkey(nc) >= 0, upd = act && !none;
            zd *ac = A + (size_t)c * ld;
            zd acj = zmk(0, 0), s = zmk(0, 0);
            if (upd && qlig == 0) {
                acj = ac[j];
                s = zmul(g, zcfma(vj, acj, dots[c]));
            }
            s.re = __shfl_sync(0xffffffffu, s.re, lane & ~(D - 1));
            s.im = __shfl_sync(0xffffffffu, s.im, lane & ~(D - 1));
            double nn = 0;
            bool redo = false;
            if (act) {
                if (upd)
                    for (int i = j + 1 + ((qlig - (j + 1)) & (D - 1)); i < k; i += D) ac[i] = zfms(s, ap[i], ac[i]);
                if (qlig == 0) {
                    const zd r = upd ? zfms(s, vj, acj) : ac[j];
                    ac[j] = r;
                    nn = nc - zabs2(r);
                    redo = !(zkey(nn) > 0) || zbelow_pow2(nn, s_w[c], 10);
                }
            }
            if (__any_sync(0xffffffffu, redo)) {
                redo = __shfl_sync(0xffffffffu, (int)redo, lane & ~(D - 1)) != 0;
                const double q = zgroup_norm<D>(redo, ac, j + 1, k, qlig);
                if (redo && qlig == 0) {
                    nn = q;
                    s_w[c] = q;
                }
            }
            if (c < k && qlig == 0) nr2[c] = act ? nn : -1.0;
        }
        __syncthreads();
    }
    {
        // columns that the deflation left: positions kk.. in column order
        const double *nr = (kk & 1) ? X1 : X0;
        if (kk < k)
            for (int c = tid; c < k; c += nthr)
                if (zkey(nr[c]) >= 0) {
                    int pos = kk;
                    for (int q = 0; q < c; ++q) pos += zkey(nr[q]) >= 0;
                    s_pcol[pos] = (short)c;
                }
    }
    __syncthreads();
    // Q's reflectors to the workspace, B = R^H (its columns kk.. are zero), A = I
    for (int h = warp; h < k; h += nw) {
        const zd *ah = A + (size_t)s_pcol[h] * ld;
        for (int i = lane; i < k; i += 32) {
            const zd x = ah[i], rd = h < kk ? s_rd[h] : zmk(0, 0);
            if (h < kk && cr == 0) Yg[(size_t)h * k + i] = i > h ? x : (i == h ? zsub(x, rd) : zmk(0, 0));
            B[(size_t)i * ld + h] = i < kk ? (i < h ? zconj(x) : (i == h ? zconj(rd) : zmk(0, 0))) : zmk(0, 0);
        }
    }
    __syncthreads();
    for (int c = warp; c < k; c += nw)
        for (int i = lane; i < k; i += 32) A[(size_t)c * ld + i] = zmk(i == c ? 1.0 : 0.0, 0);
    double *s_nrm = X0, *s_sig = X1;
    auto column_norm = [&](int c, bool fold) {   // of column c, by its group
        double w = 1;
        zd *xj = B + (size_t)c * ld;
        if (c < kk && fold) {
            w = s_w[c];
            if (w < 1e-120) {   // fold a scale before it underflows
                const double f = sqrt(w);
                zd *vj = A + (size_t)c * ld;
                for (int i = lig; i < k; i += G) {
                    xj[i] = zscal(f, xj[i]);
                    vj[i] = zscal(f, vj[i]);
                }
                w = 1;
            }
        }
        const double s = zgroup_norm<G>(c < kk, xj, 0, k, lig);
        if (c < k && lig == 0) {
            s_nrm[c] = c < kk ? w * s : 0.0;
            s_w[c] = w;
        }
    };
    for (int c0 = 0; c0 < k; c0 += ngrp) column_norm(c0 + grp, false);
    if constexpr (CL) cluster_sync(); else __syncthreads();

    // ---- one-sided Jacobi on B, rotations accumulated in A ---------------------------
    // (columns kk.. of B are zero and take no part, V_J's rows kk.. stay zero)
    const int n = kk + (kk & 1), np = n / 2;
    const int active = CL ? max(1, min(cs, np)) : 1;
    const int pi0 = CL ? min(cr, active) * np / active : 0, pi1 = CL ? min(cr + 1, active) * np / active : np;
    const unsigned left = CL && pi0 > 0 && cr < active ? peer_delta(zsm, cr - 1) : 0;
    const unsigned right = CL && pi1 < np ? peer_delta(zsm, cr + 1) : 0;
    const float tol = (float)(k > 8 ? k : 8) * (float)DBL_EPSILON;
    bool converged = kk <= 1;
    for (int sweep = 0; sweep < kMaxSweeps && !converged; ++sweep) {
        bool big = false;   // this thread rotated a pair above sqrt(tol)
        for (int round = 0; round < n - 1; ++round) {
            for (int b0 = pi0; b0 < pi1; b0 += ngrp) {
                const int pi = b0 + grp;
                int p = round + pi, q = round - pi;
                if (p >= n - 1) p -= n - 1;
                if (q < 0) q += n - 1;
                if (pi == 0) p = n - 1;
                const bool valid = pi < pi1 && p < kk && q < kk;
                zd *xp = B + (size_t)p * ld, *xq = B + (size_t)q * ld;
                double app = 0, aqq = 0, wp = 1, wq = 1;
                if (valid) {
                    app = s_nrm[p];
                    aqq = s_nrm[q];
                    wp = s_w[p];
                    wq = s_w[q];
                }
                const zd dot = zgroup_dot<G>(valid, xp, xq, 0, k, lig);
                bool rot = false, redo_p = false, redo_q = false;
                double np_ = 0, nq_ = 0, wp2 = 1, wq2 = 1;
                if (valid) {
                    const double m2 = (wp * wq) * zabs2(dot);
                    bool bigp = false;
                    rot = zkey(app) > zkey(DBL_MIN / DBL_EPSILON) && zkey(aqq) > zkey(DBL_MIN / DBL_EPSILON) &&
                          zpair_test(app, aqq, m2, tol, bigp);
                    if (rot) {
                        big |= bigp;
                        const double rm = inv_sqrt(m2), m = m2 * rm, t = tangent(app, aqq, m), tm = t * rm;
                        const zd f1 = zscal(tm * wq, zconj(dot)), f2_ = zscal(tm * wp, dot);
                        np_ = fma(-t, m, app);
                        nq_ = fma(t, m, aqq);
                        redo_p = zbelow_pow2(np_, app, 6);
                        redo_q = zbelow_pow2(nq_, aqq, 6);
                        zd *vp = A + (size_t)p * ld, *vq = A + (size_t)q * ld;
                        int i = lig;
                        for (; i < kk; i += G) {
                            const zd a = xp[i], b = xq[i], u = vp[i], v = vq[i];
                            xp[i] = zfms(f1, b, a);
                            xq[i] = zfma(f2_, a, b);
                            vp[i] = zfms(f1, v, u);
                            vq[i] = zfma(f2_, u, v);
                        }
                        for (; i < k; i += G) {
                            const zd a = xp[i], b = xq[i];
                            xp[i] = zfms(f1, b, a);
                            xq[i] = zfma(f2_, a, b);
                        }
                        const double c2 = inv(fma(t, t, 1.0));
                        wp2 = wp * c2;
                        wq2 = wq * c2;
                    }
                }
                if (__any_sync(0xffffffffu, redo_p || redo_q)) {   // strong cancellation in a tracked norm
                    const double sp = zgroup_norm<G>(redo_p, xp, 0, k, lig);
                    const double sq = zgroup_norm<G>(redo_q, xq, 0, k, lig);
                    if (redo_p) np_ = wp2 * sp;
                    if (redo_q) nq_ = wq2 * sq;
                }
                if (rot && lig == 0) {
                    s_nrm[p] = np_;
                    s_nrm[q] = nq_;
                    s_w[p] = wp2;
                    s_w[q] = wq2;
                }
                if constexpr (CL) {
                    // the next round has p in pair pi - 1 and q in pair pi + 1
                    auto send = [&](int c, unsigned to) {
                        zd *x = B + (size_t)c * ld, *v = A + (size_t)c * ld;
                        for (int i = lig; i < k; i += G) {
                            peer_store(&x[i].re, to, x[i].re);
                            peer_store(&x[i].im, to, x[i].im);
                            if (i < kk) {
                                peer_store(&v[i].re, to, v[i].re);
                                peer_store(&v[i].im, to, v[i].im);
                            }
                        }
                        if (lig == 0) {
                            peer_store(s_nrm + c, to, s_nrm[c]);
                            peer_store(s_w + c, to, s_w[c]);
                        }
                    };
                    if (pi == pi0 && pi > 0 && p < kk) send(p, left);
                    if (pi == pi1 - 1 && pi1 < np && q < kk) send(q, right);
                    __syncwarp();
                }
            }
            if constexpr (CL) cluster_sync(); else __syncthreads();
        }
        // exact norms once per sweep (every column is back in its first pair)
        if constexpr (CL) {
            for (int b0 = pi0; b0 < pi1; b0 += ngrp) {
                const int pi = b0 + grp;
                column_norm(pi < pi1 ? (pi == 0 ? n - 1 : pi) : k, true);
                column_norm(pi < pi1 ? (pi == 0 ? 0 : n - 1 - pi) : k, true);
            }
            const int any = __syncthreads_or(big);
            if (tid < cs) peer_store(&s_big[sweep & 1][cr], peer_delta(zsm, tid), any);
            cluster_sync();
            converged = true;
            for (int t = 0; t < cs; ++t) converged = converged && !s_big[sweep & 1][t];
        } else {
            for (int c0 = 0; c0 < k; c0 += ngrp) column_norm(c0 + grp, true);
            converged = !__syncthreads_or(big);
        }
    }
    auto owner = [&](int j) {   // the CTA that holds column j
        const int pi = j == n - 1 ? 0 : (j < np ? j : n - 1 - j);
        int o = 0;
        while (o + 1 < active && (o + 1) * np / active <= pi) ++o;
        return j < kk ? o : 0;
    };
    if constexpr (CL) {
        for (int j = warp; j < kk; j += nw)
            if (owner(j) == cr && lane < cs && lane != cr) {
                const unsigned to = peer_delta(zsm, lane);
                peer_store(s_nrm + j, to, s_nrm[j]);
                peer_store(s_w + j, to, s_w[j]);
            }
        cluster_sync();
    }

    // singular values, sorted descending (ties by index, NaN last), rank rule
    bool nonfinite = false;
    for (int j = tid; j < k; j += nthr) {
        const double s = sqrt(s_nrm[j]);
        nonfinite = nonfinite || !isfinite(s);
        s_sig[j] = s == s ? s : -1.0;
    }
    if (tid == 0) s_rank = k;
    const bool finite = !__syncthreads_or(nonfinite);
    for (int j = tid; j < k; j += nthr) {
        const long long sj = zkey(s_sig[j]);
        int pos = 0;
        for (int i = 0; i < k; ++i) {
            const long long si = zkey(s_sig[i]);
            pos += (si > sj) || (si == sj && i < j);
        }
        s_perm[pos] = (short)j;
    }
    __syncthreads();
    for (int t = tid; t < k; t += nthr) {
        const double s = s_sig[s_perm[t]], v = s < 0 ? NAN : mul_exp2(s, sexp);
        if (cr == 0) base[L.sig + t] = zmk(v, 0);
        if (d.rk == 0 && t >= 1 && v < d.acc) atomicMin(&s_rank, t);
    }
    __syncthreads();
    const int r = d.rk != 0 ? (d.rk < k ? d.rk : k) : s_rank;
    int st = HCORE_GPU_S_OK;
    if (!converged || !finite) st = HCORE_GPU_S_NOCONV;
    else if (r > d.max_rank) st = HCORE_GPU_S_RANK_MAX;
    if (st == HCORE_GPU_S_OK) {
        // Vo = conj(W_r S_r), W S = P (B's columns), scaled back
        zd *Uo = base + L.Uo, *Vo = base + L.Vo;
        for (int t = warp; t < r; t += nw) {
            const int j = s_perm[t];
            if (CL && owner(j) != cr) continue;
            const double f = sqrt(s_w[j]);
            for (int i = lane; i < k; i += 32) {
                const zd w = zscal(f, B[(size_t)j * ld + i]);
                Vo[(size_t)t * k + s_pcol[i]] = zmk(mul_exp2(w.re, sexp), -mul_exp2(w.im, sexp));
            }
        }
        int nown = r;   // the columns of U_r that this CTA forms
        if constexpr (CL) {
            nown = 0;
            for (int t = 0; t < r; ++t) {
                const bool mine = owner(s_perm[t]) == cr;
                if (mine && tid == 0) s_own[nown] = (short)t;
                nown += mine;
            }
        }
        __syncthreads();
        // U_r = Q (V_J's columns), Q = H_0 ... H_{kk-1}: the reflectors come into B's
        // place, each group applies them, last to first, to its columns
        for (int h = warp; h < kk; h += nw)
            for (int i = lane; i < k; i += 32) B[(size_t)h * ld + i] = Yg[(size_t)h * k + i];
        __syncthreads();
        for (int t0 = 0; t0 < nown; t0 += ngrp) {
            const bool act = t0 + grp < nown;
            const int t = !act ? 0 : (CL ? s_own[t0 + grp] : t0 + grp);
            const int j = act ? s_perm[t] : 0;
            zd *x = A + (size_t)j * ld;   // each group owns the column of its own j
            if (act) {
                const double f = sqrt(s_w[j]);
                for (int i = lig; i < k; i += G) x[i] = zscal(f, x[i]);
            }
            for (int h = kk - 1; h >= 0; --h) {
                const zd g = s_tau[h];
                if (g.re == 0.0 && g.im == 0.0) continue;
                const zd *y = B + (size_t)h * ld;
                const zd s = zmul(zconj(g), zgroup_dot<G>(act, y, x, h, k, lig));
                if (act)
                    for (int i = h + ((lig - h) & (G - 1)); i < k; i += G) x[i] = zfms(s, y[i], x[i]);
            }
            if (act)
                for (int i = lig; i < k; i += G) Uo[(size_t)t * k + i] = x[i];
        }
    }
    if (tid == 0 && cr == 0) {
        rank[d.idx] = r;
        status[d.idx] = st;
    }
}

// ---------------------------------------------------------------------------
// phase 4: rebuild, CU = Q_A [U_r; 0] (side 0), CV = Q_B [Vo_r; 0] (side 1);
// one warp per output column, RPL complex rows per lane in registers, the
// reflectors staged through shared memory kZApplyChunk at a time
// ---------------------------------------------------------------------------
template <int RPL>
__global__ void __launch_bounds__(256, 1) zapply_kernel(const ZDesc *__restrict__ descs,
                                                        const zd *__restrict__ ws,
                                                        const int *__restrict__ rank,
                                                        const int *__restrict__ status) {
    extern __shared__ unsigned char zsm[];
    zd *sv = reinterpret_cast<zd *>(zsm);
    __shared__ zd s_tau[kZApplyChunk];
    const ZDesc d = descs[blockIdx.x];
    if (d.status0 || status[d.idx] != HCORE_GPU_S_OK) return;
    const int r = rank[d.idx];
    const int col = blockIdx.z * 8 + (threadIdx.x >> 5);
    if (blockIdx.z * 8 >= r) return;
    const int side = blockIdx.y, M = d.M, k = d.k;
    const ZLayout L = zlayout(M, d.a, d.b, k);
    const zd *base = ws + d.ws;
    const zd *Y = base + (side ? L.VB : L.UA);
    const zd *tau = base + (side ? L.tauB : L.tauA);
    const zd *X0 = base + (side ? L.Vo : L.Uo);
    zd *out = side ? d.CVo : d.CUo;
    const int ldo = d.ldco;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool active = col < r;
    constexpr int ROWS = 32 * RPL;
    zd x[RPL];
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
        const int i = lane + 32 * t;
        x[t] = (active && i < k) ? X0[(size_t)col * k + i] : zmk(0, 0);
    }
    const int nch = (k + kZApplyChunk - 1) / kZApplyChunk;
    for (int ch = nch - 1; ch >= 0; --ch) {
        const int j0 = ch * kZApplyChunk, nj = min(kZApplyChunk, k - j0);
        __syncthreads();
        for (int e = tid; e < nj * ROWS; e += 256) {
            const int c = e / ROWS, i = e % ROWS, j = j0 + c;
            zd v = zmk(0, 0);
            if (i > j && i < M) v = Y[(size_t)j * M + i];
            else if (i == j) v = zmk(1, 0);
            sv[c * ROWS + i] = v;
        }
        if (tid < nj) s_tau[tid] = tau[j0 + tid];
        __syncthreads();
        if (!active) continue;
        for (int c = nj - 1; c >= 0; --c) {
            const zd tj = s_tau[c];
            if (tj.re == 0.0 && tj.im == 0.0) continue;
            const zd *v = sv + c * ROWS;
            zd s = zmk(0, 0);
#pragma unroll
            for (int t = 0; t < RPL; ++t) s = zcfma(v[lane + 32 * t], x[t], s);
            s = zmul(tj, zwarp_sum(s));
#pragma unroll
            for (int t = 0; t < RPL; ++t) x[t] = zfms(s, v[lane + 32 * t], x[t]);
        }
    }
    if (active) {
#pragma unroll
        for (int t = 0; t < RPL; ++t) {
            const int i = lane + 32 * t;
            if (i < M) out[(size_t)col * ldo + i] = x[t];
        }
    }
}

template <int RPL>
static void launch_zapply(const ZDesc *d_desc, int n, const zd *ws, const int *d_rank,
                          const int *d_status, int maxR, cudaStream_t s) {
    const size_t smem = (size_t)kZApplyChunk * 32 * RPL * sizeof(zd);
    allow_smem(zapply_kernel<RPL>);
    zapply_kernel<RPL><<<dim3(n, 2, (maxR + 7) / 8), 256, smem, s>>>(d_desc, ws, d_rank,
                                                                      d_status);
}

// CTAs per cluster: enough that two CTAs share an SM, and more while SMs are idle
// and every CTA keeps 64 rows (48 updates of order 512, ranks 16-32: four 1.75,
// eight 1.72 ms)
static cudaError_t launch_zgeqrf(const ZDesc *d_desc, int n, zd *ws, int maxM, int maxK, int sms, int optin,
                                 cudaStream_t s) {
    auto rows = [&](int cs) { return (maxM + 32 * cs - 1) / (32 * cs) * 32; };
    int cs = 1;
    while (cs < kZqMaxCluster && (2 * (zqr_smem_bytes(maxK, rows(cs)) + 1024) > (size_t)optin ||
                                  (4 * n * cs <= 2 * sms && rows(2 * cs) >= 64)))
        cs *= 2;
    const int R = rows(cs);
    const size_t smem = zqr_smem_bytes(maxK, R);
    cudaError_t e = allow_smem(zgeqrf_kernel);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n * cs, 2);
    cfg.blockDim = dim3(kZqThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, zgeqrf_kernel, d_desc, ws, cs, R, maxK);
}

int zsvd_kmax() {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
            cudaSuccess)
        return 0;
    int kmax = 0;
    while (kmax < 256 && zsvd_smem_bytes(kmax + 1) + 1024 <= (size_t)optin) ++kmax;
    return kmax;
}

// While SMs are idle, a cluster per update of more than 12 column pairs: up to eight
// pairs a CTA (16 lanes each, a warp a sub-partition), else eight lanes a pair.  SVD
// phase, one CTA and a cluster, us: one update of k = 17 324, 337, of 64 4182, 2266;
// 20 of k 24-32 779, 655 (two CTAs); 48 of k 32-64 3422, 2870 (three); 70 3416, 2899
// (two).  Eight lanes also with more updates than SMs: 600 of k 16-32 1.44 ms, four
// lanes 1.63; 600 of k 32-64 8.07, four lanes with V_J in the workspace, so that
// three CTAs share an SM, 9.01.
static cudaError_t launch_zgesvd(const ZDesc *d_desc, int n, zd *ws, int *d_rank, int *d_status, int K, int sms,
                                 cudaStream_t s) {
    const int np = (K + 1) / 2;
    int cs = np > 12 ? std::max(1, std::min({8, (np + 7) / 8, sms / n})) : 1;
    const size_t smem = zsvd_smem_bytes(K);
    auto go = [&](auto kernel, int G, int pairs, int *fit) {
        cudaError_t e = allow_smem(kernel);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)n * cs);
        cfg.blockDim = dim3(std::max(n > sms ? 32 : 256, (pairs * G + 31) / 32 * 32));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = cs > 1 ? 1 : 0;
        if (fit) return cudaOccupancyMaxActiveClusters(fit, kernel, &cfg);
        return cudaLaunchKernelEx(&cfg, kernel, d_desc, ws, d_rank, d_status, K, cs);
    };
    for (; cs > 1; --cs) {   // all clusters at once, or smaller ones
        const int pairs = (np + cs - 1) / cs;
        int fit = 0;
        const cudaError_t e = pairs <= 8 ? go(zgesvd_kernel<16, true>, 16, pairs, &fit)
                                         : go(zgesvd_kernel<8, true>, 8, pairs, &fit);
        if (e != cudaSuccess) return e;
        if (fit < n) continue;
        return pairs <= 8 ? go(zgesvd_kernel<16, true>, 16, pairs, nullptr)
                          : go(zgesvd_kernel<8, true>, 8, pairs, nullptr);
    }
    return np <= 8 && n <= sms ? go(zgesvd_kernel<16, false>, 16, np, nullptr)
                               : go(zgesvd_kernel<8, false>, 8, np, nullptr);
}

cudaError_t launch_zrecompress(const ZDesc *d_desc, int n, zd *ws, int *d_rank, int *d_status,
                               int maxM, int maxK, int maxB, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int rpl = (maxM + 31) / 32;
    if (rpl > 32 || maxK > zsvd_kmax()) return cudaErrorInvalidValue;
    int dev = 0, sms = 1, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // F: the z axis splits a column's rows while the grid is below two CTAs an SM
    const int fy = std::min((maxB + 7) / 8, 65535);
    const int fz = (int)std::max(1LL, std::min<long long>((maxK + kZf - 1) / kZf, 2 * sms / std::max(1LL, (long long)n * fy)));
    zstack_inner_kernel<<<dim3(n, fy, fz), 256, 0, s>>>(d_desc, ws);
    zstack_outer_kernel<<<dim3(n, (maxM + kZsRows - 1) / kZsRows), 256, 0, s>>>(d_desc, ws);
    if (cudaError_t e = launch_zgeqrf(d_desc, n, ws, maxM, maxK, sms, optin, s)) return e;
    if (cudaError_t e = launch_zgesvd(d_desc, n, ws, d_rank, d_status, maxK, sms, s)) return e;
    if (rpl <= 4) launch_zapply<4>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else if (rpl <= 8) launch_zapply<8>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else if (rpl <= 16) launch_zapply<16>(d_desc, n, ws, d_rank, d_status, maxK, s);
    else launch_zapply<32>(d_desc, n, ws, d_rank, d_status, maxK, s);
    return cudaGetLastError();
}

}  // namespace hc
