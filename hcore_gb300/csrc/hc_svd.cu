// hcore-gb300 — the core SVD of an update: T = R_A R_B^T (k x k), QR with column
// pivoting, one-sided Jacobi, rank rule, U_r and V_r S_r (reference step:
// src/compute/hcore_dgemm.c:296-503, __svd).  Two kernels: svd_smem_kernel, one
// CTA, both k x k matrices in its shared memory (k <= 119 in FP64, 168 in FP32),
// and svd_cluster_kernel for larger k.
//
// Method (QR-preconditioned one-sided Jacobi, Drmac and Veselic 2008): T P = Q R
// with column pivoting, then one-sided Jacobi on R^T, whose columns are graded
// by the pivoting, so the sweeps are few.  With R^T V_J = U' S (U' orthonormal),
// T = (Q V_J) S (P U')^T, hence U_T = Q V_J (V_J accumulated by the rotations)
// and V_T S = P (R^T V_J).  The rotations are scaled ("fast"): column j is d_j
// x_j in both R^T and V_J, so a rotation costs two FMAs per row and matrix.
// Squared norms are tracked (exact in exact arithmetic), recomputed on strong
// cancellation and after every sweep.  A pair is rotated when a_pq^2 > tol^2 a_pp
// a_qq, tol = k eps (LAPACK dgesvj's criterion); the sweeps stop after one whose
// largest relative off-diagonal was at most sqrt(tol): cyclic Jacobi converges
// quadratically, so the next would only rotate by angles near tol.
//
// Deflation (FP64 updates ranked by accuracy): the QR stops at the first step j
// whose trailing block R22 = R(j:k, j:k) has ||R22||_F <= delta, and the Jacobi
// runs on the first j rows of R only.  Dropping R22 moves every singular value
// by at most delta (Weyl), with delta = min(1e-13 thr, 1e-16 ||T||_F), thr the
// truncation threshold (acc, or for the relative rule its lower bound acc
// ||T||_F / sqrt(k)): a rank decision can change only for a singular value within
// 1e-13 of the threshold, relative, and every singular value stays within a few
// eps sigma_max of the full one (the accuracy of dgesvd's small singular
// values).  The dropped directions come out with singular value 0.  (The core
// of a compressed tile's range has the compressor's larger budget, kCoreShare.)
//
// Range safety (as LAPACK's dgesvd scales the matrix first): T is scaled by 2^-e
// so that its largest entry lies in [1, 2) (exact; the singular values and V S
// are scaled back by 2^e), and a column whose squared norm is below safmin is
// negligible (< 2^-485 relative in FP64, 2^-51 in FP32) and not rotated.  In FP32 a
// pair whose inner product is below 2^-75 counts as orthogonal too, its square being
// out of range: columns of norms 2^-38 or so, far below the 2^-24 of T's rounding.  A
// non-finite T or singular value marks the update NOCONV.
//
// svd_smem_kernel is written for latency, because a CTA's serial chain of Jacobi
// rounds and QR steps is what the SVD phase waits for.  One FP64 warp
// instruction holds a sub-partition's FP64 pipe for about 64 cycles and a
// dependent one cannot start earlier, so what counts is the number of FP64
// warp instructions in a round's chain, not the bytes or the lanes:
//   * a rotation's tangent is computed in FP32 from the leading bits of the
//     three FP64 inner products (integer instructions extract them).  The
//     tangent only has to bring the pair's inner product down by 2^-20 or so
//     (the sweeps converge quadratically, and the last sweep starts below
//     sqrt(tol)); what has to hold in FP64 is c^2 + s^2 = 1 for the tangent
//     used, and that is done in FP64;
//   * square roots and reciprocals in FP64 take an FP32 seed and one
//     third-order Householder iteration (A. S. Householder, "The Numerical
//     Treatment of a Single Nonlinear Equation", 1970), 5 and 3 instructions;
//   * the scales keep their reciprocals, so no rotation divides;
//   * comparisons of non-negative values run on the integer pipe;
//   * the pivoted QR moves no column (a permutation instead), every warp
//     finds the pivot itself, and the inner products with the remaining
//     columns run beside the reflector's parameters (which only warp 0 forms:
//     every warp doing so took 1453 us, not 1403, below); up to eight lanes
//     share a column there, G lanes in U_r = Q V_J as in the Jacobi.
// SVD phase, with the kernel before (its parameters about 65 FP64 instructions a
// round, two and, alone, four lanes per pair) and now, one GB300,
// us: one update of k = 64 2388 -> 1403; 16 of k 8-24 485 -> 249; 384 of k
// 12-68 4524 -> 3200; 1900 of the same 7272 -> 5747; FP32, 256 of k 10-48
// 1139 -> 1069.  What bounds it with one CTA is the FP64 pipe of the one SM: in a round
// at k = 64 each of eight warps issues about 8 instructions of inner product,
// 22 of rotation parameters and 32 of rows, two warps a sub-partition, at 64
// cycles each (4.0 us of the 4.3 us measured).  Few updates of k > 48 therefore run
// on a cluster of CTAs each (CL): 2.6 us a round at k = 64 with four CTAs, 0.8 of
// them the exchange; the phase 1175 us.
#include <cfloat>
#include <climits>

#include "hc_internal.h"
#include "hc_scalar.cuh"

namespace hc {
namespace {

// integer keys that order non-negative values (a negative value's key is
// negative), and the key of x / 2^n for a value far above the smallest normal
__device__ __forceinline__ long long key(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ int key(float x) { return __float_as_int(x); }
__device__ __forceinline__ bool below_pow2(double x, double y, int n) {  // x < y 2^-n, y >= 0
    return __double2hiint(x) < __double2hiint(y) - (n << 20);
}
__device__ __forceinline__ bool below_pow2(float x, float y, int n) {
    return __float_as_int(x) < __float_as_int(y) - (n << 23);
}

template <typename T>
struct SvLim;
template <>
struct SvLim<double> {
    static constexpr double safmin = DBL_MIN / DBL_EPSILON;
    static constexpr double tiny_scale = 1e-60;   // fold a column scale below this
};
template <>
struct SvLim<float> {
    static constexpr float safmin = FLT_MIN / FLT_EPSILON;
    static constexpr float tiny_scale = 1e-12f;
};

// Is the pair to be rotated, a_pq^2 > tol^2 a_pp a_qq (rot), and was it above
// the stopping level, a_pq^2 > tol a_pp a_qq (big)?
__device__ __forceinline__ bool pair_test(double app, double aqq, double apq, float tol, bool &big) {
    float mp, mq, ma;
    int ep, eq, ea;
    split(app, mp, ep);
    split(aqq, mq, eq);
    split(apq, ma, ea);
    // at most about 2^2 (Cauchy-Schwarz); below 2^-110 < tol^2 no rotation
    const int ex = 2 * ea - ep - eq;
    if (ea == 0 || ex < -110) return false;
    const float x = ma * ma * __int_as_float((min(ex, 60) + 127) << 23), y = mp * mq;
    big = x > tol * y;
    return x > tol * tol * y;
}
__device__ __forceinline__ bool pair_test(float app, float aqq, float apq, float tol, bool &big) {
    const float x = apq * apq, y = app * aqq;
    big = x > tol * y;
    return apq != 0.f && x > tol * tol * y;
}

// Sum of f(i) over start <= i < k by a group of G lanes (rows i = lig mod G
// each): eight partial sums by i mod 8, added in one fixed tree, so the result
// does not depend on G.
template <int G, typename T, typename F>
__device__ __forceinline__ T group_sum(bool act, int start, int k, int lig, F f) {
    constexpr int NA = 8 / G;
    T a[NA];
#pragma unroll
    for (int m = 0; m < NA; ++m) a[m] = 0;
    if (act) {
        int i = (start & ~7) + lig;
#pragma unroll
        for (int m = 0; m < NA; ++m)   // the first eight rows may begin before start
            if (i + G * m >= start && i + G * m < k) a[m] += f(i + G * m);
        for (i += 8; i + G * (NA - 1) < k; i += 8)
#pragma unroll
            for (int m = 0; m < NA; ++m) a[m] += f(i + G * m);
#pragma unroll
        for (int m = 0; m + 1 < NA; ++m)
            if (i + G * m < k) a[m] += f(i + G * m);
    }
#pragma unroll
    for (int h = NA / 2; h > 0; h /= 2)
#pragma unroll
        for (int m = 0; m < h; ++m) a[m] += a[m + h];
    T v = a[0];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// dlarfg's reflector of (alpha, x), ss = ||x||^2.  The scaled form, with tau as a sum
// and v's first entry 1, because of what it does to row j when x is small beside
// alpha (most columns of a graded T): tau is 2 and y_j becomes -y_j with one
// rounding.  With an unscaled v = (alpha - beta, x) and 1 / (beta (beta - alpha)) the
// factor 2 comes out of four rounded operations, and the QR's backward error was four
// times as large (products of FP32 updates 1.83e-7 from their 64-bit values, 1.42e-7
// so).
template <typename T>
__device__ __forceinline__ T reflector_scal(T alpha, T beta) {
    return copysign(inv(abs(alpha - beta)), alpha);
}
template <typename T>
__device__ __forceinline__ void reflector(T alpha, T ss, T &beta, T &tau, T &scal) {
    const T n2 = fma(alpha, alpha, ss), rs = inv_sqrt(n2);
    T nb = n2 * rs;
    nb = fma(fma(-nb, nb, n2) * T(0.5), rs, nb);
    beta = -copysign(nb, alpha);
    tau = fma(abs(alpha), rs, T(1));
    scal = reflector_scal(alpha, beta);
}

constexpr int kSvThreads = 512;
constexpr int kSvRows = 6;   // 32-row pieces of the largest k (168)
template <typename T>
constexpr int kSvMaxK = sizeof(T) == 8 ? 119 : 168;

// CL: cs CTAs (a cluster) per update.  Each of them computes T and its pivoted QR
// (the same bits), then takes a share of the pairs of every Jacobi round, pairs pi0
// .. pi1 - 1 of the tournament, and so holds the current values of those pairs'
// columns only.  From one round to the next a column moves by one pair, so a CTA
// sends two columns to its neighbours' shared memory and one cluster barrier ends
// the round.  Sums and rotations are the same as with one CTA, bit for bit: sums
// over a column take up to eight lanes (D), rows G.
template <typename T, int G, bool CL>
__global__ void __launch_bounds__(kSvThreads, 1)
    svd_smem_kernel(const Desc *__restrict__ descs, T *__restrict__ ws, int *__restrict__ rank,
                    int *__restrict__ status, int *__restrict__ info, int maxK, int cs) {
    static_assert(CL || G <= 8, "a column's sum has eight parts");
    constexpr int D = G < 8 ? G : 8;
    __shared__ int s_big[2][CL ? 8 : 1];
    __shared__ unsigned char s_own[CL ? kSvMaxK<T> : 1];   // (static: every byte takes from k <= 119)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T s_wmax[kSvThreads / 32];
    __shared__ T s_scal;
    __shared__ int s_rank;
    const Desc d = descs[CL ? blockIdx.x / cs : blockIdx.x];
    const int cr = CL ? blockIdx.x % cs : 0;   // this CTA's rank in the cluster
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int nw = nthr >> 5;
    if (d.status0) {
        if (tid == 0 && cr == 0) {
            status[d.idx] = d.status0;
            rank[d.idx] = 0;
            if (info) info[d.idx] = 0;
        }
        return;
    }
    const int M = d.M, k = d.k;
    const WsLayout L = ws_layout(d);
    T *base = ws + d.ws;
    const T *UA = base + L.UA, *VB = base + L.VB;
    // column-major with an odd leading dimension: lanes that walk a column
    // are free of bank conflicts
    const int ld = svd_ld(k);
    const size_t mat = (size_t)maxK * svd_ld(maxK);
    T *A = reinterpret_cast<T *>(smem_raw);   // R_A, T, its QR, then V_J
    T *B = A + mat;                           // R_B, then R^T, rotated; at the end Q's reflectors
    T *X0 = B + mat, *X1 = X0 + (maxK + 1), *s_d = X1 + (maxK + 1);
    T *s_rd = s_d + (maxK + 1);               // R's diagonal, then 1 / s_d
    T *s_tau = s_rd + (maxK + 1);             // of reflector j, H = I - tau v v^T
    short *s_perm = reinterpret_cast<short *>(s_tau + (maxK + 1));
    short *s_pcol = s_perm + (maxK + 1);
    T *Yg = base + L.Uo;   // reflectors of Q (k x k, ld k) in the Uo slot until U_r is written
    const int grp = tid / G, lig = tid & (G - 1), ngrp = nthr / G;
    const int qgrp = tid / D, dlig = tid & (D - 1), nqgrp = nthr / D;   // the QR's groups

    // ---- T = triu(R_A) triu(R_B)^T (hcore_dgemm.c:330-387): a warp per row,
    // the row of T replaces the row of R_A that only it reads --------------------
    for (int l = warp; l < k; l += nw)
        for (int i = lane; i < k; i += 32) {
            A[(size_t)l * ld + i] = i <= l ? UA[(size_t)l * M + i] : T(0);
            B[(size_t)l * ld + i] = i <= l ? VB[(size_t)l * M + i] : T(0);
        }
    __syncthreads();
    T amax = 0;
    bool bad = false;
    for (int i = warp; i < k; i += nw) {
        T acc[kSvRows];
#pragma unroll
        for (int c = 0; c < kSvRows; ++c) {
            acc[c] = 0;
            if (32 * c < k) {
                const T *b = B + min(lane + 32 * c, k - 1);
                T s0 = 0, s1 = 0;
                int l = max(i, 32 * c);
                for (; l + 1 < k; l += 2) {
                    s0 += A[(size_t)l * ld + i] * b[(size_t)l * ld];
                    s1 += A[(size_t)(l + 1) * ld + i] * b[(size_t)(l + 1) * ld];
                }
                if (l < k) s0 += A[(size_t)l * ld + i] * b[(size_t)l * ld];
                acc[c] = s0 + s1;
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kSvRows; ++c) {
            const int j = lane + 32 * c;
            if (j < k) {
                A[(size_t)j * ld + i] = acc[c];
                amax = max(amax, abs(acc[c]));
                bad = bad || !isfinite(acc[c]);
            }
        }
    }
    amax = warp_max(amax);
    if (lane == 0) s_wmax[warp] = amax;
    if (__syncthreads_or(bad)) {
        // a NaN or infinity: no decomposition; the update is not written
        if (cr != 0) return;
        for (int t = tid; t < k; t += nthr) base[L.sig + t] = T(NAN);
        if (tid == 0) {
            int r = d.rk != 0 && d.rk < k ? d.rk : k;
            if ((d.rule & kRuleCapRank) && r > d.max_rank) r = d.max_rank;
            rank[d.idx] = r;
            status[d.idx] = HCORE_GPU_S_NOCONV;
            if (info) info[d.idx] = 0;
        }
        return;
    }
    // scale T by 2^-sexp, sexp the exponent of its largest entry
    amax = 0;
    for (int w = 0; w < nw; ++w) amax = max(amax, s_wmax[w]);
    const int sexp = amax > T(0) ? binary_exponent(amax) : 0;

    // squared column norms (G lanes per column), scaled columns
    for (int c0 = 0; c0 < k; c0 += ngrp) {
        const int c = c0 + grp;
        T *ac = A + (size_t)c * ld;
        if (c < k && sexp != 0)
            for (int i = lig; i < k; i += G) ac[i] = mul_exp2(ac[i], -sexp);
        if (G > D) __syncwarp();
        const T s = group_sum<D, T>(c < k, 0, k, dlig, [&](int i) { return ac[i] * ac[i]; });
        if (c < k && lig == 0) {
            X0[c] = s;    // norms of rows j.. of column c, squared; -1: pivoted already
            s_d[c] = s;   // the same at the last exact computation
        }
    }
    __syncthreads();
    // squared deflation bound, the same in every thread
    T f2 = 0;
    for (int c = lane; c < k; c += 32) f2 += X0[c];
    const T defl2 = deflation_bound2(warp_sum(f2), k, M, d.rk, d.rule, d.acc, sexp);
    const int kfloor = d.rank_start < k ? (d.rank_start > 0 ? d.rank_start : 0) : k;

    // ---- QR with column pivoting, T P = Q R ------------------------------------
    int kk = k;
    for (int j = 0; j < k; ++j) {
        const T *nr = (j & 1) ? X1 : X0;
        T *nr2 = (j & 1) ? X0 : X1;
        // pivot: the largest remaining norm, the lowest column on a tie
        auto best = key(T(-1));
        int pv = 0;
        for (int c = lane; c < k; c += 32) {
            const auto x = key(nr[c]);
            if (x > best) {
                best = x;
                pv = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const auto ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, pv, o);
            if (ob > best || (ob == best && oi < pv)) {
                best = ob;
                pv = oi;
            }
        }
        if (j >= kfloor && defl2 >= T(0) && best <= key(defl2)) {
            T tail = 0;
            for (int c = lane; c < k; c += 32) tail += max(nr[c], T(0));
            if (warp_sum(tail) <= defl2) {
                kk = j;
                break;
            }
        }
        // the reflector of column pv, rows j.., dlarfg's: beta = -sign(alpha) ||(alpha,
        // x)||, v = (1, scal x) (x itself stays as it is), scal = 1 / (alpha - beta),
        // tau = (beta - alpha) / beta = 1 + |alpha| / ||(alpha, x)||, by warp 0 while the
        // others form x^T y for the remaining columns y
        const T *ap = A + (size_t)pv * ld;
        if (warp == 0) {
            const T alpha = ap[j];
            T ss = 0;
            for (int i = j + 1 + lane; i < k; i += 32) ss += ap[i] * ap[i];
            ss = warp_sum(ss);
            T beta = alpha, scal = 0, tau = 0;
            if (ss > SvLim<T>::safmin) reflector(alpha, ss, beta, tau, scal);
            if (lane == 0) {
                s_pcol[j] = (short)pv;
                s_rd[j] = beta;
                s_tau[j] = tau;
                s_scal = scal;
            }
        }
        for (int c0 = 0; c0 < k; c0 += nqgrp) {
            const int c = c0 + qgrp;
            const bool act = c < k && c != pv && key(nr[c]) >= 0;
            const T *ac = A + (size_t)c * ld;
            const T w = group_sum<D, T>(act, j + 1, k, dlig, [&](int i) { return ap[i] * ac[i]; });
            if (act && dlig == 0) nr2[c] = w;   // (kept where the column's new norm goes)
        }
        __syncthreads();
        // apply it to them and downdate their norms (dlaqp2's rule), D lanes per column
        const T tau = s_tau[j], scal = s_scal;
        const int i0 = j + 1 + ((dlig - (j + 1)) & (D - 1));
        for (int c0 = 0; c0 < k; c0 += nqgrp) {
            const int c = c0 + qgrp;
            const T nc = c < k ? nr[c] : T(-1);
            const bool act = c < k && c != pv && key(nc) >= 0;
            T *ac = A + (size_t)c * ld;
            const bool upd = act && tau != T(0);
            // (row j's term, in lane 0's hands, is added to the sum of the rows below;
            // s = tau v^T y itself leaves row j, s scal times x the rows below)
            T r = act && dlig == 0 ? ac[j] : T(0), s = 0;
            if (upd && dlig == 0) {
                s = tau * fma(scal, nr2[c], r);
                r -= s;
                s *= scal;
            }
            s = __shfl_sync(0xffffffffu, s, lane & ~(D - 1));
            T nn = 0;
            bool redo = false;
            if (act) {
                if (upd)
                    for (int i = i0; i < k; i += D) ac[i] -= s * ap[i];
                if (dlig == 0) {
                    ac[j] = r;
                    nn = nc - r * r;
                    redo = !(key(nn) > 0) || below_pow2(nn, s_d[c], 10);
                }
            }
            if (__any_sync(0xffffffffu, redo)) {
                redo = __shfl_sync(0xffffffffu, (int)redo, lane & ~(D - 1)) != 0;
                const T q = group_sum<D, T>(redo, j + 1, k, dlig, [&](int i) { return ac[i] * ac[i]; });
                if (redo && dlig == 0) {
                    nn = q;
                    s_d[c] = q;
                }
            }
            if (c < k && dlig == 0) nr2[c] = act ? nn : T(-1);
        }
        __syncthreads();
    }
    {
        // columns that the deflation left: positions kk.. in column order
        const T *nr = (kk & 1) ? X1 : X0;
        if (kk < k)
            for (int c = tid; c < k; c += nthr)
                if (key(nr[c]) >= 0) {
                    int pos = kk;
                    for (int q = 0; q < c; ++q) pos += key(nr[q]) >= 0;
                    s_pcol[pos] = (short)c;
                }
    }
    __syncthreads();
    // Q's reflectors to the workspace, B = R^T (its columns kk.. are zero)
    for (int h = warp; h < k; h += nw) {
        const T *ah = A + (size_t)s_pcol[h] * ld;
        // v = (1, scal x); scal once more (no use without a reflector)
        const T scal = h < kk && s_tau[h] != T(0) ? reflector_scal(ah[h], s_rd[h]) : T(0);
        for (int i = lane; i < k; i += 32) {
            const T x = ah[i];
            if (h < kk && cr == 0) Yg[(size_t)h * k + i] = i > h ? x * scal : (i == h ? T(1) : T(0));
            // R(i, h)
            B[(size_t)i * ld + h] = i < kk ? (i < h ? x : (i == h ? s_rd[h] : T(0))) : T(0);
        }
    }
    __syncthreads();
    for (int c = warp; c < k; c += nw)
        for (int i = lane; i < k; i += 32) A[(size_t)c * ld + i] = i == c ? T(1) : T(0);
    T *s_nrm = X0, *s_sig = X1;
    auto column_norm = [&](int c, bool fold) {   // of column c, by its group
        T dj = 1;
        T *xj = B + (size_t)c * ld;
        if (c < kk && fold) {
            dj = s_d[c];
            if (dj < SvLim<T>::tiny_scale) {   // fold a scale before it underflows
                T *vj = A + (size_t)c * ld;
                for (int i = lig; i < k; i += G) {
                    xj[i] *= dj;
                    vj[i] *= dj;
                }
                dj = 1;
            }
        }
        __syncwarp();
        const T s = group_sum<D, T>(c < kk, 0, k, dlig, [&](int i) { return xj[i] * xj[i]; });
        if (c < k && lig == 0) {
            s_nrm[c] = c < kk ? dj * dj * s : T(0);
            s_d[c] = dj;
            s_rd[c] = fold && c < kk ? inv(dj) : T(1);
        }
    };
    auto column_norms = [&](bool fold) {
        for (int c0 = 0; c0 < k; c0 += ngrp) column_norm(c0 + grp, fold);
    };
    column_norms(false);
    if constexpr (CL) cluster_sync(); else __syncthreads();

    // ---- one-sided Jacobi on B = R^T, rotations accumulated in A ----------------
    // (columns kk.. of B are zero and take no part, V_J's rows kk.. stay zero)
    const int n = kk + (kk & 1), np = n / 2;
    // this CTA's pairs (a CTA without any only takes part in the barriers)
    const int active = CL ? max(1, min(cs, np)) : 1;
    const int pi0 = CL ? min(cr, active) * np / active : 0, pi1 = CL ? min(cr + 1, active) * np / active : np;
    const unsigned left = CL && pi0 > 0 && cr < active ? peer_delta(A, cr - 1) : 0;
    const unsigned right = CL && pi1 < np ? peer_delta(A, cr + 1) : 0;
    const float tol = (float)(k > 8 ? k : 8) * (sizeof(T) == 8 ? (float)DBL_EPSILON : FLT_EPSILON);
    bool converged = kk <= 1;
    int sweeps = 0;
    for (; sweeps < kMaxSweeps && !converged; ++sweeps) {
        bool big = false;   // this thread rotated a pair above sqrt(tol)
        for (int round = 0; round < n - 1; ++round) {
            for (int b0 = pi0; b0 < pi1; b0 += ngrp) {
                // circle-method tournament: pair 0 is (n - 1, round), pair i
                // (round + i, round - i) mod n - 1
                const int pi = b0 + grp;
                int p = round + pi, q = round - pi;
                if (p >= n - 1) p -= n - 1;
                if (q < 0) q += n - 1;
                if (pi == 0) p = n - 1;
                const bool valid = pi < pi1 && p < kk && q < kk;
                T *xp = B + (size_t)p * ld, *xq = B + (size_t)q * ld;
                T app = 0, aqq = 0, dp = 1, dq = 1;
                if (valid) {
                    app = s_nrm[p];
                    aqq = s_nrm[q];
                    dp = s_d[p];
                    dq = s_d[q];
                }
                const T dot = group_sum<D, T>(valid, 0, k, dlig, [&](int i) { return xp[i] * xq[i]; });
                bool rot = false, redo_p = false, redo_q = false;
                T np_ = 0, nq_ = 0, dp2 = 1, dq2 = 1, rdp2 = 1, rdq2 = 1;
                if (valid) {
                    const T apq = (dp * dq) * dot;
                    bool bigp = false;
                    rot = key(app) > key(SvLim<T>::safmin) && key(aqq) > key(SvLim<T>::safmin) &&
                          pair_test(app, aqq, apq, tol, bigp);
                    if (rot) {
                        big |= bigp;
                        // true columns p' = c (p - t q), q' = c (q + t p), in B and
                        // V_J; with column scales d: f1 = t dq / dp, f2 = t dp / dq
                        const T t = tangent(app, aqq, apq);
                        // (FP32 divides: it is cheap there, and the tracked
                        // reciprocals' drift of one rounding a rotation is not)
                        const T rdp = sizeof(T) == 8 ? s_rd[p] : inv(dp);
                        const T rdq = sizeof(T) == 8 ? s_rd[q] : inv(dq);
                        const T u = fma(t, t, T(1)), cs = inv_sqrt(u);
                        const T f1 = t * (dq * rdp), f2 = t * (dp * rdq);
                        np_ = app - t * apq;
                        nq_ = aqq + t * apq;
                        dp2 = dp * cs;
                        dq2 = dq * cs;
                        redo_p = below_pow2(np_, app, 6);
                        redo_q = below_pow2(nq_, aqq, 6);
                        T *vp = A + (size_t)p * ld, *vq = A + (size_t)q * ld;
                        int i = lig;
                        for (; i < kk; i += G) {
                            const T a = xp[i], b = xq[i], c = vp[i], e = vq[i];
                            xp[i] = a - f1 * b;
                            xq[i] = b + f2 * a;
                            vp[i] = c - f1 * e;
                            vq[i] = e + f2 * c;
                        }
                        for (; i < k; i += G) {
                            const T a = xp[i], b = xq[i];
                            xp[i] = a - f1 * b;
                            xq[i] = b + f2 * a;
                        }
                        const T ics = u * cs;   // 1 / c
                        rdp2 = rdp * ics;
                        rdq2 = rdq * ics;
                    }
                }
                // strong cancellation in a tracked norm: recompute
                if (__any_sync(0xffffffffu, redo_p || redo_q)) {
                    if (G > D) __syncwarp();
                    const T sp = group_sum<D, T>(redo_p, 0, k, dlig, [&](int i) { return xp[i] * xp[i]; });
                    const T sq = group_sum<D, T>(redo_q, 0, k, dlig, [&](int i) { return xq[i] * xq[i]; });
                    if (redo_p) np_ = dp2 * dp2 * sp;
                    if (redo_q) nq_ = dq2 * dq2 * sq;
                }
                if (rot && lig == 0) {
                    s_nrm[p] = np_;
                    s_nrm[q] = nq_;
                    s_d[p] = dp2;
                    s_d[q] = dq2;
                    s_rd[p] = rdp2;
                    s_rd[q] = rdq2;
                }
                if constexpr (CL) {
                    // the next round has p in pair pi - 1 and q in pair pi + 1
                    auto send = [&](int c, unsigned to) {
                        T *x = B + (size_t)c * ld, *v = A + (size_t)c * ld;
                        for (int i = lig; i < k; i += G) {
                            peer_store(x + i, to, x[i]);
                            if (i < kk) peer_store(v + i, to, v[i]);
                        }
                        if (lig == 0) {
                            peer_store(s_nrm + c, to, s_nrm[c]);
                            peer_store(s_d + c, to, s_d[c]);
                            peer_store(s_rd + c, to, s_rd[c]);
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
            if (tid < cs) peer_store(&s_big[sweeps & 1][cr], peer_delta(A, tid), any);
            cluster_sync();
            converged = true;
            for (int t = 0; t < cs; ++t) converged = converged && !s_big[sweeps & 1][t];
        } else {
            column_norms(true);
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
                const unsigned to = peer_delta(A, lane);
                peer_store(s_nrm + j, to, s_nrm[j]);
                peer_store(s_d + j, to, s_d[j]);
            }
        cluster_sync();
    }

    // singular values = true column norms of B (of the scaled T), descending,
    // ties by index, NaN last: a total order whatever the values
    bool nonfinite = false;
    for (int j = tid; j < k; j += nthr) {
        const T s = sqrt(s_nrm[j]);
        nonfinite = nonfinite || !isfinite(s);
        s_sig[j] = s == s ? s : T(-1);
    }
    if (tid == 0) s_rank = k;
    const bool finite = !__syncthreads_or(nonfinite);
    for (int j = tid; j < k; j += nthr) {
        const auto sj = key(s_sig[j]);
        int pos = 0;
        for (int i = 0; i < k; ++i) {
            const auto si = key(s_sig[i]);
            pos += (si > sj) || (si == sj && i < j);
        }
        s_perm[pos] = (short)j;
    }
    __syncthreads();
    // rank rule (hcore_dgemm.c:444-464; the fast rules start at i = 2; the
    // compressor's starts at 0, may compare with acc * sigma_max and caps the
    // rank at max_rank)
    const T thr = (d.rule & kRuleRelative) ? (T)d.acc * mul_exp2(s_sig[s_perm[0]], sexp) : (T)d.acc;
    for (int t = tid; t < k; t += nthr) {
        const T s = s_sig[s_perm[t]];
        const T v = key(s) < 0 ? T(NAN) : mul_exp2(s, sexp);
        if (cr == 0) base[L.sig + t] = v;
        if (d.rk == 0 && t >= d.rank_start && v < thr) atomicMin(&s_rank, t);
    }
    __syncthreads();
    int r = d.rk != 0 ? (d.rk < k ? d.rk : k) : s_rank;
    if ((d.rule & kRuleCapRank) && r > d.max_rank) r = d.max_rank;
    int st = HCORE_GPU_S_OK;
    if (!converged || !finite) st = HCORE_GPU_S_NOCONV;
    else if (r > d.max_rank) st = HCORE_GPU_S_RANK_MAX;
    else if (r > d.storage_rank) st = HCORE_GPU_S_STORAGE;

    // U_r and V_r S_r of an accepted update, and of one whose rank only
    // exceeds its storage limit (rebuilt later into larger storage)
    if (st == HCORE_GPU_S_OK || st == HCORE_GPU_S_STORAGE) {
        // V_r S_r = P (B's true columns): row P(i) of the output is row i of B
        // (the rows S V^T of hcore_dgemm.c:484-489, transposed)
        T *Uo = base + L.Uo, *Vo = base + L.Vo;
        for (int t = warp; t < r; t += nw) {
            const int j = s_perm[t];
            if (CL && owner(j) != cr) continue;
            const T f = s_d[j];
            for (int i = lane; i < k; i += 32)
                Vo[(size_t)t * k + s_pcol[i]] = mul_exp2(f * B[(size_t)j * ld + i], sexp);
        }
        int nown = r;   // the columns of U_r that this CTA forms
        if constexpr (CL) {
            nown = 0;
            for (int t = 0; t < r; ++t) {
                const bool mine = owner(s_perm[t]) == cr;
                if (mine && tid == 0) s_own[nown] = (unsigned char)t;
                nown += mine;
            }
        }
        __syncthreads();
        // U_r = Q (V_J's true columns), Q = H_0 ... H_{kk-1}: the reflectors
        // come into B's place, each group applies them, last to first, to its
        // columns of V_J
        for (int h = warp; h < kk; h += nw)
            for (int i = lane; i < k; i += 32) B[(size_t)h * ld + i] = Yg[(size_t)h * k + i];
        if constexpr (CL) cluster_sync(); else __syncthreads();   // Yg is Uo's place
        for (int t0 = 0; t0 < nown; t0 += ngrp) {
            const bool act = t0 + grp < nown;
            const int t = !act ? 0 : (CL ? s_own[t0 + grp] : t0 + grp);
            const int j = act ? s_perm[t] : 0;
            T *x = A + (size_t)j * ld;   // each group owns the column of its own j
            if (act) {
                const T dj = s_d[j];
                for (int i = lig; i < k; i += G) x[i] *= dj;
            }
            for (int h = kk - 1; h >= 0; --h) {
                const T gi = s_tau[h];
                if (gi == T(0)) continue;
                const T *y = B + (size_t)h * ld;
                const int i0 = h + ((lig - h) & (G - 1));
                if (G > D) __syncwarp();
                const T s = gi * group_sum<D, T>(act, h, k, dlig, [&](int i) { return y[i] * x[i]; });
                if (act)
                    for (int i = i0; i < k; i += G) x[i] -= s * y[i];
            }
            if (act)
                for (int i = lig; i < k; i += G) Uo[(size_t)t * k + i] = x[i];
        }
    }
    if (tid == 0 && cr == 0) {
        rank[d.idx] = r;
        status[d.idx] = st;
        if (info) info[d.idx] = sweeps;
    }
}

// matrices, five arrays of k + 1 values, two index arrays
template <typename T>
size_t smem_bytes(int K) {
    return (size_t)2 * K * svd_ld(K) * sizeof(T) + (size_t)5 * (K + 1) * sizeof(T) +
           (size_t)2 * (K + 1) * sizeof(short) + 16;
}


// ---- larger cores: a cluster per update ----------------------------------------
// k beyond shared memory (119 in FP64, 168 in FP32) up to kMaxK.  The matrices
// sit in the workspace (L2-resident), column-major, and the CTAs of a cluster
// share an update: columns (QR with column pivoting, norms, U_r), column pairs
// (Jacobi), rows (T).  What one of them writes the others read after a cluster
// barrier, past the L1 (ld.global.cg).  The arithmetic is the shared-memory
// kernel's.
//
// What bounds it: a Jacobi round is 5 k FP64 FMAs per pair, 22 instructions of
// rotation parameters and a barrier, and the FP64 pipe of one SM made it 38 us
// at k = 220 (one CTA, 440 threads); over eight SMs it is about 7.  G lanes
// hold a pair's two columns of B and of V_J in registers, R rows each, loaded
// once a round, so that L2 latency is paid once.
// SVD phase with one CTA per update (1024 threads, R^T in shared memory up to k =
// 167) and now: 3 updates of k 160-220 65.1, 9.8 ms; 24 of k 80-220 57.1, 11.8;
// 40 of k 200-256 109, 60; 6 of k 360-500 508, 90; 200 of k 120-140, where one
// CTA an update fills the GPU either way, 32.1, 34.6 (their whole plan 52.4,
// 45.8).
constexpr int kClThreads = 256, kClMax = 8;

template <typename T, int G, int R>
__global__ void __launch_bounds__(kClThreads, R <= 10 ? 2 : 1)
    svd_cluster_kernel(const Desc *__restrict__ descs, T *__restrict__ ws, int *__restrict__ rank,
                       int *__restrict__ status, int *__restrict__ info) {
    __shared__ T s_tau[kMaxK], s_rdiag[kMaxK], s_sig[kMaxK];
    __shared__ short s_perm[kMaxK], s_pcol[kMaxK];
    __shared__ T s_wmax[kClThreads / 32];
    __shared__ int s_rank;
    unsigned cr, cs;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(cr));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs));
    const Desc d = descs[blockIdx.x / cs];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lig = tid & (G - 1);
    const bool first = cr == 0 && tid == 0;
    if (d.status0) {
        if (first) {
            status[d.idx] = d.status0;
            rank[d.idx] = 0;
            if (info) info[d.idx] = 0;
        }
        return;
    }
    const int M = d.M, k = d.k;
    const WsLayout L = ws_layout(d);
    T *base = ws + d.ws;
    const T *UA = base + L.UA, *VB = base + L.VB;
    T *A = base + L.W, *B = base + L.V;   // T, its QR, V_J; R^T, rotated (ld k)
    T *X0 = base + L.sv, *X1 = X0 + k, *s_d = X1 + k, *s_rd = s_d + k, *slots = s_rd + k;
    T *Yg = base + L.Uo;
    // this thread's warp and group among the cluster's
    const int gw = (int)cr * (kClThreads / 32) + warp, ngw = (int)cs * (kClThreads / 32);
    const int gg = ((int)cr * kClThreads + tid) / G, ngg = (int)cs * kClThreads / G;
    auto sum_group = [](T v) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    // rows lig, lig + G, ... of a column, zero outside [lo, hi)
    auto load = [&](T (&x)[R], const T *col, int lo, int hi, bool act) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = lig + G * r;
            x[r] = act && i >= lo && i < hi ? __ldcg(col + i) : T(0);
        }
    };
    auto store = [&](const T (&x)[R], T *col, int lo, int hi) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = lig + G * r;
            if (i >= lo && i < hi) col[i] = x[r];
        }
    };
    auto dot = [&](const T (&x)[R], const T (&y)[R]) {
        T a0 = 0, a1 = 0;
#pragma unroll
        for (int r = 0; r < R; r += 2) {
            a0 += x[r] * y[r];
            a1 += x[r + 1] * y[r + 1];
        }
        return sum_group(a0 + a1);
    };

    // ---- T = triu(R_A) triu(R_B)^T: a warp per row, 32 columns at a time -----------
    T amax = 0;
    bool bad = false;
    for (int i = gw; i < k; i += ngw)
        for (int c = 0; c < k; c += 32) {
            const int j = c + lane, jr = min(j, k - 1);
            T s0 = 0, s1 = 0;
            int l = max(i, c);
#pragma unroll 4
            for (; l + 1 < k; l += 2) {
                s0 += UA[(size_t)l * M + i] * (l >= jr ? VB[(size_t)l * M + jr] : T(0));
                s1 += UA[(size_t)(l + 1) * M + i] * (l + 1 >= jr ? VB[(size_t)(l + 1) * M + jr] : T(0));
            }
            if (l < k) s0 += UA[(size_t)l * M + i] * (l >= jr ? VB[(size_t)l * M + jr] : T(0));
            s0 += s1;
            if (j < k) {
                A[(size_t)j * k + i] = s0;
                amax = max(amax, abs(s0));
                bad = bad || !isfinite(s0);
            }
        }
    amax = warp_max(amax);
    if (lane == 0) s_wmax[warp] = amax;
    const bool cta_bad = __syncthreads_or(bad);
    if (tid == 0) {
        for (int w = 1; w < kClThreads / 32; ++w) amax = max(amax, s_wmax[w]);
        slots[cr] = cta_bad ? T(-1) : amax;
    }
    cluster_sync();
    amax = 0;
    bad = false;
    for (unsigned q = 0; q < cs; ++q) {
        const T x = __ldcg(slots + q);
        bad = bad || x < T(0);
        amax = max(amax, x);
    }
    if (bad) {   // a NaN or infinity: no decomposition; the update is not written
        if (cr == 0)
            for (int t = tid; t < k; t += kClThreads) base[L.sig + t] = T(NAN);
        if (first) {
            int r = d.rk != 0 && d.rk < k ? d.rk : k;
            if ((d.rule & kRuleCapRank) && r > d.max_rank) r = d.max_rank;
            rank[d.idx] = r;
            status[d.idx] = HCORE_GPU_S_NOCONV;
            if (info) info[d.idx] = 0;
        }
        return;
    }
    const int sexp = amax > T(0) ? binary_exponent(amax) : 0;
    // scaled columns, their squared norms
    for (int c0 = 0; c0 < k; c0 += ngg) {
        const int c = c0 + gg;
        T x[R];
        load(x, A + (size_t)c * k, 0, k, c < k);
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = mul_exp2(x[r], -sexp);
        const T s = dot(x, x);
        if (c < k) {
            store(x, A + (size_t)c * k, 0, k);
            if (lig == 0) {
                X0[c] = s;
                s_d[c] = s;
            }
        }
    }
    cluster_sync();
    T f2 = 0;
    for (int c = lane; c < k; c += 32) f2 += __ldcg(X0 + c);
    const T defl2 = deflation_bound2(warp_sum(f2), k, M, d.rk, d.rule, d.acc, sexp);
    const int kfloor = d.rank_start < k ? (d.rank_start > 0 ? d.rank_start : 0) : k;

    // ---- QR with column pivoting (as in svd_smem_kernel) ---------------------------
    int kk = k;
    for (int j = 0; j < k; ++j) {
        const T *nr = (j & 1) ? X1 : X0;
        T *nr2 = (j & 1) ? X0 : X1;
        auto best = key(T(-1));
        int pv = 0;
#pragma unroll 4
        for (int c = lane; c < k; c += 32) {
            const auto x = key(__ldcg(nr + c));
            if (x > best) {
                best = x;
                pv = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const auto ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, pv, o);
            if (ob > best || (ob == best && oi < pv)) {
                best = ob;
                pv = oi;
            }
        }
        if (j >= kfloor && defl2 >= T(0) && best <= key(defl2)) {
            T tail = 0;
            for (int c = lane; c < k; c += 32) tail += max(__ldcg(nr + c), T(0));
            if (warp_sum(tail) <= defl2) {
                kk = j;
                break;
            }
        }
        T p[R];
        load(p, A + (size_t)pv * k, j + 1, k, true);
        const T alpha = __ldcg(A + (size_t)pv * k + j), ss = dot(p, p);
        T beta = alpha, scal = 0, tau = 0;
        if (ss > SvLim<T>::safmin) reflector(alpha, ss, beta, tau, scal);
        if (tid == 0) {
            s_pcol[j] = (short)pv;
            s_rdiag[j] = beta;
            s_tau[j] = tau;
        }
        for (int c0 = 0; c0 < k; c0 += ngg) {
            const int c = c0 + gg;
            const T nc = c < k ? __ldcg(nr + c) : T(-1);
            const bool act = c < k && c != pv && key(nc) >= 0;
            T *ac = A + (size_t)c * k;
            T x[R];
            load(x, ac, j + 1, k, act);
            const T acj = act ? __ldcg(ac + j) : T(0);
            const T s = tau * fma(scal, dot(x, p), acj);
            T nn = 0;
            bool redo = false;
            if (act) {
                if (tau != T(0)) {
                    const T sx = s * scal;
#pragma unroll
                    for (int r = 0; r < R; ++r) x[r] -= sx * p[r];
                    store(x, ac, j + 1, k);
                }
                const T r = acj - s;
                if (lig == 0 && tau != T(0)) ac[j] = r;
                nn = nc - r * r;
                redo = !(key(nn) > 0) || below_pow2(nn, __ldcg(s_d + c), 10);
            }
            if (__any_sync(0xffffffffu, redo)) {
                const T q = dot(x, x);
                if (redo) {
                    nn = q;
                    if (lig == 0) s_d[c] = q;
                }
            }
            if (c < k && lig == 0) nr2[c] = act ? nn : T(-1);
        }
        cluster_sync();
    }
    if (kk < k) {   // columns that the deflation left: positions kk.. in column order
        const T *nr = (kk & 1) ? X1 : X0;
        for (int c = tid; c < k; c += kClThreads)
            if (key(__ldcg(nr + c)) >= 0) {
                int pos = kk;
                for (int q = 0; q < c; ++q) pos += key(__ldcg(nr + q)) >= 0;
                s_pcol[pos] = (short)c;
            }
    }
    __syncthreads();
    for (int h = gw; h < k; h += ngw) {
        const T *ah = A + (size_t)s_pcol[h] * k;
        const T scal = h < kk && s_tau[h] != T(0) ? reflector_scal(__ldcg(ah + h), s_rdiag[h]) : T(0);
        for (int i = lane; i < k; i += 32) {
            const T x = __ldcg(ah + i);
            if (h < kk) Yg[(size_t)h * k + i] = i > h ? x * scal : (i == h ? T(1) : T(0));
            B[(size_t)i * k + h] = i < kk ? (i < h ? x : (i == h ? s_rdiag[h] : T(0))) : T(0);
        }
    }
    cluster_sync();
    for (int c = gw; c < k; c += ngw)
        for (int i = lane; i < k; i += 32) A[(size_t)c * k + i] = i == c ? T(1) : T(0);
    T *s_nrm = X0;
    auto column_norms = [&](bool fold) {
        for (int c0 = 0; c0 < k; c0 += ngg) {
            const int c = c0 + gg;
            T dj = fold && c < kk ? __ldcg(s_d + c) : T(1);
            T x[R];
            load(x, B + (size_t)c * k, 0, k, c < kk);
            if (fold && c < kk && dj < SvLim<T>::tiny_scale) {   // fold a scale before it underflows
                T v[R];
                load(v, A + (size_t)c * k, 0, k, true);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    x[r] *= dj;
                    v[r] *= dj;
                }
                store(x, B + (size_t)c * k, 0, k);
                store(v, A + (size_t)c * k, 0, k);
                dj = 1;
            }
            const T s = dot(x, x);
            if (c < k && lig == 0) {
                s_nrm[c] = c < kk ? dj * dj * s : T(0);
                s_d[c] = dj;
                s_rd[c] = fold && c < kk ? inv(dj) : T(1);
            }
        }
    };
    column_norms(false);
    cluster_sync();

    // ---- one-sided Jacobi ------------------------------------------------------------
    const int n = kk + (kk & 1), np = n / 2;
    const float tol = (float)(k > 8 ? k : 8) * (sizeof(T) == 8 ? (float)DBL_EPSILON : FLT_EPSILON);
    bool converged = kk <= 1;
    int sweeps = 0;
    for (; sweeps < kMaxSweeps && !converged; ++sweeps) {
        bool big = false;
        for (int round = 0; round < n - 1; ++round) {
            for (int b0 = 0; b0 < np; b0 += ngg) {
                const int pi = b0 + gg;
                int p = round + pi, q = round - pi;
                if (p >= n - 1) p -= n - 1;
                if (q < 0) q += n - 1;
                if (pi == 0) p = n - 1;
                const bool valid = pi < np && p < kk && q < kk;
                T *xp = B + (size_t)p * k, *xq = B + (size_t)q * k;
                T *vp = A + (size_t)p * k, *vq = A + (size_t)q * k;
                T x[R], y[R], v[R], w[R];
                load(x, xp, 0, k, valid);
                load(y, xq, 0, k, valid);
                load(v, vp, 0, kk, valid);
                load(w, vq, 0, kk, valid);
                T app = 0, aqq = 0, dp = 1, dq = 1, rdp = 1, rdq = 1;
                if (valid) {
                    app = __ldcg(s_nrm + p);
                    aqq = __ldcg(s_nrm + q);
                    dp = __ldcg(s_d + p);
                    dq = __ldcg(s_d + q);
                    rdp = sizeof(T) == 8 ? __ldcg(s_rd + p) : inv(dp);
                    rdq = sizeof(T) == 8 ? __ldcg(s_rd + q) : inv(dq);
                }
                const T dt = dot(x, y);
                bool rot = false, redo_p = false, redo_q = false;
                T np_ = 0, nq_ = 0, cs_ = 1, ics = 1;
                if (valid) {
                    const T apq = (dp * dq) * dt;
                    bool bigp = false;
                    rot = key(app) > key(SvLim<T>::safmin) && key(aqq) > key(SvLim<T>::safmin) &&
                          pair_test(app, aqq, apq, tol, bigp);
                    if (rot) {
                        big |= bigp;
                        const T t = tangent(app, aqq, apq);
                        const T u = fma(t, t, T(1));
                        cs_ = inv_sqrt(u);
                        ics = u * cs_;
                        const T f1 = t * (dq * rdp), f2 = t * (dp * rdq);
                        np_ = app - t * apq;
                        nq_ = aqq + t * apq;
                        redo_p = below_pow2(np_, app, 6);
                        redo_q = below_pow2(nq_, aqq, 6);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const T a = x[r], c = v[r];
                            x[r] = a - f1 * y[r];
                            y[r] = y[r] + f2 * a;
                            v[r] = c - f1 * w[r];
                            w[r] = w[r] + f2 * c;
                        }
                        store(x, xp, 0, k);
                        store(y, xq, 0, k);
                        store(v, vp, 0, kk);
                        store(w, vq, 0, kk);
                    }
                }
                const T dp2 = dp * cs_, dq2 = dq * cs_;
                if (__any_sync(0xffffffffu, redo_p || redo_q)) {
                    const T sp = dot(x, x), sq = dot(y, y);
                    if (redo_p) np_ = dp2 * dp2 * sp;
                    if (redo_q) nq_ = dq2 * dq2 * sq;
                }
                if (rot && lig == 0) {
                    s_nrm[p] = np_;
                    s_nrm[q] = nq_;
                    s_d[p] = dp2;
                    s_d[q] = dq2;
                    s_rd[p] = rdp * ics;
                    s_rd[q] = rdq * ics;
                }
            }
            cluster_sync();
        }
        column_norms(true);
        const bool cta_big = __syncthreads_or(big);
        if (tid == 0) slots[(sweeps & 1) * kClMax + cr] = cta_big ? T(1) : T(0);
        cluster_sync();
        converged = true;
        for (unsigned q = 0; q < cs; ++q)
            if (__ldcg(slots + (sweeps & 1) * kClMax + q) != T(0)) converged = false;
    }

    // singular values, order and rank (as in svd_smem_kernel, in every CTA)
    bool nonfinite = false;
    for (int j = tid; j < k; j += kClThreads) {
        const T s = sqrt(__ldcg(s_nrm + j));
        nonfinite = nonfinite || !isfinite(s);
        s_sig[j] = s == s ? s : T(-1);
    }
    if (tid == 0) s_rank = k;
    const bool finite = !__syncthreads_or(nonfinite);
    for (int j = tid; j < k; j += kClThreads) {
        const auto sj = key(s_sig[j]);
        int pos = 0;
        for (int i = 0; i < k; ++i) {
            const auto si = key(s_sig[i]);
            pos += (si > sj) || (si == sj && i < j);
        }
        s_perm[pos] = (short)j;
    }
    __syncthreads();
    const T thr = (d.rule & kRuleRelative) ? (T)d.acc * mul_exp2(s_sig[s_perm[0]], sexp) : (T)d.acc;
    for (int t = tid; t < k; t += kClThreads) {
        const T s = s_sig[s_perm[t]];
        const T v = key(s) < 0 ? T(NAN) : mul_exp2(s, sexp);
        if (cr == 0) base[L.sig + t] = v;
        if (d.rk == 0 && t >= d.rank_start && v < thr) atomicMin(&s_rank, t);
    }
    __syncthreads();
    int r = d.rk != 0 ? (d.rk < k ? d.rk : k) : s_rank;
    if ((d.rule & kRuleCapRank) && r > d.max_rank) r = d.max_rank;
    int st = HCORE_GPU_S_OK;
    if (!converged || !finite) st = HCORE_GPU_S_NOCONV;
    else if (r > d.max_rank) st = HCORE_GPU_S_RANK_MAX;
    else if (r > d.storage_rank) st = HCORE_GPU_S_STORAGE;
    if (first) {
        rank[d.idx] = r;
        status[d.idx] = st;
        if (info) info[d.idx] = sweeps;
    }
    if (st != HCORE_GPU_S_OK && st != HCORE_GPU_S_STORAGE) return;
    T *Uo = base + L.Uo, *Vo = base + L.Vo;
    for (int t = gw; t < r; t += ngw) {
        const int j = s_perm[t];
        const T f = __ldcg(s_d + j);
        for (int i = lane; i < k; i += 32)
            Vo[(size_t)t * k + s_pcol[i]] = mul_exp2(f * __ldcg(B + (size_t)j * k + i), sexp);
    }
    cluster_sync();
    // the reflectors leave the slot that U_r is written to
    for (int h = gw; h < kk; h += ngw)
        for (int i = lane; i < k; i += 32) B[(size_t)h * k + i] = __ldcg(Yg + (size_t)h * k + i);
    cluster_sync();
    for (int t0 = 0; t0 < r; t0 += ngg) {
        const int t = t0 + gg;
        const bool act = t < r;
        const int j = act ? s_perm[t] : 0;
        T x[R], y[R];
        load(x, A + (size_t)j * k, 0, k, act);
        const T dj = act ? __ldcg(s_d + j) : T(0);
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] *= dj;
        for (int h = kk - 1; h >= 0; --h) {
            const T gi = s_tau[h];
            if (gi == T(0)) continue;
            load(y, B + (size_t)h * k, h, k, true);
            const T s = gi * dot(y, x);
#pragma unroll
            for (int q = 0; q < R; ++q) x[q] -= s * y[q];
        }
        if (act) store(x, Uo + (size_t)t * k, 0, k);
    }
}

}  // namespace

template <typename T>
cudaError_t configure_svd_smem(int optin, int *kmax) {
    using K = void (*)(const Desc *, T *, int *, int *, int *, int, int);
    const K kernels[] = {svd_smem_kernel<T, 1, false>, svd_smem_kernel<T, 2, false>, svd_smem_kernel<T, 4, false>,
                         svd_smem_kernel<T, 8, false>, svd_smem_kernel<T, 8, true>, svd_smem_kernel<T, 16, true>};
    int dyn = optin;
    for (K f : kernels) {
        cudaFuncAttributes fa;
        const cudaError_t e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
        dyn = dyn < optin - (int)fa.sharedSizeBytes ? dyn : optin - (int)fa.sharedSizeBytes;
    }
    int k = 0;
    while (k < kSvMaxK<T> && smem_bytes<T>(k + 1) <= (size_t)dyn) ++k;
    *kmax = k;
    for (K f : kernels) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename T, int G>
static void launch_svd_g(const Desc *d_desc, int n, T *ws, int *d_rank, int *d_status, int *d_info,
                         int K, cudaStream_t s) {
    const int np = (K + 1) / 2, t = (np * G + 31) / 32 * 32;
    svd_smem_kernel<T, G, false><<<n, t < kSvThreads ? t : kSvThreads, smem_bytes<T>(K), s>>>(
        d_desc, ws, d_rank, d_status, d_info, K, 1);
}

// cs CTAs per update
template <typename T, typename F>
static auto with_spread(int K, int cs, unsigned grid, cudaStream_t s, F f) {
    const int pairs = ((K + 1) / 2 + cs - 1) / cs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem_bytes<T>(K);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return pairs <= 8 ? f(cfg, svd_smem_kernel<T, 16, true>) : f(cfg, svd_smem_kernel<T, 8, true>);
}
template <typename T>
int svd_spread_fit(int K, int cs) {
    int n = 0;
    const cudaError_t e = with_spread<T>(K, cs, (unsigned)cs, nullptr, [&](const cudaLaunchConfig_t &cfg, auto kernel) {
        return cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    });
    if (e == cudaSuccess) return n;
    cudaGetLastError();
    return 0;
}
template <typename T>
cudaError_t launch_svd_spread(const Desc *d_desc, int n, T *ws, int *d_rank, int *d_status, int *d_info, int K,
                              int cs, cudaStream_t s) {
    return with_spread<T>(K, cs, (unsigned)n * cs, s, [&](const cudaLaunchConfig_t &cfg, auto kernel) {
        return cudaLaunchKernelEx(&cfg, kernel, d_desc, ws, d_rank, d_status, d_info, K, cs);
    });
}

template <typename T>
void launch_svd_smem(const Desc *d_desc, int n, T *ws, int *d_rank, int *d_status, int *d_info, int K,
                     int G, cudaStream_t s) {
    if (G >= 8) launch_svd_g<T, 8>(d_desc, n, ws, d_rank, d_status, d_info, K, s);
    else if (G >= 4) launch_svd_g<T, 4>(d_desc, n, ws, d_rank, d_status, d_info, K, s);
    else if (G >= 2) launch_svd_g<T, 2>(d_desc, n, ws, d_rank, d_status, d_info, K, s);
    else launch_svd_g<T, 1>(d_desc, n, ws, d_rank, d_status, d_info, K, s);
}

// One cluster per update: as many CTAs (a power of two, at most eight, the
// portable limit) as give every update's cluster its own SMs.
template <typename T>
cudaError_t launch_svd_cluster(const Desc *d_desc, int n, T *ws, int *d_rank, int *d_status, int *d_info,
                               int K, int updates, cudaStream_t s) {
    unsigned cs = 1;
    while (cs < kClMax && 2 * cs * (unsigned)(updates > n ? updates : n) <= 152) cs *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n * cs);
    cfg.blockDim = dim3(kClThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // rows past k cost instructions: the smallest G x R that holds them
    auto go = [&](auto kernel) { return cudaLaunchKernelEx(&cfg, kernel, d_desc, ws, d_rank, d_status, d_info); };
    if (K <= 160) return go(svd_cluster_kernel<T, 16, 10>);
    if (K <= 224) return go(svd_cluster_kernel<T, 16, 14>);
    if (K <= 256) return go(svd_cluster_kernel<T, 32, 8>);
    if (K <= 384) return go(svd_cluster_kernel<T, 32, 12>);
    return go(svd_cluster_kernel<T, 32, 16>);
}

template cudaError_t configure_svd_smem<double>(int, int *);
template cudaError_t configure_svd_smem<float>(int, int *);
template void launch_svd_smem<double>(const Desc *, int, double *, int *, int *, int *, int, int,
                                      cudaStream_t);
template void launch_svd_smem<float>(const Desc *, int, float *, int *, int *, int *, int, int,
                                     cudaStream_t);

template int svd_spread_fit<double>(int, int);
template int svd_spread_fit<float>(int, int);
template cudaError_t launch_svd_spread<double>(const Desc *, int, double *, int *, int *, int *, int, int,
                                               cudaStream_t);
template cudaError_t launch_svd_spread<float>(const Desc *, int, float *, int *, int *, int *, int, int,
                                              cudaStream_t);

template cudaError_t launch_svd_cluster<double>(const Desc *, int, double *, int *, int *, int *, int, int,
                                                cudaStream_t);
template cudaError_t launch_svd_cluster<float>(const Desc *, int, float *, int *, int *, int *, int, int,
                                               cudaStream_t);

}  // namespace hc
