// hcore-gb300 — the steps either side of the Schur update in a tile low-rank
// Cholesky, on sm_103a:
//   HCORE_dtrsm  (src/compute/hcore_dtrsm.c:24-48): B = alpha op(A)^-1 B or
//                alpha B op(A)^-1, A triangular; in the TLR Cholesky B is a
//                tile's V factor and A the panel's diagonal Cholesky factor
//   HCORE_dpotrf (src/compute/hcore_dpotrf.c:23-34): Cholesky factor of a
//                dense diagonal tile
//
// TRSM.  Every task is cut into groups of up to S right-hand-side vectors
// (columns of B for the left side, rows of B for the right side), one CTA
// per group.  The CTA keeps its S vectors in shared memory for the whole
// solve and turns every case into a forward substitution with a lower
// triangular T' (transposing and/or reversing the index order of A).  T' is
// walked in 32-column blocks: the block's diagonal part is solved by one warp
// per vector (lane i holds x_i; 32 steps with a shuffle), then the rows below
// are updated with the block's 32 solved values, 64 or 128 rows at a time through a
// shared-memory tile of T' that every vector of the CTA reuses.  Tiles are
// read along A's contiguous dimension, so a transposed A is read coalesced
// too.  A task's groups share A, which stays in L2.  Large triangles are solved
// that way block by block, with products on the tensor cores between the blocks
// (trsm_block_step).
//
// POTRF.  Blocked right-looking Cholesky on the lower view of the tile (the
// transposed view for uplo 'U'), 64 columns per block, three parts per block:
// the diagonal block (sub-blocks of 16 columns; the reference LAPACK's pivot
// test: a pivot that is not > 0, or is NaN, stops the factorization and is left
// in place), the panel below it (A_ik = A_ik L_kk^-T, 32 rows per CTA, four lanes
// a row), and the trailing lower triangle (A_ij -= A_ik A_jk^T: products on the
// tensor cores while it is large, else 32 x 32 tiles with 2 x 2 register blocks).
// Every launch first reads the task's info and returns once a pivot has failed.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstring>
#include <vector>

#include "hc_host.h"
#include "hc_products.h"
#include "hc_scalar.cuh"
#include "hcore.h"
#include "hcore_d.h"

namespace hc {

constexpr int kTrBs = 32;  // diagonal block of T'
constexpr int kTrThreads = 256;

struct TrsmWork {
    int task, v0, nv, pad;
};

// T' = the lower triangular form of the task's system (see the file comment):
// element (i, j) of T' is A(p, q) or A(q, p), p and q the indices i, j taken
// in reverse order when the effective triangle is upper.
struct TrsmView {
    const double *A;
    int lda, n;
    bool tflag, rev;
    __device__ double at(int i, int j) const {
        const int p = rev ? n - 1 - i : i, q = rev ? n - 1 - j : j;
        return tflag ? A[(size_t)p * lda + q] : A[(size_t)q * lda + p];
    }
};

// T'(r0 + r, c0 + c) for r < rows, c < cols into T (zero elsewhere, R rows)
template <int R>
__device__ __forceinline__ void trsm_tile(double (*T)[kTrBs + 1], const TrsmView &v, int r0, int rows, int c0,
                          int cols) {
#pragma unroll 8
    for (int e = threadIdx.x; e < R * kTrBs; e += kTrThreads) {
        int r, c;
        if (v.tflag) {  // A(q, p): contiguous in q, i.e. along a row of T'
            c = e % kTrBs; r = e / kTrBs;
        } else {        // A(p, q): contiguous in p, i.e. along a column of T'
            r = e % R; c = e / R;
        }
        T[r][c] = (r < rows && c < cols) ? v.at(r0 + r, c0 + c) : 0.0;
    }
}

// RC rows of T' per trailing chunk
template <int RC>
__global__ void __launch_bounds__(kTrThreads) trsm_kernel(const hcore_trsm_task *tasks,
                                                          const TrsmWork *work, int S) {
    extern __shared__ double X[];  // X[i * S + v]
    __shared__ double Tt[RC][kTrBs + 1];
    __shared__ double Td[kTrBs][kTrBs + 1];
    const TrsmWork w = work[blockIdx.x];
    const hcore_trsm_task t = tasks[w.task];
    const bool left = t.side == HCORE_Left;
    TrsmView v;
    v.A = t.A;
    v.lda = t.lda;
    v.n = left ? t.M : t.N;
    v.tflag = left ? t.trans != HCORE_NoTrans : t.trans == HCORE_NoTrans;
    v.rev = (t.uplo == HCORE_Lower) == v.tflag;  // effective triangle is upper
    const int n = v.n;
    const bool unit = t.diag == HCORE_Unit;
    // element i of vector u: B[i * es + u * vs]
    const size_t es = left ? 1 : (size_t)t.ldb, vs = left ? (size_t)t.ldb : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (t.alpha == 0.0) {  // B = 0 without reading A (BLAS convention)
        for (int e = tid; e < n * w.nv; e += kTrThreads) {
            const int i = left ? e % n : e / w.nv, u = left ? e / n : e % w.nv;
            t.B[(size_t)i * es + (size_t)(w.v0 + u) * vs] = 0.0;
        }
        return;
    }
    for (int e = tid; e < n * S; e += kTrThreads) {
        const int i = left ? e % n : e / S, u = left ? e / n : e % S;
        double x = 0.0;
        if (u < w.nv) {
            const int ia = v.rev ? n - 1 - i : i;
            x = t.alpha * t.B[(size_t)ia * es + (size_t)(w.v0 + u) * vs];
        }
        X[i * S + u] = x;
    }
    __syncthreads();
    for (int b0 = 0; b0 < n; b0 += kTrBs) {
        const int bs = min(kTrBs, n - b0);
        trsm_tile<kTrBs>(Td, v, b0, bs, b0, bs);
        __syncthreads();
        if (warp < w.nv) {  // one warp per vector: forward substitution in the block
            double x = lane < bs ? X[(b0 + lane) * S + warp] : 0.0;
            // x_j = b_j / T'_jj as a product with the reciprocal (one division
            // per lane and block instead of one per step)
            const double rd = (unit || lane >= bs) ? 1.0 : 1.0 / Td[lane][lane];
            for (int j = 0; j < bs; ++j) {
                if (lane == j) x *= rd;
                const double xj = __shfl_sync(0xffffffffu, x, j);
                if (lane > j) x -= Td[lane][j] * xj;
            }
            if (lane < bs) X[(b0 + lane) * S + warp] = x;
        }
        __syncthreads();
        for (int r0 = b0 + bs; r0 < n; r0 += RC) {
            const int rc = min(RC, n - r0);
            trsm_tile<RC>(Tt, v, r0, rc, b0, bs);
            __syncthreads();
            for (int o = tid; o < RC * S; o += kTrThreads) {
                const int u = o % S, r = o / S;
                if (r < rc && u < w.nv) {
                    double acc = X[(r0 + r) * S + u];
#pragma unroll 8
                    for (int j = 0; j < bs; ++j) acc -= Tt[r][j] * X[(b0 + j) * S + u];
                    X[(r0 + r) * S + u] = acc;
                }
            }
            __syncthreads();
        }
    }
    for (int e = tid; e < n * w.nv; e += kTrThreads) {
        const int i = left ? e % n : e / w.nv, u = left ? e / n : e % w.nv;
        const int ia = v.rev ? n - 1 - i : i;
        t.B[(size_t)ia * es + (size_t)(w.v0 + u) * vs] = X[i * S + u];
    }
}

// ---------------------------------------------------------------------------
// POTRF
// ---------------------------------------------------------------------------
constexpr int kPb = 64;  // block width

// element (i, j), i >= j, of the lower view
struct PotrfView {
    double *A;
    int lda;
    bool up;
    __device__ double &at(int i, int j) const {
        return up ? A[(size_t)i * lda + j] : A[(size_t)j * lda + i];
    }
};

constexpr int kSb = 16;

// 1 / sqrt(d) of a positive pivot, and sqrt(d) from both.  The short forms hold for
// finite normal d; +Inf passes LAPACK's pivot test (not d <= 0, not NaN) and gives
// L_jj = Inf and a column of zeros, as there.
__device__ __forceinline__ bool plain_pivot(double d) {
    return d >= 2.2250738585072014e-308 && d <= 1.7976931348623157e308;
}
__device__ __forceinline__ double pivot_rsqrt(double d) {
    return plain_pivot(d) ? inv_sqrt(d) : 1.0 / sqrt(d);
}
__device__ __forceinline__ double pivot_sqrt(double d, double r) {
    if (!plain_pivot(d)) return sqrt(d);
    const double l = d * r;
    return fma(fma(-l, l, d) * 0.5, r, l);
}

// The 16 x 16 block at (j0, j0) of S, by one warp in registers: lanes i and i + 16
// hold the even and the odd columns of row i.  One reciprocal square root and one
// scaling a column, no barrier; the pivots' square roots together at the end.
__device__ __forceinline__ void factor16(double (*S)[kPb + 1], int j0, int bs, double *rL, int *fail) {
    const int lane = threadIdx.x & 31, i = lane & 15, h = lane >> 4;
    double a[8], dd = 1.0, rr = 1.0;
#pragma unroll
    for (int m = 0; m < 8; ++m) a[m] = S[j0 + i][j0 + 2 * m + h];
    int bad = -1;
#pragma unroll
    for (int j = 0; j < kSb; ++j) {
        const double d = __shfl_sync(0xffffffffu, a[j / 2], j + 16 * (j & 1));
        double v = 0.0;
        if (bad < 0 && j0 + j < bs) {   // uniform in the warp
            if (!(d > 0.0)) {           // not positive, or NaN
                bad = j;
            } else {
                const double r = pivot_rsqrt(d);
                if (i == j) {
                    dd = d;
                    rr = r;
                }
                v = a[j / 2] * r;
                if (h == (j & 1) && i > j) a[j / 2] = v;
            }
        }
        v = __shfl_sync(0xffffffffu, v, i + 16 * (j & 1));   // L(i, j)
#pragma unroll
        for (int m = j / 2; m < 8; ++m) {
            const int c = 2 * m + h;
            const double lc = __shfl_sync(0xffffffffu, v, c);
            if (bad < 0 && c > j && i >= c) a[m] -= v * lc;
        }
    }
    const double l = pivot_sqrt(dd, rr);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int c = 2 * m + h;
        const bool done = c == i && j0 + i < bs && (bad < 0 || i < bad);
        if (c <= i) S[j0 + i][j0 + c] = done ? l : a[m];
    }
    if (h == 0) rL[j0 + i] = rr;
    if (lane == 0 && bad >= 0) *fail = j0 + bad;
}

// Solve rows of X L16^T = A16 in place: Q lanes a row (lane q of them holds
// columns q, q + Q, ... of the sixteen), L16's rows and reciprocal pivots in
// shared memory.  x_j goes around the lanes by a shuffle.
template <int Q>
__device__ __forceinline__ void solve16(double (&a)[kSb / Q], const double (*L)[kPb + 1], int j0, const double *rL,
                                        int q) {
#pragma unroll
    for (int j = 0; j < kSb; ++j) {
        double x = a[j / Q] * rL[j0 + j];
        x = __shfl_sync(0xffffffffu, x, j % Q, Q);
        if (q == j % Q) a[j / Q] = x;
#pragma unroll
        for (int m = j / Q; m < kSb / Q; ++m)
            if (q + Q * m > j) a[m] -= x * L[j0 + q + Q * m][j0 + j];
    }
}

// S(i, c) less the products of columns [l0, l0 + 16) of rows i and c
__device__ __forceinline__ void update16(double (*S)[kPb + 1], int i, int c, int l0) {
    double s0 = S[i][c], s1 = 0.0;
#pragma unroll
    for (int l = 0; l < kSb; l += 2) {
        s0 -= S[i][l0 + l] * S[c][l0 + l];
        s1 -= S[i][l0 + l + 1] * S[c][l0 + l + 1];
    }
    S[i][c] = s0 + s1;
}

// diagonal block [kb, kb + bs): right-looking over sub-blocks of 16 columns; a
// failing pivot is stored in place and ends the task (info = column + 1).  Bound by
// the chain of pivots: an FP64 instruction takes a warp 65 cycles, and a column 6
// of them and its updates.  So only the next sub-block's diagonal part is updated
// before its factorization (warp 0), the rest beside it (six warps that share no
// sub-partition with warp 0).  A block took 121 us with two barriers a column, 102
// with sub-blocks one after the other; 60 now.
__global__ void __launch_bounds__(256) potrf_diag_kernel(const hcore_potrf_task *tasks, int *info,
                                                         int kb) {
    __shared__ double S[kPb][kPb + 1];
    __shared__ double rL[kPb];
    __shared__ int fail;
    const hcore_potrf_task t = tasks[blockIdx.x];
    if (info[blockIdx.x] != 0 || kb >= t.n) return;
    const int bs = min(kPb, t.n - kb);
    const PotrfView V{t.A, t.lda, t.uplo == 'U' || t.uplo == 'u'};
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 16
    for (int e = tid; e < kPb * kPb; e += 256) {
        const int i = V.up ? e / kPb : e % kPb, j = V.up ? e % kPb : e / kPb;
        S[i][j] = (i < bs && j <= i) ? V.at(kb + i, kb + j) : 0.0;
    }
    if (tid == 0) fail = -1;
    __syncthreads();
    for (int j0 = 0; j0 < bs; j0 += kSb) {
        if (warp == 0) {
            factor16(S, j0, bs, rL, &fail);
        } else if (warp != 4 && j0 > 0) {
            // rows from j0 + 16 on, columns from j0 on: 16 columns, then a triangle
            const int r0 = j0 + kSb, nr = max(0, bs - r0), box = kSb * nr;
            for (int e = (warp - 1 - (warp > 4)) * 32 + lane; e < box + nr * (nr + 1) / 2; e += 192) {
                if (e < box) {
                    update16(S, r0 + e % nr, j0 + e / nr, j0 - kSb);
                } else {
                    const int x = e - box;
                    int i = (int)((sqrtf(8.f * x + 1.f) - 1.f) * 0.5f);
                    i += (i + 1) * (i + 2) / 2 <= x;
                    i -= i * (i + 1) / 2 > x;
                    update16(S, r0 + i, r0 + x - i * (i + 1) / 2, j0 - kSb);
                }
            }
        }
        __syncthreads();
        if (fail >= 0) break;
        const int below = j0 + kSb;
        if (below >= bs) break;
        // rows below (64 rows a pass, four lanes each; all lanes take part in the shuffles)
        {
            const int row = below + (tid >> 2), q = tid & 3;
            const bool in = row < kPb;
            double a[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) a[m] = in ? S[row][j0 + q + 4 * m] : 0.0;
            solve16<4>(a, S, j0, rL, q);
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (in) S[row][j0 + q + 4 * m] = a[m];
        }
        __syncthreads();
        {
            const int i = below + (tid >> 4), c = below + (tid & 15);   // the next diagonal part
            if (c <= i && i < bs) update16(S, i, c, j0);
        }
        __syncthreads();
    }
    for (int e = tid; e < kPb * kPb; e += 256) {
        const int i = V.up ? e / kPb : e % kPb, j = V.up ? e % kPb : e / kPb;
        if (i < bs && j <= i) V.at(kb + i, kb + j) = S[i][j];
    }
    if (tid == 0 && fail >= 0) info[blockIdx.x] = kb + fail + 1;
}

// panel rows below the diagonal block: X L_kk^T = A_ik, Q lanes a row, 128 / Q
// rows a CTA.  Sixteen columns at a time are solved in registers and taken out of
// the columns on their right (64 steps with a barrier each, 64 rows a CTA, took 126
// us a block, eight tiles of order 1024; this 48 us).  Bound by FP64 issue: about
// 630 instructions a warp with four lanes a row, 360 with eight, which do the same
// for half as many rows and so serve while all CTAs have an SM of their own (one
// tile of order 300: 40 and 28 us).
constexpr int kPrThreads = 128;
template <int Q>
__global__ void __launch_bounds__(kPrThreads) potrf_panel_kernel(const hcore_potrf_task *tasks,
                                                                 const int *info, int kb) {
    constexpr int PR = kPrThreads / Q;
    __shared__ double Ls[kPb][kPb + 1];
    __shared__ double Xs[PR][kPb + 1];
    __shared__ double rL[kPb];
    const hcore_potrf_task t = tasks[blockIdx.y];
    if (info[blockIdx.y] != 0 || kb >= t.n) return;
    const int bs = min(kPb, t.n - kb);
    const int r0 = kb + bs + blockIdx.x * PR;
    if (r0 >= t.n) return;   // (rows below exist, so bs = kPb)
    const int rows = min(PR, t.n - r0);
    const PotrfView V{t.A, t.lda, t.uplo == 'U' || t.uplo == 'u'};
    const int tid = threadIdx.x;
#pragma unroll 16
    for (int e = tid; e < kPb * kPb; e += kPrThreads) {
        const int i = V.up ? e / kPb : e % kPb, j = V.up ? e % kPb : e / kPb;
        Ls[i][j] = j <= i ? V.at(kb + i, kb + j) : 0.0;
    }
#pragma unroll 16
    for (int e = tid; e < PR * kPb; e += kPrThreads) {
        const int i = V.up ? e / kPb : e % PR, j = V.up ? e % kPb : e / PR;
        Xs[i][j] = i < rows ? V.at(r0 + i, kb + j) : 0.0;
    }
    if (tid < kPb) rL[tid] = 1.0 / V.at(kb + tid, kb + tid);
    __syncthreads();
    const int r = tid / Q, q = tid % Q;
#pragma unroll 1
    for (int j0 = 0; j0 < kPb; j0 += kSb) {
        double a[kSb / Q];
#pragma unroll
        for (int m = 0; m < kSb / Q; ++m) a[m] = Xs[r][j0 + q + Q * m];
        solve16<Q>(a, Ls, j0, rL, q);
#pragma unroll
        for (int m = 0; m < kSb / Q; ++m) Xs[r][j0 + q + Q * m] = a[m];
        __syncwarp();   // a row's lanes share a warp
        for (int c = j0 + kSb + q; c < kPb; c += Q) {
            double s0 = Xs[r][c], s1 = 0.0;
#pragma unroll
            for (int l = 0; l < kSb; l += 2) {
                s0 -= Xs[r][j0 + l] * Ls[c][j0 + l];
                s1 -= Xs[r][j0 + l + 1] * Ls[c][j0 + l + 1];
            }
            Xs[r][c] = s0 + s1;
        }
        __syncwarp();
    }
    __syncthreads();
    for (int e = tid; e < PR * kPb; e += kPrThreads) {
        const int i = V.up ? e / kPb : e % PR, j = V.up ? e % kPb : e / PR;
        if (i < rows) V.at(r0 + i, kb + j) = Xs[i][j];
    }
}

// small trailing lower triangle from row/column t0 = kb + bs: A_ij -= A_ik A_jk^T,
// one CTA per 32 x 32 tile (bi >= bj), 2 x 2 outputs per thread, K = bs
// staged 16 at a time.  Small tiles keep each CTA short: the update is on the
// factorization's critical path once per block.
constexpr int kUt = 32;
// From this many tiles in a step (two for each SM) the products go to the tensor
// cores: about 25 us a step with their slicing, where potrf_update_kernel takes 17
// us per tile and SM (all updates of eight tiles of order 1024: 2.6 ms, then 0.9).
// Their error is half that of FP64 FMAs.
constexpr int kTcUpdateTiles = 304;
__global__ void __launch_bounds__(256) potrf_update_kernel(const hcore_potrf_task *tasks,
                                                           const int *info, int kb, int tiles) {
    __shared__ double sP[16][kUt + 1];
    __shared__ double sQ[16][kUt + 1];
    const hcore_potrf_task t = tasks[blockIdx.y];
    if (info[blockIdx.y] != 0 || kb >= t.n) return;
    const int bs = min(kPb, t.n - kb), t0 = kb + bs;
    const int bi = blockIdx.x % tiles, bj = blockIdx.x / tiles;
    if (bj > bi) return;
    const int i0 = t0 + bi * kUt, j0 = t0 + bj * kUt;
    if (i0 >= t.n) return;
    const PotrfView V{t.A, t.lda, t.uplo == 'U' || t.uplo == 'u'};
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[2][2] = {};
    for (int k0 = 0; k0 < bs; k0 += 16) {
        for (int e = threadIdx.x; e < 2 * 16 * kUt; e += 256) {
            const int which = e / (16 * kUt), f = e % (16 * kUt);
            int kk, rr;
            if (V.up) { kk = f % 16; rr = f / 16; } else { rr = f % kUt; kk = f / kUt; }
            const int kg = k0 + kk, base = which ? j0 : i0;
            const double x = (kg < bs && base + rr < t.n) ? V.at(base + rr, kb + kg) : 0.0;
            if (which) sQ[kk][rr] = x; else sP[kk][rr] = x;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const double p0 = sP[kk][tx], p1 = sP[kk][tx + 16];
            const double q0 = sQ[kk][ty], q1 = sQ[kk][ty + 16];
            acc[0][0] += p0 * q0; acc[0][1] += p0 * q1;
            acc[1][0] += p1 * q0; acc[1][1] += p1 * q1;
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int i = i0 + tx + 16 * u, j = j0 + ty + 16 * w;
            if (i < t.n && j <= i) V.at(i, j) -= acc[u][w];
        }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// Vectors per CTA for `vectors` of them in all (tasks' last groups aside): up to 8
// while the CTA's vectors take at most 64 KB of shared memory (two or more CTAs per
// SM), fewer for longer vectors and while the CTAs do not outnumber the SMs: a
// CTA's time is its vectors' FP64 multiply-adds (order 300, 16 vectors: 214 us with
// eight a CTA, 131 with one; order 1024, 100 vectors: 1742, 803).  0 if not even one fits.
static int trsm_stride(int maxn, long long vectors) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const long long stat = (64 + kTrBs) * (kTrBs + 1) * (long long)sizeof(double);
    const long long per = (long long)maxn * (long long)sizeof(double);
    if (per + stat > optin) return 0;
    int S = 8;
    while (S > 1 && (per * S > 65536 || 2 * vectors <= 152LL * S)) S >>= 1;
    return S;
}

static int order_of(const hcore_trsm_task &t) { return t.side == HCORE_Left ? t.M : t.N; }
static int vectors_of(const hcore_trsm_task &t) { return t.side == HCORE_Left ? t.N : t.M; }

static bool trsm_valid(const hcore_trsm_task &t) {
    const bool side = t.side == HCORE_Left || t.side == HCORE_Right;
    const bool uplo = t.uplo == HCORE_Upper || t.uplo == HCORE_Lower;
    const bool tr = t.trans == HCORE_NoTrans || t.trans == HCORE_Trans || t.trans == HCORE_ConjTrans;
    const bool dg = t.diag == HCORE_Unit || t.diag == HCORE_NonUnit;
    if (!side || !uplo || !tr || !dg || t.M < 0 || t.N < 0) return false;
    const int na = t.side == HCORE_Left ? t.M : t.N;
    if (t.M == 0 || t.N == 0) return true;
    return t.A && t.B && t.lda >= std::max(1, na) && t.ldb >= std::max(1, t.M);
}

// Triangles from this order on may be solved by blocks: the vectors against a
// diagonal block of kTrTb (trsm_kernel), then one product on the tensor cores
// takes them out of all rows (columns) that follow.  The whole solve in one CTA
// is bound by the FP64 issue of its vectors and its chain of n / 32 blocks; a block
// step costs about 45 us however few the vectors.  Both ways, whole and by blocks,
// us (one GB300), by the vectors of all such tasks: order 448: 16 210, 356; 800 390,
// 414; 1920 615, 510; order 512: 160 278, 444; 800 487, 477; 1920 773, 589; order
// 1024: 160 879, 926; 480 1147, 901; 1920 2744, 1297.  So by blocks where CTAs of
// eight vectors outnumber the SMs, or where order and vectors a CTA (trsm_stride)
// make the whole solve as long as at order 512 with eight.
constexpr int kTrTcOrder = 448, kTrTb = 64;

// Step `blk` of a task solved by blocks: the diagonal block's task, and the
// product that follows (false when it is the last block).
static bool trsm_block_step(const hcore_trsm_task &t, int blk, hcore_trsm_task &diag, DenseProducts *pr) {
    const bool left = t.side == HCORE_Left, notrans = t.trans == HCORE_NoTrans;
    const int n = left ? t.M : t.N;
    // op(A)'s triangle: lower is solved forwards, upper backwards (left side; the
    // other way round on the right)
    const bool lower = (t.uplo == HCORE_Lower) == notrans, forward = left == lower;
    const int b0 = blk * kTrTb, b1 = std::min(n, b0 + kTrTb);
    const int p0 = forward ? b0 : n - b1, p1 = forward ? b1 : n - b0;
    const int r0 = forward ? p1 : 0, nr = forward ? n - p1 : p0;   // what is not solved yet
    const size_t lda = t.lda, ldb = t.ldb;
    diag = t;
    diag.alpha = blk == 0 ? t.alpha : 1.0;
    diag.A = t.A + p0 * (lda + 1);
    diag.B = t.B + (left ? (size_t)p0 : p0 * ldb);
    (left ? diag.M : diag.N) = p1 - p0;
    if (nr == 0) return false;
    if (!pr) return true;
    const double beta = blk == 0 ? t.alpha : 1.0;
    using DP = DenseProducts;
    const double *Ablk = notrans == left ? t.A + p0 * lda + r0 : t.A + r0 * lda + p0;
    const int trA = notrans == left ? 0 : 1;   // op(A)(rest, block), or its transpose on the right
    if (left)
        pr->add_one(DP::product(Ablk, t.lda, t.B + p0, t.ldb, trA | 2, p1 - p0, -1.0, beta), nr, t.N, t.B + r0,
                    t.ldb);
    else
        pr->add_one(DP::product(t.B + p0 * ldb, t.ldb, Ablk, t.lda, trA << 1, p1 - p0, -1.0, beta), t.M, nr,
                    t.B + r0 * ldb, t.ldb);
    return true;
}

// Run n TRSM tasks (device-accessible pointers) on stream s and wait.
static int run_trsm(int n, const hcore_trsm_task *tasks, cudaStream_t s) {
    int maxn = 1;
    for (int i = 0; i < n; ++i) {
        const hcore_trsm_task &t = tasks[i];
        if (!trsm_valid(t)) {
            set_error("hcore_gpu_trsm_batched: invalid task %d", i);
            return HCORE_GPU_EINVAL;
        }
        if (t.M == 0 || t.N == 0) continue;
        maxn = std::max(maxn, t.side == HCORE_Left ? t.M : t.N);
    }
    if (trsm_stride(maxn, 0) == 0) {
        set_error("hcore_gpu_trsm_batched: triangle of order %d does not fit shared memory", maxn);
        return HCORE_GPU_EINVAL;
    }
    // the launches of trsm_kernel: the small triangles, then the diagonal blocks
    // of the others, step by step, each followed by a stage of products
    struct Launch {
        size_t work0, count;
        long long vectors;
        int S, maxn, stage;
    };
    std::vector<hcore_trsm_task> solve;
    std::vector<TrsmWork> work;
    std::vector<Launch> launches;
    DenseProducts pr;
    int steps = 0;
    long long large = 0;   // vectors of the tasks that may go by blocks
    for (int i = 0; i < n; ++i)
        if (tasks[i].M > 0 && tasks[i].N > 0 && order_of(tasks[i]) >= kTrTcOrder)
            large += vectors_of(tasks[i]);
    const int large_S = trsm_stride(kTrTcOrder, large);
    auto by_blocks = [&](const hcore_trsm_task &t) {
        return t.alpha != 0.0 && t.M > 0 && t.N > 0 && order_of(t) >= kTrTcOrder &&
               (large > 8 * 152 || (long long)order_of(t) * large_S >= 8 * 512);
    };
    for (int blk = -1; blk < steps; ++blk) {
        Launch l{work.size(), 0, 0, 0, 1, -1};
        std::vector<int> todo;
        const size_t first = solve.size();
        bool any = false;
        for (int i = 0; i < n; ++i) {
            const hcore_trsm_task &t = tasks[i];
            if (t.M == 0 || t.N == 0) continue;
            const int order = order_of(t);
            hcore_trsm_task d = t;
            if (by_blocks(t)) {
                steps = std::max(steps, (order + kTrTb - 1) / kTrTb);
                if (blk < 0 || blk * kTrTb >= order) continue;
                any = trsm_block_step(t, blk, d, nullptr) || any;
                todo.push_back(i);
            } else if (blk >= 0) {
                continue;
            }
            l.maxn = std::max(l.maxn, order_of(d));
            l.vectors += vectors_of(d);
            solve.push_back(d);
        }
        l.S = trsm_stride(l.maxn, l.vectors);
        for (size_t q = first; q < solve.size(); ++q) {
            const int nvec = vectors_of(solve[q]);
            for (int v0 = 0; v0 < nvec; v0 += l.S) work.push_back({(int)q, v0, std::min(l.S, nvec - v0), 0});
        }
        l.count = work.size() - l.work0;
        if (any) {
            l.stage = pr.nstages();
            pr.stage(kBalanceP);   // (many right-hand sides share a triangle)
            for (int i : todo) {
                hcore_trsm_task d;
                trsm_block_step(tasks[i], blk, d, &pr);
            }
        }
        if (l.count) launches.push_back(l);
    }
    if (work.empty()) return HCORE_GPU_OK;
    if (work.size() > (size_t)INT_MAX || solve.size() > (size_t)INT_MAX) {
        set_error("hcore_gpu_trsm_batched: too many vector groups");
        return HCORE_GPU_EINVAL;
    }
    ThreadCtx &tc = thread_ctx();
    const size_t bt = al256(solve.size() * sizeof(hcore_trsm_task)), bw = al256(work.size() * sizeof(TrsmWork));
    size_t up = bt + bw;
    pr.place_host(up);
    size_t all = up;
    pr.place_device(all);
    char *arena = (char *)tc.dev_ensure(all);
    char *pin = (char *)tc.pin_ensure(up);
    pr.gave_up = tc.wait_word();
    if (!arena || !pin || !pr.gave_up) {
        set_error("hcore_gpu_trsm_batched: out of memory");
        return HCORE_GPU_ENOMEM;
    }
    cudaStreamSynchronize(s);  // the previous call may still read the pinned buffer
    memcpy(pin, solve.data(), solve.size() * sizeof(hcore_trsm_task));
    memcpy(pin + bt, work.data(), work.size() * sizeof(TrsmWork));
    pr.pack(pin);
    cudaMemcpyAsync(arena, pin, up, cudaMemcpyHostToDevice, s);
    cudaError_t e = configure_dense_tc();
    for (const Launch &l : launches) {
        const size_t smem = (size_t)l.maxn * l.S * sizeof(double);
        // (few vectors: larger chunks, fewer barriers)
        auto kernel = l.S <= 2 && smem <= 65536 ? trsm_kernel<128> : trsm_kernel<64>;
        if (e == cudaSuccess) e = allow_smem(kernel);
        if (e != cudaSuccess) break;
        kernel<<<(unsigned)l.count, kTrThreads, smem, s>>>((const hcore_trsm_task *)arena,
                                                           (const TrsmWork *)(arena + bt) + l.work0, l.S);
        e = cudaGetLastError();
        if (e == cudaSuccess && l.stage >= 0) e = pr.launch_stage(arena, l.stage, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error("hcore_gpu_trsm_batched: %s", cudaGetErrorString(e));
        return HCORE_GPU_ECUDA;
    }
    return check_waits(pr.gave_up, "hcore_gpu_trsm_batched");
}

// LAPACKE_dpotrf_work's argument checks (its info is LAPACK's minus one)
static int potrf_arg_info(const hcore_potrf_task &t) {
    const char u = (char)t.uplo;
    if (u != 'L' && u != 'l' && u != 'U' && u != 'u') return -2;
    if (t.n < 0) return -3;
    if (t.lda < std::max(1, t.n)) return -5;
    return 0;
}

// Run n POTRF tasks on stream s and wait; info[i] as LAPACKE_dpotrf_work.
static int run_potrf(int n, const hcore_potrf_task *tasks, int *info, cudaStream_t s) {
    std::vector<hcore_potrf_task> run;
    std::vector<int> slot;
    int maxn = 0;
    for (int i = 0; i < n; ++i) {
        info[i] = potrf_arg_info(tasks[i]);
        if (info[i] != 0 || tasks[i].n == 0) continue;
        if (!tasks[i].A) {
            set_error("hcore_gpu_potrf_batched: task %d has no matrix", i);
            return HCORE_GPU_EINVAL;
        }
        run.push_back(tasks[i]);
        slot.push_back(i);
        maxn = std::max(maxn, tasks[i].n);
    }
    if (run.empty()) return HCORE_GPU_OK;
    const int nr = (int)run.size();
    if (nr > 65535) {
        set_error("hcore_gpu_potrf_batched: more than 65535 tiles in one call");
        return HCORE_GPU_EINVAL;
    }
    ThreadCtx &tc = thread_ctx();
    const size_t bt = al256(nr * sizeof(hcore_potrf_task)), bi = al256(nr * sizeof(int));
    // The trailing updates of a block step, A_ij -= A_ik A_jk^T, run as products
    // on the tensor cores (hc_dense_tc.cu) while they are large.  Their rounding is
    // relative to the rows' largest entries, at most sqrt(a_ii) and sqrt(a_jj):
    // the backward error of a Cholesky factorization.
    DenseProducts pr;
    std::vector<int> stage_of;   // per block step: its stage of pr, or -1
    size_t up = bt + bi;
    std::vector<int> tile_of_job;
    {
        for (int kb = 0; kb < maxn; kb += kPb) {
            long long tiles = 0;
            for (const auto &t : run) {
                const long long x = t.n > kb + kPb ? (t.n - kb - kPb + kUt - 1) / kUt : 0;
                tiles += x * (x + 1) / 2;
            }
            stage_of.push_back(tiles >= kTcUpdateTiles ? pr.nstages() : -1);
            if (tiles < kTcUpdateTiles) continue;
            pr.stage(kNoBalance);   // (P and Q are the same rows)
            for (int q = 0; q < nr; ++q) {
                const hcore_potrf_task &t = run[q];
                const int n1 = t.n - kb - kPb;
                if (n1 <= 0) continue;
                const size_t ld = t.lda, k1 = kb + kPb;
                const bool up_ = t.uplo == 'U' || t.uplo == 'u';
                const double *p = up_ ? t.A + k1 * ld + kb : t.A + (size_t)kb * ld + k1;
                pr.add_one(DenseProducts::product(p, t.lda, p, t.lda, up_ ? 3 : 0, kPb, -1.0, 1.0), n1, n1,
                           t.A + k1 * (ld + 1), t.lda, up_ ? 2 : 1);
                tile_of_job.resize(pr.jobs.size(), q);
            }
        }
    }
    pr.place_host(up);
    size_t all = up;
    pr.place_device(all);
    char *arena = (char *)tc.dev_ensure(all);
    char *pin = (char *)tc.pin_ensure(up);
    pr.gave_up = tc.wait_word();
    if (!arena || !pin || !pr.gave_up) {
        set_error("hcore_gpu_potrf_batched: out of memory");
        return HCORE_GPU_ENOMEM;
    }
    const hcore_potrf_task *d_t = (const hcore_potrf_task *)arena;
    int *d_info = (int *)(arena + bt);
    for (size_t j = 0; j < pr.jobs.size(); ++j) pr.jobs[j].skip = d_info + tile_of_job[j];
    cudaStreamSynchronize(s);
    memcpy(pin, run.data(), nr * sizeof(hcore_potrf_task));
    memset(pin + bt, 0, nr * sizeof(int));
    pr.pack(pin);
    cudaMemcpyAsync(arena, pin, up, cudaMemcpyHostToDevice, s);
    cudaError_t e = configure_dense_tc();
    for (int kb = 0; kb < maxn && e == cudaSuccess; kb += kPb) {
        potrf_diag_kernel<<<nr, 256, 0, s>>>(d_t, d_info, kb);
        const int below = maxn - std::min(maxn, kb + kPb), stage = stage_of[kb / kPb];
        if (below > 0) {
            const int tiles = (below + kUt - 1) / kUt;
            if ((below + 15) / 16 * (long long)nr <= 152)
                potrf_panel_kernel<8><<<dim3((below + 15) / 16, nr), kPrThreads, 0, s>>>(d_t, d_info, kb);
            else
                potrf_panel_kernel<4><<<dim3((below + 31) / 32, nr), kPrThreads, 0, s>>>(d_t, d_info, kb);
            if (stage < 0)
                potrf_update_kernel<<<dim3(tiles * tiles, nr), 256, 0, s>>>(d_t, d_info, kb, tiles);
        }
        e = cudaGetLastError();
        if (e == cudaSuccess && stage >= 0) e = pr.launch_stage(arena, stage, s);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(pin + bt, d_info, nr * sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error("hcore_gpu_potrf_batched: %s", cudaGetErrorString(e));
        return HCORE_GPU_ECUDA;
    }
    if (const int rc = check_waits(pr.gave_up, "hcore_gpu_potrf_batched")) return rc;   // (NaN fails a pivot's test)
    for (int q = 0; q < nr; ++q) info[slot[q]] = ((const int *)(pin + bt))[q];
    return HCORE_GPU_OK;
}

// stage a host block (rows x cols, ld) into dst (ld rows) / back
static void stage_in(double *dst, const double *src, int rows, int cols, int ld, cudaStream_t s) {
    if (rows > 0 && cols > 0)
        cudaMemcpy2DAsync(dst, rows * sizeof(double), src, (size_t)ld * sizeof(double),
                          rows * sizeof(double), cols, cudaMemcpyHostToDevice, s);
}
static cudaError_t stage_out(double *dst, int ld, const double *src, int rows, int cols,
                             cudaStream_t s) {
    if (rows > 0 && cols > 0)
        cudaMemcpy2DAsync(dst, (size_t)ld * sizeof(double), src, rows * sizeof(double),
                          rows * sizeof(double), cols, cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
}

// per-thread device buffer for the drop-ins' host operands
static double *tlr_buffer(size_t n, const char *fn) {
    static thread_local double *buf = nullptr;
    static thread_local size_t buf_n = 0;
    if (buf_n < n) {
        if (buf) {
            cudaStreamSynchronize(thread_ctx().stream);
            cudaFree(buf);
        }
        buf = nullptr;
        buf_n = 0;
        if (cudaMalloc(&buf, std::max<size_t>(n, 1) * sizeof(double)) != cudaSuccess)
            fatal("%s: cannot allocate %zu bytes of device memory\n", fn, n * sizeof(double));
        buf_n = n;
    }
    return buf;
}

}  // namespace hc

using namespace hc;

extern "C" {

int hcore_gpu_trsm_batched(int n, const hcore_trsm_task *tasks, void *stream) {
    if (n < 0 || (n > 0 && !tasks)) {
        set_error("hcore_gpu_trsm_batched: invalid argument");
        return HCORE_GPU_EINVAL;
    }
    std::vector<hcore_trsm_task> tt(tasks, tasks + n);
    for (auto &t : tt) {
        if (t.M == 0 || t.N == 0) continue;
        t.A = (const double *)device_alias(t.A);
        t.B = (double *)device_alias(t.B);
        if (!t.A || !t.B) {
            set_error("hcore_gpu_trsm_batched: pointers must be device or pinned memory");
            return HCORE_GPU_EINVAL;
        }
    }
    return run_trsm(n, tt.data(), (cudaStream_t)stream);
}

int hcore_gpu_potrf_batched(int n, const hcore_potrf_task *tasks, int *info, void *stream) {
    if (n < 0 || (n > 0 && (!tasks || !info))) {
        set_error("hcore_gpu_potrf_batched: invalid argument");
        return HCORE_GPU_EINVAL;
    }
    std::vector<hcore_potrf_task> tt(tasks, tasks + n);
    for (auto &t : tt) {
        if (t.n <= 0) continue;
        t.A = (double *)device_alias(t.A);
        if (!t.A) {
            set_error("hcore_gpu_potrf_batched: pointers must be device or pinned memory");
            return HCORE_GPU_EINVAL;
        }
    }
    return run_potrf(n, tt.data(), info, (cudaStream_t)stream);
}

// cblas_dtrsm(ColMajor, side, uplo, transA, diag, M, Brank, alpha, A, LDA,
// BV, LDBV) on the GPU; flops as hcore_dtrsm.c:41-46 (an invalid side is the
// reference's failed assert).
void HCORE_dtrsm(HCORE_enum side, HCORE_enum uplo, HCORE_enum transA, HCORE_enum diag, int M,
                 int Brank, double alpha, double *A, int LDA, double *BV, int LDBV,
                 flop_counter *flops) {
    if (side != HCORE_Left && side != HCORE_Right)
        fatal("HCORE_dtrsm: side is not CblasLeft or CblasRight\n");
    hcore_trsm_task t{};
    t.side = side; t.uplo = uplo; t.trans = transA; t.diag = diag; t.M = M; t.N = Brank;
    t.alpha = alpha; t.A = A; t.lda = LDA; t.B = BV; t.ldb = LDBV;
    const bool ok = trsm_valid(t);  // as cblas_dtrsm: report, leave BV, return
    if (!ok) fprintf(stderr, "HCORE_dtrsm: invalid argument, BV left unchanged\n");
    if (ok && M > 0 && Brank > 0) {
        ThreadCtx &tc = thread_ctx();
        const int na = side == HCORE_Left ? M : Brank;
        const bool dev = is_device_memory(A) && is_device_memory(BV);
        if (!dev) {
            double *buf = tlr_buffer((size_t)na * na + (size_t)M * Brank, "HCORE_dtrsm");
            stage_in(buf, A, na, na, LDA, tc.stream);
            stage_in(buf + (size_t)na * na, BV, M, Brank, LDBV, tc.stream);
            t.A = buf; t.lda = na; t.B = buf + (size_t)na * na; t.ldb = M;
        }
        if (run_trsm(1, &t, tc.stream)) fatal("HCORE_dtrsm: %s\n", last_error());
        if (!dev && stage_out(BV, LDBV, t.B, M, Brank, tc.stream) != cudaSuccess)
            fatal("HCORE_dtrsm: %s\n", cudaGetErrorString(cudaGetLastError()));
    }
    if (flops) flops->trsm += flop_counts('t', M, Brank, side == HCORE_Left ? 1 : 2, 0);
}

// *info = LAPACKE_dpotrf_work(LAPACK_COL_MAJOR, uplo, N, A, LDA) on the GPU;
// uplo is LAPACK's character ('L' or 'U'), as the reference passes it through
// unchanged; flops as hcore_dpotrf.c:33.
void HCORE_dpotrf(HCORE_enum uplo, int N, double *A, int LDA, int *info, flop_counter *flops) {
    hcore_potrf_task t{};
    t.uplo = uplo; t.n = N; t.A = A; t.lda = LDA;
    int r = potrf_arg_info(t);
    if (r != 0) {
        fprintf(stderr, " ** On entry to DPOTRF parameter number %d had an illegal value\n", -r - 1);
    } else if (N > 0) {
        ThreadCtx &tc = thread_ctx();
        const bool dev = is_device_memory(A);
        if (!dev) {
            t.A = tlr_buffer((size_t)N * N, "HCORE_dpotrf");
            t.lda = N;
            stage_in(t.A, A, N, N, LDA, tc.stream);
        }
        if (run_potrf(1, &t, &r, tc.stream)) fatal("HCORE_dpotrf: %s\n", last_error());
        if (!dev && stage_out(A, LDA, t.A, N, N, tc.stream) != cudaSuccess)
            fatal("HCORE_dpotrf: %s\n", cudaGetErrorString(cudaGetLastError()));
    }
    if (info) *info = r;
    if (flops) flops->potrf += flop_counts('c', N, 0, 0, 0);
}

}  // extern "C"
