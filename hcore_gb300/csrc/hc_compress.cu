// hcore-gb300 — batched tile compression on sm_103a: a dense M x M tile D
// becomes U (M x r) and V (M x r) with D ~ U V^T, U the first r left singular
// vectors and V = (S V^T)^T.  This is the reference's compressor semantics
// (generate_compress, testing/testing_dgemm.c:119-236: keep the leading
// singular values sigma_i >= acc, cap the rank at storage_maxrank), with an
// optional relative rule (sigma_i >= acc * sigma_max) for TLR matrices whose
// tiles span many orders of magnitude.
//
// Method.  The reference runs a full dgesvd of the tile.  Here the tile's
// numerical range is found first,
//     D = Q B^T + E,   ||E||_F <= delta,
// with delta = 1e-3 of the truncation threshold (at least 64 eps ||D||_F), so
// that every singular value of the k-column product Q B^T is within delta of
// D's.  That product is exactly the low-rank form the recompression plan takes
// (UA = Q, VB = B), so the plan's QR, Jacobi SVD and rebuild phases finish the
// job with the compressor's rank rule.  Ranks agree with the reference's
// except where a singular value lies within delta of the threshold.
//
// The range comes from blocks of random test vectors whose products run on the
// tensor cores (find_ranges): the tile is read and written a few times per 32
// columns.  A truncated Householder QR with column pivoting (qrcp_kernel) does
// the same one column at a time; it applies 3 M^2 FP64 FMAs per column on one
// SM (98 ms for 48 tiles of 1024 and ranks 8-40 at 1e-8, where the blocks take
// 5 ms and the whole call went from 120.7 to 13.9 ms), so it is kept for what
// the blocks leave: small tiles, wide ranges, non-finite tiles.
//
// qrcp_kernel: one CTA per tile; the tile is copied into a workspace and
// factored there, one pivot column per step (argmax of the trailing column
// norms, which are recomputed exactly while the reflector is applied, so no
// norm downdating is needed).  The reflector is staged in shared memory; a
// warp applies it to one trailing column at a time.  At most kcap steps.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "hc_host.h"
#include "hc_products.h"
#include "hc_scalar.cuh"

namespace hc {

struct QrcpTask {
    const double *D;
    int ldd, M, kcap, relative;
    double acc;
    double *W;     // M x M, ld M
    double *tau;   // kcap
    int *perm;     // M
    double *vn;    // M: squared norms of the trailing column parts
};

struct FormWork {
    const double *W;
    const double *tau;
    const int *perm;
    double *UA, *VB;  // the plan workspace's UA and VB regions (M x k, ld M)
    int M, k;
    const double *Q, *B;  // a range found by products: M x k each (else null)
};

// ---- the range by products ---------------------------------------------------
// A tile of the blocked range finder: its residual E, the basis Q and B = E^T Q
// found so far (M x k, ld M).
struct RangeTile {
    const double *D;
    int ldd, M;
    double *E, *Q, *B;
};
constexpr int kSumParts = 32;   // partial sums of squares per tile

// E = D (load) and the partial sums of E's squares
__global__ void __launch_bounds__(256) range_norm_kernel(const RangeTile *tiles, const int *list, bool load,
                                                         double *part) {
    __shared__ double s_sum[8];
    const int q = list[blockIdx.x];
    const RangeTile t = tiles[q];
    const long long n = (long long)t.M * t.M, step = (long long)kSumParts * 256;
    double s = 0.0;
    for (long long e = (long long)blockIdx.y * 256 + threadIdx.x; e < n; e += step) {
        double x;
        if (load) {
            x = t.D[(size_t)(e / t.M) * t.ldd + e % t.M];
            t.E[e] = x;
        } else {
            x = t.E[e];
        }
        s += x * x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s += s_sum[w];
        part[(size_t)q * kSumParts + blockIdx.y] = s;
    }
}

// test vectors of one block: n values in (-1, 1), a fixed sequence (the
// SplitMix64 mixing function of Steele, Lea and Flood, 2014)
__global__ void range_test_vectors_kernel(double *omega, int n, int base) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long z = (unsigned long long)(base + i + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    omega[i] = (double)(long long)z * 0x1p-63;
}

// Columns c0 .. c0 + nc of each listed tile's Q made orthonormal among
// themselves (Gram-Schmidt, column by column).  Twice: a block spans several
// decades of singular values, and what one pass leaves (about 1e-9) would stay in E
// far above delta and be found again as new directions (160 columns instead of 80
// for 1024-tiles of rank 40 at 1e-8).  They need not be orthogonal to the
// earlier ones to rounding: E = D - Q B holds whatever Q is, and the plan
// factors Q.
// A cluster of CTAs per tile, R rows each in shared memory; a column's products
// with itself and the later ones are summed over the cluster in one exchange, then
// every CTA updates its rows (the arithmetic is bound by FP64 issue: one CTA per
// tile, its columns in registers, took 670 us for 32 columns of 48 tiles of order
// 1024; 340 now, three CTAs a tile).
constexpr int kOrCols = 32, kOrMaxCluster = 8;
static size_t orth_smem(int R) { return ((size_t)kOrCols * R + (2 * kOrMaxCluster + 2) * kOrCols) * sizeof(double); }

__global__ void __launch_bounds__(256) range_orth_kernel(const RangeTile *tiles, const int *list, int c0,
                                                         int nc, int cs, int R) {
    extern __shared__ __align__(16) double or_sm[];
    const RangeTile t = tiles[list[blockIdx.x / cs]];
    const int cta = blockIdx.x % cs, M = t.M, r0 = cta * R, nr = R / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *Q = t.Q + (size_t)c0 * M;
    double *Y = or_sm;                                          // column c, row i: Y[c R + i]
    double *part = Y + (size_t)kOrCols * R;                     // [parity][source CTA][column]
    double *coef = part + 2 * kOrMaxCluster * kOrCols, *scale = coef + kOrCols;
    for (int c = warp; c < nc; c += 8)
        for (int i = lane; i < R; i += 32) Y[c * R + i] = r0 + i < M ? Q[(size_t)c * M + r0 + i] : 0.0;
    cluster_sync();   // (every CTA has started before the first remote store)
    int par = 0;
    for (int pass = 0; pass < 2; ++pass) {
        for (int j = 0; j < nc; ++j, par ^= 1) {
            const double *x = Y + j * R;
            for (int g = j + 4 * warp; g < nc; g += 32) {
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                const double *y[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) y[h] = Y + min(g + h, nc - 1) * R + lane;
                for (int r = 0; r < nr; ++r) {
                    const double xi = x[lane + 32 * r];
#pragma unroll
                    for (int h = 0; h < 4; ++h) v[h] = fma(xi, y[h][32 * r], v[h]);
                }
                // lane l comes to hold sum l >> 3
#pragma unroll
                for (int n = 2, o = 16; n >= 1; n /= 2, o /= 2) {
                    const bool up = lane & o;
#pragma unroll
                    for (int e = 0; e < n; ++e) {
                        const double keep = up ? v[e + n] : v[e], send = up ? v[e] : v[e + n];
                        v[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
                const int c = g + (lane >> 3), to = lane & 7;
                if (c < nc && to < cs)
                    peer_store(part + (par * kOrMaxCluster + cta) * kOrCols + c, peer_delta(or_sm, to), v[0]);
            }
            cluster_sync();
            if (warp == 0) {   // lane c: column c
                double ss = 0.0, w = 0.0;
                for (int q = 0; q < cs; ++q) {
                    const double *p = part + (par * kOrMaxCluster + q) * kOrCols;
                    ss += p[j];
                    w += p[lane];
                }
                const double f = ss > 0.0 ? rsqrt(ss) : 0.0;   // (a zero column stays zero)
                if (lane > j && lane < nc) coef[lane] = f * (f * w);
                if (lane == j) scale[j] = f;
            }
            __syncthreads();
            for (int g = j + 1 + 4 * warp; g < nc; g += 32) {
                double *y[4], s[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    y[h] = Y + min(g + h, nc - 1) * R + lane;
                    s[h] = coef[min(g + h, nc - 1)];
                }
                for (int r = 0; r < nr; ++r) {
                    const double xi = x[lane + 32 * r];
#pragma unroll
                    for (int h = 0; h < 4; ++h)
                        if (g + h < nc) y[h][32 * r] -= s[h] * xi;
                }
            }
            __syncthreads();
        }
        for (int c = warp; c < nc; c += 8)
            for (int i = lane; i < R; i += 32) Y[c * R + i] *= scale[c];
        __syncthreads();
    }
    for (int c = warp; c < nc; c += 8)
        for (int i = lane; i < R && r0 + i < M; i += 32) Q[(size_t)c * M + r0 + i] = Y[c * R + i];
}

// CTAs per tile: at least two CTAs an SM, and as many as leave every tile's cluster
// SMs of its own
static cudaError_t launch_range_orth(const RangeTile *tiles, const int *list, int n, int c0, int nc, int maxM,
                                     cudaStream_t s) {
    auto rows = [&](int cs) { return (maxM + 32 * cs - 1) / (32 * cs) * 32; };
    int cs = 1;
    while (cs < kOrMaxCluster && (orth_smem(rows(cs)) > 110 * 1024 || (n * (cs + 1) <= 152 && rows(cs + 1) >= 64))) ++cs;
    const size_t smem = orth_smem(rows(cs));
    const cudaError_t e = allow_smem(range_orth_kernel);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n * cs);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, range_orth_kernel, tiles, list, c0, nc, cs, rows(cs));
}

// ---- the range by a pivoted QR ---------------------------------------------------
__device__ __forceinline__ double wsum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(256) qrcp_kernel(const QrcpTask *tasks, int *k_out,
                                                   int *st_out) {
    extern __shared__ double v[];  // the current reflector (rows j..M-1)
    __shared__ double r_sum[8], r_max[8];
    __shared__ int r_arg[8];
    __shared__ double s_sum, s_tau, s_scal, s_beta, s_delta2;
    __shared__ int s_piv;
    const QrcpTask t = tasks[blockIdx.x];
    const int M = t.M, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *W = t.W;
    bool bad = false;
    for (long long e = tid; e < (long long)M * M; e += 256) {
        const int i = (int)(e % M), j = (int)(e / M);
        const double x = t.D[(size_t)j * t.ldd + i];
        bad = bad || !isfinite(x);
        W[e] = x;
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) {
            k_out[blockIdx.x] = 0;
            st_out[blockIdx.x] = HCORE_GPU_S_NOCONV;
        }
        return;
    }
    for (int l = warp; l < M; l += 8) {
        const double *col = W + (size_t)l * M;
        double s = 0.0;
        for (int i = lane; i < M; i += 32) s += col[i] * col[i];
        s = wsum_d(s);
        if (lane == 0) t.vn[l] = s;
    }
    for (int l = tid; l < M; l += 256) t.perm[l] = l;
    __syncthreads();
    int k = 0, st = HCORE_GPU_S_OK;
    for (int j = 0;; ++j) {
        // remaining Frobenius norm^2 and the pivot (largest trailing norm,
        // lowest index on ties)
        double sum = 0.0, best = -1.0;
        int arg = j;
        for (int l = j + tid; l < M; l += 256) {
            const double x = t.vn[l];
            sum += x;
            if (x > best) { best = x; arg = l; }
        }
        sum = wsum_d(sum);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
        }
        if (lane == 0) { r_sum[warp] = sum; r_max[warp] = best; r_arg[warp] = arg; }
        __syncthreads();
        if (tid == 0) {
            double s = 0.0, b = -1.0;
            int a = j;
            for (int w = 0; w < 8; ++w) {
                s += r_sum[w];
                if (r_max[w] > b || (r_max[w] == b && r_arg[w] < a)) { b = r_max[w]; a = r_arg[w]; }
            }
            if (j == 0) {
                // truncation threshold: acc, or acc * sigma_max with
                // sigma_max >= ||D||_F / sqrt(M); delta 1e-3 of it, at
                // least 64 eps ||D||_F (what the arithmetic can resolve)
                const double thr = t.relative ? t.acc * sqrt(s / M) : t.acc;
                const double d1 = 1e-3 * thr, d2 = 64.0 * 2.220446049250313e-16 * sqrt(s);
                s_delta2 = fmax(d1 * d1, d2 * d2);
            }
            s_sum = s;
            s_piv = a;
        }
        __syncthreads();
        if (s_sum <= s_delta2) { k = j; break; }
        if (j >= t.kcap || j >= M) { k = j; st = HCORE_GPU_S_RANK_MAX; break; }
        const int p = s_piv;
        if (p != j) {
            double *cj = W + (size_t)j * M, *cp = W + (size_t)p * M;
            for (int i = tid; i < M; i += 256) {
                const double x = cj[i];
                cj[i] = cp[i];
                cp[i] = x;
            }
            if (tid == 0) {
                const double x = t.vn[j]; t.vn[j] = t.vn[p]; t.vn[p] = x;
                const int q = t.perm[j]; t.perm[j] = t.perm[p]; t.perm[p] = q;
            }
        }
        __syncthreads();
        // reflector of W[j:M, j] (dlarfg conventions: beta = -sign(alpha) ||x||)
        double *cj = W + (size_t)j * M;
        double xs = 0.0;
        for (int i = j + 1 + tid; i < M; i += 256) xs += cj[i] * cj[i];
        xs = wsum_d(xs);
        if (lane == 0) r_sum[warp] = xs;
        __syncthreads();
        if (tid == 0) {
            double x2 = 0.0;
            for (int w = 0; w < 8; ++w) x2 += r_sum[w];
            const double alpha = cj[j];
            if (x2 == 0.0) {
                s_tau = 0.0; s_scal = 0.0; s_beta = alpha;
            } else {
                const double beta = -copysign(sqrt(alpha * alpha + x2), alpha);
                s_tau = (beta - alpha) / beta;
                s_scal = 1.0 / (alpha - beta);
                s_beta = beta;
            }
            t.tau[j] = s_tau;
        }
        __syncthreads();
        for (int i = j + tid; i < M; i += 256) {
            const double x = i == j ? 1.0 : cj[i] * s_scal;
            v[i] = x;
            cj[i] = i == j ? s_beta : x;
        }
        __syncthreads();
        // apply H = I - tau v v^T to the trailing columns; their norms below
        // row j come out of the same pass
        const double tau = s_tau;
        for (int l = j + 1 + warp; l < M; l += 8) {
            double *col = W + (size_t)l * M;
            double nrm = 0.0;
            if (tau != 0.0) {
                double dot = 0.0;
                for (int i = j + lane; i < M; i += 32) dot += v[i] * col[i];
                const double s = tau * wsum_d(dot);
                for (int i = j + lane; i < M; i += 32) {
                    const double y = col[i] - s * v[i];
                    col[i] = y;
                    if (i > j) nrm += y * y;
                }
            } else {
                for (int i = j + 1 + lane; i < M; i += 32) nrm += col[i] * col[i];
            }
            nrm = wsum_d(nrm);
            if (lane == 0) t.vn[l] = nrm;
        }
        __syncthreads();
    }
    if (tid == 0) {
        k_out[blockIdx.x] = k;
        st_out[blockIdx.x] = st;
    }
}

// UA = Q1 = H_0 ... H_{k-1} [I_k; 0] (dorg2r: a warp per column, reflectors
// applied last to first), VB = P R~^T with R~ the first k rows of the
// factored tile (upper trapezoidal).
__global__ void __launch_bounds__(256) compress_form_kernel(const FormWork *work) {
    const FormWork f = work[blockIdx.x];
    const int M = f.M, k = f.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (f.Q) {
        for (long long e = tid; e < (long long)M * k; e += 256) {
            f.UA[e] = f.Q[e];
            f.VB[e] = f.B[e];
        }
        return;
    }
    for (long long e = tid; e < (long long)M * k; e += 256) {
        const int l = (int)(e % M), i = (int)(e / M);
        f.VB[(size_t)i * M + f.perm[l]] = i <= l ? f.W[(size_t)l * M + i] : 0.0;
    }
    for (int c = warp; c < k; c += 8) {
        double *x = f.UA + (size_t)c * M;
        for (int i = lane; i < M; i += 32) x[i] = i == c ? 1.0 : 0.0;
        __syncwarp();
        for (int h = c; h >= 0; --h) {  // H_h with h > c leaves e_c unchanged
            const double th = f.tau[h];
            if (th == 0.0) continue;
            const double *vh = f.W + (size_t)h * M;  // v_h[h] = 1, below it W
            double dot = 0.0;
            for (int i = h + lane; i < M; i += 32) dot += (i == h ? 1.0 : vh[i]) * x[i];
            const double s = th * wsum_d(dot);
            for (int i = h + lane; i < M; i += 32) x[i] -= s * (i == h ? 1.0 : vh[i]);
            __syncwarp();
        }
    }
}


static size_t al256c(size_t x) { return (x + 255) & ~(size_t)255; }

// Which tiles take the range finder, and its widest range: smaller tiles (and
// wider ranges) are cheap for (need) the pivoted QR.
constexpr int kRangeMinM = 128, kRangeMaxK = 256;
static int range_cap(int M) { return M < kRangeMinM ? 0 : std::min(kRangeMaxK, M / 2 / 32 * 32); }

// The range of tiles [0, nt) by products: blocks of columns Y = E Omega (random
// test vectors), orthonormalised to Q_i, B_i = E^T Q_i, E <- E - Q_i B_i^T until
// ||E||_F <= kRangeShare * delta (the blocked scheme of Martinsson and Voronin,
// "A randomized blocked algorithm for efficiently computing rank-revealing
// factorizations of matrices", 2016; the residual is formed, so what is found
// does not depend on chance, only how soon).  k[q] becomes the columns found;
// -1 leaves the tile to the pivoted QR (not finite, out of the range of squares,
// or wider than its cap).
static cudaError_t find_ranges(int nt, const RangeTile *tiles, const hcore_compress_task *const *tasks,
                               const RangeTile *d_tiles, int maxM, std::vector<int> &k, cudaStream_t s) {
    k.assign(nt, -1);
    if (nt == 0) return cudaSuccess;
    std::vector<int> active(nt);
    for (int q = 0; q < nt; ++q) active[q] = q;
    char *buf = nullptr;   // list, partial sums, test vectors
    const size_t b_list = al256c(nt * sizeof(int)), b_part = al256c((size_t)nt * kSumParts * sizeof(double));
    cudaError_t e = cudaMalloc(&buf, b_list + b_part + (size_t)maxM * 32 * sizeof(double));
    if (e != cudaSuccess) return e;
    int *d_list = (int *)buf;
    double *d_part = (double *)(buf + b_list), *d_omega = (double *)(buf + b_list + b_part);
    std::vector<double> part((size_t)nt * kSumParts), limit(nt);
    int *word = thread_ctx().wait_word();
    if (!word) {
        cudaFree(buf);
        return cudaErrorMemoryAllocation;
    }
    auto norms = [&](bool load) -> cudaError_t {
        cudaError_t r = cudaMemcpyAsync(d_list, active.data(), active.size() * sizeof(int),
                                        cudaMemcpyHostToDevice, s);
        if (r == cudaSuccess) {
            range_norm_kernel<<<dim3((unsigned)active.size(), kSumParts), 256, 0, s>>>(d_tiles, d_list, load,
                                                                                       d_part);
            r = cudaGetLastError();
        }
        if (r == cudaSuccess)
            r = cudaMemcpyAsync(part.data(), d_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, s);
        if (r == cudaSuccess) r = cudaStreamSynchronize(s);
        // a product whose wait gave up left NaN: an error, not a tile for the pivoted QR
        return r == cudaSuccess && *(volatile int *)word ? cudaErrorLaunchTimeout : r;
    };
    auto sum_of = [&](int q) {
        double x = 0.0;
        for (int y = 0; y < kSumParts; ++y) x += part[(size_t)q * kSumParts + y];
        return x;
    };
    char *arena = nullptr;
    size_t arena_bytes = 0;
    std::vector<char> host;
    // run a list of products: upload its layout and launch it
    auto products = [&](DenseProducts &p) -> cudaError_t {
        size_t up = 0;
        p.place_host(up);
        size_t all = up;
        p.place_device(all);
        if (all > arena_bytes) {
            cudaError_t r = cudaStreamSynchronize(s);
            cudaFree(arena);
            arena = nullptr;
            arena_bytes = 0;
            if (r == cudaSuccess) r = cudaMalloc(&arena, all);
            if (r != cudaSuccess) return r;
            arena_bytes = all;
        }
        host.resize(up);
        p.pack(host.data());
        p.gave_up = word;
        // (from pageable memory: the copy has left `host` when it returns)
        const cudaError_t r = cudaMemcpyAsync(arena, host.data(), up, cudaMemcpyHostToDevice, s);
        return r == cudaSuccess ? p.launch(arena, s) : r;
    };
    e = configure_dense_tc();
    if (e == cudaSuccess) e = norms(true);
    std::vector<int> found(nt, 0);
    for (int c0 = 0; e == cudaSuccess;) {
        // tiles that are done, refused or full leave the list
        std::vector<int> next;
        for (int q : active) {
            const hcore_compress_task &t = *tasks[q];
            const double x = sum_of(q);
            if (c0 == 0) {
                if (!(x == 0.0 || (x > 1e-280 && x < 1e280))) continue;
                const double d = kRangeShare * range_delta(sqrt(x), t.M, t.relative != 0, t.acc);
                limit[q] = d * d;
            }
            if (!(x <= limit[q])) {
                if (found[q] + 16 <= range_cap(t.M)) next.push_back(q);
            } else {
                k[q] = found[q];
            }
        }
        active.swap(next);
        if (active.empty()) break;
        // 32 columns (a tile's width in the products) at first; 16 later, where a
        // wider core costs the SVD more than another block costs here
        const int nc = c0 < 64 ? 32 : 16;
        range_test_vectors_kernel<<<(maxM * nc + 255) / 256, 256, 0, s>>>(d_omega, maxM * nc, c0 * maxM);
        DenseProducts y, b;
        y.slice_limit = b.slice_limit = (size_t)384 << 20;   // few tiles a product: fill the GPU instead
        y.stage(kNoBalance);
        using DP = DenseProducts;
        for (int q : active) {
            const RangeTile &t = tiles[q];
            y.add_one(DP::product(t.E, t.M, d_omega, maxM, 2, t.M, 1.0, 0.0), t.M, nc, t.Q + (size_t)c0 * t.M, t.M);
        }
        b.stage(kNoBalance);
        for (int q : active) {
            const RangeTile &t = tiles[q];
            b.add_one(DP::product(t.E, t.M, t.Q + (size_t)c0 * t.M, t.M, 3, t.M, 1.0, 0.0), t.M, nc,
                      t.B + (size_t)c0 * t.M, t.M);
        }
        b.stage(kNoBalance);
        for (int q : active) {
            const RangeTile &t = tiles[q];
            b.add_one(DP::product(t.Q + (size_t)c0 * t.M, t.M, t.B + (size_t)c0 * t.M, t.M, 0, nc, -1.0, 1.0), t.M,
                      t.M, t.E, t.M);
        }
        e = products(y);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(d_list, active.data(), active.size() * sizeof(int), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) {
            e = launch_range_orth(d_tiles, d_list, (int)active.size(), c0, nc, maxM, s);
        }
        // (both lists use one arena: the second's layout is copied after the
        // first's launches in stream order)
        if (e == cudaSuccess) e = products(b);
        c0 += nc;
        for (int q : active) found[q] = c0;
        if (e == cudaSuccess) e = norms(false);
    }
    cudaStreamSynchronize(s);
    cudaFree(arena);
    cudaFree(buf);
    return e;
}

// Compress tasks [0, n) (device-accessible pointers, validated) in chunks
// whose QR workspaces fit `budget` bytes.
static int run_compress(int n, const hcore_compress_task *tasks, int *ranks, int *status,
                        cudaStream_t s) {
    const size_t budget = (size_t)4 << 30;
    int i0 = 0;
    while (i0 < n) {
        // chunk [i0, i1)
        size_t bytes = 0;
        int i1 = i0;
        while (i1 < n) {
            const size_t M = tasks[i1].M;
            const size_t need = al256c(M * M * 8) + 3 * al256c(M * 8) + al256c(kMaxK * 8) +
                                2 * al256c(M * range_cap((int)M) * 8);
            if (i1 > i0 && bytes + need > budget) break;
            bytes += need;
            ++i1;
        }
        const int nc = i1 - i0;
        std::vector<QrcpTask> qt(nc);
        std::vector<RangeTile> rt;
        std::vector<const hcore_compress_task *> rtask;
        std::vector<int> rq;   // the range finder's tiles
        char *qa = nullptr;
        const size_t b_qt = al256c(nc * sizeof(QrcpTask)), b_rt = al256c(nc * sizeof(RangeTile));
        const size_t b_meta = b_qt + b_rt + 2 * al256c(nc * sizeof(int));
        if (cudaMalloc(&qa, bytes + b_meta) != cudaSuccess) {
            cudaGetLastError();
            set_error("hcore_gpu_compress_batched: cudaMalloc of %zu bytes failed", bytes + b_meta);
            return HCORE_GPU_ENOMEM;
        }
        char *p = qa + b_meta;
        int maxM = 1, rangeM = 1;
        for (int q = 0; q < nc; ++q) {
            const hcore_compress_task &t = tasks[i0 + q];
            QrcpTask &u = qt[q];
            const size_t M = t.M;
            u.D = t.D; u.ldd = t.ldd; u.M = t.M; u.acc = t.acc; u.relative = t.relative;
            u.kcap = std::min(t.M, kMaxK);
            u.W = (double *)p; p += al256c(M * M * 8);
            u.vn = (double *)p; p += al256c(M * 8);
            u.perm = (int *)p; p += al256c(M * 8);
            p += al256c(M * 8);
            u.tau = (double *)p; p += al256c(kMaxK * 8);
            maxM = std::max(maxM, t.M);
            // (without a threshold every column of the range counts: the pivoted QR
            // finds no more of them than there are)
            if (const int cap = t.acc > 0.0 ? range_cap(t.M) : 0) {
                RangeTile r{t.D, t.ldd, t.M, u.W, (double *)p, nullptr};
                p += al256c(M * cap * 8);
                r.B = (double *)p; p += al256c(M * cap * 8);
                rt.push_back(r);
                rtask.push_back(&t);
                rq.push_back(q);
                rangeM = std::max(rangeM, t.M);
            }
        }
        QrcpTask *d_qt = (QrcpTask *)qa;
        RangeTile *d_rt = (RangeTile *)(qa + b_qt);
        int *d_k = (int *)(qa + b_qt + b_rt);
        int *d_st = d_k + al256c(nc * sizeof(int)) / sizeof(int);
        cudaError_t e = cudaSuccess;
        if (!rt.empty())
            e = cudaMemcpyAsync(d_rt, rt.data(), rt.size() * sizeof(RangeTile), cudaMemcpyHostToDevice, s);
        std::vector<int> rk, hk(nc, -1), hst(nc, HCORE_GPU_S_OK), slot(nc, -1);
        if (e == cudaSuccess) e = find_ranges((int)rt.size(), rt.data(), rtask.data(), d_rt, rangeM, rk, s);
        // the tiles it did not take: the pivoted QR
        std::vector<QrcpTask> rest;
        std::vector<int> rest_q;
        if (e == cudaSuccess) {
            for (size_t x = 0; x < rq.size(); ++x) {
                hk[rq[x]] = rk[x];
                slot[rq[x]] = (int)x;
            }
            for (int q = 0; q < nc; ++q)
                if (hk[q] < 0) {
                    rest.push_back(qt[q]);
                    rest_q.push_back(q);
                    slot[q] = -1;
                }
        }
        const int nq = (int)rest.size();
        if (e == cudaSuccess && nq > 0) {
            std::vector<int> k1(nq), st1(nq);
            const size_t smem = (size_t)maxM * sizeof(double);
            e = cudaMemcpyAsync(d_qt, rest.data(), nq * sizeof(QrcpTask), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) {   // (at most 16 KB of shared memory)
                qrcp_kernel<<<nq, 256, smem, s>>>(d_qt, d_k, d_st);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) e = cudaMemcpyAsync(k1.data(), d_k, nq * sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaMemcpyAsync(st1.data(), d_st, nq * sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            for (int x = 0; x < nq && e == cudaSuccess; ++x) {
                hk[rest_q[x]] = k1[x];
                hst[rest_q[x]] = st1[x];
            }
        }
        if (e == cudaErrorLaunchTimeout && thread_ctx().word && *(volatile int *)thread_ctx().word) {
            cudaFree(qa);
            return check_waits(thread_ctx().word, "hcore_gpu_compress_batched");
        }
        if (e != cudaSuccess) {
            set_error("hcore_gpu_compress_batched: %s", cudaGetErrorString(e));
            cudaFree(qa);
            if (e == cudaErrorMemoryAllocation) {
                cudaGetLastError();
                return HCORE_GPU_ENOMEM;
            }
            return HCORE_GPU_ECUDA;
        }
        // the plan phases for the tiles with a range of k >= 1 columns,
        // sorted by decreasing k (rank buckets)
        std::vector<int> order;
        for (int q = 0; q < nc; ++q) {
            ranks[i0 + q] = 0;
            status[i0 + q] = hst[q];
            if (hst[q] == HCORE_GPU_S_OK && hk[q] > 0) order.push_back(q);
        }
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return hk[a] > hk[b]; });
        const int nd = (int)order.size();
        if (nd > 0) {
            std::vector<Desc> descs(nd);
            std::vector<FormWork> fw(nd);
            long long ws = 0;
            int maxK = 1, pM = 1;
            for (int x = 0; x < nd; ++x) {
                const int q = order[x];
                const hcore_compress_task &t = tasks[i0 + q];
                Desc &d = descs[x];
                d = Desc{};
                d.M = t.M; d.a = 0; d.b = 0; d.c = hk[q]; d.k = hk[q];
                d.alpha = 1.0; d.beta = 1.0; d.acc = t.acc;
                d.CUo = t.U; d.CVo = t.V; d.ldco = t.ldo;
                d.rk = 0; d.max_rank = std::max(t.maxrank, 0); d.storage_rank = INT_MAX;
                d.rank_start = 0;
                d.rule = kRuleCapRank | (t.relative ? kRuleRelative : 0) |
                         (slot[q] >= 0 ? kRuleRange : 0);
                d.status0 = 0;
                d.idx = i0 + q;
                d.ws = ws;
                ws += ws_layout(d).total;
                maxK = std::max(maxK, d.k);
                pM = std::max(pM, d.M);
            }
            double *pws = nullptr;
            char *pa = nullptr;
            const size_t b_desc = al256c(nd * sizeof(Desc)), b_fw = al256c(nd * sizeof(FormWork));
            const size_t b_rs = al256c((size_t)n * sizeof(int));
            if (cudaMalloc(&pa, b_desc + b_fw + 2 * b_rs + al256c((size_t)ws * 8)) != cudaSuccess) {
                cudaGetLastError();
                cudaFree(qa);
                set_error("hcore_gpu_compress_batched: cudaMalloc of the plan workspace failed");
                return HCORE_GPU_ENOMEM;
            }
            Desc *d_desc = (Desc *)pa;
            FormWork *d_fw = (FormWork *)(pa + b_desc);
            int *d_rank = (int *)(pa + b_desc + b_fw);
            int *d_status = (int *)(pa + b_desc + b_fw + b_rs);
            pws = (double *)(pa + b_desc + b_fw + 2 * b_rs);
            for (int x = 0; x < nd; ++x) {
                const int q = order[x];
                const WsLayout L = ws_layout(descs[x]);
                const RangeTile *r = slot[q] >= 0 ? &rt[slot[q]] : nullptr;
                fw[x] = FormWork{qt[q].W, qt[q].tau, qt[q].perm, pws + descs[x].ws + L.UA,
                                 pws + descs[x].ws + L.VB, descs[x].M, descs[x].k,
                                 r ? r->Q : nullptr, r ? r->B : nullptr};
            }
            LaunchShape shape;
            shape.maxM = pM;
            shape.maxK = maxK;
            shape.updates = shape.big_updates = nd;
            fill_buckets(descs, shape);
            e = cudaMemcpyAsync(d_desc, descs.data(), nd * sizeof(Desc), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(d_fw, fw.data(), nd * sizeof(FormWork), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) {
                compress_form_kernel<<<nd, 256, 0, s>>>(d_fw);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) e = configure_recompress<double>(maxK, &shape.svd_smem_kmax);
            if (e == cudaSuccess)
                e = launch_recompress<double>(d_desc, nd, pws, d_rank, d_status, nullptr, shape, s,
                                              kPhaseQR | kPhaseSVD | kPhaseApply);
            std::vector<int> hr(n), hs(n);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(hr.data(), d_rank, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(hs.data(), d_status, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            cudaFree(pa);
            if (e != cudaSuccess) {
                cudaFree(qa);
                set_error("hcore_gpu_compress_batched: %s", cudaGetErrorString(e));
                return HCORE_GPU_ECUDA;
            }
            for (int x = 0; x < nd; ++x) {
                const int u = descs[x].idx;
                ranks[u] = hr[u];
                status[u] = hs[u];
            }
        }
        cudaFree(qa);
        i0 = i1;
    }
    return HCORE_GPU_OK;
}

}  // namespace hc

using namespace hc;

extern "C" int hcore_gpu_compress_batched(int n, const hcore_compress_task *tasks, int *ranks,
                                          int *status, void *stream) {
    if (n < 0 || (n > 0 && (!tasks || !ranks || !status))) {
        set_error("hcore_gpu_compress_batched: invalid argument");
        return HCORE_GPU_EINVAL;
    }
    std::vector<hcore_compress_task> tt(tasks, tasks + n);
    for (int i = 0; i < n; ++i) {
        hcore_compress_task &t = tt[i];
        if (t.M < 1 || t.M > kMaxRowsPerLane * 32 || t.ldd < t.M || t.ldo < t.M ||
            !(t.acc >= 0.0) || t.maxrank < 0) {
            set_error("hcore_gpu_compress_batched: invalid task %d", i);
            return HCORE_GPU_EINVAL;
        }
        t.D = (const double *)device_alias(t.D);
        t.U = (double *)device_alias(t.U);
        t.V = (double *)device_alias(t.V);
        if (!t.D || !t.U || !t.V) {
            set_error("hcore_gpu_compress_batched: pointers must be device or pinned memory");
            return HCORE_GPU_EINVAL;
        }
    }
    const int rc = run_compress(n, tt.data(), ranks, status, (cudaStream_t)stream);
    if (rc) return rc;
    for (int i = 0; i < n; ++i)
        if (status[i]) return HCORE_GPU_ETASK;
    return HCORE_GPU_OK;
}
