// hcore-gb300 — dense-C tile updates on sm_103a:
//   HCORE_dsyrk   (src/compute/hcore_dsyrk.c:47-189)
//       CD = alpha * AU (AV^T AV) AU^T + CD, strict upper triangle := 0
//   HCORE_dgemmcd (src/compute/hcore_dgemmcd.c:36-106)
//       CD = CD - Au (Av^T Bv) Bu^T (associated by the smaller rank, :72)
//   HCORE_duncompress (src/compute/hcore_duncompress.c:33-84)
//       CD = AU BV^T
//   HCORE_dgemmbdcd (src/compute/hcore_dgemmbdcd.c:35-122)
//       CD = alpha AU (AV^T BD) + beta CD
//   HCORE_dgemm_dense (src/compute/hcore_dgemm.c:1701-1715)
//       C = alpha op(A) op(B) + beta C
//
// Every contribution is first reduced to a rank-K' product beta CD +
// coef * P Q^T with P of size M x K' and Q of size N x K' (syrk and gemmcd: the
// kernels below; gemmbdcd's Q = BD^T AV is a product of the next kind itself;
// uncompress needs none), and all tasks that hit the same tile are then
// applied in list order on the tensor cores (hc_dense_tc.cu).  Zeroing
// the strict upper triangle where a run of syrk tasks ends is the reference's
// sequential semantics; the syrk's own products strictly above the diagonal
// are not computed since they are overwritten by zero.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "hc_internal.h"

namespace hc {

// A task's inner product S = X^T Y (p x q over n rows): AV^T AV over lda rows
// for syrk (hcore_dsyrk.c:57,103), Av^T Bv over M rows for gemmcd
// (hcore_dgemmcd.c:66-70); then the factor that it makes:
//   syrk:                       P = AU S                 (M x a)
//   gemmcd, a > b:              P = Au S                 (M x b)
//   gemmcd, a <= b:             Q = Bu S^T               (M x a)
//
// Both kernels are bound by FP64 issue (one warp instruction per 64 cycles and
// sub-partition), so what was saved is instructions: a warp takes four entries
// of S at a time, whose sums are reduced together (6 shuffled additions
// instead of 20 beside 4 M / 32 FMAs), and syrk's S is formed on and above the
// diagonal only.  Tasks are split over CTAs (entries of S, rows of the factor)
// so that uneven ranks and short lists fill the GPU.  768 tasks of ranks 8-32,
// M = 1024: 2097 us in one kernel of a CTA per task, 825 + 723 us in these two.
// Long lists form the factors as products on the tensor cores instead (DensePrep).
__global__ void __launch_bounds__(256) dense_inner_kernel(const hcore_dense_task *tasks,
                                                          const DenseWork *work, double *ws) {
    const hcore_dense_task t = tasks[blockIdx.x];
    if (t.kind > 1) return;  // uncompress: no prep; gemmbdcd: its own product
    double *S = ws + work[blockIdx.x].ws;
    const bool syrk = t.kind == 0;
    const double *X = t.Av, *Y = syrk ? t.Av : t.Bv;
    const int p = t.a, q = syrk ? t.a : t.b, n = syrk ? t.lda : t.M;
    const int lane = threadIdx.x & 31, warp = blockIdx.y * 8 + (threadIdx.x >> 5);
    const int quads = (p + 3) / 4;
    for (int e = warp; e < quads * q; e += gridDim.y * 8) {
        const int i0 = e % quads * 4, j = e / quads;
        if (syrk && i0 > j) continue;
        const double *y = Y + (size_t)j * n;
        const double *x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = X + (size_t)min(i0 + u, p - 1) * n;
        double s[4] = {};
#pragma unroll 2
        for (int l = lane; l < n; l += 32) {
            const double yv = y[l];
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += x[u][l] * yv;
        }
        // lanes 8 u .. 8 u + 7 end with sum u
        const bool h16 = lane & 16, h8 = lane & 8;
        double a = (h16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, h16 ? s[0] : s[2], 16);
        double b = (h16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, h16 ? s[1] : s[3], 16);
        double c = (h8 ? b : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        const int i = i0 + (lane >> 3);
        if ((lane & 7) == 0 && i < p && (!syrk || i <= j)) {
            S[(size_t)j * p + i] = c;
            if (syrk) S[(size_t)i * p + j] = c;
        }
    }
}

// out(i, j) = sum_l F(i, l) S'(l, j), a thread per row, four columns at a time
__global__ void __launch_bounds__(128) dense_factor_kernel(const hcore_dense_task *tasks,
                                                           const DenseWork *work, double *ws) {
    const hcore_dense_task t = tasks[blockIdx.x];
    if (t.kind > 1) return;
    const int i = blockIdx.y * 128 + threadIdx.x;
    if (i >= t.M) return;
    const bool syrk = t.kind == 0, left = syrk || t.a > t.b;
    const int p = t.a, q = syrk ? t.a : t.b;
    const double *S = ws + work[blockIdx.x].ws;
    double *out = ws + work[blockIdx.x].ws + (size_t)p * q;
    // S'(l, j) = S(l, j), or S(j, l) for Bu S^T
    const double *F = (left ? t.Au : t.Bu) + i;
    const size_t ldf = syrk ? t.lda : t.M;
    const int inner = left ? p : q, cols = left ? q : p;
    const size_t sl = left ? 1 : p, sj = left ? p : 1;
    for (int j = 0; j < cols; j += 4) {
        double s[4] = {};
        const double *b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = S + (size_t)min(j + u, cols - 1) * sj;
#pragma unroll 4
        for (int l = 0; l < inner; ++l) {
            const double f = F[(size_t)l * ldf];
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += f * b[u][(size_t)l * sl];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u < cols) out[(size_t)(j + u) * t.M + i] = s[u];
    }
}


cudaError_t launch_dense_prep(const hcore_dense_task *d_tasks, const DenseWork *d_work, int n,
                              int maxM, bool factors, double *ws, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    // about four CTAs an SM and more: a task's entries over up to eight CTAs
    const int split = std::max(1, std::min(8, 1216 / n));
    dense_inner_kernel<<<dim3(n, split), 256, 0, s>>>(d_tasks, d_work, ws);
    if (factors) dense_factor_kernel<<<dim3(n, (maxM + 127) / 128), 128, 0, s>>>(d_tasks, d_work, ws);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// plain dense GEMM, C = alpha op(A) op(B) + beta C (HCORE_dgemm_dense)
// ---------------------------------------------------------------------------
// Tiles of 64 x 64: thread (tx, ty) owns a 4 x 4 register block; the inner
// dimension is staged in chunks of 16 through shared memory.
constexpr int TB = 64, TK = 16;
template <typename T>
__global__ void __launch_bounds__(256) gemm_dense_kernel(int ta, int tb, int M, int N, int K,
                                                         T alpha, const T *A, int lda, const T *B,
                                                         int ldb, T beta, T *C, int ldc) {
    __shared__ T sA[TK][TB + 1];
    __shared__ T sB[TK][TB + 1];
    const int row0 = blockIdx.x * TB, col0 = blockIdx.y * TB;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    T acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += TK) {
        for (int e = threadIdx.x; e < TK * TB; e += 256) {
            const int kk = e / TB, r = e % TB;
            const int kg = k0 + kk, i = row0 + r, j = col0 + r;
            T av = 0, bv = 0;
            if (kg < K && i < M) av = ta ? A[(size_t)i * lda + kg] : A[(size_t)kg * lda + i];
            if (kg < K && j < N) bv = tb ? B[(size_t)kg * ldb + j] : B[(size_t)j * ldb + kg];
            sA[kk][r] = av;
            sB[kk][r] = bv;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            T pv[4], qv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) pv[u] = sA[kk][tx + 16 * u];
#pragma unroll
            for (int v = 0; v < 4; ++v) qv[v] = sB[kk][ty + 16 * v];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] += pv[u] * qv[v];
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int i = row0 + tx + 16 * u, j = col0 + ty + 16 * v;
            if (i < M && j < N) {
                T *c = C + (size_t)j * ldc + i;
                *c = alpha * acc[u][v] + (beta == T(0) ? T(0) : beta * *c);
            }
        }
}

template <typename T>
cudaError_t launch_gemm_dense(int ta, int tb, int M, int N, int K, T alpha, const T *A, int lda,
                              const T *B, int ldb, T beta, T *C, int ldc, cudaStream_t s) {
    if (M <= 0 || N <= 0) return cudaSuccess;
    dim3 grid((M + TB - 1) / TB, (N + TB - 1) / TB);
    gemm_dense_kernel<T><<<grid, 256, 0, s>>>(ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    return cudaGetLastError();
}
template cudaError_t launch_gemm_dense<double>(int, int, int, int, int, double, const double *, int,
                                               const double *, int, double, double *, int,
                                               cudaStream_t);
template cudaError_t launch_gemm_dense<float>(int, int, int, int, int, float, const float *, int,
                                              const float *, int, float, float *, int, cudaStream_t);

}  // namespace hc
