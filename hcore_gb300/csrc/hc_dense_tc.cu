// hcore-gb300: the dense-C tile updates' products on the tensor cores,
// FP64-accurate.
//
// hc_dense.cu reduces every task (HCORE_dsyrk, HCORE_dgemmcd, HCORE_duncompress,
// HCORE_dgemmbdcd) to CD = beta CD + coef P Q^T with P of M x K' and Q of
// N x K'.  The tasks on one tile are laid one after the other along K: the
// tile then takes one product per chunk of up to 128 columns, whatever tasks
// they come from, as exact digit products (hc_digits.cuh) in tensor-memory
// accumulators, combined in 64-bit integers and added to CD in FP64 once per
// chunk.  A chunk ends where a later task scales CD (beta != 1) and where
// syrk tasks, which leave the strict upper triangle zero, change to others.
//
// Scales.  Column l of a task is balanced first: P's column takes 2^-s_l and
// Q's 2^s_l, s_l half the difference of their largest exponents, so that only
// the size of a column's product matters, as in an FP64 sum.  Then each row of
// P and of Q takes one power of two per chunk.  The error per term is 2^-55 of
// the largest product of a row of P with a row of Q.  A NaN or an infinity in
// a row of P or Q sends the entries it reaches to an FP64 loop, so they come
// out as in IEEE arithmetic.
//
// Entries of graded rows.  Where a row's large entries meet small ones of the other
// row only, an entry's terms are all far below the product of the two scales, and
// 2^-55 of that product may be all of the entry.  So each row notes which columns are
// within 2^-kNear of its top; an entry whose rows share such a column has a term of
// 2^-(2 kNear + 2) of the scales at least, and its error is below (1.25 K + 1) 2^-45 of the
// sum of its terms' magnitudes; so it is if the result or CD's entry is that large.
// The others, 2e-6 of the entries of low-rank updates with singular values over 16
// decades (1e-4 with kNear = 3), are summed in FP64.  Stages without balance are left
// out (kNoBalance): the compressor's products only have to be small in norm, and a
// Cholesky factorization's backward error is relative to sqrt(a_ii a_jj), the rows'
// scales, in FP64 too (of a covariance tile two thirds of the entries would be slow).
// Cost: 12 gemmbdcd tasks of 777 x 650 x 900 482 -> 500 us, 32 tiles of 1024 with 24
// updates each 2595 -> 2752, the factorization and solves of 8 tiles of 1024 with 12
// factors each 4279 -> 4370; 4094 updates of covariance tiles, whose singular vectors
// fall by many decades from point to point, so that most entries of the factors AU S
// are slow, 10.2 -> 12.0 ms (the factors 2.4 of them, as long as in FP64 alone).
//
// Measured on one GB300 (tiles and their preparation): 384 products of 1024 x
// 1024 x 17 21.9 -> 2.56 ms (3.2 GB written: 1.3 TB/s), 32 tiles of 1024 with
// 24 syrk or gemmcd updates each of ranks 8-32 25.9 -> 2.75 ms, 12 gemmbdcd
// tasks of 777 x 650 x 900, rank 40, 1.77 -> 0.50 ms; one 32 x 32 x 4 product
// alone 25 -> 19 us (so no size keeps the FP64 kernel that this replaced).
//
// What bounds it.  In FP64 a term costs 1/2 clock of an SM (the FP64 pipe), so
// a rank-24 product is 12 clocks an entry.  Here an entry costs one FP64
// addition per chunk and about 70 integer instructions (0.55 clocks); the MMAs
// of a chunk are 7 per 16 columns (N = 256, 90 clocks each: 0.15 clocks an
// entry and 16 columns).  Slicing a value into its seven digits takes some 60
// instructions, so it is not done by the CTAs that use it: a kernel of its own
// writes the slices in the MMA's core-matrix layout, and a tile's CTA fetches
// a block (128 x 16 of P, 32 x 16 of Q, all seven slices contiguous) with one
// bulk copy each.  A tile is 128 x 32 entries (256 tensor-memory columns); two
// CTAs share an SM, so one drains while the other multiplies, and each runs
// many tiles, its producer one or more blocks ahead (a CTA per tile took 4.3 ms
// where this takes 2.56).  Sixteen worker warps a CTA, because a worker's chain
// (tensor-memory loads, integer combination, one store) is latency-bound: with
// eight it took 3.2 ms.  The slice buffer is kept below the L2's size by
// running the tiles in batches.
#include <cuda_runtime.h>

#include <climits>

#include "hc_digits.cuh"
#include "hc_internal.h"

namespace hc {
namespace {
using namespace dg;

constexpr int kRowsA = 128, kRowsB = 32, kKb = 16;   // block rows of P and Q, block columns
constexpr int kSliceA = kRowsA * kKb * 2, kSliceB = kRowsB * kKb * 2;
constexpr int kBlockA = 7 * kSliceA, kBlockB = 7 * kSliceB;
constexpr int kSbo = kKb / 8 * 128;                  // row-group stride inside a block
constexpr int kStages = 3;
constexpr int kStage = kBlockA + kBlockB + kSliceB;  // Q's eighth slice stays zero
constexpr int kMisc = 1024;                          // barriers, the units' ring
// the library's tensor-memory rule: at least 113 KB with 256 columns
constexpr int kSmem = 113 * 1024;
static_assert(kStages * kStage + kMisc <= kSmem, "shared memory of a tile's CTA");
constexpr int kWorkers = 512, kThreadsTc = kWorkers + 64;
constexpr int kTmem = 256;
// T = value 2^(110 - E_r - E_c - S), |value| < 128 2^(E_r + E_c): T < 2^62
constexpr int kShift = 55;
// Columns "near the top" of a row: scaled entry within kNear binades of the row's
// largest, among 32 columns of the chunk (those with the largest products, so that
// one word a row holds them).  An entry of the product whose rows share no such column
// is formed in FP64 if both the digits' result and CD's entry are below 2^-(2 kNear + 2)
// of the rows' scales (kFar, in T's units shifted by 32).  See the file comment.
constexpr int kNear = 4;
constexpr int kFarBits = kShift - 2 * kNear - 2, kFar = 1 << (kFarBits - 32);
constexpr int kNonFinite = INT_MAX / 4;   // (more than any sum of two other scales, less than INT_MAX)
constexpr int kSms = 152;
// blocks of a chunk's columns; a chunk without columns takes one of zeros
__host__ __device__ constexpr int dense_blocks(int ncol) { return ncol > 0 ? (ncol + kKb - 1) / kKb : 1; }

// balance of P's and Q's column l from their largest exponent fields (a warp per
// column), or of P's alone: 2^s brings its largest entry near 1; a zero column
// or one with a non-finite entry is left as it is
__global__ void __launch_bounds__(256) dense_balance_kernel(const DenseWork *work, const int2 *cols,
                                                            const int2 *dims, int n, bool p_only, int *shift,
                                                            int *mag) {
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= n) return;
    const int2 tl = cols[c], mn = dims[tl.x];
    const DenseWork w = work[tl.x];
    const bool tp = w.tr & 1, tq = w.tr & 2;
    const double *p = w.P + (tp ? (size_t)tl.y : (size_t)tl.y * w.ldp);
    const double *q = w.Q + (tq ? (size_t)tl.y : (size_t)tl.y * w.ldq);
    const size_t sp = tp ? w.ldp : 1, sq = tq ? w.ldq : 1;
    int ep = 0, eq = 0;
#pragma unroll 4
    for (int i = lane; i < mn.x; i += 32) ep = max(ep, exp_field(p[i * sp]));
#pragma unroll 4
    for (int i = lane; i < mn.y && !p_only; i += 32) eq = max(eq, exp_field(q[i * sq]));
    ep = __reduce_max_sync(0xffffffffu, ep);
    eq = __reduce_max_sync(0xffffffffu, eq);
    if (lane == 0) mag[c] = p_only ? 0 : ep + eq;
    if (lane == 0 && p_only) shift[c] = ep == 0 || ep == 0x7FF ? 0 : ep - 1023;
    else if (lane == 0) shift[c] = ep == 0 || eq == 0 || ep == 0x7FF || eq == 0x7FF ? 0 : (ep - eq) / 2;
}

// the same for operands stored transposed: a thread per column (64 a block,
// four threads each), so that the loads are coalesced
__global__ void __launch_bounds__(256) dense_balance_t_kernel(const DenseWork *work, const int2 *cols,
                                                              const int2 *dims, int n, int *shift, int *mag) {
    __shared__ int s_p[64], s_q[64];
    const int tid = threadIdx.x, lc = tid & 63, rg = tid >> 6, c = blockIdx.x * 64 + lc;
    if (tid < 64) s_p[tid] = s_q[tid] = 0;
    __syncthreads();
    if (c < n) {
        const int2 tl = cols[c], mn = dims[tl.x];
        const DenseWork w = work[tl.x];
        int ep = 0, eq = 0;
#pragma unroll 8
        for (int i = rg; i < mn.x; i += 4) ep = max(ep, exp_field(w.P[(size_t)i * w.ldp + tl.y]));
#pragma unroll 8
        for (int i = rg; i < mn.y; i += 4) eq = max(eq, exp_field(w.Q[(size_t)i * w.ldq + tl.y]));
        atomicMax(&s_p[lc], ep);
        atomicMax(&s_q[lc], eq);
    }
    __syncthreads();
    if (tid < 64 && c < n) {
        const int ep = s_p[tid], eq = s_q[tid];
        shift[c] = ep == 0 || eq == 0 || ep == 0x7FF || eq == 0x7FF ? 0 : (ep - eq) / 2;
        mag[c] = ep + eq;
    }
}

// the digit slices and row scales of one chunk's P (blockIdx.x < mb: 128 rows)
// or Q (the others: 128 rows, four blocks).  No FP64 instruction for a factor of 1
// or -1 (two comparisons and a product an element held the FP64 pipe 62% of the
// time), and the loads of 16 columns, then of the next eight, in flight together:
// the compressor's products of 48 tiles of order 1024 2.31 ms of slicing, 1.58 now;
// a panel of dense tiles 0.53, 0.23.  What is left is the latency of a block's two
// reads, then the 14 bytes an element that it writes.
__global__ void __launch_bounds__(256) dense_slice_kernel(const DenseWork *work, const int2 *cols,
                                                          const int *shift, const int *mag,
                                                          const DenseChunk *chunks, unsigned char *slices, int *exps,
                                                          unsigned *near_cols) {
    __shared__ __align__(16) int s_key[128];
    __shared__ int2 s_near[128];   // a column's shift, and its bit among the 32 of near_cols
    __shared__ const double *s_col[128];
    __shared__ int s_shift[128], s_e[kRowsA], s_ld[128];   // s_ld: distance of two rows
    __shared__ double s_coef[128];
    __shared__ int s_sign[128];   // what +-1 does to the sign bit, 1 for any other factor
    const DenseChunk ch = chunks[blockIdx.y];
    const int mb = (ch.M + kRowsA - 1) / kRowsA;
    const bool q = (int)blockIdx.x >= mb;
    const int rb = q ? blockIdx.x - mb : blockIdx.x, n = q ? ch.N : ch.M;
    if (rb * kRowsA >= n || (!q && ch.shared_p)) return;
    const int tid = threadIdx.x, lrow = tid & 127, half = tid >> 7;
    if (tid < ch.ncol) {
        const int2 tl = cols[ch.col0 + tid];
        const DenseWork w = work[tl.x];
        const bool tr = w.tr & (q ? 2 : 1);
        const double *x = q ? w.Q : w.P;
        const int ld = q ? w.ldq : w.ldp;
        s_col[tid] = x + (tr ? (size_t)tl.y : (size_t)tl.y * ld);
        s_ld[tid] = tr ? ld : 1;
        s_shift[tid] = q ? -shift[ch.col0 + tid] : shift[ch.col0 + tid];
        s_coef[tid] = q ? 1.0 : w.coef;
        s_sign[tid] = q || w.coef == 1.0 ? 0 : (w.coef == -1.0 ? (int)0x80000000 : 1);
    }
    // order of the columns: by the size of their products, then every second, third or
    // fourth column first (a solve's triangle is balanced by itself: no sizes)
    const int stride = (ch.ncol + 31) / 32;
    if (near_cols && tid < ch.ncol)
        s_key[tid] = (mag[ch.col0 + tid] << 14) | ((3 - tid % max(stride, 1)) << 7) | (127 - tid);
    if (tid < kRowsA) s_e[tid] = INT_MIN;
    __syncthreads();
    if (near_cols && tid < 128) {
        int place = tid < ch.ncol ? tid : 32;
        if (ch.ncol > 32 && tid < ch.ncol) {
            place = 0;
#pragma unroll 8
            for (int c = 0; c < ch.ncol; ++c) place += s_key[c] > s_key[tid];
        }
        s_near[tid] = make_int2(s_shift[tid], place < 32 ? 1 << place : 0);
    }
    const int row = rb * kRowsA + lrow;
    const bool in = row < n;
    auto entry = [&](int c) -> double { return in && c < ch.ncol ? s_col[c][(size_t)row * s_ld[c]] : 0.0; };
    auto scaled = [&](int c, double x) -> double {
        if (s_sign[c] == 1) return s_coef[c] * x;
        return __hiloint2double(__double2hiint(x) ^ s_sign[c], __double2loint(x));
    };
    int e = INT_MIN;
    for (int c0 = half; c0 < ch.ncol; c0 += 32) {   // 16 loads in flight
        double v[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) v[t] = entry(c0 + 2 * t);
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int c = c0 + 2 * t;
            if (c >= ch.ncol) break;
            const double x = scaled(c, v[t]);
            const int ef = exp_field(x);
            if (ef == 0x7FF) e = kNonFinite;
            else if ((__double2hiint(x) & 0x7FFFFFFF) | __double2loint(x)) e = max(e, max(ef, 1) - s_shift[c]);
        }
    }
    if (e != INT_MIN) atomicMax(&s_e[lrow], e);
    __syncthreads();
    e = s_e[lrow];
    // |x 2^-s| < 2^E; a row of zeros takes any scale
    const int E = e == kNonFinite ? kNonFinite : (e == INT_MIN ? 0 : e - 1022);
    if (half == 0 && in) exps[(q ? ch.eq : ch.ep) + row] = E;
    const int kblocks = dense_blocks(ch.ncol);
    const int pad = q ? kRowsB : kRowsA;      // rows of the last block past n hold zeros
    if (row >= (n + pad - 1) / pad * pad) return;
    unsigned char *dst;
    int slice, step;
    if (q) {
        const int blk = row / kRowsB, r = row % kRowsB;
        dst = slices + ch.q + (size_t)blk * kblocks * kBlockB + (r >> 3) * kSbo + (r & 7) * 16;
        slice = kSliceB;
        step = kBlockB;
    } else {
        dst = slices + ch.p + (size_t)rb * kblocks * kBlockA + (lrow >> 3) * kSbo + (lrow & 7) * 16;
        slice = kSliceA;
        step = kBlockA;
    }
    const bool zero = E == kNonFinite;
    // which columns are near the row's top (a row of zeros, or one that goes to FP64
    // anyway, has all of them)
    unsigned near = zero || e == INT_MIN ? ~0u : 0u;
    double next[8];   // the next columns, loaded while the digits of these are formed
#pragma unroll
    for (int t = 0; t < 8; ++t) next[t] = zero ? 0.0 : entry(8 * half + t);
    for (int g = half; g < 2 * kblocks; g += 2) {
        unsigned char *d = dst + (size_t)(g >> 1) * step + (g & 1) * 128;
        double x[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            x[t] = 8 * g + t < ch.ncol ? scaled(8 * g + t, next[t]) : 0.0;
            next[t] = zero ? 0.0 : entry(8 * g + 16 + t);
        }
        if (near_cols)
#pragma unroll
            for (int t = 0; t < 8; ++t) {   // (a zero is not near: its exponent field is 0)
                const int2 col = s_near[min(8 * g + t, 127)];
                if (exp_field(x[t]) >= max(1, e - kNear + col.x)) near |= (unsigned)col.y;
            }
        uint32_t w[7][4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int c = 8 * g + 2 * h;
            uint32_t f0[7], f1[7];
            digits7_fast(fixed55(x[2 * h], E + (c < ch.ncol ? s_shift[c] : 0)), f0);
            digits7_fast(fixed55(x[2 * h + 1], E + (c + 1 < ch.ncol ? s_shift[c + 1] : 0)), f1);
#pragma unroll
            for (int s = 0; s < 7; ++s) w[s][h] = pack_bf16(f0[s], f1[s]);
        }
#pragma unroll
        for (int s = 0; s < 7; ++s)
            *reinterpret_cast<uint4 *>(d + s * slice) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
    if (near_cols && in) near_cols[2 * ((size_t)(q ? ch.eq : ch.ep) + row) + half] = near;
}

// Entries that a NaN, an infinity, a subnormal result or graded rows send to FP64: those
// of the mask `slow`, of this lane's row and 8 columns from `col`, added to acc.  A
// lane's sum over the K axis is a chain of loads, which the CTA's other warps wait for:
// a few entries are formed one after the other by the whole warp, a column of the K
// axis a lane, many by their own lanes, the eight columns at the same time.
__device__ __noinline__ void slow_entries(const DenseWork *work, const int2 *cols, int ncol, int row, int col,
                                          unsigned slow, double *acc) {
    const int lane = threadIdx.x & 31;
    const int all = __reduce_add_sync(0xffffffffu, __popc(slow));
    if (all * (ncol / 32 + 2) > ncol + 3) {
        if (slow) {
            const int last = 31 - __clz(slow);   // (the columns after it may not exist)
            double v[8] = {};
            for (int l = 0; l < ncol;) {   // a task's columns are consecutive
                const int2 tl = cols[l];
                const DenseWork w = work[tl.x];
                const bool tp = w.tr & 1, tq = w.tr & 2;
                const double *p = w.P + (tp ? (size_t)row * w.ldp + tl.y : (size_t)tl.y * w.ldp + row);
                const double *q = w.Q + (tq ? (size_t)col * w.ldq + tl.y : (size_t)tl.y * w.ldq + col);
                const size_t sp = tp ? 1 : w.ldp, sq = tq ? 1 : w.ldq, sc = tq ? w.ldq : 1;
                const int run = min(ncol - l, w.kk - tl.y);
#pragma unroll 1
                for (int i = 0; i < run; ++i, p += sp, q += sq) {
                    const double x = w.coef * *p;
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = fma(x, q[min(e, last) * sc], v[e]);
                }
                l += run;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (slow >> e & 1) acc[e] += v[e];
        }
        __syncwarp();
        return;
    }
#pragma unroll 1
    for (int e = 0; e < 8; ++e)
        for (unsigned left = __ballot_sync(0xffffffffu, slow >> e & 1); left; left &= left - 1) {
            const int s = __ffs(left) - 1, r = row - lane + s, c = col + e;
            double v = 0.0;
            for (int l = lane; l < ncol; l += 32) {
                const int2 tl = cols[l];
                const DenseWork w = work[tl.x];
                const double p = w.P[w.tr & 1 ? (size_t)r * w.ldp + tl.y : (size_t)tl.y * w.ldp + r];
                const double q = w.Q[w.tr & 2 ? (size_t)c * w.ldq + tl.y : (size_t)tl.y * w.ldq + c];
                v += w.coef * p * q;
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == s) acc[e] += v;
        }
}

// The eight planes of 4 columns combined, sum of plane_d 2^(96 - 8 d - 55 - 8)
// with the last pair rounded to nearest.  SMALL: every accumulator is below 2^22
// in magnitude (chunks of up to 32 columns: 7 * 32 * 2^14), so that an FP32
// addition of 1.5 2^23 leaves the integer in the low bits: two instructions at
// full rate where a conversion takes one at an eighth of it; the additions'
// constants come off at the end (mod 2^64).
template <bool SMALL>
__device__ __forceinline__ void combine4(long long (&acc)[4], uint32_t taddr) {
    constexpr unsigned long long C = 0x4B400000ull;
    constexpr unsigned long long K0 = (C * 257ull << 33) + (C * 257ull << 17) + (C * 257ull << 1);
    auto bits = [](float v) { return __float_as_uint(v + 12582912.f); };
    __syncwarp();   // (the loads are .aligned, and what comes before branches by lane)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        float v0[4], v1[4];
        tc::tmem_ld4(taddr + (2 * m) * kRowsB, v0);
        tc::tmem_ld4(taddr + (2 * m + 1) * kRowsB, v1);
        tc::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (SMALL && m < 3) {
                const unsigned long long q = (unsigned long long)bits(v0[e]) * 256u + bits(v1[e]);
                acc[e] = (long long)(m == 0 ? q : ((unsigned long long)acc[e] << 16) + q);
            } else if (SMALL) {
                const int q = (int)(bits(v0[e]) - (unsigned)C) * 256 + (int)(bits(v1[e]) - (unsigned)C);
                acc[e] = (long long)(((unsigned long long)acc[e] << 1) - K0) + ((q + (1 << 14)) >> 15);
            } else {
                const long long q = (long long)__float2int_rn(v0[e]) * 256 + __float2int_rn(v1[e]);
                acc[e] = m == 0 ? q : (m < 3 ? acc[e] * 65536 + q : acc[e] * 2 + ((q + (1 << 14)) >> 15));
            }
        }
    }
}

// A unit: one chunk of one 128 x 32 tile, as the workers need it.
struct Unit {
    double *cd;         // the tile's first entry
    const int *ep, *eq; // row scales of P and Q from the tile's first row and column
    const uint2 *np, *nq;   // their columns near the top (of each half of the columns)
    double beta;
    int ldcd, rows, cols;
    int row0, col0;     // the tile's place in CD
    int kcol0, ncol;    // its columns of the K axis
    int flags;          // kFirst ...
};
constexpr int kFirst = 1, kLast = 2, kZeroUpper = 4, kFromZero = 8, kScale = 16, kBetaZero = 32, kStop = 64,
              kKeepUpper = 128, kKeepLower = 256;
constexpr int kRing = 8;

// The producer's walk over a CTA's units: tiles blockIdx.x, blockIdx.x +
// gridDim.x, ... of the batch's jobs, the chunks of each.
struct Walk {
    int t, j, c, c1;
    DenseJob job;
    int row0, col0;
    bool first, from_zero;
};
__device__ __forceinline__ void walk_tile(Walk &w, const DenseJob *jobs, int njobs, const DenseChunk *chunks) {
    int lo = w.j, hi = njobs;   // the last job that starts at or before the tile
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (jobs[mid].tile0 <= w.t) lo = mid;
        else hi = mid;
    }
    w.j = lo;
    w.job = jobs[lo];
    const int nb = (w.job.N + kRowsB - 1) / kRowsB, i = w.t - w.job.tile0;
    w.row0 = i / nb * kRowsA;   // neighbouring CTAs share a block of P
    w.col0 = i % nb * kRowsB;
    w.c = w.job.chunk0;
    w.c1 = w.job.chunk0 + w.job.nchunks;
    w.first = true;
    w.from_zero = false;
    // strictly above the diagonal only what follows the last zeroing counts (if
    // nothing does, one block of that chunk, to leave the zeros)
    if (w.row0 + kRowsA <= w.col0)
        for (int c = w.c1 - 1; c >= w.job.chunk0; --c)
            if (chunks[c].zero_upper) {
                w.c = min(c + 1, w.c1 - 1);
                w.from_zero = true;
                break;
            }
}

// tiles that a job's mask or its skip word leaves out
__device__ __forceinline__ bool tile_left_out(const Walk &w) {
    return (w.job.mask == 1 && w.row0 + kRowsA <= w.col0) ||
           (w.job.mask == 2 && w.row0 >= w.col0 + kRowsB) || (w.job.skip && *w.job.skip != 0);
}

// A wait gave up: NaN in every tile of this CTA, never stale or half-summed ones
// (thread: one row, 8 columns), and a word that the host reads (in its pinned memory).
__device__ __noinline__ void poison_tiles(const DenseJob *jobs, int njobs, const DenseChunk *chunks,
                                          int ntiles, int lrow, int cw, int *gave_up) {
    *gave_up = 1;
    Walk w;
    w.j = 0;
    for (w.t = blockIdx.x; w.t < ntiles; w.t += gridDim.x) {
        walk_tile(w, jobs, njobs, chunks);
        if (tile_left_out(w)) continue;
        const int row = w.row0 + lrow;
        for (int col = w.col0 + cw; col < min(w.col0 + cw + 8, w.job.N); ++col)
            if (row < w.job.M && !(w.job.mask == 1 && row < col) && !(w.job.mask == 2 && row > col))
                w.job.cd[(size_t)col * w.job.ldcd + row] = __longlong_as_double(-1LL);
    }
}

// Two CTAs of 18 warps per SM: 16 workers (thread: one row, 8 columns), a
// producer that walks the units, fetches their blocks and describes them, and
// an issuer of MMAs.  All waits are bounded: after `limit` clock cycles a role gives
// up, and so in turn do those that wait for it; the workers are the last, and fill
// the tiles with NaN.  What a role has in flight by then, copies or MMAs, it waits
// for with the full limit, whatever `limit` is.
__global__ void __launch_bounds__(kThreadsTc, 2)
    dense_tile_tc_kernel(const DenseWork *work, const int2 *cols, const DenseChunk *chunks,
                         const DenseJob *jobs, int njobs, int ntiles, const unsigned char *slices,
                         const int *exps, const uint2 *near_cols, int *gave_up, long long limit) {
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char *misc = sm + kStages * kStage;
    uint64_t *full = reinterpret_cast<uint64_t *>(misc), *empty = full + kStages;
    uint64_t *done = empty + kStages, *drained = done + 1, *info = drained + 1;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(info + kRing);
    int *s_block = reinterpret_cast<int *>(tslot + 1);   // per stage: kFirst, kLast, kStop
    Unit *s_unit = reinterpret_cast<Unit *>(misc + 256);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tc::tmem_alloc(tslot, kTmem);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(full + s, 1);
            tc::mbar_init(empty + s, 1);
        }
        for (int s = 0; s < kRing; ++s) tc::mbar_init(info + s, 1);
        tc::mbar_init(done, 1);
        tc::mbar_init(drained, kWorkers);
    }
    for (int e = tid; e < kStages * kSliceB / 16; e += kThreadsTc) {
        const int s = e / (kSliceB / 16), o = e % (kSliceB / 16);
        reinterpret_cast<uint4 *>(sm + s * kStage + kBlockA + kBlockB)[o] = make_uint4(0, 0, 0, 0);
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *tslot;

    if (tid == kWorkers) {
        // ---- producer ------------------------------------------------------------
        Walk w;
        w.j = 0;
        int b = 0, u = 0;
        bool ok = true;
        for (w.t = blockIdx.x; w.t < ntiles && ok; w.t += gridDim.x) {
            walk_tile(w, jobs, njobs, chunks);
            if (tile_left_out(w)) continue;
            double *cd = w.job.cd + (size_t)w.col0 * w.job.ldcd + w.row0;
            const int ldcd = w.job.ldcd;
            for (; w.c < w.c1 && ok; ++w.c, ++u) {
                const DenseChunk ch = chunks[w.c];
                const int kblocks = dense_blocks(ch.ncol);
                const int nblocks = w.from_zero && ch.zero_upper ? 1 : kblocks;
                for (int kb = 0; kb < nblocks && ok; ++kb, ++b) {
                    const int s = b % kStages;
                    if (b >= kStages)
                        ok = tc::mbar_wait(empty + s, (b / kStages - 1) & 1, limit);
                    if (!ok) break;
                    if (kb == 0) {
                        // slot u % kRing is free: three blocks back the unit before
                        // that block's was drained
                        Unit &x = s_unit[u % kRing];
                        x.cd = cd;
                        x.ldcd = ldcd;
                        x.ep = exps + ch.ep + w.row0;
                        x.eq = exps + ch.eq + w.col0;
                        x.np = near_cols ? near_cols + ch.ep + w.row0 : nullptr;
                        x.nq = near_cols + ch.eq + w.col0;
                        x.beta = ch.beta;
                        x.rows = w.job.M - w.row0;
                        x.cols = w.job.N - w.col0;
                        x.row0 = w.row0;
                        x.col0 = w.col0;
                        x.kcol0 = ch.col0;
                        x.ncol = ch.ncol;
                        x.flags = (w.first ? kFirst : 0) | (w.c + 1 == w.c1 ? kLast : 0) |
                                  (ch.zero_upper ? kZeroUpper : 0) | (w.from_zero ? kFromZero : 0) |
                                  (ch.scale != 0 ? kScale : 0) | (ch.scale == 2 ? kBetaZero : 0) |
                                  (w.job.mask == 1 ? kKeepUpper : 0) | (w.job.mask == 2 ? kKeepLower : 0);
                        tc::mbar_arrive(info + u % kRing);
                        w.first = false;
                    }
                    s_block[s] = (kb == 0 ? kFirst : 0) | (kb + 1 == nblocks ? kLast : 0);
                    unsigned char *dst = sm + s * kStage;
                    tc::mbar_expect(full + s, kBlockA + kBlockB);
                    tc::bulk_load(dst, slices + ch.p + ((size_t)(w.row0 / kRowsA) * kblocks + kb) * kBlockA,
                                  kBlockA, full + s);
                    tc::bulk_load(dst + kBlockA,
                                  slices + ch.q + ((size_t)(w.col0 / kRowsB) * kblocks + kb) * kBlockB,
                                  kBlockB, full + s);
                }
            }
        }
        // the end, for the issuer and the workers
        const int s = b % kStages;
        if (ok && b >= kStages) ok = tc::mbar_wait(empty + s, (b / kStages - 1) & 1, limit);
        if (ok) {
            s_block[s] = kStop;
            tc::mbar_arrive(full + s);
            s_unit[u % kRing].flags = kStop;
            tc::mbar_arrive(info + u % kRing);
        }
        // copies in flight land before the CTA gives its memory up, also where the issuer
        // no longer waits for them (after the stop, block b - kStages has been read and
        // its barrier serves the stop)
        const int flight = ok ? kStages - 1 : kStages;
        for (int k = max(0, b - flight); k < b; ++k)
            tc::mbar_wait(full + k % kStages, (k / kStages) & 1, kTcWaitCycles);
    } else if (tid == kWorkers + 32) {
        // ---- issuer --------------------------------------------------------------
        int u = 0;
        bool first_block = true;
        for (int b = 0;; ++b) {
            const int s = b % kStages;
            bool ok = tc::mbar_wait(full + s, (b / kStages) & 1, limit);
            const int fl = ok ? s_block[s] : kStop;
            if (ok && (fl & kFirst) && u > 0) {   // the accumulators are free again
                ok = tc::mbar_wait(drained, (u - 1) & 1, limit);
                tc::fence_after_sync();
            }
            if (!ok || (fl & kStop)) {
                if (!ok && b > 0)   // MMAs in flight end first
                    tc::mbar_wait(empty + (b - 1) % kStages, ((b - 1) / kStages) & 1, kTcWaitCycles);
                break;
            }
            first_block = fl & kFirst;
            const uint32_t a0 = tc::smem_u32(sm + s * kStage), b0 = a0 + kBlockA;
#pragma unroll 1
            for (int i = 0; i < 7; ++i)   // slice i of P, slices 0 .. 7 - i of Q: planes i .. 7
                tc::mma_bf16(tbase + i * kRowsB, tc::make_desc(a0 + i * kSliceA, tc::kLbo, kSbo),
                             tc::make_desc(b0, tc::kLbo, kSbo),
                             tc::idesc_bf16_f32(kRowsA, (kPlanes - i) * kRowsB), i > 0 || !first_block);
            tc::mma_commit(empty + s);
            if (fl & kLast) {
                tc::mma_commit(done);
                ++u;
            }
        }
    } else if (tid < kWorkers) {
        // ---- workers: combine the accumulators and update CD ----------------------
        const int lrow = tid & 127, cw = tid >> 7 << 3;   // this thread's row and first column
        const uint32_t tw = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + cw;
        double acc[8];
        bool unset = true;   // the first product is stored as it is, without an FP64 addition
        for (int u = 0;; ++u) {
            bool ok = tc::mbar_wait(info + u % kRing, (u / kRing) & 1, limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                poison_tiles(jobs, njobs, chunks, ntiles, lrow, cw, gave_up);
                break;
            }
            const Unit &x = s_unit[u % kRing];
            const int flags = x.flags;
            if (flags & kStop) break;
            const bool in = lrow < x.rows;
            const int nc = min(8, x.cols - cw);
            if (flags & kFirst) {
                unset = (flags & (kFromZero | kBetaZero)) != 0;
                const double *p = x.cd + (size_t)cw * x.ldcd + lrow;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    acc[e] = !unset && in && e < nc ? *p : 0.0;
                    p += x.ldcd;
                }
            }
            if (flags & kScale) {   // beta = 0 does not read CD (BLAS convention)
                unset = (flags & kBetaZero) != 0;
                const double beta = x.beta;
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = unset ? 0.0 : beta * acc[e];
            }
            const int Er = in ? x.ep[lrow] + kShift - 110 : 0;
            const int Ecl = (lane & 7) < nc ? x.eq[cw + (lane & 7)] : 0;
            unsigned nr = ~0u, ncl = ~0u;
            if (x.np) {
                if (in) nr = x.np[lrow].x | x.np[lrow].y;
                if ((lane & 7) < nc) ncl = x.nq[cw + (lane & 7)].x | x.nq[cw + (lane & 7)].y;
            }
            ok = tc::mbar_wait(done, u & 1, limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {   // (no later unit: its phase of `done` would be taken for this one's)
                poison_tiles(jobs, njobs, chunks, ntiles, lrow, cw, gave_up);
                break;
            }
            tc::fence_after_sync();
            unsigned slow = 0;   // entries that FP64 forms: NaN, infinity, subnormal, no large term
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                long long a4[4];
                if (x.ncol <= 32) combine4<true>(a4, tw + 4 * h);
                else combine4<false>(a4, tw + 4 * h);
                double v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int p = Er + __shfl_sync(0xffffffffu, Ecl, 4 * h + e);
                    bool fits;
                    v[e] = i64_times_pow2(a4[e], p, fits);
                    // no column near both tops, |T| < kFar 2^32, CD's entry small too
                    const unsigned common = nr & __shfl_sync(0xffffffffu, ncl, 4 * h + e);
                    const bool far = common == 0 && (unsigned)((int)(a4[e] >> 32) + kFar) < 2u * kFar &&
                                     exp_field(acc[4 * h + e]) - 1023 < p + kFarBits;
                    if (!fits || p >= kNonFinite / 2 || far) {
                        v[e] = 0.0;
                        slow |= 1u << (4 * h + e);
                    }
                }
                // (the FP64 pipe is skipped, not only its result, where nothing is to be added to)
                if (unset) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[4 * h + e] = v[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        asm("add.rn.f64 %0, %0, %1;" : "+d"(acc[4 * h + e]) : "d"(v[e]));
                }
            }
            unset = false;
            slow &= in && nc > 0 ? (1u << nc) - 1 : 0u;
            if (flags & kZeroUpper)   // (what becomes zero anyway)
                slow &= (1u << max(0, min(8, x.row0 + lrow - x.col0 - cw + 1))) - 1;
            if (__any_sync(0xffffffffu, slow != 0)) {
                double v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = acc[e];
                slow_entries(work, cols + x.kcol0, x.ncol, x.row0 + lrow, x.col0 + cw, slow, v);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = v[e];
            }
            if (flags & kZeroUpper) {
                const int up = x.col0 + cw - (x.row0 + lrow);   // entry e lies above the diagonal if e + up > 0
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (e + up > 0) acc[e] = 0.0;
            }
            if ((flags & kLast) && in) {
                double *p = x.cd + (size_t)cw * x.ldcd + lrow;
                // entry e lies e + up columns right of the diagonal; lo .. hi are written
                const int up = x.col0 + cw - (x.row0 + lrow);
                const int lo = flags & kKeepLower ? -up : 0, hi = flags & kKeepUpper ? min(nc, 1 - up) : nc;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (e >= lo && e < hi) *p = acc[e];
                    p += x.ldcd;
                }
            }
            tc::fence_before_sync();
            tc::mbar_arrive(drained);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, kTmem);
}

}  // namespace

size_t dense_slice_bytes(int M, int N, int ncol) {
    const size_t kb = dense_blocks(ncol);
    return kb * ((size_t)((M + kRowsA - 1) / kRowsA) * kBlockA + (size_t)((N + kRowsB - 1) / kRowsB) * kBlockB);
}
int dense_tiles(int M, int N) { return ((M + kRowsA - 1) / kRowsA) * ((N + kRowsB - 1) / kRowsB); }
size_t dense_slice_q_offset(int M, int ncol) {
    return (size_t)dense_blocks(ncol) * ((M + kRowsA - 1) / kRowsA) * kBlockA;
}

static thread_local long long t_wait_cycles = dg::kTcWaitCycles;
extern "C" void hcore_gpu_test_wait_cycles(long long cycles) {
    t_wait_cycles = cycles > 0 ? cycles : dg::kTcWaitCycles;
}

cudaError_t configure_dense_tc() {
    return cudaFuncSetAttribute(dense_tile_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
}

cudaError_t launch_dense_balance(const DenseWork *d_work, const int2 *d_cols, const int2 *d_dims, int ncols,
                                 DenseBalance how, int *d_shift, int *d_mag, cudaStream_t s) {
    if (ncols <= 0) return cudaSuccess;
    if (how == kNoBalance) return cudaMemsetAsync(d_shift, 0, (size_t)ncols * sizeof(int), s);
    if (how == kBalanceByThread)
        dense_balance_t_kernel<<<(ncols + 63) / 64, 256, 0, s>>>(d_work, d_cols, d_dims, ncols, d_shift, d_mag);
    else
        dense_balance_kernel<<<(ncols + 7) / 8, 256, 0, s>>>(d_work, d_cols, d_dims, ncols, how == kBalanceP,
                                                             d_shift, d_mag);
    return cudaGetLastError();
}

cudaError_t launch_dense_tiles_tc(const DenseWork *d_work,
                                  const int2 *d_cols, const int *d_shift, const int *d_mag, const DenseChunk *d_chunks,
                                  const DenseJob *d_jobs, const DenseBatch &b, unsigned char *d_slices,
                                  int *d_exps, unsigned *d_near, int *gave_up, cudaStream_t s) {
    const int mb = (b.maxM + kRowsA - 1) / kRowsA, nq = (b.maxN + kRowsA - 1) / kRowsA;
    dense_slice_kernel<<<dim3(mb + nq, b.nchunks), 256, 0, s>>>(d_work, d_cols, d_shift, d_mag,
                                                                d_chunks + b.chunk0, d_slices, d_exps, d_near);
    const int grid = b.ntiles < 2 * kSms ? b.ntiles : 2 * kSms;   // two CTAs per SM
    dense_tile_tc_kernel<<<grid, kThreadsTc, kSmem, s>>>(d_work, d_cols, d_chunks,
                                                         d_jobs + b.job0, b.njobs, b.ntiles, d_slices, d_exps,
                                                         reinterpret_cast<const uint2 *>(d_near), gave_up,
                                                         t_wait_cycles);
    return cudaGetLastError();
}

}  // namespace hc
