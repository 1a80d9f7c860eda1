// hcore-gb300 — host side of the tensor-core products (hc_dense_tc.cu): lists of
// products CD = beta CD + coef P Q^T, laid out as chunks, jobs and batches in
// one arena and launched stage after stage.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "hc_internal.h"

namespace hc {

struct DenseProducts {
    // a batch's digit slices stay in the L2 (129 MB; the tiles pass through it
    // too), and 96 MB more than that held costs 2.5%: 384 products of 1024 x
    // 1024 x 17 took 2873, 2625, 2557, 2538 and 2493 us with limits of 16, 48,
    // 96, 160 and 400 MB
    size_t slice_limit = (size_t)96 << 20;
    std::vector<DenseWork> work;
    std::vector<int2> dims;      // M, N of each product
    std::vector<int2> cols;      // the K axes of all tiles: (product, its column)
    std::vector<DenseChunk> chunks;
    std::vector<DenseJob> jobs;
    std::vector<DenseBatch> batches;
    // set to 1 by a launch one of whose bounded waits gave up (its tiles are NaN
    // then): device-accessible, zeroed and read by the caller
    int *gave_up = nullptr;

    // a product; its kk columns are laid out by add_tile
    int add(const DenseWork &w, int M, int N) {
        work.push_back(w);
        dims.push_back(make_int2(M, N));
        return (int)work.size() - 1;
    }

    // the tiles added from here on run after those before
    void stage(DenseBalance b) { stages.push_back(Stage{(int)cols.size(), (int)batches.size(), b}); }

    // lay a tile's tasks out along K: a chunk ends after 128 columns, where a
    // task scales CD, and where syrk tasks change to others (a run of syrk
    // tasks may zero the strict upper triangle at its end: it writes nothing
    // else there)
    void add_tile(const std::vector<int> &g) {
        const int2 mn = dims[g[0]];
        const int first = (int)chunks.size();
        auto open = [&](double beta, int syrk) {
            chunks.push_back(DenseChunk{0, 0, 0, 0, (int)cols.size(), 0, mn.x, mn.y, beta, syrk,
                                        beta == 1.0 ? 0 : (beta == 0.0 ? 2 : 1), 0});
        };
        for (size_t x = 0; x < g.size(); ++x) {
            const DenseWork &w = work[g[x]];
            if (x == 0 || w.beta != 1.0 || w.syrk != chunks.back().zero_upper) open(w.beta, w.syrk);
            for (int l = 0; l < w.kk; ++l) {
                if (chunks.back().ncol == 128) open(1.0, w.syrk);
                cols.push_back(make_int2(g[x], l));
                ++chunks.back().ncol;
            }
        }
        const int tiles = dense_tiles(mn.x, mn.y);
        // jobs: the tile's chunks, split where a batch's slice buffer is full
        for (int c = first; c < (int)chunks.size(); ++c) {
            DenseChunk &ch = chunks[c];
            // P's slices serve the next product too if it has the same P (and they
            // do not depend on Q)
            const size_t p_bytes = dense_slice_q_offset(mn.x, ch.ncol);
            size_t need = dense_slice_bytes(mn.x, mn.y, ch.ncol);
            const DenseChunk *same = last_p(g[0], c, first);
            if (same && cur_slices + need - p_bytes <= slice_limit) need -= p_bytes;
            else same = nullptr;
            if ((int)batches.size() == stages.back().batches0 ||
                (cur_slices > 0 && cur_slices + need > slice_limit) || batches.back().ntiles > INT_MAX - tiles ||
                batches.back().nchunks == 65535) {
                batches.push_back(DenseBatch{(int)jobs.size(), 0, 0, c, 0, 1, 1});
                cur_slices = cur_exps = 0;
            }
            DenseBatch &b = batches.back();
            if (c == first || b.nchunks == 0) {
                jobs.push_back(DenseJob{nullptr, nullptr, 0, g[0], 0, mn.x, mn.y, c, 0, b.ntiles});
                ++b.njobs;
                b.ntiles += tiles;
            }
            ++jobs.back().nchunks;
            ++b.nchunks;
            b.maxM = std::max(b.maxM, mn.x);
            b.maxN = std::max(b.maxN, mn.y);
            ch.shared_p = same != nullptr;
            ch.p = same ? same->p : (long long)cur_slices;
            ch.ep = same ? same->ep : (int)cur_exps;
            ch.q = (long long)(cur_slices + (same ? 0 : p_bytes));
            ch.eq = (int)cur_exps + (same ? 0 : mn.x);
            cur_slices += need;
            cur_exps += (size_t)(same ? 0 : mn.x) + mn.y;
            slice_bytes = std::max(slice_bytes, cur_slices);
            max_exps = std::max(max_exps, cur_exps);
        }
    }

    // the arena: what pack() writes at `at`, and the device's own arrays
    void place_host(size_t &at) {
        place(at, o_work, work.size() * sizeof(DenseWork));
        place(at, o_cols, cols.size() * sizeof(int2));
        place(at, o_dims, dims.size() * sizeof(int2));
        place(at, o_chunks, chunks.size() * sizeof(DenseChunk));
        place(at, o_jobs, jobs.size() * sizeof(DenseJob));
    }
    void place_device(size_t &at) {
        place(at, o_shift, cols.size() * sizeof(int));
        place(at, o_exps, max_exps * sizeof(int));
        place(at, o_near, max_exps * sizeof(uint2));
        place(at, o_mag, cols.size() * sizeof(int));
        place(at, o_slices, slice_bytes);
    }
    void pack(char *host) const {
        auto put = [host](size_t o, const void *src, size_t bytes) {
            if (bytes) memcpy(host + o, src, bytes);
        };
        put(o_work, work.data(), work.size() * sizeof(DenseWork));
        put(o_cols, cols.data(), cols.size() * sizeof(int2));
        put(o_dims, dims.data(), dims.size() * sizeof(int2));
        put(o_chunks, chunks.data(), chunks.size() * sizeof(DenseChunk));
        put(o_jobs, jobs.data(), jobs.size() * sizeof(DenseJob));
    }
    const DenseWork *device_work(const char *arena) const { return (const DenseWork *)(arena + o_work); }

    // the chunk before chunk c, if c is its product's only one and has the same P
    // in the same batch
    const DenseChunk *last_p(int prod, int c, int first) const {
        if (c == 0 || c != first || c + 1 != (int)chunks.size() || stages.back().balance == kBalanceByWarp ||
            stages.back().balance == kBalanceByThread || (int)batches.size() == stages.back().batches0)
            return nullptr;
        const DenseBatch &b = batches.back();
        if (b.nchunks == 0 || b.chunk0 + b.nchunks != c || b.nchunks == 65535) return nullptr;
        const DenseChunk &q = chunks[c - 1], &x = chunks[c];
        if (q.ncol != x.ncol || q.M != x.M || q.ncol == 0) return nullptr;
        const int2 l = cols[q.col0], m = cols[x.col0];
        const DenseWork &w = work[l.x], &v = work[prod];
        const bool same = l.y == 0 && m.y == 0 && w.kk == v.kk && w.kk == x.ncol && w.P == v.P && w.P != nullptr &&
                          w.ldp == v.ldp && (w.tr & 1) == (v.tr & 1) && w.coef == v.coef;
        return same ? &q : nullptr;
    }

    int nstages() const { return (int)stages.size(); }
    cudaError_t launch_stage(char *arena, int q, cudaStream_t s) const {
        const DenseWork *d_work = device_work(arena);
        const int2 *d_cols = (const int2 *)(arena + o_cols), *d_dims = (const int2 *)(arena + o_dims);
        int *d_shift = (int *)(arena + o_shift), *d_mag = (int *)(arena + o_mag);
        const bool last = q + 1 == nstages();
        const int c0 = stages[q].cols0, c1 = last ? (int)cols.size() : stages[q + 1].cols0;
        const int b1 = last ? (int)batches.size() : stages[q + 1].batches0;
        cudaError_t e = launch_dense_balance(d_work, d_cols + c0, d_dims, c1 - c0, stages[q].balance,
                                             d_shift + c0, d_mag + c0, s);
        for (int b = stages[q].batches0; b < b1 && e == cudaSuccess; ++b)
            e = launch_dense_tiles_tc(d_work, d_cols, d_shift, d_mag, (const DenseChunk *)(arena + o_chunks),
                                      (const DenseJob *)(arena + o_jobs), batches[b],
                                      (unsigned char *)(arena + o_slices), (int *)(arena + o_exps),
                                      stages[q].balance == kNoBalance ? nullptr : (unsigned *)(arena + o_near),
                                      gave_up, s);
        return e;
    }
    cudaError_t launch(char *arena, cudaStream_t s) const {
        cudaError_t e = cudaSuccess;
        for (int q = 0; q < nstages() && e == cudaSuccess; ++q) e = launch_stage(arena, q, s);
        return e;
    }

    // a product alone on its output
    void add_one(const DenseWork &w, int M, int N, double *cd, int ldcd, int mask = 0, const int *skip = nullptr) {
        const size_t first = jobs.size();
        add_tile({add(w, M, N)});
        for (size_t j = first; j < jobs.size(); ++j) {
            jobs[j].cd = cd;
            jobs[j].ldcd = ldcd;
            jobs[j].mask = mask;
            jobs[j].skip = skip;
        }
    }
    static DenseWork product(const double *P, int ldp, const double *Q, int ldq, int tr, int kk, double coef,
                             double beta) {
        DenseWork w{};
        w.P = P; w.ldp = ldp; w.Q = Q; w.ldq = ldq; w.tr = tr; w.kk = kk; w.coef = coef; w.beta = beta;
        return w;
    }

private:
    struct Stage {
        int cols0, batches0;
        DenseBalance balance;
    };
    std::vector<Stage> stages;
    size_t slice_bytes = 0, max_exps = 0, cur_slices = 0, cur_exps = 0;
    size_t o_work = 0, o_cols = 0, o_dims = 0, o_chunks = 0, o_jobs = 0, o_shift = 0, o_exps = 0, o_near = 0, o_mag = 0, o_slices = 0;

    static void place(size_t &at, size_t &o, size_t bytes) {
        o = at;
        at += (std::max<size_t>(bytes, 1) + 255) & ~(size_t)255;
    }
};

}  // namespace hc
