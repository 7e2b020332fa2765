// scan_rows.cu — exact FP32 scan of a few queries, reading only the rows
// their filter passes.
//
// For at most 8 queries the scan is bound by HBM, so the rows it does not
// read are what counts: a warp looks at the filter of its share of rows
// first (the batch's bitmap, or, for one range-form filter shared by all
// queries, the attribute values themselves, which saves the bitmap kernel),
// queues the passing rows and reads them R = 32 / QT at a time, so every
// read is of a row that is wanted and every batch is full whatever the
// selectivity. Distances are those of scan_f32.cu bit for bit (a lane's
// dims, then the transposing butterfly). The K best keys stay in each warp's
// registers (sorted across the lanes, folded in 32 at a time), a block's
// warps fold into one list, and the blocks' lists are merged like the
// tensor-core scan's runs; no block barrier and no shared-memory sort while
// rows stream.
//
// Rows are split evenly over all warps of a grid of two blocks per SM, by
// 32-row words. Measured on one B200, one query, 70 % of 1M x 128 rows pass:
// scan 0.070 ms (366 MB, 5.2 TB/s) and merge 0.010, where bitmap, full scan
// and merge took 0.007 + 0.094 + 0.023; 2 % of 100,000 rows: 0.012 + 0.009
// against 0.007 + 0.034 (49 blocks, for lists long enough to sort) + 0.009.
#include <algorithm>

#include "launch.cuh"
#include "pv_internal.h"
#include "tc_core.cuh"

namespace pv {

struct RowScanArgs {
    const float *__restrict__ vecs;
    uint64_t nrows;
    int dpad;
    const float *__restrict__ queries;
    int nq, K;
    const int32_t *__restrict__ qprog;
    const uint32_t *__restrict__ bitmaps;  // null: no filter, or `fused`
    uint64_t bm_words;
    // fused: program 0, a range form whose terms the host checked, is tested
    // on the columns and counted into popcnt[0]
    int fused, shared_prog;
    const double *__restrict__ cols;
    const PredInsn *__restrict__ insns;
    const PredProg *__restrict__ progs;
    const double *__restrict__ consts;
    unsigned long long *popcnt;
    uint64_t words_per_warp;
    uint64_t *dense;  // [nq][dcap]
    uint32_t *dcnt;
    uint64_t dcap;
};

constexpr int RS_WARPS = 8;

// 32 partial sums per lane -> lane L holds total L (scan_f32.cu).
__device__ __forceinline__ float rs_butterfly(float (&p)[32], int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool upper = (lane & s) != 0;
#pragma unroll
        for (int j = 0; j < s; j++) {
            const float send = upper ? p[j] : p[j + s];
            const float keep = upper ? p[j + s] : p[j];
            p[j] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    return p[0];
}

template <int QT, int DCH, int W>
__global__ void __launch_bounds__(32 * RS_WARPS, 2) scan_rows_kernel(RowScanArgs a) {
    constexpr int R = 32 / QT;  // rows of a butterfly
    // butterflies whose rows are read together (with 8 queries one has only four)
    constexpr int NB = QT == 8 && W == 1 ? 2 : 1;
    __shared__ uint32_t s_queue[RS_WARPS][64];
    __shared__ uint64_t s_new[RS_WARPS][QT][64];  // keys not yet folded in
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    float4 qr[QT][DCH];
#pragma unroll
    for (int qq = 0; qq < QT; qq++)
#pragma unroll
        for (int c = 0; c < DCH; c++) {
            const int j = c * 128 + lane * 4;
            qr[qq][c] = (qq < a.nq && j < a.dpad)
                            ? __ldg((const float4 *)(a.queries + (size_t)qq * a.dpad + j))
                            : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    uint64_t best[QT][W];
#pragma unroll
    for (int qq = 0; qq < QT; qq++)
#pragma unroll
        for (int h = 0; h < W; h++) best[qq][h] = KEY_MAX;
    uint32_t *queue = s_queue[warp];
    const int my_r = lane / QT, my_q = lane % QT;
    const int my_pg = my_q < a.nq && a.bitmaps ? a.qprog[my_q] : -1;
    unsigned head = 0, tail = 0;
    // this lane's query (the same in all lanes of the query): keys waiting,
    // and the K-th of its list
    int fill = 0;
    uint64_t thr = KEY_MAX;
    uint64_t *mynew = s_new[warp][my_q];
    unsigned qlanes = 0;
#pragma unroll
    for (int r = 0; r < R; r++) qlanes |= 1u << (r * QT);
    qlanes <<= my_q;
    auto ballot_of = [&](bool p) { return __ballot_sync(0xffffffffu, p) & qlanes; };
    // folds the waiting keys of every query that has more than `most`
    auto fold = [&](int most) {
        __syncwarp();
#pragma unroll
        for (int qq = 0; qq < QT; qq++) {
            const int n = __shfl_sync(0xffffffffu, fill, qq);
            if (n <= most) continue;
            for (int b = 0; b < n; b += 32) {
                const uint64_t k = b + lane < n ? s_new[warp][qq][b + lane] : KEY_MAX;
                warp_fold32<W>(best[qq], warp_sort32(k, lane, true), lane);
            }
            const uint64_t last = W == 1 || a.K <= 32 ? best[qq][0] : best[qq][W - 1];
            const uint64_t kth = __shfl_sync(0xffffffffu, last, (a.K - 1) & 31);
            if (my_q == qq) {
                thr = kth;
                fill = 0;
            }
        }
        __syncwarp();
    };

    auto take = [&](int cnt) {  // the queue's first cnt <= R * NB rows
        float4 x[NB][NB > 1 ? R : 1][DCH];  // NB > 1: all rows' reads first
        auto read = [&](int r, float4 (&v)[DCH]) {
            const uint32_t row = queue[(head + (r < cnt ? r : 0)) & 63];
#pragma unroll
            for (int c = 0; c < DCH; c++) {
                const int j = c * 128 + lane * 4;
                v[c] = j < a.dpad
                           ? __ldg((const float4 *)(a.vecs + (uint64_t)row * a.dpad + j))
                           : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        if (NB > 1) {
#pragma unroll
            for (int b = 0; b < NB; b++)
#pragma unroll
                for (int r = 0; r < R; r++) read(b * R + r, x[b][NB > 1 ? r : 0]);
        }
#pragma unroll
        for (int b = 0; b < NB; b++) {
            if (b * R >= cnt) break;
            float p[32];
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (NB == 1) read(r, x[0][0]);
                const float4(&v)[DCH] = x[b][NB > 1 ? r : 0];
#pragma unroll
                for (int qq = 0; qq < QT; qq++) {
                    float s = 0.f;
#pragma unroll
                    for (int c = 0; c < DCH; c++) {
                        const float d0 = v[c].x - qr[qq][c].x, d1 = v[c].y - qr[qq][c].y;
                        const float d2 = v[c].z - qr[qq][c].z, d3 = v[c].w - qr[qq][c].w;
                        s = fmaf(d0, d0, s);
                        s = fmaf(d1, d1, s);
                        s = fmaf(d2, d2, s);
                        s = fmaf(d3, d3, s);
                    }
                    p[r * QT + qq] = s;
                }
            }
            const float dist = rs_butterfly(p, lane);
            const int at = b * R + my_r;
            const uint32_t row = queue[(head + (at < cnt ? at : 0)) & 63];
            bool ok = at < cnt && my_q < a.nq;
            // queries with filters of their own: the row passes one of them
            if (ok && !a.shared_prog && my_pg >= 0)
                ok = (__ldg(a.bitmaps + (uint64_t)my_pg * a.bm_words + (row >> 5)) >> (row & 31)) & 1u;
            // keys better than the list's K-th wait in shared memory until a
            // batch of them is worth a sort (8 queries get 4 keys each here)
            const uint64_t key = make_key(dist, row);
            const bool want = ok && key < thr;
            const unsigned same = ballot_of(want);
            if (want) mynew[fill + __popc(same & lt)] = key;
            fill += __popc(same);
            if (__any_sync(0xffffffffu, fill > 64 - R)) fold(64 - R);
        }
    };

    const uint64_t nwords = (a.nrows + 31) / 32;
    const uint64_t w0 = ((uint64_t)blockIdx.x * RS_WARPS + warp) * a.words_per_warp;
    const uint64_t w1 = min(w0 + a.words_per_warp, nwords);
    unsigned passing = 0;
    for (uint64_t ws = w0; ws < w1; ws += 32) {
        // lane j holds word ws + j of the rows any query's filter passes
        const int nw = (int)min((uint64_t)32, w1 - ws);
        uint32_t mine = 0xFFFFFFFFu;
        if (a.fused) {
            const PredInsn ri = a.insns[a.progs[0].insn0];
            mine = 0;
            for (int j0 = 0; j0 < nw; j0 += 4) {
                bool ok[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    ok[u] = j0 + u < nw && (ws + j0 + u) * 32 + lane < a.nrows;
                int ci = ri.val0;
                for (int k = 0; k < ri.n; k++) {
                    const int meta = (int)__ldg(a.consts + ci);
                    const double *c = a.cols + (uint64_t)(meta & 0xFFFF) * a.nrows;
                    double v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        v[u] = ok[u] ? __ldg(c + (ws + j0 + u) * 32 + lane) : 0.0;
                    const double lo = __ldg(a.consts + ci + 1);
                    if (meta & PV_TERM_MASK) {
                        const unsigned long long bits = (unsigned long long)__double_as_longlong(lo);
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const bool in = v[u] >= 0.0 && v[u] < 64.0;
                            const int b = in ? (int)v[u] : 64;
                            const int code = (in && (double)b == v[u]) ? b : 64;
                            ok[u] = ok[u] && code < 64 && ((bits >> (code & 63)) & 1ull);
                        }
                        ci += 2;
                    } else {
                        const double hi = __ldg(a.consts + ci + 2);
#pragma unroll
                        for (int u = 0; u < 4; u++) ok[u] = ok[u] && v[u] >= lo && v[u] <= hi;
                        ci += 3;
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t wd = __ballot_sync(0xffffffffu, ok[u]);
                    if (lane == j0 + u) mine = wd;
                }
            }
            passing += __popc(mine);
        } else if (lane < nw) {
            const uint64_t w = ws + lane;
            if (a.bitmaps) {
                mine = 0;
                for (int qq = 0; qq < a.nq; qq++) {
                    const int pg = a.qprog[qq];
                    mine |= pg >= 0 ? __ldg(a.bitmaps + (uint64_t)pg * a.bm_words + w) : 0xFFFFFFFFu;
                    if (a.shared_prog) break;
                }
            }
            if (w == nwords - 1 && (a.nrows & 31)) mine &= (1u << (a.nrows & 31)) - 1u;
        }
        for (int j = 0; j < nw; j++) {
            const uint32_t word = __shfl_sync(0xffffffffu, mine, j);
            if (!word) continue;
            if ((word >> lane) & 1u)
                queue[(tail + __popc(word & lt)) & 63] = (uint32_t)((ws + j) * 32 + lane);
            tail += __popc(word);
            __syncwarp();
            while (tail - head >= (unsigned)(R * NB)) {
                take(R * NB);
                head += R * NB;
            }
            __syncwarp();
        }
    }
    if (tail != head) take((int)(tail - head));
    fold(0);

    if (a.fused) {
        passing = __reduce_add_sync(0xffffffffu, passing);
        if (lane == 0 && passing) atomicAdd(a.popcnt, (unsigned long long)passing);
    }
    // the warps' lists meet in shared memory (the waiting keys' place); each
    // query's are folded by a warp of its own, and its K best keys join the
    // query's run
#pragma unroll
    for (int qq = 0; qq < QT; qq++)
#pragma unroll
        for (int h = 0; h < W; h++) s_new[warp][qq][h * 32 + lane] = best[qq][h];
    __syncthreads();
    if (warp < a.nq) {
        const int qq = warp;
        uint64_t all[W];
#pragma unroll
        for (int h = 0; h < W; h++) all[h] = s_new[0][qq][h * 32 + lane];
        for (int o = 1; o < RS_WARPS; o++)
#pragma unroll
            for (int h = 0; h < W; h++) {
                const uint64_t d = s_new[o][qq][h * 32 + 31 - lane];
                const uint64_t worst = __shfl_sync(0xffffffffu, all[W - 1], 31);
                if (__any_sync(0xffffffffu, d < worst)) warp_fold32<W>(all, d, lane);
            }
        int n = 0;
#pragma unroll
        for (int h = 0; h < W; h++)
            n += __popc(
                __ballot_sync(0xffffffffu, h * 32 + lane < a.K && all[h] != KEY_MAX));
        uint32_t at = 0;
        if (lane == 0 && n) at = atomicAdd(a.dcnt + qq, (uint32_t)n);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int h = 0; h < W; h++)
            if (h * 32 + lane < n) a.dense[(uint64_t)qq * a.dcap + at + h * 32 + lane] = all[h];
    }
}

// At most 8 queries (2 of rows beyond 256 dims), lists of at most 64.
bool scan_rows_fits(int nq, int dpad, uint32_t topb) {
    const int dch = dpad <= 128 ? 1 : dpad <= 256 ? 2 : 4;
    return dpad <= 512 && nq * dch <= 8 && topb <= 64;
}

// The whole batch: scan and merge (db.rows_fused: its one filter is tested by
// the scan itself, else the bitmaps are in g->scan).
int scan_rows_launch(FvGpuIndex *g, const DevBatch &db, uint32_t topb, FvHit *d_out,
                     uint32_t *d_cnt, uint8_t *d_trunc, char *errbuf, size_t errlen) {
    ScanScratch &s = g->scan;
    const char *d = db.stage_d->as<char>();
    const int nq = db.nq;
    const uint64_t nwords = (g->count + 31) / 32;
    const uint64_t warps = std::min<uint64_t>((uint64_t)g->sm_count * 2 * RS_WARPS, nwords);
    RowScanArgs a;
    a.words_per_warp = (nwords + warps - 1) / warps;
    const unsigned blocks = (unsigned)((nwords + a.words_per_warp * RS_WARPS - 1) /
                                       (a.words_per_warp * RS_WARPS));
    a.dcap = (uint64_t)blocks * topb;
    PV_CUDA_OK(s.part.ensure((size_t)nq * a.dcap * 8), errbuf, errlen);
    // [dcnt u32 x 8][filter count u64], cleared together
    PV_CUDA_OK(s.part_cnt.ensure(64), errbuf, errlen);
    PV_CUDA_OK(cudaMemsetAsync(s.part_cnt.p, 0, 64, g->stream), errbuf, errlen);
    a.vecs = g->d_vecs;
    a.nrows = g->count;
    a.dpad = g->dpad;
    a.queries = (const float *)(d + db.off_q);
    a.nq = nq;
    a.K = (int)topb;
    a.qprog = (const int32_t *)(d + db.off_qprog);
    a.bitmaps = db.rows_fused || db.P == 0 ? nullptr : s.bitmaps.as<uint32_t>();
    a.bm_words = nwords;
    a.fused = db.rows_fused ? 1 : 0;
    a.shared_prog = db.P == 0 || db.one_prog ? 1 : 0;
    a.cols = g->d_cols;
    a.insns = (const PredInsn *)(d + db.off_insns);
    a.progs = (const PredProg *)(d + db.off_progs);
    a.consts = (const double *)(d + db.off_consts);
    a.popcnt = (unsigned long long *)(s.part_cnt.as<char>() + 32);
    a.dense = s.part.as<uint64_t>();
    a.dcnt = s.part_cnt.as<uint32_t>();
    cudaError_t e = cudaErrorInvalidValue;
    const int dch = g->dpad <= 128 ? 1 : g->dpad <= 256 ? 2 : 4;
    const int qt = nq <= 1 ? 1 : nq <= 2 ? 2 : nq <= 4 ? 4 : 8, w = topb <= 32 ? 1 : 2;
#define PV_CASE(Q, D)                                                                          \
    if (qt == Q && dch == D)                                                                   \
        e = w == 1 ? launch_pdl(scan_rows_kernel<Q, D, 1>, dim3(blocks), dim3(32 * RS_WARPS),  \
                                0, g->stream, a)                                               \
                   : launch_pdl(scan_rows_kernel<Q, D, 2>, dim3(blocks), dim3(32 * RS_WARPS),  \
                                0, g->stream, a);
    PV_CASE(1, 1) PV_CASE(2, 1) PV_CASE(4, 1) PV_CASE(8, 1)
    PV_CASE(1, 2) PV_CASE(2, 2) PV_CASE(4, 2) PV_CASE(1, 4) PV_CASE(2, 4)
#undef PV_CASE
    PV_CUDA_OK(e, errbuf, errlen);
    g->launches += 2;
    const unsigned long long *pop =
        db.rows_fused ? a.popcnt : s.popcnt.as<unsigned long long>();
    PV_CUDA_OK(launch_dense_merge(a.dense, a.dcap, a.dcnt, false, nullptr, nullptr, (int)topb,
                                  a.qprog, pop, g->count, nq, d_out, d_cnt, d_trunc, nullptr,
                                  nullptr, g->stream, false, true),
               errbuf, errlen);
    return 0;
}

}  // namespace pv
