// scan_tc.cu — reduced-precision filtered L2 scan on the 5th-gen tensor
// cores (tcgen05, TMEM accumulators, TMA-fed shared memory).
//
// New path beside the exact scan (the reference has no tensor-core path;
// its approximate SQ8 scan is gpu_engine.cu:759-893 + rerank :934-992).
// Distances use the norm form ||x||^2 + ||q||^2 - 2 q.x with the dot
// products from one GEMM per 128-row tile:
//     D[128 queries][128 rows] = Q[128 x K] * X_tile[128 x K]^T
// (A = query tile, resident in shared memory; B = row tile, streamed by
// TMA in 128-byte-swizzled K-major boxes). D lives in TMEM in four
// buffers, so the MMAs of the next tiles overlap the epilogue of tile t.
// In TMEM, lane = query and column = row: each epilogue thread owns ONE
// query, walks the tile's 128 rows and keeps that query's best K' keys
// in a private shared-memory list with its threshold in a register; the
// bitmap predicate is read only for rows that beat the threshold. The
// grid-wide per-query bound in global memory lets CTAs prune with each
// other's K'-th key. Per-CTA lists are merged per query and the K'
// survivors re-ranked with exact FP32 distances (rerank_kernel).
//
// BF16 operands are exact for integers up to 256, so on integer-valued
// rows (the benchmark data) every distance is exact; FP8-E4M3 rows carry a
// per-row scale (absmax / 448) and the query a per-query scale.
//
// Warp roles (64 + 128 * EPI threads): warp 0 TMA producer, warp 1 TMEM
// allocator + MMA issuer, then EPI groups of 4 epilogue warps (warp w reads
// TMEM lanes 32*(w%4)..+31; group h owns the tiles h, h + EPI, ...).
// A batch of at most 64 (32) queries is replicated 2 (4) times down the
// 128 query slots of the A tile: the MMA costs the same, and each replica
// takes a disjoint share of every tile's rows, so the epilogue work per
// warp shrinks by the replication factor and all four SM sub-partitions
// work (without it the warps of the padding lanes idle).
// All waits are bounded by a deadline and unwind through an abort flag.
#include <math.h>

#include <algorithm>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "pv_internal.h"
#include "sm100.cuh"
#include "launch.cuh"
#include "tc_core.cuh"

namespace pv {

using namespace sm100;

template <int KIND, int EPI, bool WARM>
__global__ void __launch_bounds__(64 + 128 * EPI, 1)
scan_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmQ,
               TcArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte alignment for the swizzled operand tiles
    unsigned char *base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const TcSmem sm = tc_carve(base, a.kblocks, a.NS, a.KP, EPI, KIND == TCK_TF32 && a.qstream);
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_abort = 0;
        tc_init_barriers(sm, a.NS, EPI);
    }
    if (warp == 1) {
        tmem_alloc(&s_tmem, TC_TMEM_COLS);
        tmem_relinquish();
    }
    __syncthreads();
    tc_fence_after();
    pdl_wait();  // the previous kernel's outputs (query tile, bounds, bitmaps)
    pdl_trigger();
    TcRun run;
    tc_pass<KIND, EPI, WARM>(&tmX, &tmQ, a, sm, s_tmem, run, &s_abort, blockIdx.x % a.qtiles,
                      blockIdx.x / a.qtiles);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(s_tmem, TC_TMEM_COLS);
    }
}

}  // namespace pv

namespace pv {

// ---------------------------------------------------------------- queries
// f32 queries [nq][dpad] -> low-precision tile rows [nqpad][row_bytes] with
// zero padding, plus ||q||^2 of the rounded query (and the fp8 scale).
// Row qi holds query qi % bq (bq = nqpad without replication). Also resets
// the scan's per-query state for query qi < nq: bound tau (none), dense run
// count, full-list minimum (if tracked), and the watchdog word.
__global__ void query_prep_kernel(const float *__restrict__ q, int nq, int dpad, int dim,
                                  int nqpad, int bq, int kelems, int kind,
                                  unsigned char *__restrict__ out, float *__restrict__ qnorm,
                                  float *__restrict__ qscale, unsigned long long *__restrict__ tau,
                                  uint32_t *__restrict__ dcnt,
                                  unsigned long long *__restrict__ fullmin, int *__restrict__ err,
                                  int behind_bitmaps) {
    // behind_bitmaps: the kernel ahead is this batch's bitmap kernel, which
    // touches nothing this one reads or writes (the queries were copied
    // before it), so the work runs beside it and only the completion waits
    if (!behind_bitmaps) {
        pdl_wait();
        pdl_trigger();
    }
    const int qi = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (qi < nqpad)
        query_prep_row(qi, threadIdx.x & 31, q, nq, dpad, dim, bq, kelems, kind, out, qnorm,
                       qscale, tau, dcnt, fullmin, err);
    if (behind_bitmaps) {
        pdl_wait();
        pdl_trigger();
    }
}

// ---------------------------------------------------------------- re-rank
// Exact FP32 distances (difference form) for each query's merged candidates
// (up to TC_MAX_SUPERSET, row stride S); keeps the best topb by (dist, id).
// One CTA (8 warps) per query: 8 lanes per candidate, 128 candidates in
// flight (random rows of 512 bytes: latency, then bandwidth), then a bitonic
// sort of the keys.
template <int ORDER>
__global__ void __launch_bounds__(256)
rerank_kernel(const float *__restrict__ vecs, int dpad, const float *__restrict__ queries,
              const FvHit *__restrict__ cand, const uint32_t *__restrict__ cand_cnt, int S,
              uint32_t topb, const int32_t *__restrict__ qprog,
              const unsigned long long *__restrict__ popcnt, uint64_t nrows,
              FvHit *__restrict__ out, uint32_t *__restrict__ out_cnt,
              uint8_t *__restrict__ trunc, const RerankCert cert) {
    __shared__ uint64_t keys[TC_MAX_SUPERSET];
    __shared__ int again;
    if (threadIdx.x == 0) again = 0;
    pdl_wait();
    pdl_trigger();
    rerank_query<256, ORDER>(blockIdx.x, keys, vecs, dpad, queries, cand, cand_cnt, S, topb, qprog, popcnt,
                      nrows, out, out_cnt, trunc, cert, &again);
    if (ORDER == RR_LANES8 && again)
        rerank_again<256>(blockIdx.x, keys, vecs, dpad, queries, (int)min(cand_cnt[blockIdx.x], (uint32_t)S),
                          (int)topb, out);
}

// ---------------------------------------------------------------- merge
// Per-query merge of the tensor-core scan's kept keys (one CTA per query).
// Query q's keys are dense[q][0 .. dcnt[q]) in any order; only keys at or
// below the grid-wide bound can be in the answer. Keys are unique 64-bit
// (distance bits, row) values, so the KO-th smallest is found exactly by a
// radix select, 8 bits per pass (a histogram of the digit among the keys
// that share the digits chosen so far) until few are left, and only the at
// most KO keys at or below it are sorted, if they need to be. Runs up to stage_cap keys are staged in shared
// memory; longer ones are read from global memory on every pass (4 loads
// in flight per lane).
__global__ void __launch_bounds__(DM_THREADS)
dense_merge_kernel(const uint64_t *__restrict__ dense, uint64_t dcap, int stage_cap,
                   uint32_t *__restrict__ dcnt, int reset_cnt,
                   const unsigned long long *__restrict__ fullmin,
                   const unsigned long long *tau, int KO, const int32_t *__restrict__ qprog,
                   const unsigned long long *__restrict__ popcnt, uint64_t nrows,
                   FvHit *__restrict__ out, uint32_t *__restrict__ out_cnt,
                   uint8_t *__restrict__ trunc, unsigned long long *tau_out,
                   uint8_t *__restrict__ unc, int estimated, int mode) {
    extern __shared__ __align__(16) unsigned char dm_smem[];
    pdl_wait();
    pdl_trigger();
    dense_merge_query(blockIdx.x, (uint64_t *)dm_smem, dense, dcap, stage_cap, dcnt, reset_cnt,
                      fullmin, tau, KO, qprog, popcnt, nrows, out, out_cnt, trunc, tau_out, unc,
                      estimated != 0, mode);
}

// KO <= 32
__global__ void __launch_bounds__(DM_THREADS)
dense_top32_kernel(const uint64_t *__restrict__ dense, uint64_t dcap, uint32_t *__restrict__ dcnt,
                   int reset_cnt, const unsigned long long *__restrict__ fullmin,
                   const unsigned long long *tau, int KO, const int32_t *__restrict__ qprog,
                   const unsigned long long *__restrict__ popcnt, uint64_t nrows,
                   FvHit *__restrict__ out, uint32_t *__restrict__ out_cnt,
                   uint8_t *__restrict__ trunc, unsigned long long *tau_out,
                   uint8_t *__restrict__ unc, int estimated, int late_counts) {
    __shared__ uint64_t lists[DM_THREADS / 32][32];
    // the batch's programs and the bitmap kernel's counts were written two
    // or more kernels back (each kernel of the chain triggers the next only
    // after its own wait): read them while the kernel ahead finishes, unless
    // that is the one that counts (late_counts)
    long long passing = -1;
    if (threadIdx.x == 0 && !late_counts) {
        const int pg = qprog[blockIdx.x];
        passing = (long long)(pg >= 0 ? popcnt[pg] : nrows);
    }
    pdl_wait();
    pdl_trigger();
    dense_top32_query(blockIdx.x, lists, dense, dcap, dcnt, reset_cnt, fullmin, tau, KO, qprog,
                         popcnt, nrows, out, out_cnt, trunc, tau_out, unc, passing,
                         estimated != 0);
}

cudaError_t launch_dense_merge(const uint64_t *dense, uint64_t dcap, uint32_t *dcnt,
                               bool reset_cnt, const unsigned long long *fullmin,
                               const unsigned long long *tau, int KO, const int32_t *qprog,
                               const unsigned long long *popcnt, uint64_t nrows, int nq,
                               FvHit *out, uint32_t *out_cnt, uint8_t *trunc,
                               unsigned long long *tau_out, uint8_t *unc, cudaStream_t st,
                               bool estimated, bool late_counts, int mode) {
    if (KO < 1 || KO > DM_OUT) return cudaErrorInvalidValue;
    // The warps' lists where they hold the answer (KO 10 of 2048 runs of 200
    // and 1,000 keys: 0.0205 and 0.0225 ms, the radix select 0.031 and 0.033),
    // else the radix select (KO 48 of 1,000 keys: 0.045 ms, lists of 64 0.065;
    // KO 400 of 512 runs of 1,500 keys with the re-rank: 0.056 ms; with all
    // eight digits, a sort of 45 barriers and 32 candidates of a query in
    // flight 0.097).
    if (KO <= 32)
        return launch_pdl(dense_top32_kernel, dim3(nq), dim3(DM_THREADS), 0, st, dense, dcap, dcnt,
                          reset_cnt ? 1 : 0, fullmin, tau, KO, qprog, popcnt, nrows, out, out_cnt,
                          trunc, tau_out, unc, estimated ? 1 : 0, late_counts ? 1 : 0);
    // the stage holds a whole run when it can (runs never exceed dcap)
    const int stage_cap = (int)std::min<uint64_t>(std::max<uint64_t>(dcap, 1), DM_CAP_MAX);
    const size_t smem = (size_t)(stage_cap + DM_OUT) * 8;
    cudaError_t e = raise_smem_limit((const void *)dense_merge_kernel, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(dense_merge_kernel, dim3(nq), dim3(DM_THREADS), smem, st, dense, dcap,
                      stage_cap, dcnt, reset_cnt ? 1 : 0, fullmin, tau, KO, qprog, popcnt, nrows,
                      out, out_cnt, trunc, tau_out, unc, estimated ? 1 : 0, mode);
}

// ---------------------------------------------------------------- host side
static PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) ==
                cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 2-D row-major [rows][inner] tensor map with 128-byte swizzled boxes of
// [128 rows][128 bytes] (elements of the operand kind: fp8, bf16 or f32).
// Columns past `inner` read as zeros.
bool tc_make_tmap(CUtensorMap *m, const void *ptr, int kind, uint64_t inner, uint64_t rows) {
    auto enc = get_encode();
    if (!enc) return false;
    const uint32_t esz = (uint32_t)tck_esz(kind);
    cuuint64_t dims[2] = {inner, rows};
    cuuint64_t strides[1] = {inner * esz};
    cuuint32_t box[2] = {TC_KB_BYTES / esz, TC_BN};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapDataType dt = kind == TCK_FP8    ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                   : kind == TCK_TF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                                      : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUresult r = enc(m, dt, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Candidates kept per query before the exact re-rank (the superset): 4k
// while the scan's distances may be inexact; k itself when the upload
// certified that BF16 distances are exact (integer rows, |x| <= 256, all
// sums below 2^24), since then the scan's top-k already is the exact top-k.
// 0 = topb too large.
int tc_superset(const FvGpuIndex *g, uint32_t topb, float q_amax) {
    const bool exact = g->precision != FV_GPU_PREC_FP8 && !g->force_wide_superset &&
                       pv_bf16_exact(g->dim, g->row_amax, q_amax);
    const int s = exact ? (int)topb : 4 * (int)topb;
    return s <= TC_MAX_SUPERSET ? s : 0;  // 0: topb beyond the superset capacity
}

// The exact scan on the tensor cores reads the f32 rows as TF32 and
// re-ranks a superset exactly: S = k when the upload certified integer rows
// (TF32 keeps integers up to 2048 exactly, so the norm-form distances are
// exact as in the BF16 case), else 4k (at least 16), each query's answer
// then certified by the re-rank's error bound (RerankCert) and re-run on the
// CUDA cores when the bound does not separate it. 0 = topb too large, or
// rows (one infinite or NaN value is enough) whose norms leave no query
// certifiable: such a table is scanned on the CUDA cores at once.
int tf32_superset(const FvGpuIndex *g, uint32_t topb, float q_amax) {
    const bool exact = !g->force_wide_superset && pv_bf16_exact(g->dim, g->row_amax, q_amax);
    if (!exact && !(g->norm32_max < 0x1p126f)) return 0;
    const int s = exact ? (int)topb : std::max(4 * (int)topb, 16);
    return s <= TC_MAX_SUPERSET ? s : 0;
}

// For which k a table of rows beyond 128 dims goes through TF32 at all. Below
// that width every batch of 16+ queries does; wider rows were the CUDA-core
// scan's alone, and where the certificate then sends most queries there after
// all, the call takes half as long again: 64 real-valued queries of 60,000 x
// 512 rows in clusters of 200, k 10 0.48 ms instead of 0.37, 0.37 through
// TF32 alone for k 100. So 16 rows are looked up at upload by the exact scan,
// and for k of 1, 2, 4 .. the share of them is kept whose gap between the
// k-th and the superset's last distance the certificate's bound would leave
// open.
constexpr int TL_Q = 16, TL_K = 257;  // (a row finds itself too)
void tf32_look(FvGpuIndex *g, const float *vectors) {
    memset(g->tf32_share, 0, sizeof(g->tf32_share));
    if (g->dpad <= 128 || !tf32_supported(g) || !(g->norm32_max < 0x1p126f) ||
        tc_supported(g))  // (the low-precision rows are scanned)
        return;
    const uint64_t stride = g->count / TL_Q;  // row p * stride is query p
    std::vector<FvHit> hits((size_t)TL_Q * TL_K);
    std::vector<uint32_t> cnt(TL_Q);
    // the exact scan on scratch of its own: [queries][bounds][keys][counts]
    // [no program][filter count][hits][counts][flags]
    ScanPlan pl;
    if (!plan_scan_f32(g->count, g->dpad, TL_Q, TL_K, g->sm_count, pl)) return;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t row = (size_t)g->dpad * 4;
    const size_t o_tau = al(TL_Q * row), o_part = o_tau + al(TL_Q * 8);
    const size_t o_pcnt = o_part + al((size_t)TL_Q * pl.grow * TL_K * 8);
    const size_t o_prog = o_pcnt + al((size_t)TL_Q * pl.grow * 4), o_pop = o_prog + al(TL_Q * 4);
    const size_t o_hit = o_pop + 256, o_cnt = o_hit + al(hits.size() * sizeof(FvHit));
    const size_t o_tr = o_cnt + al(TL_Q * 4);
    char *d = nullptr;
    cudaError_t e = cudaMalloc(&d, o_tr + al(TL_Q));
    for (int p = 0; p < TL_Q && e == cudaSuccess; p++)
        e = cudaMemcpyAsync(d + p * row, g->d_vecs + p * stride * (uint64_t)g->dpad, row,
                            cudaMemcpyDeviceToDevice, g->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d + o_tau, 0xFF, TL_Q * 8, g->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d + o_prog, 0xFF, TL_Q * 4, g->stream);
    if (e == cudaSuccess) {
        ScanF32Args a;
        a.vecs = g->d_vecs;
        a.nrows = g->count;
        a.dpad = g->dpad;
        a.queries = (const float *)d;
        a.nq = TL_Q;
        a.bitmaps = nullptr;
        a.bm_words = (g->count + 31) / 32;
        a.qprog = (const int32_t *)(d + o_prog);
        a.K = TL_K;
        a.S = pl.S;
        a.CB = pl.CB;
        a.rows_per_cta = pl.rows_per_cta;
        a.grow = pl.grow;
        a.qtiles = pl.qtiles;
        a.tau = (unsigned long long *)(d + o_tau);
        a.part = (uint64_t *)(d + o_part);
        a.part_cnt = (uint32_t *)(d + o_pcnt);
        e = launch_scan_f32(a, pl, g->stream);
        if (e == cudaSuccess)
            e = launch_merge(a.part, a.part_cnt, pl.grow, TL_K, pl, a.tau, a.qprog,
                             (const unsigned long long *)(d + o_pop), g->count, TL_Q,
                             (FvHit *)(d + o_hit), (uint32_t *)(d + o_cnt), (uint8_t *)(d + o_tr),
                             g->stream);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(hits.data(), d + o_hit, hits.size() * sizeof(FvHit),
                            cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(cnt.data(), d + o_cnt, TL_Q * 4, cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    cudaFree(d);
    if (e != cudaSuccess) {  // (no room, say: the CUDA-core scan it is)
        (void)cudaGetLastError();
        return;
    }
    const double c2 = (g->dpad + 8) * 0x1p-23;
    for (int p = 0; p < TL_Q; p++) {
        double qn = 0.0, qr = 0.0;
        for (int j = 0; j < g->dim; j++) {
            const float v = vectors[p * stride * (uint64_t)g->dim + j];
            uint32_t u;
            memcpy(&u, &v, 4);
            u &= 0xFFFFE000u;
            float t;
            memcpy(&t, &u, 4);
            qn += (double)v * v;
            qr += ((double)v - t) * ((double)v - t);
        }
        double d[TL_K];  // distances, the row itself left out
        int n = 0;
        for (uint32_t i = 0; i < std::min<uint32_t>(cnt[p], TL_K); i++)
            if (hits[(size_t)p * TL_K + i].node != p * stride)
                d[n++] = hits[(size_t)p * TL_K + i].dist;
        for (int i = 0; i < FvGpuIndex::TF32_KS; i++) {
            const int k = 1 << i, S = std::min(std::max(4 * k, 16), n);
            if (k > n) break;
            const double A = d[S - 1];
            const double E = tf32_scan_error(g->dpad, g->norm32_max, g->res32_max, qn, qr, A);
            g->tf32_share[i] += (A - E) * (1.0 - c2) > d[k - 1] ? 1 : 0;
        }
    }
}

// Whether an exact batch that can take the TF32 scan (superset S) should:
// pass, the share of the rows its filters let through, thins the neighbours
// out. Three of four queries looked up must come through, for the k's on
// either side; and lists shorter than the superset lose its rows where they
// are stored cluster by cluster (250,000 x 200 such rows, 40 queries, k 100:
// all run again, 1.3 ms instead of 0.49).
bool tf32_pays(const FvGpuIndex *g, uint32_t topb, int S, double pass) {
    if (g->dpad <= 128) return true;
    if (S > TC_MAX_LIST && !g->rows_mixed) return false;
    if (S == (int)topb) return true;  // (distances are exact)
    const double k = log2((double)topb / std::max(pass, 1e-9));
    const int lo = std::min((int)k, FvGpuIndex::TF32_KS - 1);
    const int hi = std::min(lo + (k > lo ? 1 : 0), FvGpuIndex::TF32_KS - 1);
    return std::min(g->tf32_share[lo], g->tf32_share[hi]) >= TL_Q * 3 / 4;
}

// Rows of at most 512 f32 (beyond 128 the query tile streams with the rows),
// at least 8 row tiles, and not switched off for the index.
bool tf32_supported(const FvGpuIndex *g) {
    return g->exact_tc && g->d_norm32 && g->dpad <= 512 && g->count >= 8 * (uint64_t)TC_BN;
}

bool tc_supported(const FvGpuIndex *g) {
    if (g->precision == FV_GPU_PREC_FP32 || !g->d_vlow) return false;
    const int row_bytes = g->kpad * (g->precision == FV_GPU_PREC_FP8 ? 1 : 2);
    return row_bytes <= 512;  // query tile <= 64 KB of shared memory
}

// (kinds other than TF32 have at most 4 K-blocks)
static bool tc_qstream(int kblocks) { return kblocks > 4; }
static size_t tc_smem(int kblocks, int NS, int KP, int EPI) {
    return tc_smem_bytes(kblocks, NS, KP, EPI, tc_qstream(kblocks));
}

bool tc_shape_fits(const FvGpuIndex *g, uint32_t topb, int epi, int ns) {
    if (!tc_supported(g) || epi < 1 || epi > 3 || ns < 2 || ns > TC_MAX_STAGES) return false;
    const int S = tc_superset(g, topb, -1.f);
    if (!S) return false;
    const int kblocks = g->kpad * (g->precision == FV_GPU_PREC_FP8 ? 1 : 2) / TC_KB_BYTES;
    const int KP = std::min(S, tc_list_cap(epi, kblocks));
    return tc_smem(kblocks, ns, KP, epi) <= 227 * 1024;
}

template <int KIND, int EPI, bool WARM>
static cudaError_t tc_launch_kind(int grid, size_t smem, cudaStream_t st, const CUtensorMap &tmX,
                                  const CUtensorMap &tmQ, const TcArgs &a) {
    cudaError_t e = raise_smem_limit((const void *)scan_tc_kernel<KIND, EPI, WARM>, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(scan_tc_kernel<KIND, EPI, WARM>, dim3(grid), dim3(64 + 128 * EPI), smem,
                      st, tmX, tmQ, a);
}

template <int EPI, bool WARM>
static cudaError_t tc_launch(int kind, int grid, size_t smem, cudaStream_t st,
                            const CUtensorMap &tmX, const CUtensorMap &tmQ, const TcArgs &a) {
    if (kind == TCK_FP8) return tc_launch_kind<TCK_FP8, EPI, WARM>(grid, smem, st, tmX, tmQ, a);
    if (kind == TCK_TF32) return tc_launch_kind<TCK_TF32, EPI, WARM>(grid, smem, st, tmX, tmQ, a);
    return tc_launch_kind<TCK_BF16, EPI, WARM>(grid, smem, st, tmX, tmQ, a);
}

// Whether a query's `lists` of KP keys, one tile each of the `rows` that pass,
// fill little without a bound: few kept keys for the merge and few admissions
// per warp (of a list's p passing rows it keeps min(KP, p) and admits about
// KP (1 + ln(p / KP))). The sample and its merge take 8 to 20 us; 1 to 7
// queries of 50,000 to 100,000 rows with k of 1 or 2, or 1.6 % of the rows
// passing, took 10 to 20 us more with them. (The lines, over 6,000 batches of
// 1 to 300 queries: the merge takes what the sample saves from 5,000 kept keys
// on, from 4,400 with 100 admissions a warp; the pass does from 150 admissions
// on. Below, unseeded is 1 to 10 us faster; a little beyond, 2 to 10 slower.)
bool tc_fills_little(int KP, uint64_t lists, double rows, int nq, int qtiles) {
    const double p = rows / (double)lists;
    const double kept = std::min<double>(KP, p);
    const double admits = p <= KP ? p : KP * (1.0 + log(p / KP));
    const double per_warp = admits * std::min(32, qtiles > 1 ? 32 : nq);
    return per_warp <= 150.0 && kept * (double)lists + 8.0 * per_warp <= 5200.0;
}

// Launches query prep, the tensor-core scan, the per-query merge and the
// exact re-rank. Inputs: f32 queries [nq][dpad] on the device, predicate
// programs/bitmaps already built. tf32: scan the f32 rows themselves (the
// exact mode), else the upload's BF16 / FP8 rows.
int launch_scan_tc(FvGpuIndex *g, int nq, float q_amax, const float *d_q,
                   const int32_t *d_qprog,
                   const uint32_t *bitmaps, uint64_t bm_words,
                   const unsigned long long *popcnt, uint32_t topb, FvHit *d_out,
                   uint32_t *d_cnt, uint8_t *d_trunc, cudaEvent_t *ev, char *errbuf,
                   size_t errlen, const TcLazy *lz, bool tf32, const TcRowSet *rs,
                   bool behind_bitmaps, cudaEvent_t prep_done, double pass, bool redo) {
    const bool fp8 = !tf32 && g->precision == FV_GPU_PREC_FP8;
    const int kind = tf32 ? TCK_TF32 : fp8 ? TCK_FP8 : TCK_BF16;
    const int esz = tck_esz(kind);
    // elements of K per row: the low-precision row pitch, or dpad rounded up
    // to whole 32-element boxes (the f32 rows' tail boxes read zeros)
    const int kelems = tf32 ? ((g->dpad + 31) & ~31) : g->kpad;
    const int kblocks = kelems * esz / TC_KB_BYTES;
    const int S = tf32 ? tf32_superset(g, topb, q_amax) : tc_superset(g, topb, q_amax);
    g->last_superset = S;
    g->tc_unc = nullptr;
    if (!S || !(tf32 ? tf32_supported(g) : tc_supported(g)) || (rs && lz)) {
        snprintf(errbuf, errlen, "gpu: tensor-core scan not available for this batch");
        return -1;
    }
    const int qtiles = (nq + TC_BM - 1) / TC_BM;
    const int nqpad = qtiles * TC_BM;
    // query replicas: as many as the batch leaves room for, while each
    // part of a tile keeps at least 32 rows (one TMEM load)
    int R = 1;
    if (g->tune_rep > 0) R = g->tune_rep;
    else if (qtiles == 1) R = nq <= 32 ? 4 : nq <= 64 ? 2 : 1;
    while (R > 1 && (TC_BM / R < nq || TC_BN / R < 32)) R >>= 1;
    const int bq = TC_BM / R;
    // epilogue warp groups (each owning every EPI-th tile): three where every
    // warp has 128 rows of a tile to go through (more than 64 queries: 0.227
    // against 0.237 ms for 512 over 1M BF16 rows, 0.55 against 0.72 ms for
    // 512 over 2M FP8 rows with supersets of 400), else two (with 64 queries
    // three run the same: 0.0615 ms), one where a tile's rows take longer to
    // arrive than one group to look through (16 queries over BF16 rows, 64
    // over f32 rows: the same pass, half the lists to merge, 0.088 against
    // 0.094 ms in all) or the lists do not fit with two. With three, lists of
    // up to 32 keys that spill: 64 keys left room for one group (2048 queries,
    // 500,000 BF16 rows, k 64: the pass 2.25 ms, 48 keys and two groups 1.08
    // for k 48; now 0.80 and 0.76). The automatic shape stays within smem_pref,
    // which leaves each SM a few KB for a small kernel beside the scan (the
    // router's, a merge launched early).
    const size_t smem_cap = 227 * 1024;
    const size_t smem_pref = 222 * 1024;
    // stages: up to 128 KB of rows in flight
    const int ns0 = std::min(TC_MAX_STAGES, std::max(
        2, (int)(128 * 1024 / ((size_t)std::min(kblocks, TC_KBS) * TC_BOX *
                                         (tc_qstream(kblocks) ? 2 : 1)))));
    int EPI = 0, NS = 0;
    auto shape = [&](int most) {
        EPI = 0;
        for (int e = most; e >= 1 && !EPI; e--) {
            const int KPe = std::min(S, tc_list_cap(e, kblocks));
            int n = ns0;
            while (n > 2 && tc_smem(kblocks, n, KPe, e) > smem_pref) n--;
            if (tc_smem(kblocks, n, KPe, e) <= smem_pref) {
                EPI = e;
                NS = n;
            }
        }
        if (!EPI) {  // the smallest shape, within the hard limit
            EPI = 1;
            NS = 2;
        }
    };
    // (three groups' lists hold every nearest row of the query that a list
    // meets: where rows are stored cluster by cluster, only whole lists do;
    // and a run that spills may be full, which flags the query)
    const bool whole3 = S <= tc_list_cap(3, kblocks);
    const bool three = whole3 || (g->rows_mixed && redo);
    shape(kblocks * TC_KB_BYTES * R >= 1024 ? 1 : R == 1 && three ? 3 : 2);
    if (g->tune_epi || g->tune_ns) {  // a tuned shape, if it fits
        const int e = std::min(g->tune_epi ? g->tune_epi : EPI, whole3 || redo ? 3 : 2);
        const int n = g->tune_ns ? g->tune_ns : NS;
        if (e >= 1 && n >= 2 && n <= TC_MAX_STAGES &&
            tc_smem(kblocks, n, std::min(S, tc_list_cap(e, kblocks)), e) <= smem_cap) {
            EPI = e;
            NS = n;
        }
    }
    int KP = std::min(S, tc_list_cap(EPI, kblocks));
    // rows scanned: the index's, or a compacted set
    const uint64_t nrows_scan = rs ? rs->nrows : g->count;
    const uint64_t ntiles_all = (nrows_scan + TC_BN - 1) / TC_BN;
    bool certify = KP < S;  // lists shorter than the superset
    int grow = std::max(1, g->tune_grow > 0 ? g->tune_grow : g->sm_count / qtiles);
    auto split = [&](uint64_t most) {  // CTAs along the rows, evenly loaded
        if ((uint64_t)grow > most) grow = (int)most;
        const uint64_t per = (ntiles_all + grow - 1) / grow;
        grow = (int)((ntiles_all + per - 1) / per);
        return per;
    };
    uint64_t tpc = split((ntiles_all + 1) / 2);
    // Seeding pass: a few tiles per CTA from an evenly strided sample; the
    // rank-th key of the sample bounds the S-th key of the whole scan, so the
    // main pass admits only rows that can still matter. Tiles per CTA, spread
    // over its own range: a tile more costs the sample one tile's time, and a
    // list of the main pass admits about S * tpc / (m * grow) rows; the sum is
    // least near sqrt(S tpc / grow) times a constant measured at 1 (batch 512,
    // 128 and 64 of 1M rows: half and twice as many tiles are both slower or
    // the same). At most 24 (graph construction, 2048 queries with lists of
    // 64: 62.6 ms for 60,000 rows with 24, 70.6 with 8; batch 1000 the same
    // with both), 8 where an estimated bound makes up for a short sample; and
    // chunks for four times the keys a certain bound needs.
    // A compacted set has room for more rows than pass: the tiles that exist
    // are a prefix, so the sample's are dealt round robin (every CTA has some
    // of them) and as many more are drawn as `pass` leaves empty.
    const double fill = !rs || pass > 0.9 ? 1.0 : std::max(pass, 1.0 / 64);
    const bool full = !rs || pass > 0.99;  // (what fills its last tile may be missing)
    const uint64_t region = rs ? tpc : ntiles_all / grow;
    const double best = sqrt((double)S * tpc * fill / grow);
    const bool may_est = certify && S > TC_MAX_LIST && g->rows_mixed && redo;
    const uint64_t least = may_est ? 1 : ((uint64_t)S + grow - 1) / grow;
    const double want_m = std::min<double>(may_est ? 8 : 24, std::max<double>(least, floor(best)));
    uint64_t m = (uint64_t)std::min<double>((double)region, ceil(want_m / fill));
    // The sample's S-th key is a bound for certain, but with large supersets
    // it admits S / share rows, far more than S. A sample holding `share` of
    // the rows has S * share of the S best in expectation, with a Poisson
    // spread: its key six deviations above that lies beyond the S-th key of
    // the scan but for about one query in 10^9, and the merge sees such a
    // query (fewer than S keys got through), which is then re-run exactly.
    // Only where the merge certifies anyway (lists shorter than the superset)
    // and rows lie in no order (else the best clump in the sample's tiles),
    // and not for up to 64 keys, which a certain bound costs little (512
    // queries, 500,000 rows, S 40: 0.180 against 0.170 ms).
    int rank_est = S;
    double share = 1.0;
    auto enough = [&]() {  // chunk minima for the bound's rank, twice over
        // A compacted set with room to spare: the strides reach past the
        // prefix of tiles that exist, so the sample holds every step-th of
        // them and one more, not m of the room (which gave 256 queries of 1M
        // FP8 rows, k 75, a bound below their superset when half of the room
        // was used; all were run twice). Right down to half of the expected
        // tiles.
        share =
            full ? std::min(1.0, (double)m * grow * TC_BN / (double)nrows_scan)
                 : std::min(1.0, 1.0 / (double)std::max<uint64_t>(1, region / m) +
                                     2.0 / (fill * (double)region));
        rank_est = may_est ? (int)ceil(S * share + 6.0 * sqrt(S * share) + 8.0) : S;
        return (uint64_t)(m * fill * grow * (TC_BN / 32)) >= 2 * (uint64_t)std::min(S, rank_est);
    };
    // (a table of few tiles is sampled more of: 60,000 rows, 512 queries,
    // S 800 took 1.08 ms without a bound, 0.36 seeded)
    while (!enough() && m < region) m++;
    // Rows stored cluster by cluster: a query's nearest lie in a few chunks of
    // a few tiles, of which the sample keeps one row a chunk, so its bound is
    // loose and the pass admits cluster after cluster. Four times the tiles,
    // then, and every chunk's best row kept (k 100, 200 queries of 300,000 x
    // 32 BF16 rows: 1229 us a call without either, 490 with both; 715 behind
    // heaps of a smaller sample's best keys. 2,160 batches over such tables:
    // 1.36 times as fast as behind those heaps, 1.05 without either). Three
    // times as many are 1 % slower, eight times as many the same.
    // (Batches that may test their filters lazily cannot tell a chunk's best
    // passing row: twice their share of the best keys.)
    const bool clusters = !g->rows_mixed && !lz;
    if (clusters) m = std::min<uint64_t>(region, 4 * m);
    const bool estimated = rank_est < S;
    const int rank = std::min(S, rank_est);
    // Seeding pays from two tiles per CTA on, as long as the sample's chunk
    // minima are at least twice the keys its bound needs (enough): small tables took
    // 2 to 4 times as long filling their lists behind no bound (100,000 BF16
    // rows, 73 queries: k 2, 25, 100 in 0.106, 0.158, 0.343 ms, seeded 0.043,
    // 0.044, 0.079). Without it every tile gets its own CTA.
    // Nor does it pay when lists fill little without a bound (tc_fills_little).
    const uint64_t ugrow = std::min<uint64_t>(std::max(1, g->sm_count / qtiles), ntiles_all);
    const bool little = tc_fills_little(KP, ugrow * EPI * R, pass * (double)nrows_scan, nq, qtiles);
    const bool seed = g->tune_seed != 2 && !little && enough();
    if (!seed) {
        if (EPI == 3) {  // without a bound: lists that keep the best
            shape(2);
            KP = std::min(S, tc_list_cap(EPI, kblocks));
            certify = KP < S;
        }
        grow = std::max(1, g->tune_grow > 0 ? g->tune_grow : g->sm_count / qtiles);
        tpc = split(ntiles_all);
    }

    // A run that spills has to hold what its query's bound lets through, and
    // the sample of a large table leaves that far above S: room for 2.5 times
    // rank / share (chunk minima lie 1.15 times as deep, and six deviations of
    // 64 keys are another 1.75), or whole lists where that is more than 1 GB.
    // With 64 keys a list and no more, every query of large batches over large
    // tables was run again: 1024 queries of 4M x 64 rows, k 40 61 ms (whole
    // lists 5.0 before there were short ones, now 2.1), of 10M FP8 rows, k 10
    // 150 ms (12.5, now 5.5), graphs of 1M rows 11.7 s (3.2, now 1.0). Whole
    // lists from 3,000 keys on instead take 1.1 to 2.1 times as long.
    uint64_t run_keys = (uint64_t)grow * EPI * R * std::min(S, TC_MAX_LIST);
    if (seed && certify && EPI == 3) {
        run_keys = std::max(run_keys, (uint64_t)(2.5 * rank / share) +
                                          (uint64_t)grow * EPI * R * KP);
        if ((uint64_t)nq * run_keys * 8 > 1ull << 30) {
            shape(2);
            KP = std::min(S, tc_list_cap(EPI, kblocks));
            certify = KP < S;
        }
    }

    ScanScratch &s = g->scan;
    const size_t qbytes = (size_t)nqpad * kelems * esz;
    const size_t off_qn = (qbytes + 255) & ~(size_t)255;
    const size_t off_qs = off_qn + (((size_t)nqpad * 4 + 255) & ~(size_t)255);
    const size_t off_err = off_qs + (((size_t)nqpad * 4 + 255) & ~(size_t)255);
    // (the flags lie behind the watchdog word: one copy brings both)
    const size_t off_unc = off_err + TC_TAIL_UNC;
    const size_t off_cand = off_unc + (((size_t)nq + 255) & ~(size_t)255);
    const size_t off_ccnt = off_cand + (((size_t)nq * S * sizeof(FvHit) + 255) & ~(size_t)255);
    const size_t off_ctr = off_ccnt + (((size_t)nq * 4 + 255) & ~(size_t)255);
    const size_t cbytes = off_ctr + (size_t)nq + 256;
    PV_CUDA_OK(s.cand.ensure(cbytes), errbuf, errlen);
    PV_CUDA_OK(s.tau.ensure((size_t)nq * 8), errbuf, errlen);
    const size_t smem = tc_smem(kblocks, NS, KP, EPI);
    const int nlists = grow * EPI * R;  // lists per query
    const bool spill = seed && certify && EPI == 3;
    // a query's dense run at most
    const uint64_t dcap = spill ? run_keys : (uint64_t)nlists * KP;
    PV_CUDA_OK(s.part.ensure((size_t)nq * dcap * 8), errbuf, errlen);
    // [dcnt u32 x nq][fullmin u64 x nq]
    const size_t off_fm = ((size_t)nq * 4 + 255) & ~(size_t)255;
    PV_CUDA_OK(s.part_cnt.ensure(off_fm + (size_t)nq * 8), errbuf, errlen);
    uint32_t *d_dcnt = s.part_cnt.as<uint32_t>();
    unsigned long long *d_fullmin = (unsigned long long *)(s.part_cnt.as<char>() + off_fm);
    unsigned char *c = s.cand.as<unsigned char>();
    int *d_err = (int *)(c + off_err);
    // inexact scan distances of exact-mode batches: the re-rank certifies
    const bool num_cert = tf32 && S > (int)topb;

    g->launches += 4;  // query prep, main pass, merge, re-rank
    PV_CUDA_OK(launch_pdl(query_prep_kernel, dim3((nqpad + 7) / 8), dim3(256), 0, g->stream, d_q,
                          nq, g->dpad, g->dim, nqpad, R > 1 ? bq : nqpad, kelems, kind, c,
                          (float *)(c + off_qn),
                          fp8 || tf32 ? (float *)(c + off_qs) : nullptr,
                          s.tau.as<unsigned long long>(), d_dcnt,
                          certify ? d_fullmin : nullptr, d_err, behind_bitmaps ? 1 : 0),
               errbuf, errlen);
    if (prep_done) PV_CUDA_OK(cudaEventRecord(prep_done, g->stream), errbuf, errlen);

    static_assert(sizeof(CUtensorMap) == sizeof(g->tmap_x), "CUtensorMap size");
    CUtensorMap tmX, tmQ;
    bool &x_ok = rs ? g->tmap_c_ok : tf32 ? g->tmap_x32_ok : g->tmap_x_ok;
    unsigned char *x_map = rs ? g->tmap_c : tf32 ? g->tmap_x32 : g->tmap_x;
    if (tf32 && !rs && g->tmap_x32_rows != g->count) x_ok = false;  // encoded for the current rows
    if (rs && (g->tmap_c_ptr != rs->rows || g->tmap_c_rows != rs->nrows || g->tmap_c_kind != kind))
        x_ok = false;
    if (rs && !x_ok) {
        if (!tc_make_tmap(&tmX, rs->rows, kind, (uint64_t)(tf32 ? g->dpad : g->kpad), rs->nrows)) {
            snprintf(errbuf, errlen, "gpu: tensor map encoding failed");
            return -1;
        }
        memcpy(x_map, &tmX, sizeof(tmX));
        x_ok = true;
        g->tmap_c_ptr = rs->rows;
        g->tmap_c_rows = rs->nrows;
        g->tmap_c_kind = kind;
    }
    if (!x_ok) {
        const bool okm = tf32 ? tc_make_tmap(&tmX, g->d_vecs, kind, (uint64_t)g->dpad, g->count)
                              : tc_make_tmap(&tmX, g->d_vlow, kind, (uint64_t)g->kpad, g->count);
        if (!okm) {
            snprintf(errbuf, errlen, "gpu: tensor map encoding failed");
            return -1;
        }
        memcpy(x_map, &tmX, sizeof(tmX));
        x_ok = true;
        if (tf32) g->tmap_x32_rows = g->count;
    }
    memcpy(&tmX, x_map, sizeof(tmX));
    if (g->tmap_q_ptr != c || g->tmap_q_rows != (uint64_t)nqpad || g->tmap_q_kind != kind) {
        if (!tc_make_tmap(&tmQ, c, kind, (uint64_t)kelems, (uint64_t)nqpad)) {
            g->tmap_q_ptr = nullptr;
            snprintf(errbuf, errlen, "gpu: tensor map encoding failed");
            return -1;
        }
        memcpy(g->tmap_q, &tmQ, sizeof(tmQ));
        g->tmap_q_ptr = c;
        g->tmap_q_rows = (uint64_t)nqpad;
        g->tmap_q_kind = kind;
    }
    memcpy(&tmQ, g->tmap_q, sizeof(tmQ));
    TcArgs a;
    a.nrows = nrows_scan;
    a.kblocks = kblocks;
    a.nq = nq;
    a.qtiles = qtiles;
    a.grow = grow;
    a.tiles_per_cta = tpc;
    a.KP = KP;
    a.rep = R;
    a.bq = bq;
    a.push_tau = KP == S ? 1 : 0;
    a.spill = spill ? 1 : 0;
    a.NS = NS;
    a.qstream = tc_qstream(kblocks) ? 1 : 0;
    a.xnorm = rs ? rs->norms : tf32 ? g->d_norm32 : g->d_norm;
    a.xscale = fp8 ? (rs ? rs->scales : g->d_vscale) : nullptr;
    a.rowids = rs ? rs->rowids : nullptr;
    a.nrows_dev = rs ? rs->nrows_dev : nullptr;
    a.qnorm = (const float *)(c + off_qn);
    a.qscale = fp8 ? (const float *)(c + off_qs) : nullptr;
    a.qprog = d_qprog;
    a.bitmaps = bitmaps;
    a.bm_words = bm_words;
    a.lazy = lz ? lz->flag : nullptr;
    a.progs = lz ? lz->progs : nullptr;
    a.insns = lz ? lz->insns : nullptr;
    a.consts = lz ? lz->consts : nullptr;
    a.nconsts = lz ? lz->nconsts : 0;
    a.cols = g->d_cols;
    a.ncols = g->ncols;
    a.tau = s.tau.as<unsigned long long>();
    a.dense = s.part.as<uint64_t>();
    a.dcnt = d_dcnt;
    a.dcap = dcap;
    a.fullmin = certify ? d_fullmin : nullptr;
    a.err = d_err;
    a.timeout_ns = g->tc_timeout_ns ? g->tc_timeout_ns : 2000000000ull;
    a.drain_ns = 2000000000ull;
    a.trace = nullptr;
    a.trace_tiles = 0;
    static const bool tracing = getenv("PV_TC_TRACE") != nullptr;
    static uint64_t *d_trace = nullptr;
    if (tracing) {
        if (!d_trace) cudaMalloc(&d_trace, 64 * 4 * 8);
        if (d_trace) {
            cudaMemsetAsync(d_trace, 0, 64 * 4 * 8, g->stream);
            a.trace = d_trace;
            a.trace_tiles = 64;
        }
    }
    // warm: a seeding pass, or one that starts without a bound (see tc_pass)
    // (a warm pass with three groups would not fit its registers: it runs
    // with two, inside the same shared-memory carve and dense runs)
    auto run = [&](const TcArgs &args, bool warm) {
        const int gr = args.grow * qtiles;
        if (warm)
            return EPI >= 2 ? tc_launch<2, true>(kind, gr, smem, g->stream, tmX, tmQ, args)
                            : tc_launch<1, true>(kind, gr, smem, g->stream, tmX, tmQ, args);
        if (EPI == 3) return tc_launch<3, false>(kind, gr, smem, g->stream, tmX, tmQ, args);
        if (EPI == 2) return tc_launch<2, false>(kind, gr, smem, g->stream, tmX, tmQ, args);
        return tc_launch<1, false>(kind, gr, smem, g->stream, tmX, tmQ, args);
    };
    FvHit *cand = (FvHit *)(c + off_cand);
    uint32_t *ccnt = (uint32_t *)(c + off_ccnt);
    if (seed) {
        TcArgs sa = a;
        sa.tile0_mul = rs ? 1 : region;
        sa.tile_step = std::max<uint64_t>(1, region / m) * (rs ? grow : 1);
        sa.tiles_per_cta = m;
        // A list keeps the best key of every few of its chunks, about 4 rank
        // keys in all (the S-th key of a subset of the sample still bounds
        // the S-th key of the scan, and short runs keep the merge cheap):
        // the rank-th of 4 rank chunk minima lies about 1.15 times as deep as
        // the sample's own rank-th key. Lazy batches, which cannot tell a
        // chunk's best passing row, keep their share of the best keys; a
        // full list's last key then bounds the S-th key if it holds S. Rows in
        // clusters: as many chunks' best as a list takes.
        const int epiw = std::min(EPI, 2);
        const int chunks = (int)((m + epiw - 1) / epiw) * (TC_BN / R / 32);  // of a list
        const int lists = grow * (int)std::min<uint64_t>(m, epiw) * R;
        const int want = std::max(1, (4 * rank + lists - 1) / lists);
        sa.KP = std::min(KP * EPI / epiw, clusters ? chunks
                                          : (int)ceil(want / fill) * (g->rows_mixed ? 1 : 2));
        sa.seed_group = std::max(1, std::max(clusters ? 1 : (int)(chunks * fill) / want,
                                             (chunks + sa.KP - 1) / sa.KP));
        sa.push_tau = sa.KP == S ? 1 : 0;
        sa.spill = 0;
        sa.fullmin = nullptr;
        g->launches += 2;  // seeding pass + its merge
        PV_CUDA_OK(run(sa, true), errbuf, errlen);
        // the merge leaves the counts at zero for the main pass
        PV_CUDA_OK(launch_dense_merge(a.dense, dcap, d_dcnt, true, nullptr, a.tau, rank, d_qprog,
                                      popcnt, g->count, nq, cand, ccnt,
                                      (uint8_t *)(c + off_ctr), a.tau, nullptr, g->stream, false,
                                      false, DM_BOUND),
                   errbuf, errlen);
    }
    // stage boundary: everything before the main pass (bitmaps, query prep,
    // seeding) is stage 0, the main pass alone is stage 1
    if (ev) cudaEventRecord(ev[1], g->stream);
    // contiguous tile ranges per CTA; a compacted set's tiles are dealt
    // round robin instead, so the rows that exist (a prefix of its tiles)
    // spread over the CTAs
    a.tile0_mul = rs ? 1 : tpc;
    a.tile_step = rs ? (uint64_t)grow : 1;
    PV_CUDA_OK(run(a, !seed), errbuf, errlen);
    if (ev) cudaEventRecord(ev[2], g->stream);
    uint8_t *d_unc = (certify || num_cert) ? (uint8_t *)(c + off_unc) : nullptr;
    if (S == (int)topb) {
        // certified exact (integer rows and queries, all sums below 2^24):
        // every norm-form distance already is the exact squared L2 distance,
        // so the merged top-k is the answer and needs no re-rank
        g->launches--;
        PV_CUDA_OK(launch_dense_merge(a.dense, dcap, d_dcnt, false, a.fullmin, a.tau, S,
                                      d_qprog, popcnt, g->count, nq, d_out, d_cnt, d_trunc,
                                      nullptr, d_unc, g->stream, seed && estimated),
                   errbuf, errlen);
    } else {
        PV_CUDA_OK(launch_dense_merge(a.dense, dcap, d_dcnt, false, a.fullmin, a.tau, S,
                                      d_qprog, popcnt, g->count, nq, cand, ccnt,
                                      (uint8_t *)(c + off_ctr), nullptr, d_unc, g->stream,
                                      seed && estimated, false, DM_SET),
                   errbuf, errlen);
        RerankCert cert;
        if (num_cert) {
            cert.qnorm = (const float *)(c + off_qn);
            cert.qres = (const float *)(c + off_qs);
            cert.xnmax = g->norm32_max;
            cert.xrmax = g->res32_max;
            cert.dim = g->dpad;
            cert.unc = d_unc;
        }
        auto *rerank = rerank_kernel<RR_LANES8>;
        if (tf32 && g->dpad > 128) {
            ScanPlan pl;
            rerank = !(rs && rs->listed) &&
                             plan_scan_f32t(g->count, g->dpad, nq, (int)topb, g->sm_count, pl)
                         ? rerank_kernel<RR_THREAD> : rerank_kernel<RR_WARP>;
        }
        PV_CUDA_OK(launch_pdl(rerank, dim3(nq), dim3(256), 0, g->stream, g->d_vecs,
                              g->dpad, d_q, cand, ccnt, S, topb, d_qprog, popcnt, g->count, d_out,
                              d_cnt, d_trunc, cert),
                   errbuf, errlen);
    }
    g->tc_unc = d_unc;
    g->tc_unc_n = nq;
    if (ev) cudaEventRecord(ev[3], g->stream);
    g->tc_err = d_err;
    g->tc_err_h = nullptr;  // their host copy, if any, is queued by the caller
    g->tc_unc_h = nullptr;
    if (tracing && d_trace) {
        uint64_t h[64 * 4];
        cudaStreamSynchronize(g->stream);
        cudaMemcpy(h, d_trace, sizeof(h), cudaMemcpyDeviceToHost);
        const uint64_t t0 = h[0];
        for (int t = 0; t < 64 && h[t * 4]; t++)
            fprintf(stderr, "PVTRACE tile %d issue %.2f mma %.2f epi %.2f done %.2f us\n", t,
                    (h[t * 4] - t0) / 1e3, (h[t * 4 + 1] - t0) / 1e3,
                    (h[t * 4 + 2] - t0) / 1e3, (h[t * 4 + 3] - t0) / 1e3);
    }
    return 0;
}

}  // namespace pv

namespace pv {
// Queues the copy of the watchdog word and, where the scan certifies, its
// nq flags into pinned host memory (tc_tail_bytes(nq)) behind the batch's own
// result copy, so reading them costs no extra round trip (two copies into
// pageable memory with a synchronization each took 15 us of a batch).
void tc_tail_enqueue(FvGpuIndex *g, char *h) {
    g->tc_err_h = nullptr;
    g->tc_unc_h = nullptr;
    if (!g->tc_err) return;
    const size_t bytes = g->tc_unc ? TC_TAIL_UNC + (size_t)g->tc_unc_n : sizeof(int);
    if (cudaMemcpyAsync(h, g->tc_err, bytes, cudaMemcpyDeviceToHost, g->stream) != cudaSuccess) {
        (void)cudaGetLastError();
        return;
    }
    g->tc_err_h = (int *)h;
    if (g->tc_unc) g->tc_unc_h = (const uint8_t *)h + TC_TAIL_UNC;
}

int check_tc_watchdog(FvGpuIndex *g, char *errbuf, size_t errlen) {
    if (!g->tc_err) return 0;
    int e = 0;
    if (g->tc_err_h) {  // queued with the results
        PV_CUDA_OK(cudaStreamSynchronize(g->stream), errbuf, errlen);
        e = *(volatile int *)g->tc_err_h;
        g->tc_err_h = nullptr;
    } else {
        PV_CUDA_OK(cudaMemcpyAsync(&e, g->tc_err, 4, cudaMemcpyDeviceToHost, g->stream), errbuf,
                   errlen);
        PV_CUDA_OK(cudaStreamSynchronize(g->stream), errbuf, errlen);
    }
    if (e) {
        cudaMemsetAsync(g->tc_err, 0, 4, g->stream);
        snprintf(errbuf, errlen, "gpu: tensor-core scan wait expired (role %d)", e);
        return -1;
    }
    return 0;
}
}  // namespace pv
