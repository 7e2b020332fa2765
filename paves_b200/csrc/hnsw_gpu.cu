// hnsw_gpu.cu — HNSW graph construction on the GPU.
//
// No counterpart in the reference: its builder is a CPU thread pool that
// inserts rows one at a time (engine.cpp:698-1032). Here rows are inserted
// in batches of doubling size (64, then as many as are already in), and
// each batch takes exact candidates instead of insertion-time beam searches:
//   1. candidates: each new node's C nearest nodes among all nodes inserted
//      so far (its own batch included), exact, from this library's scans
//      with the new nodes as queries over the prefix of the rows (the BF16
//      tensor-core scan when its distances are certified exact, else the
//      exact FP32 scan). Rows are in random order, so the early batches are
//      sparse samples of the data and their lists carry the long-range
//      links an insertion order gives a navigable graph;
//   2. forward selection, one warp per new node: candidates in ascending
//      distance, a candidate is kept when it is closer to the node than to
//      every neighbour kept so far (the neighbour-selection heuristic of
//      the HNSW paper, Malkov & Yashunin, Algorithm 4), up to R; a list
//      left short is topped up with the closest rejected candidates;
//   3. reverse edges: every kept edge u -> v of a new node is offered to v
//      (in-degrees counted with atomics, a prefix sum, a scatter into
//      per-node runs);
//   4. re-selection, one warp per touched node: its current list and its
//      new reverse candidates sorted together (duplicates dropped) and
//      selected again by the same rule to R.
// Level 0 uses R = 2M over all rows, each level L >= 1 uses R = M over the
// nodes whose level is >= L (a sub-index of their rows). Node levels are
// drawn as the engine draws them (so upper levels have the usual sizes),
// the entry point is the lowest-numbered node of the top level. The result
// is a graph in the index-file layout (PvHnsw), searched by the same code
// as any other; its quality contract is search recall, not identity with
// the engine's graph.
#include <string.h>

#include <algorithm>
#include <vector>

#include "index.h"
#include "paves_ext.h"
#include "pv_internal.h"
#include "tc_core.cuh"

namespace pv {

constexpr int HG_CAP = 512;      // candidates per node in the final selection
constexpr int HG_WARPS = 8;      // warps per block of the selection kernels
constexpr int HG_RMAX = 128;     // largest R (2M with M <= 64)

template <int NV>
__device__ __forceinline__ void hg_row(float4 (&r)[NV], const float *x, uint64_t a, int dpad,
                                       int lane) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int j = i * 128 + lane * 4;
        r[i] = j < dpad ? __ldg((const float4 *)(x + a * (uint64_t)dpad + j))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// The selection rule on n ascending candidate keys of node v (smem, warp
// private): keeps up to R candidates, topping up from rejected ones; kept[]
// receives their positions in ck. Returns the number kept. Keys of v
// itself are skipped. A lane holds dims 4 lane + 128 i of a row; the kept
// rows are compared JB at a time and the next candidate's row loads
// meanwhile: one after another each waited out an L2 round trip (0.27 ms a
// batch of 2048 nodes, 64 candidates, now 0.20 ms).
template <int NV>
__device__ int hg_select(const uint64_t *ck, int n, uint32_t v, int R, const float *x, int dpad,
                         uint32_t *kept, uint32_t *rej, int lane) {
    constexpr int JB = NV == 1 ? 8 : NV == 2 ? 4 : 2;
    int nk = 0, nr = 0;
    float4 rn[NV];
    if (n > 0) hg_row<NV>(rn, x, key_row(ck[0]), dpad, lane);
    for (int i = 0; i < n && nk < R; i++) {
        const uint32_t c = key_row(ck[i]);
        float4 rc[NV];
#pragma unroll
        for (int t = 0; t < NV; t++) rc[t] = rn[t];
        if (i + 1 < n) hg_row<NV>(rn, x, key_row(ck[i + 1]), dpad, lane);
        if (c == v) continue;
        const float dc = key_dist(ck[i]);
        bool ok = true;
        for (int j0 = 0; j0 < nk && ok; j0 += JB) {
            float s[JB];
#pragma unroll
            for (int u = 0; u < JB; u++) {
                // (places past the kept ones read the last kept row again)
                float4 rk[NV];
                hg_row<NV>(rk, x, key_row(ck[kept[min(j0 + u, nk - 1)]]), dpad, lane);
                s[u] = 0.f;
#pragma unroll
                for (int t = 0; t < NV; t++) {
                    const float d0 = rc[t].x - rk[t].x, d1 = rc[t].y - rk[t].y,
                                d2 = rc[t].z - rk[t].z, d3 = rc[t].w - rk[t].w;
                    s[u] = fmaf(d0, d0, s[u]);
                    s[u] = fmaf(d1, d1, s[u]);
                    s[u] = fmaf(d2, d2, s[u]);
                    s[u] = fmaf(d3, d3, s[u]);
                }
            }
#pragma unroll
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int u = 0; u < JB; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
            for (int u = 0; u < JB; u++)
                if (s[u] < dc) ok = false;
        }
        if (lane == 0) {
            if (ok) kept[nk] = (uint32_t)i;
            else if (nr < R) rej[nr] = (uint32_t)i;
        }
        __syncwarp();
        if (ok) nk++;
        else if (nr < R) nr++;
    }
    // top up in ascending distance: merge of the kept and rejected positions
    // is not needed, the rejected ones come after (keys stay sorted only
    // within each group, and lists need no order)
    for (int i = 0; i < nr && nk < R; i++) {
        if (lane == 0) kept[nk] = rej[i];
        __syncwarp();
        nk++;
    }
    return nk;
}

// Step 2: forward selection for nodes [n0, n0 + nq) from their scan answers
// (cand [nq][topb] ascending, cnt [nq]); out: fwd keys [node][R] + counts.
template <int NV>
__global__ void __launch_bounds__(32 * HG_WARPS)
hg_forward_kernel(const FvHit *__restrict__ cand, const uint32_t *__restrict__ ccnt, int topb,
                  uint64_t n0, int nq, int R, const float *__restrict__ x, int dpad,
                  uint64_t *__restrict__ fwd, uint32_t *__restrict__ fwd_cnt) {
    __shared__ uint64_t s_ck[HG_WARPS][HG_CAP];
    __shared__ uint32_t s_kept[HG_WARPS][HG_RMAX], s_rej[HG_WARPS][HG_RMAX];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * HG_WARPS + warp;
    if (q >= nq) return;
    const uint64_t v = n0 + q;
    const int n = min((int)ccnt[q], min(topb, HG_CAP));
    for (int i = lane; i < n; i += 32) {
        const FvHit h = cand[(uint64_t)q * topb + i];
        s_ck[warp][i] = make_key(h.dist, (uint32_t)h.node);
    }
    __syncwarp();
    const int nk = hg_select<NV>(s_ck[warp], n, (uint32_t)v, R, x, dpad, s_kept[warp],
                                 s_rej[warp], lane);
    for (int j = lane; j < nk; j += 32) fwd[v * R + j] = s_ck[warp][s_kept[warp][j]];
    if (lane == 0) fwd_cnt[v] = (uint32_t)nk;
}

// Step 3: in-degrees, then the scatter of reverse edges into per-node runs.
// (edges of the sources [u0, u0 + nu))
__global__ void hg_count_kernel(const uint64_t *__restrict__ fwd,
                                const uint32_t *__restrict__ fwd_cnt, uint64_t u0, uint64_t nu,
                                int R, uint32_t *__restrict__ in_cnt) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nu * (uint64_t)R) return;
    const uint64_t u = u0 + i / R;
    if ((uint32_t)(i % R) >= fwd_cnt[u]) return;
    atomicAdd(&in_cnt[key_row(fwd[u * R + i % R])], 1u);
}

// Each node's run among the reverse edges, anywhere (one claim per warp).
__global__ void hg_runs_kernel(const uint32_t *__restrict__ in_cnt, uint64_t n,
                               uint64_t *__restrict__ in_off,
                               unsigned long long *__restrict__ total) {
    const uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const uint32_t c = v < n ? in_cnt[v] : 0u;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t w = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += w;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(total, (unsigned long long)incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (v < n) in_off[v] = base + incl - c;
}

__global__ void hg_scatter_kernel(const uint64_t *__restrict__ fwd,
                                  const uint32_t *__restrict__ fwd_cnt, uint64_t u0, uint64_t nu,
                                  int R, const uint64_t *__restrict__ in_off,
                                  uint32_t *__restrict__ cursor, uint64_t *__restrict__ rev) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nu * (uint64_t)R) return;
    const uint64_t u = u0 + i / R;
    if ((uint32_t)(i % R) >= fwd_cnt[u]) return;
    const uint64_t k = fwd[u * R + i % R];
    const uint32_t v = key_row(k);
    const uint32_t pos = atomicAdd(&cursor[v], 1u);
    rev[in_off[v] + pos] = make_key(key_dist(k), (uint32_t)u);
}

// Step 4: re-selection over a node's list and its new reverse candidates,
// for the nodes [0, n) touched by this batch (new nodes >= lo, or with
// reverse edges); the list (keys, in place) and its count are rewritten.
template <int NV>
__global__ void __launch_bounds__(32 * HG_WARPS)
hg_final_kernel(uint64_t *__restrict__ fwd, uint32_t *__restrict__ fwd_cnt,
                const uint64_t *__restrict__ rev, const uint64_t *__restrict__ in_off,
                const uint32_t *__restrict__ in_cnt, uint64_t n, uint64_t lo, int R,
                const float *__restrict__ x, int dpad) {
    __shared__ uint64_t s_ck[HG_WARPS][HG_CAP];
    __shared__ uint32_t s_kept[HG_WARPS][HG_RMAX], s_rej[HG_WARPS][HG_RMAX];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t v = (uint64_t)blockIdx.x * HG_WARPS + warp;
    if (v >= n || (v < lo && in_cnt[v] == 0)) return;
    uint64_t *ck = s_ck[warp];
    const int nf = (int)fwd_cnt[v];
    // reverse runs longer than the buffer keep their first entries (rare:
    // in-degrees of a pruned neighbour graph stay a small multiple of R)
    const int nr = min((int)in_cnt[v], HG_CAP - nf);
    for (int i = lane; i < nf; i += 32) ck[i] = fwd[v * R + i];
    for (int i = lane; i < nr; i += 32) ck[nf + i] = rev[in_off[v] + i];
    const int n1 = nf + nr;
    int n2 = 1;
    while (n2 < n1) n2 <<= 1;
    for (int i = n1 + lane; i < n2; i += 32) ck[i] = KEY_MAX;
    __syncwarp();
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < (n2 >> 1); i += 32) {
                const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1));
                const int hi = lo | j;
                const uint64_t a = ck[lo], b = ck[hi];
                if ((a > b) == ((lo & k) == 0)) {
                    ck[lo] = b;
                    ck[hi] = a;
                }
            }
            __syncwarp();
        }
    // drop duplicates (an edge present both ways has one key: distances
    // are symmetric)
    int m = 0;
    uint64_t last = KEY_MAX;  // the previous chunk's last key (pads are beyond n1)
    for (int base = 0; base < n1; base += 32) {
        const int i = base + lane;
        const uint64_t k = i < n1 ? ck[i] : KEY_MAX;
        uint64_t p = __shfl_up_sync(0xffffffffu, k, 1);
        if (lane == 0) p = last;
        last = __shfl_sync(0xffffffffu, k, 31);
        const bool keep = i < n1 && k != p;
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        __syncwarp();  // every lane has read its keys before the compaction writes
        if (keep) ck[m + __popc(bal & ((1u << lane) - 1u))] = k;
        m += __popc(bal);
        __syncwarp();
    }
    const int nk = hg_select<NV>(ck, m, (uint32_t)v, R, x, dpad, s_kept[warp], s_rej[warp], lane);
    for (int j = lane; j < nk; j += 32) fwd[v * R + j] = ck[s_kept[warp][j]];
    if (lane == 0) fwd_cnt[v] = (uint32_t)nk;
}

// The rows of an upper level, out of the table's: f32 rows and, where the
// scans read them, the BF16 rows and norms (kpad16: 16-byte pieces of one).
__global__ void hg_gather_kernel(const float *__restrict__ x, int dpad,
                                 const unsigned char *__restrict__ lo, int kpad16,
                                 const float *__restrict__ norm, const uint32_t *__restrict__ ids,
                                 uint64_t n, float *__restrict__ xs, unsigned char *__restrict__ los,
                                 float *__restrict__ norms) {
    const int d16 = dpad / 4, per = d16 + kpad16;
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n * per) return;
    const uint64_t i = p / per, r = ids[i];
    const int j = (int)(p % per);
    if (j < d16)
        ((uint4 *)xs)[i * d16 + j] = __ldg((const uint4 *)x + r * d16 + j);
    else
        ((uint4 *)los)[i * kpad16 + j - d16] = __ldg((const uint4 *)lo + r * kpad16 + j - d16);
    if (j == 0 && norm) norms[i] = __ldg(norm + r);
}

// The lists in the file layout: [cnt, ids...] of stride R + 1.
__global__ void hg_export_kernel(const uint64_t *__restrict__ lst,
                                 const uint32_t *__restrict__ cnt, uint64_t n, int R,
                                 uint32_t *__restrict__ lists) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * (uint64_t)(R + 1)) return;
    const uint64_t v = i / (R + 1);
    const int j = (int)(i % (R + 1));
    const uint32_t c = cnt[v];
    lists[i] = j == 0 ? c : (uint32_t)(j - 1) < c ? key_row(lst[v * R + j - 1]) : 0u;
}

namespace {

struct DevArr {  // a part of HgWork's allocation
    void *p = nullptr;
    template <typename T>
    T *as() const {
        return (T *)p;
    }
};

#define HG_OK(call)                                                                  \
    do {                                                                             \
        cudaError_t e__ = (call);                                                    \
        if (e__ != cudaSuccess) {                                                    \
            if (errbuf && errlen)                                                    \
                snprintf(errbuf, errlen, "hnsw gpu: %s: %s", #call,                  \
                         cudaGetErrorString(e__));                                   \
            return -1;                                                               \
        }                                                                            \
    } while (0)

template <int NV>
void launch_forward(const FvHit *cand, const uint32_t *ccnt, int topb, uint64_t n0, int nq, int R,
                    const float *x, int dpad, uint64_t *fwd, uint32_t *fwd_cnt, cudaStream_t st) {
    hg_forward_kernel<NV><<<(nq + HG_WARPS - 1) / HG_WARPS, 32 * HG_WARPS, 0, st>>>(
        cand, ccnt, topb, n0, nq, R, x, dpad, fwd, fwd_cnt);
}
template <int NV>
void launch_final(uint64_t *fwd, uint32_t *fwd_cnt, const uint64_t *rev, const uint64_t *in_off,
                  const uint32_t *in_cnt, uint64_t n, uint64_t lo, int R, const float *x,
                  int dpad, cudaStream_t st) {
    hg_final_kernel<NV><<<(unsigned)((n + HG_WARPS - 1) / HG_WARPS), 32 * HG_WARPS, 0, st>>>(
        fwd, fwd_cnt, rev, in_off, in_cnt, n, lo, R, x, dpad);
}

// Exact nearest neighbours of rows [r0, r0 + nq) of g among all rows of g:
// the tensor-core scan when its BF16 distances are certified exact for
// these rows, else the exact FP32 scan (queries read in place from g's f32
// rows). out [nq][topb] ascending, cnt [nq]; tail (zeroed by the caller): the
// scan's watchdog word and flags as tc_tail_bytes lays them out, a query's
// flag nonzero where short lists may have dropped a neighbour (the batch is
// then run again, `exact`).
int knn_batch(FvGpuIndex *g, uint64_t r0, int nq, uint32_t topb, const int32_t *d_qprog,
              const unsigned long long *d_popcnt, FvHit *d_out, uint32_t *d_cnt, uint8_t *d_tr,
              uint8_t *d_tail, bool exact, char *errbuf, size_t errlen) {
    const float *d_q = g->d_vecs + r0 * (uint64_t)g->dpad;
    const uint64_t bm_words = (g->count + 31) / 32;
    g->tc_unc = nullptr;
    if (!exact && g->precision != FV_GPU_PREC_FP32 && tc_supported(g) &&
        tc_superset(g, topb, g->row_amax) == (int)topb) {
        if (launch_scan_tc(g, nq, g->row_amax, d_q, d_qprog, nullptr, bm_words, d_popcnt, topb,
                           d_out, d_cnt, d_tr, nullptr, errbuf, errlen))
            return -1;
        // (each batch's own: the next one's query prep clears the word, and
        // may have it elsewhere)
        PV_CUDA_OK(cudaMemcpyAsync(d_tail, g->tc_err,
                                   g->tc_unc ? tc_tail_bytes(nq) : sizeof(int),
                                   cudaMemcpyDeviceToDevice, g->stream),
                   errbuf, errlen);
        g->tc_err = nullptr;
        g->tc_unc = nullptr;
        return 0;
    }
    ScanPlan pl;
    const bool tiled = plan_scan_f32t(g->count, g->dpad, nq, (int)topb, g->sm_count, pl);
    if (!tiled && !plan_scan_f32(g->count, g->dpad, nq, (int)topb, g->sm_count, pl)) {
        snprintf(errbuf, errlen, "hnsw gpu: dimension %d not supported by the scan", g->dim);
        return -1;
    }
    ScanScratch &s = g->scan;
    PV_CUDA_OK(s.tau.ensure((size_t)nq * 8), errbuf, errlen);
    PV_CUDA_OK(s.part.ensure((size_t)nq * pl.grow * topb * 8), errbuf, errlen);
    PV_CUDA_OK(s.part_cnt.ensure((size_t)nq * pl.grow * 4), errbuf, errlen);
    PV_CUDA_OK(cudaMemsetAsync(s.tau.p, 0xFF, (size_t)nq * 8, g->stream), errbuf, errlen);
    ScanF32Args a;
    a.vecs = g->d_vecs;
    a.nrows = g->count;
    a.dpad = g->dpad;
    a.queries = d_q;
    a.nq = nq;
    a.bitmaps = nullptr;
    a.bm_words = bm_words;
    a.qprog = d_qprog;
    a.K = (int)topb;
    a.S = pl.S;
    a.CB = pl.CB;
    a.rows_per_cta = pl.rows_per_cta;
    a.grow = pl.grow;
    a.qtiles = pl.qtiles;
    a.tau = s.tau.as<unsigned long long>();
    a.part = s.part.as<uint64_t>();
    a.part_cnt = s.part_cnt.as<uint32_t>();
    PV_CUDA_OK(tiled ? launch_scan_f32t(a, pl, g->stream) : launch_scan_f32(a, pl, g->stream),
               errbuf, errlen);
    PV_CUDA_OK(launch_merge(a.part, a.part_cnt, pl.grow, (int)topb, pl, a.tau, d_qprog, d_popcnt,
                            g->count, nq, d_out, d_cnt, d_tr, g->stream),
               errbuf, errlen);
    return 0;
}

constexpr int HG_BATCH = 2048;  // scan batch (queries per call)
constexpr size_t HG_TAIL = TC_TAIL_UNC + HG_BATCH;
// scan batches of an insertion step at most (the first 64 rows, then as many
// as are in)
uint64_t hg_step_batches(uint64_t n) { return 1 + n / 2 / HG_BATCH; }
// A limit for the waits of one scan of level 0 (its number), for tests.
struct HgWait {
    uint64_t ns = 0;
    int batch = -1;
};

// Workspace of a level: one allocation (17 of them, and their frees, took 3 of
// a build's 30 ms and at times ten times that), laid out for level 0 and then
// for the upper levels, whose rows take what level 0 no longer needs.
struct HgWork {
    void *base = nullptr;
    DevArr qprog, popcnt, out, cnt, tr, tails, lst, lcnt, in_cnt, in_off, cursor, rev, lists;
    DevArr ids, xs, los, norms;  // upper levels: the rows gathered
    ~HgWork() {
        if (base) cudaFree(base);
    }
    // A level of n rows with lists of R and answers of topb, the rows gathered
    // or not (dpad f32 and lo_bytes of low-precision row each). The bytes it
    // takes from base on.
    size_t layout(uint64_t n, int topb, int R, int dpad, size_t lo_bytes, bool gathered) {
        const uint64_t n1 = gathered ? n : 0;
        const struct {
            DevArr *a;
            size_t bytes;
        } parts[] = {{&qprog, (size_t)HG_BATCH * 4},
                     {&popcnt, 8},
                     {&out, (size_t)HG_BATCH * topb * sizeof(FvHit)},
                     {&cnt, (size_t)HG_BATCH * 4},
                     {&tr, (size_t)HG_BATCH},
                     {&tails, (size_t)hg_step_batches(n) * HG_TAIL},
                     {&lst, (size_t)n * R * 8},
                     {&lcnt, (size_t)n * 4},
                     {&in_cnt, (size_t)n * 4},
                     {&cursor, (size_t)n * 4},
                     {&in_off, (size_t)(n + 1) * 8},
                     // (an insertion batch is at most the rows before it)
                     {&rev, (size_t)std::max<uint64_t>(64, (n + 1) / 2) * R * 8},
                     {&lists, (size_t)n * (R + 1) * 4},
                     {&ids, (size_t)n1 * 4},
                     {&xs, (size_t)n1 * dpad * 4},
                     {&los, (size_t)n1 * lo_bytes},
                     {&norms, (size_t)((n1 + 127) & ~127ull) * 4}};  // whole tiles
        char *at = (char *)base;
        for (const auto &p : parts) {
            p.a->p = at;
            at += (p.bytes + 255) & ~(size_t)255;
        }
        return (size_t)(at - (char *)base);
    }
};

// One level over the rows of g by batched insertion: w.lists [count][R + 1]
// of local ids.
int build_level(FvGpuIndex *g, HgWork &w, int R, int C, const HgWait &wait, char *errbuf,
                size_t errlen) {
    const uint64_t n = g->count;
    const int dpad = g->dpad;
    const int NVn = (dpad + 127) / 128;
    const int B = HG_BATCH;
    // first insertion batch: a few rows spread over the whole data set, so
    // the earliest lists link distant regions (then doubling batches)
    const uint64_t first = 64;
    cudaStream_t st = g->stream;
    // the rows' tensor map covers all rows, whatever prefix is scanned
    if (g->precision != FV_GPU_PREC_FP32 && !g->tmap_x_ok) {
        CUtensorMap m;
        if (!tc_make_tmap(&m, g->d_vlow, g->precision == FV_GPU_PREC_FP8 ? TCK_FP8 : TCK_BF16,
                          (uint64_t)g->kpad,
                          g->count)) {
            snprintf(errbuf, errlen, "hnsw gpu: tensor map encoding failed");
            return -1;
        }
        memcpy(g->tmap_x, &m, sizeof(m));
        g->tmap_x_ok = true;
    }
    DevArr &qprog = w.qprog, &popcnt = w.popcnt, &out = w.out, &cnt = w.cnt, &tr = w.tr,
           &tails = w.tails, &lst = w.lst, &lcnt = w.lcnt, &in_cnt = w.in_cnt, &in_off = w.in_off,
           &cursor = w.cursor, &rev = w.rev;
    HG_OK(cudaMemsetAsync(qprog.p, 0xFF, (size_t)B * 4, st));  // no filter
    HG_OK(cudaMemsetAsync(lcnt.p, 0, (size_t)n * 4, st));
    std::vector<uint8_t> h_tails;
    int rc = 0, nbatch = 0;
    for (uint64_t lo = 0; lo < n && rc == 0;) {
        const uint64_t hi = lo == 0 ? std::min(n, first) : std::min(n, 2 * lo);
        // 1-2: candidates among the inserted prefix [0, hi), forward selection
        g->count = hi;
        const int topb = (int)std::min<uint64_t>((uint64_t)C + 1, hi);
        const size_t steps = (hi - lo + B - 1) / B;
        HG_OK(cudaMemsetAsync(tails.p, 0, steps * HG_TAIL, st));
        auto batch = [&](uint64_t r0, bool exact) {
            const int nq = (int)std::min<uint64_t>(B, hi - r0);
            const uint64_t limit = g->tc_timeout_ns;
            if (nbatch++ == wait.batch) g->tc_timeout_ns = wait.ns;
            const int bad = knn_batch(
                g, r0, nq, (uint32_t)topb, qprog.as<int32_t>(), popcnt.as<unsigned long long>(),
                out.as<FvHit>(), cnt.as<uint32_t>(), tr.as<uint8_t>(),
                tails.as<uint8_t>() + (r0 - lo) / B * HG_TAIL, exact, errbuf, errlen);
            g->tc_timeout_ns = limit;
            if (bad) return -1;
            if (NVn <= 1)
                launch_forward<1>(out.as<FvHit>(), cnt.as<uint32_t>(), topb, r0, nq, R, g->d_vecs,
                                  dpad, lst.as<uint64_t>(), lcnt.as<uint32_t>(), st);
            else if (NVn <= 2)
                launch_forward<2>(out.as<FvHit>(), cnt.as<uint32_t>(), topb, r0, nq, R, g->d_vecs,
                                  dpad, lst.as<uint64_t>(), lcnt.as<uint32_t>(), st);
            else
                launch_forward<4>(out.as<FvHit>(), cnt.as<uint32_t>(), topb, r0, nq, R, g->d_vecs,
                                  dpad, lst.as<uint64_t>(), lcnt.as<uint32_t>(), st);
            return cudaGetLastError() == cudaSuccess ? 0 : -1;
        };
        for (uint64_t r0 = lo; r0 < hi && rc == 0; r0 += B) rc = batch(r0, false);
        if (!rc) {
            h_tails.resize(steps * HG_TAIL);
            if (cudaMemcpyAsync(h_tails.data(), tails.p, h_tails.size(), cudaMemcpyDeviceToHost,
                                st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                rc = -1;
        }
        for (size_t i = 0; i < steps && rc == 0; i++) {
            int e;
            memcpy(&e, &h_tails[i * HG_TAIL], sizeof(e));
            if (e) {
                snprintf(errbuf, errlen, "hnsw gpu: tensor-core scan wait expired (role %d)", e);
                rc = -1;
            }
        }
        for (uint64_t r0 = lo; r0 < hi && rc == 0; r0 += B) {
            const auto f = h_tails.begin() + (r0 - lo) / B * HG_TAIL + TC_TAIL_UNC;
            if (std::any_of(f, f + std::min<uint64_t>(B, hi - r0), [](uint8_t u) { return u != 0; }))
                rc = batch(r0, true);
        }
        g->count = n;
        if (rc) break;
        // 3: reverse edges of the new nodes' lists
        const uint64_t nu = hi - lo;
        HG_OK(cudaMemsetAsync(in_cnt.p, 0, (size_t)hi * 4, st));
        HG_OK(cudaMemsetAsync(cursor.p, 0, (size_t)hi * 4, st));
        const unsigned eb = (unsigned)((nu * R + 255) / 256);
        hg_count_kernel<<<eb, 256, 0, st>>>(lst.as<uint64_t>(), lcnt.as<uint32_t>(), lo, nu, R,
                                            in_cnt.as<uint32_t>());
        HG_OK(cudaGetLastError());
        // (the batch's edges fit rev; in_off's last word counts them)
        unsigned long long *tot = w.in_off.as<unsigned long long>() + n;
        HG_OK(cudaMemsetAsync(tot, 0, 8, st));
        hg_runs_kernel<<<(unsigned)((hi + 255) / 256), 256, 0, st>>>(
            in_cnt.as<uint32_t>(), hi, in_off.as<uint64_t>(), tot);
        HG_OK(cudaGetLastError());
        hg_scatter_kernel<<<eb, 256, 0, st>>>(lst.as<uint64_t>(), lcnt.as<uint32_t>(), lo, nu, R,
                                              in_off.as<uint64_t>(), cursor.as<uint32_t>(),
                                              rev.as<uint64_t>());
        HG_OK(cudaGetLastError());
        // 4: re-selection of every touched list
        if (NVn <= 1)
            launch_final<1>(lst.as<uint64_t>(), lcnt.as<uint32_t>(), rev.as<uint64_t>(),
                            in_off.as<uint64_t>(), in_cnt.as<uint32_t>(), hi, lo, R, g->d_vecs,
                            dpad, st);
        else if (NVn <= 2)
            launch_final<2>(lst.as<uint64_t>(), lcnt.as<uint32_t>(), rev.as<uint64_t>(),
                            in_off.as<uint64_t>(), in_cnt.as<uint32_t>(), hi, lo, R, g->d_vecs,
                            dpad, st);
        else
            launch_final<4>(lst.as<uint64_t>(), lcnt.as<uint32_t>(), rev.as<uint64_t>(),
                            in_off.as<uint64_t>(), in_cnt.as<uint32_t>(), hi, lo, R, g->d_vecs,
                            dpad, st);
        HG_OK(cudaGetLastError());
        lo = hi;
    }
    g->count = n;
    if (rc) return -1;
    const uint64_t total = n * (uint64_t)(R + 1);
    hg_export_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
        lst.as<uint64_t>(), lcnt.as<uint32_t>(), n, R, w.lists.as<uint32_t>());
    HG_OK(cudaGetLastError());
    HG_OK(cudaStreamSynchronize(st));
    return 0;
}

// All levels of the graph, over the uploaded rows: level 0 all of them, R =
// 2M; levels 1..top the rows of each level, R = M, gathered on the device
// into one set of buffers that stands in for the table's (an upload of its
// own per level took 8 of a build's 50 ms, 60,000 rows).
int build_levels(PvHnsw *h, FvGpuIndex *g, int M, int candidates, int top, const HgWait &wait,
                 char *errbuf, size_t errlen) {
    std::lock_guard<std::mutex> lk(g->mu);
    const uint64_t count = g->count;
    const uint8_t *lev = hnsw_levels(h);
    std::vector<uint32_t> ids;
    for (uint64_t i = 0; i < count; i++)
        if (lev[i] >= 1) ids.push_back((uint32_t)i);
    // upper levels are small: twice the candidates (with self: one more)
    auto upper = [&](uint64_t n) {
        return (int)std::min<uint64_t>((uint64_t)std::min(2 * candidates + 1, 1023), n - 1);
    };
    HgWork w;
    const bool low = g->d_vlow != nullptr;
    const size_t lo_bytes = low ? (size_t)g->kpad * (g->precision == FV_GPU_PREC_FP8 ? 1 : 2) : 0;
    auto lay_upper = [&]() {
        return w.layout(ids.size(), upper(ids.size()) + 1, M, g->dpad, lo_bytes, true);
    };
    auto lay_level0 = [&]() {
        return w.layout(count, (int)std::min<uint64_t>((uint64_t)candidates + 1, count), 2 * M,
                        g->dpad, lo_bytes, false);
    };
    HG_OK(cudaMalloc(&w.base, std::max(ids.size() >= 2 ? lay_upper() : 0, lay_level0())));
    lay_level0();
    if (g->precision != FV_GPU_PREC_FP32 && tc_supported(g)) {
        // the tensor-core scans' scratch at its largest batch: growing with
        // the doubling batches, it was freed and allocated anew ten times
        // (query tiles x CTAs along the rows are at most the SMs)
        const uint64_t nq = std::min<uint64_t>(HG_BATCH, count);
        const uint64_t topb = std::min<uint64_t>((uint64_t)candidates + 1, count);
        ScanScratch &s = g->scan;
        const uint64_t tiles = std::min<uint64_t>(
            g->sm_count, ((nq + TC_BM - 1) / TC_BM) * ((count + TC_BN - 1) / TC_BN));
        HG_OK(s.part.ensure((size_t)(TC_BM * tiles * 3 * TC_MAX_LIST * 8)));
        HG_OK(s.part_cnt.ensure(nq * 12 + 512));
        HG_OK(s.tau.ensure(nq * 8));
        HG_OK(s.cand.ensure((nq + TC_BM) * ((size_t)g->kpad * 2 + 16) +
                            nq * (topb * sizeof(FvHit) + 8) + 4096));
    }
    if (build_level(g, w, 2 * M, candidates, wait, errbuf, errlen)) return -1;
    HG_OK(cudaMemcpy(hnsw_l0(h), w.lists.p, (size_t)count * (2 * M + 1) * 4,
                     cudaMemcpyDeviceToHost));
    if (ids.size() < 2) return 0;  // a single node has no neighbours
    lay_upper();
    HG_OK(cudaMemsetAsync(w.norms.p, 0, ((ids.size() + 127) & ~127ull) * 4, g->stream));
    const auto vecs = g->d_vecs;
    const auto vlow = g->d_vlow;
    const auto norm = g->d_norm;
    std::vector<uint32_t> lists;
    int rc = 0;
    for (int L = 1; L <= top && !rc; L++) {
        if (L > 1) {
            ids.erase(std::remove_if(ids.begin(), ids.end(),
                                     [&](uint32_t i) { return lev[i] < L; }),
                      ids.end());
            if (ids.size() < 2) break;
        }
        const uint64_t n = ids.size();
        const uint64_t pieces = n * (g->dpad / 4 + lo_bytes / 16);
        if (cudaMemcpyAsync(w.ids.p, ids.data(), n * 4, cudaMemcpyHostToDevice, g->stream) !=
            cudaSuccess) {
            rc = -1;
            break;
        }
        hg_gather_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, g->stream>>>(
            vecs, g->dpad, (const unsigned char *)vlow, (int)(lo_bytes / 16), low ? norm : nullptr,
            w.ids.as<uint32_t>(), n, w.xs.as<float>(), (unsigned char *)w.los.p, w.norms.as<float>());
        if (cudaGetLastError() != cudaSuccess) rc = -1;
        // the gathered rows stand in for the table's while the level is built
        g->d_vecs = w.xs.as<float>();
        if (low) {
            g->d_vlow = (decltype(g->d_vlow))w.los.p;
            g->d_norm = w.norms.as<float>();
        }
        g->count = n;
        g->tmap_x_ok = false;
        if (!rc) rc = build_level(g, w, M, upper(n), HgWait(), errbuf, errlen);
        g->d_vecs = vecs;
        g->d_vlow = vlow;
        g->d_norm = norm;
        g->count = count;
        g->tmap_x_ok = false;
        if (rc) break;
        lists.resize(n * (M + 1));
        if (cudaMemcpy(lists.data(), w.lists.p, lists.size() * 4, cudaMemcpyDeviceToHost) !=
            cudaSuccess) {
            rc = -1;
            break;
        }
        for (uint64_t i = 0; i < n; i++) {
            uint32_t *dst = hnsw_upper_list(h, ids[i], L);
            const uint32_t *src = &lists[i * (M + 1)];
            dst[0] = src[0];
            for (uint32_t j = 0; j < src[0]; j++) dst[1 + j] = ids[src[1 + j]];
        }
    }
    return rc;
}

}  // namespace
}  // namespace pv

using namespace pv;

extern "C" PvHnsw *pv_hnsw_build_gpu(const float *vectors, uint64_t count, int dim, int M,
                                     int candidates, int device, int precision, char *errbuf,
                                     size_t errlen) {
    return pv_hnsw_build_gpu_wait(vectors, count, dim, M, candidates, device, precision, 0, -1,
                                  errbuf, errlen);
}

extern "C" PvHnsw *pv_hnsw_build_gpu_wait(const float *vectors, uint64_t count, int dim, int M,
                                          int candidates, int device, int precision,
                                          uint64_t wait_ns, int wait_batch, char *errbuf,
                                          size_t errlen) {
    if (!vectors || count == 0 || dim <= 0 || dim > 512 || M < 2 || M > HG_RMAX / 2 ||
        candidates < 2 * M || candidates > 1023 || wait_ns > 10000000000ull ||
        (precision != FV_GPU_PREC_FP32 && precision != FV_GPU_PREC_BF16)) {
        if (errbuf && errlen) snprintf(errbuf, errlen, "hnsw gpu: bad build parameters");
        return nullptr;
    }
    if (count >= 0xFFFFFFFFull) {
        if (errbuf && errlen) snprintf(errbuf, errlen, "hnsw gpu: too many rows");
        return nullptr;
    }
    PvHnsw *h = hnsw_sections(vectors, count, dim, M);
    const uint8_t *lev = hnsw_levels(h);
    int top = 0;
    uint64_t entry = 0;
    for (uint64_t i = 0; i < count; i++)
        if (lev[i] > top) {
            top = lev[i];
            entry = i;
        }
    auto fail = [&]() -> PvHnsw * {
        pv_hnsw_free(h);
        return nullptr;
    };
    FvGpuIndex *g = upload_rows(vectors, count, dim, device, precision, errbuf, errlen);
    if (!g) return fail();
    const int rc = build_levels(h, g, M, candidates, top, HgWait{wait_ns, wait_batch}, errbuf, errlen);
    fv_gpu_index_free(g);
    if (rc) {
        if (errbuf && errlen && !errbuf[0]) snprintf(errbuf, errlen, "hnsw gpu: build failed");
        return fail();
    }
    hnsw_set_entry(h, entry, top, candidates);
    return h;
}
