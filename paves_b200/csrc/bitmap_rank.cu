// bitmap_rank.cu — bitmaps of batches with many range-form filters.
//
// The posting rows of an attribute column list its rows in value order, so
// the rows of a closed f64 interval are the positions [lo, hi) of that list
// (NaN rows, listed last, are in none), and every row's position is known
// from upload (the list's inverse). The ends of a batch's intervals on a
// column cut the positions into elementary pieces on which no filter
// changes; a table gives each piece the word of every 32 filters it lies
// in. A row then costs one binary search among the ends, one table word per
// 32 filters and column (small-integer sets: a second table, by the row's
// code), and its share of a 32 x 32 bit transposition, instead of one test
// per filter:
//   bitmap_resolve_kernel  each program's [lo, hi), a warp per program, 32
//                          probes of the sorted values at a time
//   bitmap_table_kernel    sorted ends and the tables, a block per column
//                          and 32 programs
//   bitmap_rank_kernel     the bitmaps and their counts: a warp takes 256
//                          rows through all tables of its group
//
// Bound: instruction issue, about 26 per 32 rows x 32 filters (one test per
// filter, on positions in shared memory, took 100 to 150). Measured on one
// B200, 2M rows, a price interval per filter and a category set on a third
// of them: 512 filters 0.121 ms (0.144 with the two kernels before it; the
// general kernel 2.80 ms, one position test per filter 0.55 ms; writing the
// words alone, 128 MB, takes 0.02 ms), 29 filters 0.022 ms (0.037; general
// kernel 0.157 ms). Six filters over 1M rows take these three 0.022 ms,
// bitmap_few_kernel 0.014. Where they pay: rank_pays.
#include <string.h>

#include <algorithm>

#include "launch.cuh"
#include "pv_internal.h"

namespace pv {

constexpr uint32_t RK_FULL = 0xFFFFFFFFu;  // interval of a column the program does not test
constexpr int RK_OTHER = 31;               // code of values that are no integer in [0, 31)
constexpr int RK_ENDS = 2 * PV_RANK_MAX_PROGS;  // interval ends of a column at most
constexpr int RK_W = 8;                    // 32-row words a warp holds at a time
// shared memory of a block of bitmap_rank_kernel: the ends of four columns
// and at least one table word of each piece fit (66 KB); two blocks share an
// SM (118 registers)
constexpr int RK_SMEM = 72 * 1024;

struct __align__(16) RankProg {
    uint32_t lo[PV_RANK_COLS], len[PV_RANK_COLS], set[PV_RANK_COLS];
};

// Scratch of a batch of P programs, in words: programs, then per column the
// number of ends, the sorted ends, the piece table [32-program chunk][piece]
// and the set table [chunk][32 codes].
struct RankTab {
    RankProg *prog;
    int *nends;      // [PV_RANK_COLS]; -1: no interval on the column
    int *sets;       // [PV_RANK_COLS]; 1: some set on the column
    uint32_t *ends;  // [PV_RANK_COLS][2P]
    uint32_t *piece; // [PV_RANK_COLS][nch][2P + 1]
    uint32_t *code;  // [PV_RANK_COLS][nch][32]
};
static RankTab rank_tab_at(void *p, int P) {
    const size_t nch = (size_t)(P + 31) / 32;
    RankTab t;
    t.prog = (RankProg *)p;
    t.nends = (int *)(t.prog + P);
    t.sets = t.nends + PV_RANK_COLS;
    t.ends = (uint32_t *)(t.sets + PV_RANK_COLS);
    t.piece = t.ends + (size_t)PV_RANK_COLS * 2 * P;
    t.code = t.piece + PV_RANK_COLS * nch * (2 * (size_t)P + 1);
    return t;
}
size_t rank_tab_bytes(int P) {
    const RankTab t = rank_tab_at(nullptr, P);
    return (size_t)(uintptr_t)(t.code + PV_RANK_COLS * (((size_t)P + 31) / 32) * 32);
}

// ---------------------------------------------------------------- upload
// pos[r] = place of row r in the column's posting list, and the values in
// that order. A row listed twice leaves another at RK_FULL.
__global__ void rank_scatter_kernel(const double *__restrict__ col,
                                    const uint32_t *__restrict__ prows, uint64_t n,
                                    uint32_t *__restrict__ pos, double *__restrict__ sorted) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t r = prows[i];
    if (r < n) pos[r] = (uint32_t)i;
    sorted[i] = r < n ? col[r] : __longlong_as_double(0x7ff8000000000000ll);
}

// res[0]: values that are numbers; res[1]: faults (rows missing from the
// list, neighbours out of order); res[2]: integers in [31, 64), which a
// 31-code byte cannot tell apart
__global__ void rank_check_kernel(const double *__restrict__ col,
                                  const uint32_t *__restrict__ pos,
                                  const double *__restrict__ sorted, uint64_t n,
                                  uint8_t *__restrict__ code, unsigned *__restrict__ res) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool num = false, bad = false, wide = false;
    if (i < n) {
        const double s = sorted[i];
        num = s == s;
        if (i + 1 < n) {
            const double t = sorted[i + 1];
            bad = t == t && !(s <= t);  // a number after NaN or after a larger one
        }
        bad = bad || pos[i] == RK_FULL;
        const double v = col[i];
        const bool in = v >= 0.0 && v < 64.0;
        const int b = in ? (int)v : 64;
        const bool whole = in && (double)b == v;
        code[i] = (uint8_t)(whole && b < RK_OTHER ? b : RK_OTHER);
        wide = whole && b >= RK_OTHER;
    }
    const int c0 = __syncthreads_count(num), c1 = __syncthreads_count(bad),
              c2 = __syncthreads_count(wide);
    if (threadIdx.x == 0) {
        if (c0) atomicAdd(res, (unsigned)c0);
        if (c1) atomicAdd(res + 1, (unsigned)c1);
        if (c2) atomicAdd(res + 2, (unsigned)c2);
    }
}

// Whether the arrays below may be made: only batches of many filters are
// faster with them, so they leave the calls' own scratch its room (bitmaps
// and visited sets of the largest batch, a gathered set, lists and runs) and
// another index or process a quarter of the device.
bool rank_tables_fit(uint64_t free_bytes, uint64_t total_bytes, uint64_t count, int ncols) {
    if (ncols < 1 || ncols > PV_RANK_COLS) return false;
    const uint64_t tables = (uint64_t)ncols * count * 13 + PV_RANK_COLS * 16;
    const uint64_t calls = (2ull << 30) + 2ull * FV_GPU_MAX_BATCH * ((count + 31) / 32) * 4;
    return free_bytes >= tables + std::max(calls, total_bytes / 4);
}

// Positions, sorted values and codes of every column (tables of at most
// PV_RANK_COLS columns); a column whose posting rows are no ordering of its
// values is left out. Runs on g's stream and waits for it.
cudaError_t build_rank_cols(FvGpuIndex *g) {
    g->rank_cols = g->code_cols = 0;
    const uint64_t n = g->count;
    size_t room = 0, total = 0;
    if (g->ncols < 1 || g->ncols > PV_RANK_COLS) return cudaSuccess;
    if (cudaMemGetInfo(&room, &total) != cudaSuccess ||
        !rank_tables_fit(room, total, n, g->ncols)) {
        (void)cudaGetLastError();
        return cudaSuccess;
    }
    const size_t words = (size_t)g->ncols * n;
    cudaError_t e = cudaMalloc(&g->d_rank, words * 4 + PV_RANK_COLS * 16);
    if (e == cudaSuccess) e = cudaMalloc(&g->d_sorted, words * 8);
    if (e == cudaSuccess) e = cudaMalloc(&g->d_code, words);
    if (e != cudaSuccess) {  // no room: filters stay on the f64 columns
        (void)cudaGetLastError();
        cudaFree(g->d_rank);
        cudaFree(g->d_sorted);
        g->d_rank = nullptr;
        g->d_sorted = nullptr;
        return cudaSuccess;
    }
    unsigned *res = (unsigned *)(g->d_rank + words);
    if ((e = cudaMemsetAsync(g->d_rank, 0xFF, words * 4, g->stream)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(res, 0, PV_RANK_COLS * 16, g->stream)) != cudaSuccess) return e;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    for (int c = 0; c < g->ncols; c++) {
        const uint64_t o = (uint64_t)c * n;
        rank_scatter_kernel<<<blocks, 256, 0, g->stream>>>(g->d_cols + o, g->d_prows + o, n,
                                                           g->d_rank + o, g->d_sorted + o);
        rank_check_kernel<<<blocks, 256, 0, g->stream>>>(g->d_cols + o, g->d_rank + o,
                                                         g->d_sorted + o, n, g->d_code + o,
                                                         res + c * 4);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    unsigned h[PV_RANK_COLS * 4] = {};
    e = cudaMemcpyAsync(h, res, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) return e;
    for (int c = 0; c < g->ncols; c++) {
        g->rank_nv[c] = h[c * 4];
        if (h[c * 4 + 1] == 0) g->rank_cols |= 1 << c;
        if (h[c * 4 + 2] == 0) g->code_cols |= 1 << c;
    }
    return cudaSuccess;
}

// Whether the three kernels are faster than the general one for P programs:
// that takes 2.3 ps a row and program beyond its first wave, these take 5 us
// of launches and 0.04 us a program (ends, tables and their loads) whatever
// the rows are. Measured, in us with the batch's query prep, general kernel
// against these: 9 programs over 200,000 rows 20 and 22, over 400,000 26 and
// 22; 32 over 60,000 27 and 29, 100,000 33 and 31; 128 over 20,000 31 and
// 39, 60,000 42 and 40; 1000 over 20,000 75 and 77, 2,000 31 and 71.
bool rank_pays(uint64_t rows, int P) {
    return P >= PV_RANK_MIN_PROGS && P <= PV_RANK_MAX_PROGS &&
           rows * (uint64_t)P >= 2400000ull + 25000ull * (uint64_t)P;
}

// Whether every program of a batch has the form these kernels take.
bool rank_batch_ok(const FvGpuIndex *g, const PredBatch &pb) {
    if (!g->rank_cols) return false;
    const int nc = (int)pb.consts.size();
    for (const PredProg &p : pb.progs) {
        if (p.ninsn != 1 || p.insn0 < 0 || p.insn0 >= (int)pb.insns.size()) return false;
        const PredInsn &r = pb.insns[p.insn0];
        if (r.kind != PV_NODE_RANGE || r.n < 0 || r.n > PV_RANGE_MAX_TERMS) return false;
        int ci = r.val0;
        for (int k = 0; k < r.n; k++) {
            if (ci < 0 || ci + 2 > nc) return false;
            const int meta = (int)pb.consts[ci], col = meta & 0xFFFF;
            const bool set = meta & PV_TERM_MASK;
            if (col >= g->ncols || (!set && ci + 3 > nc)) return false;
            if (!((set ? g->code_cols : g->rank_cols) >> col & 1)) return false;
            ci += set ? 2 : 3;
        }
    }
    return true;
}

// ---------------------------------------------------------------- batch
// By a warp: x[0] = values of s[0, n) (ascending) below x0, x[1] = values at
// most x1; both searches' probes are in flight together.
__device__ __forceinline__ void warp_counts(const double *__restrict__ s, uint32_t n, double x0,
                                            double x1, int lane, uint32_t &c0, uint32_t &c1) {
    uint32_t b[2] = {0, 0}, e[2] = {n, n};
    while (e[0] - b[0] > 32 || e[1] - b[1] > 32) {
        double v[2];
#pragma unroll
        for (int k = 0; k < 2; k++)
            v[k] = __ldg(s + b[k] + (uint32_t)((uint64_t)(lane + 1) * (e[k] - b[k]) / 33));
#pragma unroll
        for (int k = 0; k < 2; k++) {
            // (a search that is down to 32 values goes on with repeated
            // probes: those before the first miss are still below)
            const uint64_t w = e[k] - b[k];
            const int c = __popc(__ballot_sync(0xffffffffu, k ? v[k] <= x1 : v[k] < x0));
            if (w <= 32) continue;
            const uint32_t lo = c ? b[k] + (uint32_t)((uint64_t)c * w / 33) + 1 : b[k];
            if (c < 32) e[k] = b[k] + (uint32_t)((uint64_t)(c + 1) * w / 33);
            b[k] = lo;
        }
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const bool in = b[k] + lane < e[k];
        const double v = in ? __ldg(s + b[k] + lane) : 0.0;
        (k ? c1 : c0) =
            b[k] + __popc(__ballot_sync(0xffffffffu, in && (k ? v <= x1 : v < x0)));
    }
}

struct RankCols {
    const uint32_t *pos;
    const double *sorted;
    const uint8_t *code;
    uint64_t nrows;
    int ncols;
    uint32_t nv[PV_RANK_COLS];
};

// A warp per program; also zeroes the program's count. dP, if given, holds
// the batch's program count in device memory (at most P).
__global__ void __launch_bounds__(256, 2)
bitmap_resolve_kernel(RankCols t, const PredInsn *__restrict__ insns,
                      const PredProg *__restrict__ progs, const double *__restrict__ consts,
                      int P, const int *__restrict__ dP, RankProg *__restrict__ out,
                      unsigned long long *__restrict__ popcnt) {
    pdl_wait();
    pdl_trigger();
    if (dP) P = min(P, *dP);
    const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= P) return;
    const PredInsn r = insns[progs[p].insn0];
    uint32_t lo[PV_RANK_COLS], len[PV_RANK_COLS], set[PV_RANK_COLS];
#pragma unroll
    for (int c = 0; c < PV_RANK_COLS; c++) {
        lo[c] = 0;
        len[c] = set[c] = RK_FULL;
    }
    int ci = r.val0;
    for (int k = 0; k < r.n; k++) {
        const int meta = (int)consts[ci], col = meta & 0xFFFF;
        uint32_t a = 0, n = RK_FULL, m = RK_FULL;
        if (meta & PV_TERM_MASK) {
            m = (uint32_t)__double_as_longlong(consts[ci + 1]) & ~(1u << RK_OTHER);
            ci += 2;
        } else {
            const double x0 = consts[ci + 1], x1 = consts[ci + 2];
            n = 0;
            if (x0 == x0 && x1 == x1) {
                const double *s = t.sorted + (uint64_t)col * t.nrows;
                uint32_t b;
                warp_counts(s, t.nv[col], x0, x1, lane, a, b);
                n = b > a ? b - a : 0;
            }
            ci += 3;
        }
#pragma unroll
        for (int c = 0; c < PV_RANK_COLS; c++)
            if (c == col) {
                if (meta & PV_TERM_MASK) {
                    set[c] = m;
                } else {
                    lo[c] = a;
                    len[c] = n;
                }
            }
    }
    if (lane == 0) {
        RankProg o;
#pragma unroll
        for (int c = 0; c < PV_RANK_COLS; c++) {
            o.lo[c] = lo[c];
            o.len[c] = len[c];
            o.set[c] = set[c];
        }
        out[p] = o;
        popcnt[p] = 0;
    }
}

// grid (32-program chunks, columns): the column's ends in order (each block
// sorts them, only chunk 0 stores them) and the chunk's words of every piece
// and code.
__global__ void __launch_bounds__(256)
bitmap_table_kernel(RankTab t, int P_cap, const int *__restrict__ dP) {
    __shared__ uint32_t s_end[RK_ENDS];
    __shared__ uint32_t s_lo[32], s_len[32], s_set[32];
    __shared__ int s_n, s_any;
    pdl_wait();
    pdl_trigger();
    const int P = dP ? min(P_cap, *dP) : P_cap;
    const int chunk = blockIdx.x, c = blockIdx.y, tid = threadIdx.x;
    const int nch_cap = (P_cap + 31) / 32;
    if (chunk * 32 >= P) return;
    if (tid == 0) s_n = s_any = 0;
    __syncthreads();
    for (int p = tid; p < P; p += 256) {
        const uint32_t len = t.prog[p].len[c], lo = t.prog[p].lo[c];
        if (len != RK_FULL) {
            const int at = atomicAdd(&s_n, 2);
            s_end[at] = lo;
            s_end[at + 1] = lo + len;
        }
        if (t.prog[p].set[c] != RK_FULL) s_any = 1;
    }
    if (tid < 32) {
        const int p = chunk * 32 + tid;
        s_lo[tid] = p < P ? t.prog[p].lo[c] : 0;
        s_len[tid] = p < P ? t.prog[p].len[c] : 0;
        s_set[tid] = p < P ? t.prog[p].set[c] : 0;
    }
    __syncthreads();
    const int n = s_n;
    int n2 = 2;
    while (n2 < n) n2 <<= 1;
    for (int i = n + tid; i < n2; i += 256) s_end[i] = RK_FULL;
    __syncthreads();
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < (n2 >> 1); i += 256) {
                const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1)), b = a | j;
                const uint32_t x = s_end[a], y = s_end[b];
                if ((x > y) == ((a & k) == 0)) {
                    s_end[a] = y;
                    s_end[b] = x;
                }
            }
            __syncthreads();
        }
    if (chunk == 0) {
        for (int i = tid; i < n; i += 256) t.ends[(size_t)c * 2 * P_cap + i] = s_end[i];
        if (tid == 0) {
            t.nends[c] = n ? n : -1;
            t.sets[c] = s_any;
        }
    }
    // piece e holds the positions [end e - 1, end e)
    uint32_t *piece = t.piece + ((size_t)c * nch_cap + chunk) * (2 * (size_t)P_cap + 1);
    for (int e = tid; n && e <= n; e += 256) {
        const uint32_t at = e ? s_end[e - 1] : 0u;
        uint32_t w = 0;
#pragma unroll 8
        for (int p = 0; p < 32; p++)
            if (at - s_lo[p] < s_len[p]) w |= 1u << p;
        piece[e] = w;
    }
    if (tid < 32 && s_any) {
        uint32_t w = 0;
        for (int p = 0; p < 32; p++) w |= ((s_set[p] >> tid) & 1u) << p;
        t.code[((size_t)c * nch_cap + chunk) * 32 + tid] = w;
    }
}

// 32 x 32 bits across a warp: lane r's bit p becomes lane p's bit r. Step s
// trades the off-diagonal s x s blocks of lanes s apart: a rotation lines the
// partner's block up whichever side the lane is on, a mask takes it in.
struct Transpose32 {
    uint32_t keep[5];
    int rot[5];
    __device__ __forceinline__ explicit Transpose32(int lane) {
        const uint32_t m[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const int s = 16 >> i;
            keep[i] = lane & s ? ~m[i] : m[i];
            rot[i] = lane & s ? 32 - s : s;
        }
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 16 >> i);
            x = (x & keep[i]) | (__funnelshift_l(y, y, rot[i]) & ~keep[i]);
        }
        return x;
    }
};

// Groups of as many 32-program chunks as the tables of one block's shared
// memory hold; a block keeps one group's tables and takes every ng-th part
// of the row tiles (8 warps x 256 rows).
__global__ void __launch_bounds__(256, 2)
bitmap_rank_kernel(RankCols t, RankTab tab, int P_cap, const int *__restrict__ dP,
                   uint32_t *__restrict__ bitmaps, uint64_t bm_words,
                   unsigned long long *__restrict__ popcnt) {
    extern __shared__ __align__(16) uint32_t rk_smem[];
    __shared__ unsigned s_cnt[PV_RANK_MAX_PROGS];
    pdl_wait();
    pdl_trigger();
    const int P = dP ? min(P_cap, *dP) : P_cap;
    if (P <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nch = (P + 31) / 32, nch_cap = (P_cap + 31) / 32;
    // carve: ends of each interval column, then the chunks' tables
    int nend[PV_RANK_COLS], off_end[PV_RANK_COLS], off_tab[PV_RANK_COLS], off_set[PV_RANK_COLS];
    int w_ends = 0, w_chunk = 0;
#pragma unroll
    for (int c = 0; c < PV_RANK_COLS; c++) {
        nend[c] = c < t.ncols ? tab.nends[c] : -1;
        off_end[c] = w_ends;
        off_tab[c] = w_chunk;
        if (nend[c] >= 0) {
            w_ends += nend[c];
            w_chunk += nend[c] + 1;
        }
        const bool set = c < t.ncols && tab.sets[c];
        off_set[c] = set ? w_chunk : -1;
        if (set) w_chunk += 32;
    }
    const int cg = w_chunk ? min(nch, (RK_SMEM / 4 - w_ends) / w_chunk) : nch;
    const int ng = (nch + cg - 1) / cg;
    const int grp = blockIdx.x % ng;
    const int ch0 = grp * cg, nc = min(cg, nch - ch0);
    const int nblk = (gridDim.x - grp + ng - 1) / ng;  // blocks of this group
    uint32_t *s_tab = rk_smem + w_ends;
#pragma unroll
    for (int c = 0; c < PV_RANK_COLS; c++) {
        if (nend[c] >= 0) {
            for (int i = tid; i < nend[c]; i += 256)
                rk_smem[off_end[c] + i] = tab.ends[(size_t)c * 2 * P_cap + i];
            for (int k = 0; k < nc; k++) {
                const uint32_t *src =
                    tab.piece + ((size_t)c * nch_cap + ch0 + k) * (2 * (size_t)P_cap + 1);
                for (int i = tid; i <= nend[c]; i += 256)
                    s_tab[k * w_chunk + off_tab[c] + i] = src[i];
            }
        }
        if (off_set[c] >= 0)
            for (int i = tid; i < nc * 32; i += 256)
                s_tab[(i >> 5) * w_chunk + off_set[c] + (i & 31)] =
                    tab.code[((size_t)c * nch_cap + ch0) * 32 + i];
    }
    for (int i = tid; i < nc * 32; i += 256) s_cnt[i] = 0;
    __syncthreads();
    const Transpose32 transpose(lane);
    const bool wide = (bm_words & 3) == 0;  // 16-byte stores of a program's words
    const uint64_t nunits = (bm_words + RK_W - 1) / RK_W;
    for (uint64_t u = (uint64_t)(blockIdx.x / ng) * 8 + warp; u < nunits; u += (uint64_t)nblk * 8) {
        const uint64_t r0 = u * (RK_W * 32) + lane;
        // each row's table places: piece in the low, code in the high half
        uint32_t pc[PV_RANK_COLS][RK_W];
#pragma unroll
        for (int c = 0; c < PV_RANK_COLS; c++) {
            if (nend[c] >= 0) {
                uint32_t pos[RK_W];
#pragma unroll
                for (int w = 0; w < RK_W; w++) {
                    pos[w] = r0 + w * 32 < t.nrows
                                 ? __ldg(t.pos + (uint64_t)c * t.nrows + r0 + w * 32) : RK_FULL;
                    pc[c][w] = 0;
                }
                // ends at most the position, by halving
                const uint32_t *end = rk_smem + off_end[c];
                for (int n = nend[c]; n > 0;) {
                    const int h = n >> 1;
#pragma unroll
                    for (int w = 0; w < RK_W; w++)
                        if (end[pc[c][w] + h] <= pos[w]) pc[c][w] += n - h;
                    n = h;
                }
            }
            if (off_set[c] >= 0) {
#pragma unroll
                for (int w = 0; w < RK_W; w++) {
                    const uint32_t k = r0 + w * 32 < t.nrows
                                           ? __ldg(t.code + (uint64_t)c * t.nrows + r0 + w * 32)
                                           : (uint32_t)RK_OTHER;
                    pc[c][w] = (nend[c] >= 0 ? pc[c][w] : 0u) | k << 16;
                }
            }
        }
        uint32_t live[RK_W];
#pragma unroll
        for (int w = 0; w < RK_W; w++) live[w] = r0 + w * 32 < t.nrows ? 0xFFFFFFFFu : 0u;
        for (int k = 0; k < nc; k++) {
            const uint32_t *tb = s_tab + k * w_chunk;
            uint32_t m[RK_W];
            unsigned cnt = 0;
#pragma unroll
            for (int w = 0; w < RK_W; w++) m[w] = live[w];
#pragma unroll
            for (int c = 0; c < PV_RANK_COLS; c++) {
                if (nend[c] >= 0) {
#pragma unroll
                    for (int w = 0; w < RK_W; w++) m[w] &= tb[off_tab[c] + (pc[c][w] & 0xFFFF)];
                }
                if (off_set[c] >= 0) {
#pragma unroll
                    for (int w = 0; w < RK_W; w++) m[w] &= tb[off_set[c] + (pc[c][w] >> 16)];
                }
            }
#pragma unroll
            for (int w = 0; w < RK_W; w++) {
                m[w] = transpose(m[w]);
                cnt += __popc(m[w]);
            }
            const int p = (ch0 + k) * 32 + lane;
            if (p < P) {
                uint32_t *dst = bitmaps + (uint64_t)p * bm_words + u * RK_W;
                if (wide && (u + 1) * RK_W <= bm_words) {
#pragma unroll
                    for (int w = 0; w < RK_W; w += 4)
                        *(uint4 *)(dst + w) = make_uint4(m[w], m[w + 1], m[w + 2], m[w + 3]);
                } else {
#pragma unroll
                    for (int w = 0; w < RK_W; w++)
                        if (u * RK_W + w < bm_words) dst[w] = m[w];
                }
                if (cnt) atomicAdd(&s_cnt[k * 32 + lane], cnt);
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < nc * 32; i += 256)
        if (ch0 * 32 + i < P && s_cnt[i])
            atomicAdd(popcnt + ch0 * 32 + i, (unsigned long long)s_cnt[i]);
}

// The bitmaps and counts of P programs that rank_batch_ok accepted; tab:
// rank_tab_bytes(P) of scratch. dP: the program count in device memory
// (<= P; 0: nothing is done), so one launch serves every batch of a CUDA
// graph.
cudaError_t launch_bitmaps_rank(const FvGpuIndex *g, const PredInsn *insns, const PredProg *progs,
                                const double *consts, int P, const int *dP, void *tab,
                                uint32_t *bitmaps, uint64_t bm_words, unsigned long long *popcnt,
                                cudaStream_t st) {
    RankCols t;
    t.pos = g->d_rank;
    t.sorted = g->d_sorted;
    t.code = g->d_code;
    t.nrows = g->count;
    t.ncols = g->ncols;
    memcpy(t.nv, g->rank_nv, sizeof(t.nv));
    const RankTab rt = rank_tab_at(tab, P);
    cudaError_t e = launch_pdl(bitmap_resolve_kernel, dim3((P + 7) / 8), dim3(256), 0, st, t,
                               insns, progs, consts, P, dP, rt.prog, popcnt);
    if (e == cudaSuccess)
        e = launch_pdl(bitmap_table_kernel, dim3((P + 31) / 32, g->ncols), dim3(256), 0, st, rt, P,
                       dP);
    if (e == cudaSuccess) e = raise_smem_limit((const void *)bitmap_rank_kernel, RK_SMEM);
    if (e != cudaSuccess) return e;
    const uint64_t units = (bm_words + RK_W * 8 - 1) / (RK_W * 8);
    const uint64_t groups = (uint64_t)(P + 31) / 32;  // at most
    const unsigned blocks =
        (unsigned)std::max(std::min<uint64_t>(units * groups, (uint64_t)g->sm_count * 2), groups);
    return launch_pdl(bitmap_rank_kernel, dim3(blocks), dim3(256), RK_SMEM, st, t, rt, P, dP,
                      bitmaps, bm_words, popcnt);
}

}  // namespace pv

extern "C" int pv_rank_tables_fit(uint64_t free_bytes, uint64_t total_bytes, uint64_t count,
                                  int ncols) {
    return pv::rank_tables_fit(free_bytes, total_bytes, count, ncols) ? 1 : 0;
}
