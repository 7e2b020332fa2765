// sparse.cu — selective filters scan only their matching rows.
//
// The reference answers a selective filter through its posting-list
// driver: the spans of the sorted attribute values that can match bound
// the candidate rows (engine.cpp:464-599, fv_pred_estimate :640-643), and
// its GPU router sends a query to the span path when that total is small
// (gpu_engine.cu:2249-2260). Here the same bound decides the route:
//  * at upload each attribute column's values are kept sorted on the host
//    (from the posting rows), so a comparison or IN list is counted exactly
//    by binary search, and AND / OR / NOT combine lower / upper bounds;
//  * a batch whose queries share one filter bounded by a small count
//    compacts that filter's bitmap into a row-id list on the device and
//    either gathers those rows into a contiguous set for the tensor-core
//    scan (2048+ rows, when the batch's mode scans on the tensor cores),
//    or computes the exact FP32 distance of every (query, listed row) and
//    selects each query's top-k from those keys (a radix select).
// Results equal the full scan's: same rows, same FP32 distances.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "pv_internal.h"
#include "sm100.cuh"

namespace pv {

void build_sorted_cols(FvGpuIndex *g, const double *cols, const uint32_t *post_rows) {
    g->sorted_cols.assign(g->ncols, {});
    for (int c = 0; c < g->ncols; c++) {
        std::vector<double> &v = g->sorted_cols[c];
        v.reserve(g->count);
        const double *col = cols + (uint64_t)c * g->count;
        const uint32_t *pr = post_rows + (uint64_t)c * g->count;
        for (uint64_t i = 0; i < g->count; i++) {
            const double x = col[pr[i] < g->count ? pr[i] : 0];
            if (x == x) v.push_back(x);  // NaN sorts last and matches nothing
        }
        // posting rows are ordered by value; keep the copy sorted regardless
        if (!std::is_sorted(v.begin(), v.end())) std::sort(v.begin(), v.end());
    }
}

namespace {

uint64_t count_cmp(const std::vector<double> &v, int op, double c) {
    const uint64_t n = v.size();
    if (c != c) return op == FV_CMP_NE ? n : 0;  // NaN constant
    const uint64_t lo = std::lower_bound(v.begin(), v.end(), c) - v.begin();
    const uint64_t hi = std::upper_bound(v.begin(), v.end(), c) - v.begin();
    switch (op) {
        case FV_CMP_LT: return lo;
        case FV_CMP_LE: return hi;
        case FV_CMP_EQ: return hi - lo;
        case FV_CMP_GE: return n - lo;
        case FV_CMP_GT: return n - hi;
        case FV_CMP_NE: return n - (hi - lo);
    }
    return n;
}

}  // namespace

// Estimated fraction of rows a range-form program passes: the product of
// its terms' exact fractions (independent columns); 0 for other programs or
// without sorted columns.
double prog_pass_estimate(const FvGpuIndex *g, const PredInsn *ins, int n, const double *consts) {
    if (n != 1 || ins[0].kind != PV_NODE_RANGE || g->count == 0 ||
        (int)g->sorted_cols.size() != g->ncols)
        return 0.0;
    const double N = (double)g->count;
    double f = 1.0;
    int ci = ins[0].val0;
    for (int k = 0; k < ins[0].n; k++) {
        const int meta = (int)consts[ci];
        const int col = meta & 0xFFFF;
        if (col >= g->ncols) return 0.0;
        const std::vector<double> &v = g->sorted_cols[col];
        uint64_t c = 0;
        if (meta & PV_TERM_MASK) {
            uint64_t bits;
            memcpy(&bits, &consts[ci + 1], 8);
            for (int b = 0; b < 64; b++)
                if ((bits >> b) & 1ull) c += count_cmp(v, FV_CMP_EQ, (double)b);
            ci += 2;
        } else {
            const double lo = consts[ci + 1], hi = consts[ci + 2];
            if (lo == lo && hi == hi) {
                const uint64_t a = std::lower_bound(v.begin(), v.end(), lo) - v.begin();
                const uint64_t b = std::upper_bound(v.begin(), v.end(), hi) - v.begin();
                c = b > a ? b - a : 0;
            }
            ci += 3;
        }
        f *= (double)c / N;
    }
    return f;
}

uint64_t prog_upper_bound(const FvGpuIndex *g, const PredInsn *ins, int n, const double *consts) {
    const uint64_t N = g->count;
    if ((int)g->sorted_cols.size() != g->ncols || g->ncols == 0) return N;
    struct B { uint64_t lo, hi; };
    std::vector<B> st;
    st.reserve(n);
    for (int i = 0; i < n; i++) {
        const PredInsn &in = ins[i];
        switch (in.kind) {
            case FV_NODE_CMP: {
                if (in.col < 0 || in.col >= g->ncols) return N;
                const uint64_t c = count_cmp(g->sorted_cols[in.col], in.op, in.value);
                st.push_back({c, c});
                break;
            }
            case FV_NODE_IN: {
                if (in.col < 0 || in.col >= g->ncols) return N;
                std::vector<double> vals(consts + in.val0, consts + in.val0 + in.n);
                std::sort(vals.begin(), vals.end());
                vals.erase(std::unique(vals.begin(), vals.end()), vals.end());
                uint64_t c = 0;
                for (double x : vals) c += count_cmp(g->sorted_cols[in.col], FV_CMP_EQ, x);
                st.push_back({c, c});
                break;
            }
            case PV_NODE_RANGE: {
                // AND of exact per-term counts: at most the smallest, at
                // least what the terms' counts force to overlap
                uint64_t hi = N, lo_sum = 0;
                int ci = in.val0;
                for (int k = 0; k < in.n; k++) {
                    const int meta = (int)consts[ci];
                    const int col = meta & 0xFFFF;
                    if (col >= g->ncols) return N;
                    const std::vector<double> &v = g->sorted_cols[col];
                    uint64_t c = 0;
                    if (meta & PV_TERM_MASK) {
                        uint64_t bits;
                        memcpy(&bits, &consts[ci + 1], 8);
                        for (int b = 0; b < 64; b++)
                            if ((bits >> b) & 1ull) c += count_cmp(v, FV_CMP_EQ, (double)b);
                        ci += 2;
                    } else {
                        const double lo = consts[ci + 1], hi_v = consts[ci + 2];
                        if (lo == lo && hi_v == hi_v) {  // closed [lo, hi]
                            const uint64_t a = std::lower_bound(v.begin(), v.end(), lo) - v.begin();
                            const uint64_t b = std::upper_bound(v.begin(), v.end(), hi_v) - v.begin();
                            c = b > a ? b - a : 0;
                        }
                        ci += 3;
                    }
                    hi = std::min(hi, c);
                    lo_sum += c;
                }
                const uint64_t over = in.n > 1 ? (uint64_t)(in.n - 1) * N : 0;
                st.push_back({lo_sum > over ? lo_sum - over : 0, hi});
                break;
            }
            case FV_NODE_AND:
            case FV_NODE_OR: {
                if (in.n == 0) {
                    st.push_back(in.kind == FV_NODE_AND ? B{N, N} : B{0, 0});
                    break;
                }
                if (st.size() < 2) return N;
                const B b = st.back();
                st.pop_back();
                const B a = st.back();
                st.pop_back();
                if (in.kind == FV_NODE_AND)
                    st.push_back({a.lo + b.lo > N ? a.lo + b.lo - N : 0, std::min(a.hi, b.hi)});
                else
                    st.push_back({std::max(a.lo, b.lo), std::min(N, a.hi + b.hi)});
                break;
            }
            default: {  // NOT
                if (st.empty()) return N;
                const B a = st.back();
                st.back() = {N - a.hi, N - a.lo};
                break;
            }
        }
    }
    return st.size() == 1 ? st.back().hi : N;
}

// Bitmap -> ascending row ids within each block of words; blocks claim
// their output range with one atomic (the list's order across blocks does
// not matter: keys carry the row id).
__global__ void __launch_bounds__(256) compact_kernel(const uint32_t *__restrict__ bm,
                                                      uint64_t bm_words, uint64_t nrows,
                                                      uint32_t *__restrict__ ids,
                                                      unsigned long long *__restrict__ count,
                                                      uint64_t cap) {
    __shared__ int s_warp[8];
    __shared__ unsigned long long s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint64_t w0 = (uint64_t)blockIdx.x * blockDim.x; w0 < bm_words;
         w0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t w = w0 + tid;
        uint32_t word = w < bm_words ? bm[w] : 0u;
        if (w == bm_words - 1 && (nrows & 31)) word &= (1u << (nrows & 31)) - 1u;
        const int c = __popc(word);
        int incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = 0, total = 0;
        for (int i = 0; i < 8; i++) {
            if (i < warp) before += s_warp[i];
            total += s_warp[i];
        }
        if (tid == 0) s_base = atomicAdd(count, (unsigned long long)total);
        __syncthreads();
        uint64_t pos = s_base + before + incl - c;
        while (word) {
            const int b = __ffs(word) - 1;
            word &= word - 1;
            if (pos < cap) ids[pos] = (uint32_t)(w * 32 + b);
            pos++;
        }
        __syncthreads();
    }
}

// Exact FP32 distances of every listed row to every query of the batch:
// keys[q][i] = (||x_rowids[i] - q||^2, rowids[i]) for i < n = min(*count,
// cap), and dcnt[q] = n. grid (row blocks, query tiles of GD_QT); a warp
// takes one row at a time: lane L holds dims [4L, 4L+4) of each 128-dim
// chunk, the GD_QT partial sums are reduced with xor-shuffles.
constexpr int GD_QT = 8;

__global__ void __launch_bounds__(256)
gather_dist_kernel(const float *__restrict__ vecs, int dpad, const float *__restrict__ queries,
                   int nq, const uint32_t *__restrict__ rowids,
                   const unsigned long long *__restrict__ count, uint64_t cap,
                   uint64_t *__restrict__ keys, uint32_t *__restrict__ dcnt) {
    extern __shared__ __align__(16) float gd_q[];  // [GD_QT][dpad]
    const int q0 = blockIdx.y * GD_QT;
    const uint64_t n = min((unsigned long long)cap, *count);
    for (int i = threadIdx.x; i < GD_QT * dpad; i += blockDim.x) {
        const int j = i / dpad, d = i - j * dpad;
        gd_q[i] = q0 + j < nq ? queries[(size_t)(q0 + j) * dpad + d] : 0.f;
    }
    if (blockIdx.x == 0 && threadIdx.x < GD_QT && q0 + (int)threadIdx.x < nq)
        dcnt[q0 + threadIdx.x] = (uint32_t)n;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t r = (uint64_t)blockIdx.x * 8 + warp; r < n; r += (uint64_t)gridDim.x * 8) {
        const uint32_t row = __ldg(rowids + r);
        const float *x = vecs + (uint64_t)row * dpad;
        float acc[GD_QT];
#pragma unroll
        for (int j = 0; j < GD_QT; j++) acc[j] = 0.f;
        for (int c = lane * 4; c < dpad; c += 128) {
            const float4 v = __ldg((const float4 *)(x + c));
#pragma unroll
            for (int j = 0; j < GD_QT; j++) {
                const float4 w = *(const float4 *)(gd_q + j * dpad + c);
                const float d0 = v.x - w.x, d1 = v.y - w.y, d2 = v.z - w.z, d3 = v.w - w.w;
                acc[j] = fmaf(d0, d0, acc[j]);
                acc[j] = fmaf(d1, d1, acc[j]);
                acc[j] = fmaf(d2, d2, acc[j]);
                acc[j] = fmaf(d3, d3, acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < GD_QT; j++)
#pragma unroll
            for (int o = 16; o; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
        float mine = acc[0];
#pragma unroll
        for (int j = 1; j < GD_QT; j++)
            if (lane == j) mine = acc[j];
        if (lane < GD_QT && q0 + lane < nq)
            keys[(uint64_t)(q0 + lane) * cap + r] = make_key(mine, row);
    }
}

// The same for larger batches of rows up to 128 dims: a block takes 64 listed
// rows x 64 queries, a thread 4 rows x 4 queries, two queries per packed
// instruction (sub / fma.rn.f32x2; the queries lie transposed in shared
// memory, four of a dim in one 16-byte read). Each distance is summed in the
// row-per-warp kernel's order, so both give the same bits: what lane L sums
// there, dims 4L .. 4L + 3, is a leaf here, and leaves join in the order of
// its shuffles (16, 8, 4, 2, 1 lanes apart): bit-reversed, pairs of equal
// depth added as they complete. Measured for 64 queries x 10,000 rows of 128
// dims: 0.022 ms; the row-per-warp kernel, which spends 5 shuffles per
// (row, query), 0.032 ms.
constexpr int GT_T = 64;         // rows and queries per block
constexpr int GT_D = 128;        // dims at most
constexpr int GT_S = GT_D + 4;   // padded stride of the rows (floats)
constexpr int GT_MIN_NQ = 12;    // smaller batches leave most of a tile empty
constexpr size_t GT_SMEM = (size_t)(GT_T * GT_S + GT_D * GT_T) * 4;

__global__ void __launch_bounds__(256)
gather_tile_kernel(const float *__restrict__ vecs, int dpad, const float *__restrict__ queries,
                   int nq, const uint32_t *__restrict__ rowids,
                   const unsigned long long *__restrict__ count, uint64_t cap,
                   uint64_t *__restrict__ keys, uint32_t *__restrict__ dcnt) {
    extern __shared__ __align__(16) float gt_smem[];
    float *sx = gt_smem, *sq = gt_smem + GT_T * GT_S;  // [row][dim], [dim][query]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int q0 = blockIdx.y * GT_T;
    const uint64_t n = min((unsigned long long)cap, *count);
    if (blockIdx.x == 0 && tid < GT_T && q0 + tid < nq) dcnt[q0 + tid] = (uint32_t)n;
    for (int i = tid; i < GT_T * (GT_D / 4); i += 256) {
        const int r = i & (GT_T - 1), c = (i / GT_T) * 4;
        const float4 v = q0 + r < nq && c < dpad
                             ? __ldg((const float4 *)(queries + (size_t)(q0 + r) * dpad + c))
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        sq[(c + 0) * GT_T + r] = v.x;
        sq[(c + 1) * GT_T + r] = v.y;
        sq[(c + 2) * GT_T + r] = v.z;
        sq[(c + 3) * GT_T + r] = v.w;
    }
    // row copies: 32 threads along a row's 16-byte pieces, 8 rows at a time,
    // all of a tile's in flight together (the rows are scattered)
    const int cr = tid >> 5, cc = (tid & 31) * 4;
    for (uint64_t r0 = (uint64_t)blockIdx.x * GT_T; r0 < n; r0 += (uint64_t)gridDim.x * GT_T) {
        __syncthreads();  // the previous tile is done with
#pragma unroll
        for (int u = 0; u < GT_T / 8; u++) {
            const uint64_t r = r0 + cr + 8 * u;
            const uint32_t row = __ldg(rowids + (r < n ? r : r0));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(sx + (cr + 8 * u) * GT_S + cc)),
                         "l"(vecs + (uint64_t)row * dpad + (cc < dpad ? cc : 0)),
                         "r"(cc < dpad ? 16 : 0));  // zeros outside
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // [row][pair of queries] packed
        uint64_t s0[4][2], s1[4][2], s2[4][2], sum[4][2];
        auto leaf = [&](int l, uint64_t (&acc)[4][2]) {
            float4 x[4];
            ulonglong2 q[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                x[i] = *(const float4 *)(sx + (tx + 16 * i) * GT_S + 4 * l);
                q[i] = *(const ulonglong2 *)(sq + (4 * l + i) * GT_T + 4 * ty);
            }
#pragma unroll
            for (int d = 0; d < 4; d++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float xv = d == 0 ? x[i].x : d == 1 ? x[i].y : d == 2 ? x[i].z : x[i].w;
                    const uint64_t x2 = sm100::f2_pack(xv, xv);
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        uint64_t t;
                        asm("sub.rn.f32x2 %0, %1, %2;"
                            : "=l"(t) : "l"(x2), "l"(j ? q[d].y : q[d].x));
                        acc[i][j] = d == 0 ? sm100::f2_fma(t, t, 0ull)
                                           : sm100::f2_fma(t, t, acc[i][j]);
                    }
                }
        };
        auto add = [](uint64_t (&d)[4][2], const uint64_t (&a)[4][2], const uint64_t (&b)[4][2]) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) d[i][j] = sm100::f2_add(a[i][j], b[i][j]);
        };
#pragma unroll 1
        for (int u = 0; u < 8; u++) {
            const int b = ((u & 1) << 2) | (u & 2) | (u >> 2);  // the leaves b + 0, 16, 8, 24
            uint64_t t[4][2], v[4][2];
            leaf(b, t);
            leaf(b + 16, v);
            add(sum, t, v);
            leaf(b + 8, t);
            leaf(b + 24, v);
            add(t, t, v);
            add(sum, sum, t);
            if (!(u & 1)) {
#pragma unroll
                for (int i = 0; i < 8; i++) s0[i >> 1][i & 1] = sum[i >> 1][i & 1];
                continue;
            }
            add(sum, s0, sum);
            if (!(u & 2)) {
#pragma unroll
                for (int i = 0; i < 8; i++) s1[i >> 1][i & 1] = sum[i >> 1][i & 1];
                continue;
            }
            add(sum, s1, sum);
            if (!(u & 4)) {
#pragma unroll
                for (int i = 0; i < 8; i++) s2[i >> 1][i & 1] = sum[i >> 1][i & 1];
                continue;
            }
            add(sum, s2, sum);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint64_t r = r0 + tx + 16 * i;
            if (r >= n) continue;
            const uint32_t row = __ldg(rowids + r);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                uint32_t lo, hi;
                sm100::f2_unpack(sum[i][j], lo, hi);
                const int q = q0 + 4 * ty + 2 * j;
                if (q < nq) keys[(uint64_t)q * cap + r] = make_key(__uint_as_float(lo), row);
                if (q + 1 < nq)
                    keys[(uint64_t)(q + 1) * cap + r] = make_key(__uint_as_float(hi), row);
            }
        }
    }
}

// The listed rows in the tensor-core scan's operand layout: compacted row i
// (i < min(*count, cap)) is index row ids[i] — its operand row (row_bytes,
// a multiple of 16), norm and fp8 scale; the rows' 16-byte pieces are dealt
// to the threads.
// valid[w] marks the compacted rows [32w, 32w + 32) that exist.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const unsigned char *__restrict__ src, size_t row_bytes,
                   const float *__restrict__ norms, const float *__restrict__ scales,
                   const uint32_t *__restrict__ ids, const unsigned long long *__restrict__ count,
                   uint64_t cap, unsigned char *__restrict__ dst, float *__restrict__ dnorm,
                   float *__restrict__ dscale, uint32_t *__restrict__ valid, uint64_t vwords) {
    const uint64_t n = min((unsigned long long)cap, *count);
    const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = gt; w < vwords; w += nthreads) {
        const uint64_t r0 = w * 32;
        valid[w] = r0 >= n ? 0u : n - r0 >= 32 ? 0xFFFFFFFFu : (1u << (n - r0)) - 1u;
    }
    // 16-byte pieces, four of a thread in flight
    const uint32_t n16 = (uint32_t)(row_bytes / 16);
    constexpr int U = 4;
    for (uint64_t p = gt; p < n * n16; p += nthreads * U) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint64_t i = p + u * nthreads;
            if (i >= n * n16) break;
            const uint64_t r = i / n16;
            v[u] = __ldg((const uint4 *)(src + (size_t)__ldg(ids + r) * row_bytes) + (i - r * n16));
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint64_t i = p + u * nthreads;
            if (i < n * n16) ((uint4 *)dst)[i] = v[u];
        }
    }
    for (uint64_t i = gt; i < n; i += nthreads) {
        const uint32_t r = __ldg(ids + i);
        dnorm[i] = __ldg(norms + r);
        if (dscale) dscale[i] = __ldg(scales + r);
    }
}

// Scratch of the gathered set of at most `bound` rows:
// [count u64][ids u32 x cap_pad][rows][norms][scales][valid words]
struct GatherPlan {
    bool fp8;
    size_t row_bytes;
    uint64_t cap, cap_pad;  // whole 128-row tiles
    size_t off_ids = 256, off_rows, off_norm, off_scale, off_valid, bytes;
    GatherPlan(const FvGpuIndex *g, uint64_t bound, bool tf32) {
        auto al = [](size_t x, size_t a) { return (x + a - 1) & ~(a - 1); };
        fp8 = !tf32 && g->precision == FV_GPU_PREC_FP8;
        row_bytes = tf32 ? (size_t)g->dpad * 4 : (size_t)g->kpad * (fp8 ? 1 : 2);
        cap = std::max<uint64_t>(bound, 1);
        cap_pad = (cap + 127) & ~127ull;
        off_rows = al(off_ids + cap_pad * 4, 1024);
        off_norm = al(off_rows + cap_pad * row_bytes, 1024);
        off_scale = al(off_norm + cap_pad * 4, 256);
        off_valid = al(off_scale + (fp8 ? cap_pad * 4 : 0), 256);
        bytes = off_valid + cap_pad / 32 * 4 + 256;
    }
};

// Whether the gathered set of a filter that passes up to `bound` rows (more
// than the sparse route's own limit) is scanned rather than the index. The
// gather reads and writes the listed rows, in 15 to 20 us of launches of its
// own, and every query tile of 128 then scans them and not the index. Speed
// of the gathered scan over dense's, 128 dims, k 10: BF16 with 64, 256 and
// 512 queries: 100,000 rows, 10 % passing 0.85, 0.96, 1.12; 300,000 rows 10 %
// 1.06, 1.36, 1.78, 30 % 0.89, 1.03, 1.26; 1M rows 10 % 1.61 (89 -> 55 us),
// 2.25, 3.04, 20 % 1.23, 1.60, 2.11, 30 % 0.98, 1.27, 1.63; f32 rows 1M 10 %
// 1.75, 2.63, 3.68, 30 % 0.96, 1.38, 1.80. The line: bytes the dense scan's
// query tiles read, less the gathered scan's and 2.5 times the listed rows',
// against 60 MB. (Rows under 256 bytes count as 256: their scan is bound by
// its epilogue.) And enough rows must pass for the seeding sample's chunk
// minima to bound the lists (`pass` of the index's rows, S kept): 300,000
// rows, 64 queries, k 60, 2 % passing took 0.105 ms against dense's 0.055.
bool gather_pays(const FvGpuIndex *g, int nq, uint64_t bound, double pass, int S, bool tf32) {
    if (!bound || bound > g->count) return false;
    if (pass * (double)g->count / 32 < 4.0 * std::min(S, 128)) return false;
    const GatherPlan gp(g, bound, tf32);
    const double tiles = std::max(1.0, nq / 128.0);
    const double rows = tiles * (double)g->count - (tiles + 2.5) * (double)bound;
    // (the copy lives in the index's scratch from then on: 1 GB at most)
    return rows * (double)std::max<size_t>(gp.row_bytes, 256) >= 60e6 && gp.bytes <= (1ull << 30);
}

// Room for the gathered set; without it the whole index is scanned as ever.
bool sparse_tc_reserve(FvGpuIndex *g, uint64_t bound, bool tf32) {
    if (g->scan.sparse.ensure(GatherPlan(g, bound, tf32).bytes) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// The sparse route on the tensor cores: the filter's bitmap is compacted to
// a row list, the listed rows are gathered into a contiguous set in the
// scan's operand layout (the upload's BF16 / FP8 rows, or the f32 rows read
// as TF32 for exact-mode batches), and the tensor-core scan runs over that
// set with the same supersets, certificates and re-rank as over the whole
// index; keys carry the index rows, so ties order as in the full scan.
int sparse_tc_launch(FvGpuIndex *g, DevBatch &db, uint32_t topb, uint64_t bound, bool tf32,
                     FvHit *d_out, uint32_t *d_cnt, uint8_t *d_trunc, cudaEvent_t *ev,
                     char *errbuf, size_t errlen) {
    const int nq = db.nq;
    char *d = db.stage_d->as<char>();
    const float *d_q = (const float *)(d + db.off_q);
    const int32_t *d_qprog = (const int32_t *)(d + db.off_qprog);
    const uint64_t bm_words = (g->count + 31) / 32;
    ScanScratch &s = g->scan;
    const GatherPlan gp(g, bound, tf32);
    const bool fp8 = gp.fp8;
    const size_t row_bytes = gp.row_bytes;
    const uint64_t cap = gp.cap, cap_pad = gp.cap_pad, vwords = gp.cap_pad / 32;
    PV_CUDA_OK(s.sparse.ensure(gp.bytes), errbuf, errlen);
    char *sp = s.sparse.as<char>();
    unsigned long long *d_count = (unsigned long long *)sp;
    uint32_t *ids = (uint32_t *)(sp + gp.off_ids);
    unsigned char *rows = (unsigned char *)(sp + gp.off_rows);
    float *norms = (float *)(sp + gp.off_norm);
    float *scales = fp8 ? (float *)(sp + gp.off_scale) : nullptr;
    uint32_t *valid = (uint32_t *)(sp + gp.off_valid);
    PV_CUDA_OK(cudaMemsetAsync(d_count, 0, 8, g->stream), errbuf, errlen);
    unsigned blocks = (unsigned)std::min<uint64_t>((bm_words + 255) / 256, (uint64_t)g->sm_count * 4);
    if (!blocks) blocks = 1;
    compact_kernel<<<blocks, 256, 0, g->stream>>>(s.bitmaps.as<uint32_t>(), bm_words, g->count,
                                                  ids, d_count, cap);
    PV_CUDA_OK(cudaGetLastError(), errbuf, errlen);
    const unsigned gblocks = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((cap * (row_bytes / 16) + 1023) / 1024, (uint64_t)g->sm_count * 8));
    const unsigned char *src = tf32 ? (const unsigned char *)g->d_vecs
                                    : (const unsigned char *)g->d_vlow;
    gather_rows_kernel<<<gblocks, 256, 0, g->stream>>>(
        src, row_bytes, tf32 ? g->d_norm32 : g->d_norm, fp8 ? g->d_vscale : nullptr, ids, d_count,
        cap, rows, norms, scales, valid, vwords);
    PV_CUDA_OK(cudaGetLastError(), errbuf, errlen);
    g->launches += 2;  // compaction, gather
    const TcRowSet rs{rows, norms, scales, cap_pad, ids, d_count, db.sparse_bound > 0};
    const double expect = std::min(1.0, db.pass * (double)g->count / (double)cap_pad);
    return launch_scan_tc(g, nq, db.q_amax, d_q, d_qprog, valid, vwords,
                          s.popcnt.as<unsigned long long>(), topb, d_out, d_cnt, d_trunc, ev,
                          errbuf, errlen, nullptr, tf32, &rs, false, nullptr, expect, db.redo);
}

// The sparse route of brute_launch: every query uses program 0, whose
// matches are at most `bound` rows. The bitmap is compacted to a row list,
// every (query, listed row) gets its exact FP32 key, and each query's
// top-topb is selected from its keys (launch_dense_merge).
int sparse_launch(FvGpuIndex *g, DevBatch &db, uint32_t topb, uint64_t bound, FvHit *d_out,
                  uint32_t *d_cnt, uint8_t *d_trunc, char *errbuf, size_t errlen) {
    const int nq = db.nq;
    char *d = db.stage_d->as<char>();
    const float *d_q = (const float *)(d + db.off_q);
    const int32_t *d_qprog = (const int32_t *)(d + db.off_qprog);
    const uint64_t bm_words = (g->count + 31) / 32;
    ScanScratch &s = g->scan;
    const uint64_t cap = std::max<uint64_t>(bound, 1);
    // scratch: [count u64][dcnt u32 x nq][ids u32 x cap][keys u64 x nq x cap]
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t off_dcnt = 256, off_ids = off_dcnt + al((size_t)nq * 4);
    const size_t off_keys = off_ids + al(cap * 4);
    PV_CUDA_OK(s.sparse.ensure(off_keys + (size_t)nq * cap * 8 + 256), errbuf, errlen);
    char *sp = s.sparse.as<char>();
    unsigned long long *d_count = (unsigned long long *)sp;
    uint32_t *dcnt = (uint32_t *)(sp + off_dcnt);
    uint32_t *ids = (uint32_t *)(sp + off_ids);
    uint64_t *keys = (uint64_t *)(sp + off_keys);
    PV_CUDA_OK(cudaMemsetAsync(d_count, 0, 8, g->stream), errbuf, errlen);
    unsigned blocks = (unsigned)std::min<uint64_t>((bm_words + 255) / 256, (uint64_t)g->sm_count * 4);
    if (!blocks) blocks = 1;
    compact_kernel<<<blocks, 256, 0, g->stream>>>(s.bitmaps.as<uint32_t>(), bm_words, g->count,
                                                  ids, d_count, cap);
    PV_CUDA_OK(cudaGetLastError(), errbuf, errlen);
    const unsigned ty = (unsigned)((nq + GT_T - 1) / GT_T);
    // (tiles for half the SMs at least, by the rows expected: 276 queries x
    // 394 rows make 35, and took 3 us longer than the row-per-warp kernel's
    // many small blocks)
    const uint64_t expect = std::min<uint64_t>(cap, (uint64_t)(db.pass * (double)g->count) + 1);
    if (nq >= GT_MIN_NQ && g->dpad <= GT_D &&
        (expect + GT_T - 1) / GT_T * ty >= (uint64_t)g->sm_count / 2) {
        const unsigned tx = (unsigned)std::max<uint64_t>(
            1, std::min<uint64_t>((cap + GT_T - 1) / GT_T, std::max(1u, 4u * g->sm_count / ty)));
        PV_CUDA_OK(raise_smem_limit((const void *)gather_tile_kernel, GT_SMEM), errbuf, errlen);
        gather_tile_kernel<<<dim3(tx, ty), 256, GT_SMEM, g->stream>>>(g->d_vecs, g->dpad, d_q, nq, ids,
                                                                d_count, cap, keys, dcnt);
        PV_CUDA_OK(cudaGetLastError(), errbuf, errlen);
        g->launches += 3;  // compaction, distances, selection
        PV_CUDA_OK(launch_dense_merge(keys, cap, dcnt, false, nullptr, nullptr, (int)topb, d_qprog,
                                      s.popcnt.as<unsigned long long>(), g->count, nq, d_out,
                                      d_cnt, d_trunc, nullptr, nullptr, g->stream),
                   errbuf, errlen);
        return 0;
    }
    const int qtiles = (nq + GD_QT - 1) / GD_QT;
    const uint64_t bx = std::max<uint64_t>(
        1, std::min<uint64_t>((cap + 63) / 64, std::max(1, 4 * g->sm_count / qtiles)));
    const size_t smem = (size_t)GD_QT * g->dpad * 4;
    PV_CUDA_OK(raise_smem_limit((const void *)gather_dist_kernel, smem), errbuf, errlen);
    gather_dist_kernel<<<dim3((unsigned)bx, (unsigned)qtiles), 256, smem, g->stream>>>(
        g->d_vecs, g->dpad, d_q, nq, ids, d_count, cap, keys, dcnt);
    PV_CUDA_OK(cudaGetLastError(), errbuf, errlen);
    g->launches += 3;  // compaction, distances, selection
    // the truncation flag counts the filter's true matches
    PV_CUDA_OK(launch_dense_merge(keys, cap, dcnt, false, nullptr, nullptr, (int)topb, d_qprog,
                                  s.popcnt.as<unsigned long long>(), g->count, nq, d_out, d_cnt,
                                  d_trunc, nullptr, nullptr, g->stream),
               errbuf, errlen);
    return 0;
}

}  // namespace pv
