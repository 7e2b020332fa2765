// graph.cu — batched filtered HNSW level-0 beam search.
//
// Replaces fv_graph_kernel / fv_gpu_graph_batch (gpu_engine.cu:1118-1485,
// 2338-2542) with the search semantics of the CPU HnswCursor
// (engine.cpp:1661-1713): traversal is unrestricted, only predicate-passing
// nodes enter the result list, the search stops when the best unexpanded
// candidate is farther than the worst of a full result list, when the
// frontier empties, or when max_visited nodes were visited.
//
// One CTA per query. Everything the search touches per step lives in
// shared memory:
//  * visited set: open-addressing hash of node ids; past half load it
//    spills into a per-query global bitmap that the kernel zeroes itself,
//    so there is no per-batch O(nq * N) memset;
//  * frontier (two arrays, recent entries and the rest) and results:
//    ascending keys (dist bits << 32 | node); each step's new keys are placed
//    by rank (a count among the new keys plus a binary search in the old
//    list), so no step sorts, and frontier entries beyond the worst of a full
//    result list are dropped;
//  * the step expands the best W frontier nodes at once (up to 16, fewer
//    only when the rest cannot beat the worst result), gathers their
//    neighbours from the fixed-width device adjacency, and computes
//    distances with 4 lanes per node (16-byte loads), whole rows in flight
//    while a step has up to 128 new nodes;
//  * the predicate is a bit of the batch bitmap, read only for candidates
//    that beat the current worst result.
#include <string.h>

#include <type_traits>
#include <vector>

#include "pv_internal.h"

namespace pv {

constexpr int G_THREADS = 256;
constexpr int G_HC = 8192;   // visited hash slots (u32)
constexpr int G_FC = 8192;   // frontier capacity (selective filters grow it)
constexpr int G_RC = 512;    // result capacity (FV_GPU_MAX_EF)
constexpr int G_NB = 512;    // new entries per step (W * deg_cap <= G_NB)
constexpr int G_BC = 1024;   // recent frontier entries kept apart from the rest
constexpr int G_WMAX = 16;   // nodes expanded per step at most
constexpr uint32_t G_EMPTY = 0xFFFFFFFFu;

struct GraphArgs {
    const float *__restrict__ vecs;
    int dpad;
    uint64_t nrows;
    const uint32_t *__restrict__ adj;
    int deg_cap;
    int dc_shift;  // log2(deg_cap) when a power of two, else -1
    const float *__restrict__ queries;  // [nq][dpad]
    const uint32_t *__restrict__ entries;
    const int32_t *__restrict__ qprog;
    const uint32_t *__restrict__ bitmaps;
    uint64_t bm_words;
    int ef;
    const uint16_t *__restrict__ efq;  // optional per-query ef (<= ef)
    uint64_t max_visited;
    int wmax;
    uint32_t *visited_bits;  // [nq][bm_words], zeroed by the kernel on spill
    FvHit *out;              // [nq][ef]
    uint32_t *out_cnt;
    uint8_t *out_exh;
    uint32_t *stats;  // [nq][4]: steps, visited, predicate probes, results
};

__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    return x;
}

// A result/frontier key carries the node's predicate bit in bit 31 of the
// row half (rows < 2^31 are required), so one sort orders the keys and
// keeps each key's bit. Among passing keys the order is (dist, node).
constexpr uint32_t G_PASS = 0x80000000u;
__device__ __forceinline__ uint32_t grow_of(uint64_t k) { return (uint32_t)k & ~G_PASS; }

// Number of keys of the ascending f[0, n) at or below k, by a warp.
__device__ __forceinline__ int warp_upper(const uint64_t *f, int n, uint64_t k, int lane) {
    int b = 0, e = n;
    while (e - b > 32) {
        const int w = e - b;
        const int c = __popc(__ballot_sync(0xffffffffu, f[b + (lane + 1) * w / 33] <= k));
        const int b0 = b;
        if (c) b = b0 + c * w / 33 + 1;
        if (c < 32) e = b0 + (c + 1) * w / 33;
    }
    return b + __popc(__ballot_sync(0xffffffffu, b + lane < e && f[b + lane] <= k));
}

// Numbers of keys of the ascending f[0, n) and g[0, m) below k, by one
// thread, the two searches' reads in flight together.
__device__ __forceinline__ void lower2(const uint64_t *f, int n, const uint64_t *g, int m,
                                       uint64_t k, int &bf, int &bg) {
    int b = 0, d = 0;
    while (n > 0 || m > 0) {
        const int h = n >> 1, j = m >> 1;
        const uint64_t x = n > 0 ? f[b + h] : KEY_MAX, y = m > 0 ? g[d + j] : KEY_MAX;
        if (x < k) {
            b += h + 1;
            n -= h + 1;
        } else {
            n = h;
        }
        if (y < k) {
            d += j + 1;
            m -= j + 1;
        } else {
            m = j;
        }
    }
    bf = b;
    bg = d;
}

// Number of keys of the ascending f[0, n) below k, by one thread.
__device__ __forceinline__ int lower(const uint64_t *f, int n, uint64_t k) {
    int b = 0;
    while (n > 0) {
        const int h = n >> 1;
        if (f[b + h] < k) {
            b += h + 1;
            n -= h + 1;
        } else {
            n = h;
        }
    }
    return b;
}

// Number of entries of the ascending places p[0, n) at or below i.
__device__ __forceinline__ int placed(const int *p, int n, int i) {
    int b = 0;
    while (n > 0) {
        const int h = n >> 1;
        if (p[b + h] <= i) {
            b += h + 1;
            n -= h + 1;
        } else {
            n = h;
        }
    }
    return b;
}

// Squared L2 of the rows nid[base + grp + r * groups], r < RPG, four lanes a
// row, all of a 128-dim (RPG 4: 64-dim) stretch's loads in flight at once;
// the sum's order does not depend on RPG.
template <int RPG>
__device__ __forceinline__ void graph_dists(const GraphArgs &a, const float *sq,
                                            const uint32_t *nid, const uint32_t *bm, int base,
                                            int nnew, float (&acc)[RPG], uint32_t (&nn)[RPG],
                                            uint32_t (&pw)[RPG]) {
    constexpr int GROUPS = G_THREADS / 4;
    constexpr int CH = RPG == 4 ? 64 : 128, U = CH / 16;
    const int grp = threadIdx.x >> 2, sub = threadIdx.x & 3;
    const float *xr[RPG];
#pragma unroll
    for (int r = 0; r < RPG; r++) {
        const int i = base + grp + r * GROUPS;
        // rows past nnew re-read row nid[0] (valid) and are discarded
        nn[r] = nid[i < nnew ? i : 0];
        xr[r] = a.vecs + (uint64_t)nn[r] * a.dpad;
        pw[r] = bm ? __ldg(bm + (nn[r] >> 5)) : ~0u;
        acc[r] = 0.f;
    }
    for (int c = 0; c < a.dpad; c += CH) {
        float4 v[RPG][U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = c + u * 16 + sub * 4;
            const bool in = j < a.dpad;
#pragma unroll
            for (int r = 0; r < RPG; r++)
                v[r][u] = in ? __ldg((const float4 *)(xr[r] + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = c + u * 16 + sub * 4;
            if (j >= a.dpad) break;
            const float4 w = *(const float4 *)(sq + j);
#pragma unroll
            for (int r = 0; r < RPG; r++) {
                const float d0 = v[r][u].x - w.x, d1 = v[r][u].y - w.y;
                const float d2 = v[r][u].z - w.z, d3 = v[r][u].w - w.w;
                acc[r] = fmaf(d0, d0, acc[r]); acc[r] = fmaf(d1, d1, acc[r]);
                acc[r] = fmaf(d2, d2, acc[r]); acc[r] = fmaf(d3, d3, acc[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RPG; r++) {
        acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 2);
        acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 1);
    }
}

// A step is a chain of latencies (two dependent gathers from HBM, and the
// shared-memory work between them) on one SM per query, so what counts is
// how many waits it makes. The frontier is two ascending arrays, the few
// recent entries (a step's keys are merged into these) and the rest, which
// only lose entries at their ends between the rare merges of the one into
// the other; every warp picks the step's nodes itself, and new keys find
// their places by counting and binary search, with no sort: four barriers a
// step, where sorting and merging into one long frontier took fourteen.
// Lists and rows are prefetched into L2 as soon as a node is known to be
// wanted. Measured on one B200, 64 queries of 1M x 128 rows: a 10 % filter at
// ef 64 (44 steps, 83 at most) 0.53 ms, 6.4 us a step, against 0.69; a 1 %
// filter at ef 64 (403 steps, a frontier of thousands) 3.3 ms against 5.4,
// 0.15 % (8 queries, 2294 steps) 17.6 ms against 43.7; 60,000 rows, 10 %:
// 0.16 ms, 3.1 us a step with every read in L2, against 0.24.
//
// WIDE: rows of so many dims that the query has no room beside the search's
// arrays; it is read where it lies.
template <bool WIDE>
__global__ void __launch_bounds__(G_THREADS) graph_kernel(GraphArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t *const fm0 = (uint64_t *)smem_raw;  // [2][G_FC] frontier: the rest
    uint64_t *const fb0 = fm0 + 2 * G_FC;        // [2][G_BC] frontier: recent entries
    uint64_t *const rs0 = fb0 + 2 * G_BC;        // [2][G_RC] results
    uint64_t *nfk = rs0 + 2 * G_RC;              // [G_NB + 2] new keys (any order)
    uint32_t *hash = (uint32_t *)(nfk + G_NB + 2);  // [G_HC]
    uint32_t *nid = hash + G_HC;                 // [G_NB] gathered neighbours
    int *rpos = (int *)(nid + G_NB);             // [G_NB] new results' places
    int *fpos = rpos + G_NB;                     // [G_NB] new frontier keys' places
    float *s_q = (float *)(fpos + G_NB);         // [dpad] query

    // a step's counts: fresh neighbours, admitted keys, passing ones (two
    // sets: the next step's are cleared while this one's are read)
    __shared__ int s_cnt[2][3];
    __shared__ int s_hcount;

    const int q = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a per-query beam width of 0: the query is answered elsewhere (a mixed
    // routed batch scans it), nothing to search
    if (a.efq && a.efq[q] == 0) {
        if (tid == 0) {
            a.out_cnt[q] = 0;
            a.out_exh[q] = 0;
            if (a.stats)
                for (int i = 0; i < 4; i++) a.stats[q * 4 + i] = 0;
        }
        return;
    }
    // per-query beam width (never above the batch's, which is the output stride)
    const int ef = a.efq ? min((int)a.efq[q], a.ef) : a.ef;
    const int pg = a.qprog[q];
    const uint32_t *bm = pg >= 0 ? a.bitmaps + (uint64_t)pg * a.bm_words : nullptr;
    uint32_t *vb = a.visited_bits + (uint64_t)q * a.bm_words;
    const float *qv = a.queries + (uint64_t)q * a.dpad;

    const float *sq = WIDE ? qv : s_q;
    if (!WIDE)
        for (int i = tid; i < a.dpad; i += blockDim.x) s_q[i] = qv[i];
    for (int i = tid; i < G_HC; i += blockDim.x) hash[i] = G_EMPTY;
    if (tid < 6) s_cnt[tid / 3][tid % 3] = 0;
    if (tid == 0) s_hcount = 1;
    // seed: entry point (engine.cpp:1651-1656), its distance by every warp
    uint32_t ep = a.entries[q];
    if (ep >= a.nrows) ep = 0;
    const bool ep_pass = !bm || ((bm[ep >> 5] >> (ep & 31)) & 1u);
    __syncthreads();
    if (warp == 0) {
        float acc = 0.f;
        const float *x = a.vecs + (uint64_t)ep * a.dpad;
        for (int j = lane * 4; j < a.dpad; j += 128) {
            float4 v = __ldg((const float4 *)(x + j));
            float4 w = *(const float4 *)(sq + j);
            float d0 = v.x - w.x, d1 = v.y - w.y, d2 = v.z - w.z, d3 = v.w - w.w;
            acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc);
            acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
        }
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            hash[hash_u32(ep) & (G_HC - 1)] = ep;
            const uint64_t key = make_key(acc, ep | (ep_pass ? G_PASS : 0u));
            fb0[0] = key;
            if (ep_pass) rs0[0] = key;
        }
    }
    __syncthreads();

    // the search's state, the same in every thread
    int cm = 0, mh = 0, me = 0;      // rest: side, [mh, me)
    int cb = 0, bh = 0, be = 1;      // recent: side, [bh, be)
    int cr = 0, nr = ep_pass ? 1 : 0;
    bool spilled = false, dropped = false;
    unsigned long long visited = 1;
    unsigned int probes = 0, steps = 0;
    int exh = 0;
    // the step's nodes; t0 > 0: the rest of a list longer than G_NB is next
    uint32_t selnode = 0;
    int nsel = 0, t0 = 0;

    for (;;) {
        // ---- selection (by every warp): the best W entries, cut at the
        // first one beyond the worst result
        const uint64_t *R = rs0 + cr * G_RC;
        const uint64_t *FM = fm0 + cm * G_FC, *FB = fb0 + cb * G_BC;
        const bool full = nr >= ef;
        const float worst = full ? key_dist(R[ef - 1]) : 0.f;
        if (full) {
            // entries beyond the worst of a full result list are never
            // expanded (the search would end first): drop them
            const uint64_t kthr = ((uint64_t)__float_as_uint(worst) << 32) | 0xFFFFFFFFull;
            if (me > mh && FM[me - 1] > kthr) {
                me = mh + warp_upper(FM + mh, me - mh, kthr, lane);
                dropped = true;
            }
            if (be > bh && FB[be - 1] > kthr) {
                be = bh + warp_upper(FB + bh, be - bh, kthr, lane);
                dropped = true;
            }
        }
        if ((me - mh) + (be - bh) > G_FC) {
            // more than the frontier holds: the largest go, x of the recent
            // ones and e - x of the rest
            const int e = (me - mh) + (be - bh) - G_FC;
            int lo = max(0, e - (me - mh)), hi = min(e, be - bh);
            while (lo < hi) {
                const int x = (lo + hi) >> 1;  // enough when what the rest loses is larger
                if (FB[be - 1 - x] < FM[me - (e - x)]) hi = x;
                else lo = x + 1;
            }
            be -= lo;
            me -= e - lo;
            dropped = true;
        }
        if (t0 == 0) {
            const int nb = be - bh, nm = me - mh, avail = nb + nm;
            // an empty frontier is exhaustion unless entries were dropped (they
            // would still sit in an unbounded candidate queue)
            if (avail <= 0) {
                exh = dropped ? 0 : 1;
                break;
            }
            if (visited >= a.max_visited) {
                exh = 1;
                break;
            }
            const int w = min(avail, a.wmax);
            const uint64_t own = lane < G_WMAX ? (lane < nb ? FB[bh + lane] : KEY_MAX)
                                               : (lane - G_WMAX < nm ? FM[mh + lane - G_WMAX] : KEY_MAX);
            uint64_t k = own;
            if (nm > 0) {
#pragma unroll
                for (int s = 16; s; s >>= 1) {  // two ascending halves: reverse one, then clean
                    const uint64_t o = s == 16 ? __shfl_sync(0xffffffffu, k, 31 - lane)
                                               : __shfl_xor_sync(0xffffffffu, k, s);
                    const bool low = (lane & s) == 0;
                    k = low ? (k < o ? k : o) : (k > o ? k : o);
                }
            }
            const bool okl = lane < w && (lane == 0 || !full || !(key_dist(k) > worst));
            const unsigned okm = __ballot_sync(0xffffffffu, okl);
            nsel = okm == 0xffffffffu ? 32 : __ffs(~okm) - 1;  // leading run
            if (full && key_dist(__shfl_sync(0xffffffffu, k, 0)) > worst) break;
            selnode = grow_of(k);
            const uint64_t klast = __shfl_sync(0xffffffffu, k, nsel - 1);
            const int fromb =
                __popc(__ballot_sync(0xffffffffu, lane < G_WMAX && lane < nb && own <= klast));
            bh += fromb;
            mh += nsel - fromb;
        }
        int *cnt = s_cnt[steps & 1];
        steps++;

        // ---- gather neighbours of the selected nodes, visited test-and-set
        // (lists are padded to deg_cap with ids no row has; G_NB of them at a
        // time, which is all unless a single list is longer)
        const int dc = a.deg_cap;
        const int total = nsel * dc;
        {
            constexpr int SL = G_NB / G_THREADS;
            uint32_t nv[SL];
            bool fresh[SL];
#pragma unroll
            for (int u = 0; u < SL; u++) {
                const int t = t0 + u * G_THREADS + tid;
                const int sidx = a.dc_shift >= 0 ? t >> a.dc_shift : t / dc;
                const uint32_t node = __shfl_sync(0xffffffffu, selnode, min(sidx, nsel - 1));
                nv[u] = t < total ? __ldg(a.adj + (uint64_t)node * dc + (t - sidx * dc)) : G_EMPTY;
            }
            int mine = 0;
            unsigned fmask[SL];
#pragma unroll
            for (int u = 0; u < SL; u++) {
                const uint32_t nbr = nv[u];
                fresh[u] = false;
                if (nbr < a.nrows) {
                    if (spilled) {
                        const uint32_t m = 1u << (nbr & 31);
                        fresh[u] = (atomicOr(vb + (nbr >> 5), m) & m) == 0;
                    } else {
                        uint32_t h = hash_u32(nbr) & (G_HC - 1);
                        for (int probe = 0; probe < G_HC; probe++) {
                            const uint32_t old = atomicCAS(hash + h, G_EMPTY, nbr);
                            if (old == G_EMPTY) { fresh[u] = true; break; }
                            if (old == nbr) break;
                            h = (h + 1) & (G_HC - 1);
                        }
                    }
                }
                fmask[u] = __ballot_sync(0xffffffffu, fresh[u]);
                mine += __popc(fmask[u]);
            }
            // one shared-memory atomic per warp for the appends
            int wb = 0;
            if (lane == 0 && mine) {
                wb = atomicAdd(&cnt[0], mine);
                if (!spilled) atomicAdd(&s_hcount, mine);
            }
            wb = __shfl_sync(0xffffffffu, wb, 0);
#pragma unroll
            for (int u = 0; u < SL; u++) {
                const int at = wb + __popc(fmask[u] & ((1u << lane) - 1u));
                if (fresh[u] && at < G_NB) {
                    nid[at] = nv[u];
                    // its row is read after the barrier
                    const char *row = (const char *)(a.vecs + (uint64_t)nv[u] * a.dpad);
                    for (int j = 0; j < a.dpad * 4; j += 128)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + j));
                }
                wb += __popc(fmask[u]);
            }
        }
        t0 = t0 + G_NB < total ? t0 + G_NB : 0;
        if (tid < 3) s_cnt[steps & 1][tid] = 0;  // the next step's
        __syncthreads();
        const int nnew = min(cnt[0], G_NB);
        visited += (unsigned long long)nnew;

        // ---- distances; admission as the reference cursor: a node enters
        // the frontier while results are short or it beats the worst result
        // (engine.cpp:1684-1690). The predicate word of each row is fetched
        // with the row.
        {
            auto admit = [&](auto rpg, int base) {
                constexpr int RPG = decltype(rpg)::value;
                float acc[RPG];
                uint32_t nn[RPG], pw[RPG];
                graph_dists<RPG>(a, sq, nid, bm, base, nnew, acc, nn, pw);
                // admitted rows of this warp (one lane of four), appended
                // with one shared-memory atomic per warp
                unsigned m[RPG], pm[RPG];
                bool ad[RPG];
                int tot = 0, pass = 0;
#pragma unroll
                for (int r = 0; r < RPG; r++) {
                    ad[r] = base + (tid >> 2) + r * (G_THREADS / 4) < nnew && (tid & 3) == 0 &&
                            (!full || acc[r] < worst);
                    m[r] = __ballot_sync(0xffffffffu, ad[r]);
                    pm[r] = __ballot_sync(0xffffffffu, ad[r] && ((pw[r] >> (nn[r] & 31)) & 1u));
                    tot += __popc(m[r]);
                    pass += __popc(pm[r]);
                }
                int wb = 0;
                if (lane == 0 && tot) {
                    wb = atomicAdd(&cnt[1], tot);
                    if (pass) atomicAdd(&cnt[2], pass);
                }
                wb = __shfl_sync(0xffffffffu, wb, 0);
                const unsigned lt = (1u << lane) - 1u;
#pragma unroll
                for (int r = 0; r < RPG; r++) {
                    if (ad[r]) {
                        const bool ps = (pm[r] >> lane) & 1u;
                        nfk[wb + __popc(m[r] & lt)] = make_key(acc[r], nn[r] | (ps ? G_PASS : 0u));
                        // its list is wanted soon if it is expanded
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(
                            a.adj + (uint64_t)nn[r] * a.deg_cap));
                    }
                    wb += __popc(m[r]);
                }
            };
            for (int base = 0; base < nnew;) {
                const int left = nnew - base;
                if (left > 2 * (G_THREADS / 4)) {
                    admit(std::integral_constant<int, 4>{}, base);
                    base += G_THREADS;
                } else if (left > G_THREADS / 4) {
                    admit(std::integral_constant<int, 2>{}, base);
                    base += G_THREADS / 2;
                } else {
                    admit(std::integral_constant<int, 1>{}, base);
                    base += G_THREADS / 4;
                }
            }
        }
        __syncthreads();
        const int nnf = cnt[1], nnr = cnt[2];
        if (bm) probes += (unsigned)nnf;

        if (nnf > 0) {
            // ---- the recent entries make room: merged into the rest
            if (be - bh + nnf > G_BC) {
                const int n0 = be - bh, n1 = me - mh;
                const uint64_t *B = fb0 + cb * G_BC + bh, *M = fm0 + cm * G_FC + mh;
                uint64_t *D = fm0 + (cm ^ 1) * G_FC;
                for (int i = tid; i < n0; i += G_THREADS) D[i + lower(M, n1, B[i])] = B[i];
                for (int i = tid; i < n1; i += G_THREADS) D[i + lower(B, n0, M[i])] = M[i];
                __syncthreads();
                cm ^= 1;
                mh = 0;
                me = n0 + n1;
                bh = be = 0;
            }
            // ---- a new key's places: its rank among the new keys by
            // counting, and binary searches in the results and the recent
            // entries (keys are unique: each node is visited once)
            const int nbn = be - bh;
            const uint64_t *B = fb0 + cb * G_BC + bh;
            uint64_t *Bn = fb0 + (cb ^ 1) * G_BC, *Rn = rs0 + (cr ^ 1) * G_RC;
            for (int i = tid; i < nnf; i += G_THREADS) {
                const uint64_t key = nfk[i];
                int r = 0, rp = 0;
                const bool pass = ((uint32_t)key & G_PASS) != 0;
                int pb, pr;
                lower2(B, nbn, R, pass ? nr : 0, key, pb, pr);
                int j = 0;
#pragma unroll 2
                for (; j + 2 <= nnf; j += 2) {
                    const ulonglong2 o = *(const ulonglong2 *)(nfk + j);
                    const int c0 = o.x < key, c1 = o.y < key;
                    r += c0 + c1;
                    rp += (c0 & (int)((uint32_t)o.x >> 31)) + (c1 & (int)((uint32_t)o.y >> 31));
                }
                if (j < nnf) {
                    const int c0 = nfk[j] < key;
                    r += c0;
                    rp += c0 & (int)((uint32_t)nfk[j] >> 31);
                }
                fpos[r] = pb;
                Bn[pb + r] = key;
                if (pass) {
                    rpos[rp] = pr;
                    if (pr + rp < ef) Rn[pr + rp] = key;
                }
            }
            __syncthreads();
            // an old entry moves up by the number of new keys placed before it
            const int nro = nnr > 0 ? nr : 0;
            for (int i = tid; i < nro + nbn; i += G_THREADS) {
                const bool res = i < nro;
                const int j = res ? i : i - nro;
                const uint64_t key = res ? R[j] : B[j];
                const int at = j + placed(res ? rpos : fpos, res ? nnr : nnf, j);
                if (!res) Bn[at] = key;
                else if (at < ef) Rn[at] = key;
            }
            cb ^= 1;
            bh = 0;
            be = nbn + nnf;
            if (nnr > 0) {
                cr ^= 1;
                nr = min(nr + nnr, ef);
            }
        }

        // ---- spill the visited set to the global bitmap at half load
        if (!spilled && s_hcount > G_HC / 2) {
            for (uint64_t i = tid; i < a.bm_words; i += blockDim.x) vb[i] = 0u;
            __syncthreads();
            for (int i = tid; i < G_HC; i += blockDim.x) {
                const uint32_t v = hash[i];
                if (v != G_EMPTY) atomicOr(vb + (v >> 5), 1u << (v & 31));
            }
            spilled = true;
        }
        __syncthreads();
    }

    // ---- emit (ascending by (dist, node))
    const uint64_t *R = rs0 + cr * G_RC;
    for (int i = tid; i < nr; i += blockDim.x) {
        FvHit h;
        h.node = grow_of(R[i]);
        h.dist = key_dist(R[i]);
        a.out[(uint64_t)q * a.ef + i] = h;
    }
    if (tid == 0) {
        a.out_cnt[q] = (uint32_t)nr;
        a.out_exh[q] = (uint8_t)exh;
        if (a.stats) {
            a.stats[q * 4 + 0] = steps;
            a.stats[q * 4 + 1] = (uint32_t)visited;
            a.stats[q * 4 + 2] = probes;
            a.stats[q * 4 + 3] = (uint32_t)nr;
        }
    }
}

constexpr int G_DIMS = 11460;  // dims at most
size_t graph_smem_bytes(int dpad) {  // without the query: 0 dims
    return (size_t)(2 * G_FC + 2 * G_BC + 2 * G_RC + G_NB + 2) * 8 +
           (size_t)(G_HC + 3 * G_NB) * 4 + (size_t)dpad * 4;
}

cudaError_t launch_graph(const GraphArgs &a, int nq, cudaStream_t st) {
    if (a.dpad > G_DIMS) return cudaErrorInvalidValue;
    const bool wide = graph_smem_bytes(a.dpad) > 227 * 1024 - 256;  // (28 bytes static)
    const size_t smem = graph_smem_bytes(wide ? 0 : a.dpad);
    auto *kernel = wide ? graph_kernel<true> : graph_kernel<false>;
    cudaError_t e = raise_smem_limit((const void *)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<nq, G_THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace pv

using namespace pv;

extern "C" int fv_gpu_graph_batch(FvGpuIndex *g, int nq, const float *queries,
                                  const FvGpuQueryDesc *qd, const FvGpuPredNode *nodes,
                                  int nnodes, const int32_t *children, int nchildren,
                                  const double *invals, int ninvals, uint32_t ef,
                                  uint64_t max_visited, FvHit *out, uint32_t *out_cnt,
                                  uint8_t *exhausted, char *errbuf, size_t errlen) {
    if (!g || !g->d_adj) {
        if (errbuf && errlen) snprintf(errbuf, errlen, "gpu: graph not uploaded");
        return -1;
    }
    if (g->count >= (1ull << 31)) {  // keys keep the predicate bit in bit 31 of the row
        if (errbuf && errlen) snprintf(errbuf, errlen, "gpu: graph search needs < 2^31 rows");
        return -1;
    }
    if (nq < 1 || nq > FV_GPU_MAX_BATCH || ef < 1 || ef > FV_GPU_MAX_EF || !queries || !qd ||
        !out || !out_cnt || !exhausted) {
        if (errbuf && errlen) snprintf(errbuf, errlen, "gpu: bad graph batch (nq=%d ef=%u)", nq, ef);
        return -1;
    }
    std::lock_guard<std::mutex> lk(g->mu);
    PV_CUDA_OK(cudaSetDevice(g->device), errbuf, errlen);
    PredBatch pb;
    if (compile_predicates(nq, &qd[0].proot, sizeof(FvGpuQueryDesc), nodes, nnodes, children,
                           nchildren, invals, ninvals, g->ncols, pb, errbuf, errlen) != 0)
        return -1;
    std::vector<uint32_t> entries(nq);
    for (int q = 0; q < nq; q++) entries[q] = qd[q].entry;
    return graph_run_host(g, nq, queries, entries.data(), pb, ef, max_visited, out, out_cnt,
                          exhausted, errbuf, errlen);
}

namespace pv {

GraphOut graph_out_layout(int nq, uint32_t ef) {
    GraphOut lo;
    const size_t hit_bytes = (size_t)nq * ef * sizeof(FvHit);
    lo.off_cnt = (hit_bytes + 255) & ~(size_t)255;
    lo.off_exh = lo.off_cnt + (((size_t)nq * 4 + 255) & ~(size_t)255);
    lo.off_st = lo.off_exh + (((size_t)nq + 255) & ~(size_t)255);
    lo.bytes = lo.off_st + (size_t)nq * 16;
    return lo;
}

int graph_launch(FvGpuIndex *g, int nq, const float *d_q, const uint32_t *d_entries,
                 const int32_t *d_qprog, const uint16_t *d_efq, uint32_t ef,
                 uint64_t max_visited, char *od, const GraphOut &lo, char *errbuf,
                 size_t errlen, cudaStream_t st) {
    if (!st) st = g->stream;
    const uint64_t bm_words = (g->count + 31) / 32;
    GraphScratch &gs = g->graph;
    PV_CUDA_OK(gs.visited.ensure((size_t)nq * bm_words * 4), errbuf, errlen);
    GraphArgs a;
    a.vecs = g->d_vecs;
    a.dpad = g->dpad;
    a.nrows = g->count;
    a.adj = g->d_adj;
    a.deg_cap = g->deg_cap;
    a.dc_shift = -1;
    for (int sh = 0; sh < 16; sh++)
        if (g->deg_cap == (1 << sh)) a.dc_shift = sh;
    a.queries = d_q;
    a.entries = d_entries;
    a.qprog = d_qprog;
    a.bitmaps = g->scan.bitmaps.as<uint32_t>();
    a.bm_words = bm_words;
    a.ef = (int)ef;
    a.efq = d_efq;
    a.max_visited = max_visited;
    int wmax = G_NB / (g->deg_cap > 0 ? g->deg_cap : 1);
    if (wmax > G_WMAX) wmax = G_WMAX;
    if (wmax < 1) wmax = 1;
    a.wmax = wmax;
    a.visited_bits = gs.visited.as<uint32_t>();
    a.out = (FvHit *)od;
    a.out_cnt = (uint32_t *)(od + lo.off_cnt);
    a.out_exh = (uint8_t *)(od + lo.off_exh);
    a.stats = (uint32_t *)(od + lo.off_st);
    g->launches++;
    PV_CUDA_OK(launch_graph(a, nq, st), errbuf, errlen);
    return 0;
}

int graph_run_host(FvGpuIndex *g, int nq, const float *queries, const uint32_t *entries,
                   const PredBatch &pb, uint32_t ef, uint64_t max_visited, FvHit *out,
                   uint32_t *out_cnt, uint8_t *exhausted, char *errbuf, size_t errlen) {
    g->launches = 0;
    DevBatch db;
    db.stage_h = &g->scan.stage_h;
    db.stage_d = &g->scan.stage_d;
    for (int q = 0; q < nq; q++)
        if (entries[q] >= g->count) {
            snprintf(errbuf, errlen, "gpu: query %d entry %u out of range", q, entries[q]);
            return -1;
        }
    // entries ride in the extra section of the staging buffer
    if (brute_prepare(g, nq, queries, pb, db, (size_t)nq * 4, errbuf, errlen)) return -1;
    const size_t off_ent = db.off_extra;
    memcpy(db.stage_h->as<char>() + off_ent, entries, (size_t)nq * 4);
    if (brute_upload(g, db, errbuf, errlen)) return -1;
    char *d = db.stage_d->as<char>();
    ScanScratch &s = g->scan;
    const int P = db.P;
    cudaEventRecord(g->ev0, g->stream);
    if (P > 0) {
        if (brute_bitmaps(g, db, errbuf, errlen)) return -1;
    }
    const GraphOut lo = graph_out_layout(nq, ef);
    const size_t off_cnt = lo.off_cnt, off_exh = lo.off_exh, off_st = lo.off_st;
    const size_t obytes = lo.bytes;
    PV_CUDA_OK(s.out_d.ensure(obytes), errbuf, errlen);
    PV_CUDA_OK(s.out_h.ensure(obytes), errbuf, errlen);
    char *od = s.out_d.as<char>();
    if (graph_launch(g, nq, (const float *)(d + db.off_q), (const uint32_t *)(d + off_ent),
                     (const int32_t *)(d + db.off_qprog), nullptr, ef, max_visited, od, lo,
                     errbuf, errlen))
        return -1;
    cudaEventRecord(g->ev1, g->stream);
    PV_CUDA_OK(cudaMemcpyAsync(s.out_h.p, od, obytes, cudaMemcpyDeviceToHost, g->stream), errbuf,
               errlen);
    PV_CUDA_OK(cudaStreamSynchronize(g->stream), errbuf, errlen);
    cudaEventElapsedTime(&g->last_kernel_ms, g->ev0, g->ev1);
    const char *oh = s.out_h.as<char>();
    const uint32_t *cnt = (const uint32_t *)(oh + off_cnt);
    for (int q = 0; q < nq; q++) {
        uint32_t c = cnt[q] > ef ? ef : cnt[q];
        memcpy(out + (size_t)q * ef, oh + (size_t)q * ef * sizeof(FvHit), c * sizeof(FvHit));
        out_cnt[q] = c;
    }
    memcpy(exhausted, oh + off_exh, (size_t)nq);
    g->graph_stats.resize((size_t)nq * 4);
    memcpy(g->graph_stats.data(), oh + off_st, (size_t)nq * 16);
    return 0;
}

}  // namespace pv
