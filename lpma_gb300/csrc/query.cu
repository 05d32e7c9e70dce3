// Read paths over the PMA: batched neighbour lists with a time window,
// edge queries, BFS and PageRank.  They read the structure in place (no CSR
// view is built): the keys of vertex v are the occupied slots strictly
// between the sentinel of v-1 and the sentinel of v in linear slot order.
#include <climits>

#include "kernels.cuh"
#include "prims.cuh"
#include "quotient.h"

namespace lpma {
namespace {

constexpr int TPB = 256;

// linear slot (32 * linear segment + lane) of a heap slot index
__device__ inline uint64_t linear_slot(uint32_t heap_slot, uint32_t H) {
    const uint64_t j = heap_slot >> 5;
    const uint32_t level = 63 - __clzll((long long)(j + 1));
    return 32 * linear_of_heap(j, level, H) + (heap_slot & 31);
}

// linear slot range [p0, p1) that holds vertex v's keys (empty slots
// included; a slot is occupied when its lane is below the segment's count)
__device__ inline void vertex_range(const uint32_t *sent, uint32_t v, uint32_t H, uint64_t &p0, uint64_t &p1) {
    p0 = v ? linear_slot(sent[v - 1], H) + 1 : 0;
    p1 = linear_slot(sent[v], H);
}

// One 8-lane group reads linear segment s: lane gl holds slots 4gl..4gl+3.
// Returns the mask of slots that are occupied and inside [p0, p1).
__device__ inline uint32_t load_seg_part(Geo g, const uint8_t *cnt, uint64_t s, uint64_t p0, uint64_t p1, int gl,
                                         uint64_t (&k)[4], uint8_t (&v)[4]) {
    const uint64_t j = heap_of_linear(s, g.H);
    const uint32_t c = cnt[s];
    const uint64_t base = 32 * s;
    const uint32_t a = p0 > base ? (uint32_t)(p0 - base) : 0u;
    const uint32_t b0 = p1 < base + 32 ? (uint32_t)(p1 - base) : 32u;
    const uint32_t b = b0 < c ? b0 : c;
    uint32_t m = 0;
    if (4 * (uint32_t)gl < b && 4 * (uint32_t)gl + 4 > a) {
        const ulonglong2 *kp = reinterpret_cast<const ulonglong2 *>(g.keys + 32 * j + 4 * gl);
        const ulonglong2 x = kp[0], y = kp[1];
        const uint32_t v4 = *reinterpret_cast<const uint32_t *>(g.vals + 32 * j + 4 * gl);
        k[0] = x.x, k[1] = x.y, k[2] = y.x, k[3] = y.y;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = (uint8_t)(v4 >> (8 * q));
            const uint32_t slot = 4 * gl + q;
            if (slot >= a && slot < b && v[q] != VAL_TOMB) m |= 1u << q;
        }
    }
    return m;
}

__device__ inline bool in_window(uint64_t key, uint32_t lb, uint32_t ub) {
    const uint32_t t = (uint32_t)(key & TIME_MASK);
    return t >= lb && t <= ub;
}

// ---------------------------------------------------------------- neighbour lists
// query_rpma (rpma.cuh:1827-2036): for query i, the neighbours of srcs[i]
// whose timestamp lies in [windows[i] >> 32, windows[i] & 0xFFFFFFFF], in
// key order.
//
// The queries' rounds (4 segments, one per 8-lane group of a warp; at least
// one round a query) are laid end to end and cut into equal shares, one a
// warp, so a hub's list is read by many warps.  The lists too lie end to end
// in that order: a share's neighbours start where those of the shares
// before it end.  Pass 1 counts each share (and, for each query that starts
// in it, the share's neighbours before that query); its last CTA sums the
// shares; pass 2 writes.  A warp per query walked the hubs serially: 4,096
// lists of a scale-20 graph, 8 hubs among them, took 240 us a count and 335 a
// fill, now 24 and 11 (and 12 to weigh the queries).
//
// A query counts as nbr_cap(n) rounds at most, so that the rounds of all n
// stay below 2^31; one of more is cut into that many equal parts.
constexpr uint32_t NBR_CTAS = 152 * 4, NBR_SHARES = NBR_CTAS * (TPB / 32);
constexpr uint32_t NBR_ONE_CTA = 8192;  // up to here one CTA weighs the queries, and one places the lists

__host__ __device__ inline uint32_t nbr_cap(uint32_t n) { return ((1u << 31) - 1) / n; }

__device__ __forceinline__ uint32_t nbr_rounds(uint32_t src, uint32_t n, uint32_t V, Geo g, const uint32_t *sent) {
    if (src >= V) return 1;
    uint64_t p0, p1;
    vertex_range(sent, src, g.H, p0, p1);
    return p1 > p0 ? min((uint32_t)(((p1 - 1) >> 5) - (p0 >> 5)) / 4 + 1, nbr_cap(n)) : 1u;
}

// rounds of every query (scanned afterwards)
__global__ void __launch_bounds__(TPB) k_nbr_weigh(const uint32_t *__restrict__ srcs, uint32_t n, Geo g,
                                                   const uint32_t *__restrict__ sent, uint32_t V, uint32_t *w) {
    for (uint32_t i = blockIdx.x * TPB + threadIdx.x; i < n; i += gridDim.x * TPB)
        w[i] = nbr_rounds(srcs[i], n, V, g, sent);
}

// the same and the exclusive scan for up to NBR_ONE_CTA queries, in one CTA
__global__ void __launch_bounds__(1024) k_nbr_weigh_scan(const uint32_t *__restrict__ srcs, uint32_t n, Geo g,
                                                         const uint32_t *__restrict__ sent, uint32_t V,
                                                         uint32_t *P) {
    constexpr uint32_t PER = NBR_ONE_CTA / 1024;
    __shared__ uint32_t ws[32];
    const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint32_t per = (n + 1023) / 1024, beg = threadIdx.x * per;
    uint32_t x[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
        x[q] = q < per && beg + q < n ? nbr_rounds(srcs[beg + q], n, V, g, sent) : 0u;
        sum += x[q];
    }
    uint32_t v = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    if (lane == 31) ws[wp] = v;
    __syncthreads();
    uint32_t off = v - sum, tot = 0;
    for (uint32_t k = 0; k < 32; k++) {
        const uint32_t y = ws[k];
        off += k < wp ? y : 0u;
        tot += y;
    }
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
        if (q < per && beg + q < n) P[beg + q] = off;
        off += x[q];
    }
    if (threadIdx.x == 0) P[n] = tot;
}

// Walks the rounds of share w: f(i, first, s0, s1, p0, p1, window) for each
// query i in it (whole warps), first when the share holds its first round;
// segments [s0, s1) of it, none for a query without slots.
template <typename F>
__device__ __forceinline__ void nbr_walk(uint32_t w, const uint32_t *__restrict__ srcs,
                                         const uint64_t *__restrict__ windows, uint32_t n, Geo g,
                                         const uint32_t *__restrict__ sent, uint32_t V,
                                         const uint32_t *__restrict__ P, F f) {
    const uint64_t T = P[n];
    const uint32_t u0 = (uint32_t)(T * w / NBR_SHARES), u1 = (uint32_t)(T * (w + 1) / NBR_SHARES);
    if (u0 >= u1) return;
    uint32_t i = forest_job_of(P, n, u0);
    for (uint32_t u = u0; u < u1; i++) {
        const uint32_t qs = P[i], qe = P[i + 1];
        const uint32_t a = u - qs, b = min(u1, qe) - qs;  // rounds [a, b) of query i
        const uint32_t src = srcs[i];
        const uint64_t win = windows[i];
        uint64_t p0 = 0, p1 = 0;
        if (src < V) vertex_range(sent, src, g.H, p0, p1);
        uint32_t s0 = 0, s1 = 0;
        if (p1 > p0) {
            const uint32_t S0 = (uint32_t)(p0 >> 5), ns = (uint32_t)((p1 - 1) >> 5) + 1 - S0;
            const uint32_t per = 4 * (((ns + 3) / 4 + qe - qs - 1) / (qe - qs));  // segments a round stands for
            s0 = S0 + (uint32_t)umin64(ns, (uint64_t)a * per);
            s1 = S0 + (uint32_t)umin64(ns, (uint64_t)b * per);
        }
        f(i, a == 0, s0, s1, p0, p1, win);
        u = qs + b;
    }
}

__global__ void __launch_bounds__(TPB) k_nbr_count(const uint32_t *__restrict__ srcs,
                                                   const uint64_t *__restrict__ windows, uint32_t n, Geo g,
                                                   const uint8_t *__restrict__ cnt, const uint32_t *__restrict__ sent,
                                                   uint32_t V, const uint32_t *__restrict__ P, uint32_t *done, uint2 *at,
                                                   uint32_t *base, uint32_t *offsets) {
    const int lane = threadIdx.x & 31, gl = lane & 7, grp = lane >> 3;
    const uint32_t w = (blockIdx.x * TPB + threadIdx.x) >> 5;
    uint32_t run = 0;  // the share's neighbours so far
    nbr_walk(w, srcs, windows, n, g, sent, V, P,
             [&](uint32_t i, bool first, uint32_t s0, uint32_t s1, uint64_t p0, uint64_t p1, uint64_t win) {
                 if (first && lane == 0) at[i] = make_uint2(w, run);
                 const uint32_t lb = (uint32_t)(win >> 32), ub = (uint32_t)win;
                 uint32_t c = 0;
                 for (uint32_t s = s0 + grp; s < s1; s += 4) {
                     uint64_t k[4];
                     uint8_t v[4];
                     const uint32_t m = load_seg_part(g, cnt, s, p0, p1, gl, k, v);
#pragma unroll
                     for (int q = 0; q < 4; q++)
                         if (((m >> q) & 1u) && in_window(k[q], lb, ub)) c++;
                 }
                 run += __reduce_add_sync(0xffffffffu, c);
             });
    if (lane == 0) base[w] = run;
    // the last CTA to finish turns the shares' counts into their starts
    __shared__ uint32_t last;
    __shared__ uint32_t ws[TPB / 32];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    constexpr uint32_t PER = NBR_SHARES / TPB;
    static_assert(NBR_SHARES % TPB == 0, "equal runs of shares a thread");
    uint32_t x[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) sum += x[q] = __ldcg(base + threadIdx.x * PER + q);
    uint32_t v = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t off = v - sum, tot = 0;
#pragma unroll
    for (uint32_t k = 0; k < TPB / 32; k++) {
        const uint32_t y = ws[k];
        off += k < (threadIdx.x >> 5) ? y : 0u;
        tot += y;
    }
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
        base[threadIdx.x * PER + q] = off;
        off += x[q];
    }
    if (threadIdx.x == 0) offsets[n] = tot;
    if (n > NBR_ONE_CTA) return;  // k_nbr_offsets places the lists
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += TPB) {
        const uint32_t sw = __ldcg(&at[i].x), sr = __ldcg(&at[i].y);
        offsets[i] = __ldcg(base + sw) + sr;
    }
}

__global__ void __launch_bounds__(TPB) k_nbr_offsets(uint32_t n, const uint2 *__restrict__ at,
                                                     const uint32_t *__restrict__ base, uint32_t *offsets) {
    const uint32_t i = blockIdx.x * TPB + threadIdx.x;
    if (i < n) offsets[i] = base[at[i].x] + at[i].y;
}

__global__ void __launch_bounds__(TPB) k_nbr_fill(const uint32_t *__restrict__ srcs,
                                                  const uint64_t *__restrict__ windows, uint32_t n, Geo g,
                                                  const uint8_t *__restrict__ cnt, const uint32_t *__restrict__ sent,
                                                  uint32_t V, const uint32_t *__restrict__ P,
                                                  const uint32_t *__restrict__ base, uint32_t *nbrs, uint8_t *vals) {
    const int lane = threadIdx.x & 31, gl = lane & 7, grp = lane >> 3;
    const uint32_t w = (blockIdx.x * TPB + threadIdx.x) >> 5;
    uint32_t out = base[w];
    nbr_walk(w, srcs, windows, n, g, sent, V, P,
             [&](uint32_t, bool, uint32_t s0, uint32_t s1, uint64_t p0, uint64_t p1, uint64_t win) {
                 const uint32_t lb = (uint32_t)(win >> 32), ub = (uint32_t)win;
                 for (uint32_t sr = s0; sr < s1; sr += 4) {
                     const uint32_t s = sr + grp;
                     uint64_t k[4];
                     uint8_t v[4];
                     uint32_t m = 0;
                     if (s < s1) m = load_seg_part(g, cnt, s, p0, p1, gl, k, v);
#pragma unroll
                     for (int q = 0; q < 4; q++)
                         if (((m >> q) & 1u) && !in_window(k[q], lb, ub)) m &= ~(1u << q);
                     // warp-wide exclusive prefix in (group, lane, slot) order = key order
                     const uint32_t c = __popc(m);
                     uint32_t incl = c;
#pragma unroll
                     for (int o = 1; o < 32; o <<= 1) {
                         const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                         if (lane >= o) incl += y;
                     }
                     uint32_t pos = out + incl - c;
#pragma unroll
                     for (int q = 0; q < 4; q++) {
                         if ((m >> q) & 1u) {
                             nbrs[pos] = (uint32_t)((k[q] & DST_MASK) >> DST_SHIFT);
                             vals[pos] = v[q];
                             pos++;
                         }
                     }
                     out += __shfl_sync(0xffffffffu, incl, 31);
                 }
             });
}

// ---------------------------------------------------------------- edge queries
// For key (src, dst, t): the number of stored keys (src, dst, t') with
// t - window <= t' <= t (the edge-query check of test.cu:46-62; window =
// 0xFFFFF with t = 0xFFFFF gives check_edge_kernel's any-time test,
// rpma.cuh:2040-2066).  One thread a query: src's sentinels give its segment
// range, a binary search over the segments' last keys the first one that
// reaches (src, dst, lb), five probes of that segment its first key >= lb,
// and the count goes forward from there.  The sentinel of src ends both
// searches (it is above every key asked for), so neither tests a bound.
//
// Bound by its random reads (sentinels, segment bounds out of L2, slots out
// of DRAM), about 10 sectors a query.  The segment's bounds stand for its
// count (an empty one has no first key): one load a step where there were
// two; the slots are halved twice and a quarter (64 bytes, one DRAM access)
// loads at once, where they were walked from the first on.  2M queries of a
// 15M-key graph 184 -> 144 us, 400K of 19M keys 60 -> 39, 4K 21 -> 13.
// Measured slower: three probes a step of the segment search (159 us for
// 2M: more L2 sectors), the three quarter bounds of a segment at once (178:
// more DRAM accesses).
__global__ void __launch_bounds__(TPB) k_edge_query(const uint64_t *__restrict__ q, uint32_t n, uint32_t window, Geo g,
                                                    const ulonglong2 *__restrict__ fl,
                                                    const uint32_t *__restrict__ sent, uint32_t V, uint32_t *res) {
    for (uint64_t i = blockIdx.x * (uint64_t)TPB + threadIdx.x; i < n; i += gridDim.x * (uint64_t)TPB) {
        const uint64_t key = q[i];
        const uint32_t src = (uint32_t)(key >> SRC_SHIFT);
        const uint32_t dst = (uint32_t)((key & DST_MASK) >> DST_SHIFT);
        uint32_t found = 0;
        if (src < V && dst < NBR_END) {
            const uint32_t t = (uint32_t)(key & TIME_MASK);
            const uint32_t lb = t > window ? t - window : 0;
            const uint64_t pre = key & ~TIME_MASK;
            const uint64_t lo = pre | lb, hi = pre | t;
            const uint32_t e1 = sent[src], e0 = src ? sent[src - 1] : 0u;
            // src's keys lie in the segments of its predecessor's sentinel to its own
            uint32_t L = src ? (uint32_t)(linear_slot(e0, g.H) >> 5) : 0u;
            const uint32_t last_seg = (uint32_t)(linear_slot(e1, g.H) >> 5);
            // first non-empty segment whose last key >= lo (last_seg is one)
            uint32_t U = last_seg, s = last_seg;
            while (L < U) {
                const uint32_t mid = (L + U) >> 1;
                uint32_t ms = mid;
                ulonglong2 b = fl[heap_of_linear32(ms, g.H)];
                while (b.x == KEY_NONE && ++ms < U) b = fl[heap_of_linear32(ms, g.H)];
                if (ms == U) {
                    U = mid;  // [mid, U) holds nothing
                } else if (b.y >= lo) {
                    s = ms;
                    U = mid;
                } else {
                    L = ms + 1;
                }
            }
            const uint64_t *sk = g.keys + 32ull * heap_of_linear32(s, g.H);
            // the first key >= lo: two probes choose a quarter of the segment,
            // whose 8 keys (64 bytes) then load together
            uint32_t pos = sk[15] < lo ? 16u : 0u;
            if (sk[pos + 7] < lo) pos += 8;
            {
                const ulonglong2 *qp = reinterpret_cast<const ulonglong2 *>(sk + pos);
                const ulonglong2 a = qp[0], b = qp[1], c = qp[2], d = qp[3];
                pos += (a.x < lo) + (a.y < lo) + (b.x < lo) + (b.y < lo) + (c.x < lo) + (c.y < lo) + (d.x < lo) +
                       (d.y < lo);
            }
            for (;;) {
                const uint64_t kk = pos < 32 ? sk[pos] : KEY_NONE;
                if (kk == KEY_NONE) {  // the segment's keys end: the next one that has any
                    uint64_t first = KEY_NONE;
                    while (s < last_seg && first == KEY_NONE) first = fl[heap_of_linear32(++s, g.H)].x;
                    if (first > hi) break;
                    sk = g.keys + 32ull * heap_of_linear32(s, g.H);
                    pos = 0;
                    continue;
                }
                if (kk > hi) break;
                if (g.vals[(uint64_t)(sk - g.keys) + pos] != VAL_TOMB) found++;
                if (kk == hi) break;  // keys are distinct
                pos++;
            }
        }
        res[i] = found;
    }
}

// ---------------------------------------------------------------- BFS
// A frontier is a list of slot ranges of at most BFS_SEGS segments each (a
// vertex of many edges makes several), so the work of a level spreads over
// the grid whatever the degrees are: one 8-lane group expands a range.  A
// vertex found at this level gets dist = level + 1 and its ranges join the
// next frontier; a warp queues what it finds and places 32 vertices with one
// atomic.
//
// With a warp per frontier vertex the hubs of an R-MAT graph were walked by
// one warp each: a 2-hop BFS from 1,024 seeds of a scale-20 graph (16.8M
// edges) took 1,697 us of expansion, a full one 3,376; now 128 and 362 (280
// and 524 with an atomic per find round: a million on one address).  Ranges
// of 1, 2, 4 and 8 segments measured within 5%; 4 keeps the lists short.
// Bound by the random reads of dist (one a stored edge, out of L2).
constexpr uint32_t BFS_SEGS = 4;

// the ranges of the vertices d of the lanes with `add` set (whole warps)
__device__ inline void bfs_append(bool add, uint32_t d, Geo g, const uint32_t *__restrict__ sent, uint2 *items,
                                  uint32_t cap, uint32_t *n_items) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t p0 = 0, p1 = 0;
    if (add) vertex_range(sent, d, g.H, p0, p1);
    const uint32_t k = p1 > p0 ? (uint32_t)(((p1 - 1) >> 5) - (p0 >> 5)) / BFS_SEGS + 1 : 0u;
    uint32_t incl = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    if (!tot) return;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(n_items, tot);
    at = __shfl_sync(0xffffffffu, at, 0) + incl - k;
    uint64_t a = p0;
    for (uint32_t i = 0; i < k; i++) {
        const uint64_t e = umin64(p1, ((a >> 5) + BFS_SEGS) << 5);
        if (at + i < cap) items[at + i] = make_uint2((uint32_t)a, (uint32_t)e);
        a = e;
    }
}

__global__ void __launch_bounds__(TPB) k_bfs_init(int32_t *dist, uint32_t V) {
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB)
        dist[v] = INT_MAX;
}

__global__ void __launch_bounds__(TPB) k_bfs_seed(const uint32_t *__restrict__ sources, uint32_t n, uint32_t V, Geo g,
                                                  const uint32_t *__restrict__ sent, int32_t *dist, uint2 *items,
                                                  uint32_t cap, uint32_t *n_items, uint32_t *n_found) {
    for (uint64_t i0 = blockIdx.x * (uint64_t)TPB; i0 < n; i0 += gridDim.x * (uint64_t)TPB) {
        const uint64_t i = i0 + threadIdx.x;
        const uint32_t s = i < n ? sources[i] : V;
        const bool add = s < V && atomicCAS(&dist[s], INT_MAX, 0) == INT_MAX;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, add));
        if (c && (threadIdx.x & 31) == 0) atomicAdd(n_found, c);
        bfs_append(add, s, g, sent, items, cap, n_items);
    }
}

__global__ void __launch_bounds__(TPB) k_bfs_expand(const uint2 *__restrict__ items, const uint32_t *__restrict__ n_p,
                                                    int32_t level, Geo g, const uint8_t *__restrict__ cnt,
                                                    const uint32_t *__restrict__ sent, int32_t *dist, uint2 *next,
                                                    uint32_t cap, uint32_t *n_next, uint32_t *n_found) {
    // vertices found by a warp wait here until they fill it once
    __shared__ uint32_t queue[TPB / 32][160];
    uint32_t *Q = queue[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, gl = lane & 7;
    const uint32_t n = min(*n_p, cap), stride = gridDim.x * (TPB / 8), lt = lanemask_lt();
    uint32_t found = 0, nq = 0;
    for (uint32_t i0 = (blockIdx.x * TPB + threadIdx.x) / 32 * 4; i0 < n; i0 += stride) {  // uniform over the warp
        const uint32_t i = i0 + (lane >> 3);
        const uint2 it = i < n ? items[i] : make_uint2(0u, 0u);
        const uint32_t s0 = it.x >> 5, ns = it.y > it.x ? ((it.y - 1) >> 5) - s0 + 1 : 0u;
        const uint32_t nmax = __reduce_max_sync(0xffffffffu, ns);
        for (uint32_t r = 0; r < nmax; r++) {
            uint64_t k[4];
            uint8_t v[4];
            uint32_t m = 0;
            if (r < ns) m = load_seg_part(g, cnt, s0 + r, it.x, it.y, gl, k, v);
            uint32_t d[4];
            // most neighbours are known already: a plain read comes before the
            // compare-and-swap (a distance is written once)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                d[q] = (uint32_t)((k[q] & DST_MASK) >> DST_SHIFT);
                if (((m >> q) & 1u) && dist[d[q]] != INT_MAX) m &= ~(1u << q);
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (((m >> q) & 1u) && atomicCAS(&dist[d[q]], INT_MAX, level + 1) != INT_MAX) m &= ~(1u << q);
            found += __popc(m);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t bal = __ballot_sync(0xffffffffu, (m >> q) & 1u);
                if ((m >> q) & 1u) Q[nq + __popc(bal & lt)] = d[q];
                nq += __popc(bal);
            }
            __syncwarp();
            while (nq >= 32) {
                nq -= 32;
                bfs_append(true, Q[nq + lane], g, sent, next, cap, n_next);
            }
            __syncwarp();
        }
    }
    bfs_append((uint32_t)lane < nq, (uint32_t)lane < nq ? Q[lane] : 0u, g, sent, next, cap, n_next);
    found = __reduce_add_sync(0xffffffffu, found);
    if (lane == 0 && found) atomicAdd(n_found, found);
}

// ---------------------------------------------------------------- PageRank
// out-degree: one 8-lane group per segment, one atomic per run of equal
// sources within a lane's four slots
__global__ void __launch_bounds__(TPB) k_outdeg(Geo g, const uint8_t *__restrict__ cnt, uint32_t *deg) {
    const uint64_t nseg = nseg_of(g.H);
    const int gl = threadIdx.x & 7;
    for (uint64_t s = (blockIdx.x * (uint64_t)TPB + threadIdx.x) >> 3; s < nseg; s += (gridDim.x * (uint64_t)TPB) >> 3) {
        uint64_t k[4];
        uint8_t v[4];
        const uint32_t m = load_seg_part(g, cnt, s, 0, ~0ull, gl, k, v);
        uint32_t run_src = 0xFFFFFFFFu, run = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (((m >> q) & 1u) && !is_sentinel(k[q])) {
                const uint32_t src = (uint32_t)(k[q] >> SRC_SHIFT);
                if (src != run_src) {
                    if (run) atomicAdd(&deg[run_src], run);
                    run_src = src;
                    run = 0;
                }
                run++;
            }
        }
        if (run) atomicAdd(&deg[run_src], run);
    }
}

// contrib[v] = rank[v] / deg[v]; the rank of vertices without out-edges is
// summed into *dangling
__global__ void __launch_bounds__(TPB) k_pr_contrib(const double *__restrict__ rank, const uint32_t *__restrict__ deg,
                                                    uint32_t V, double *contrib, double *dangling) {
    __shared__ double ws[TPB / 32];
    double d = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB) {
        const uint32_t c = deg[v];
        contrib[v] = c ? rank[v] / (double)c : 0.0;
        if (!c) d += rank[v];
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int i = 0; i < TPB / 32; i++) t += ws[i];
        if (t != 0.0) atomicAdd(dangling, t);
    }
}

__global__ void __launch_bounds__(TPB) k_pr_push(Geo g, const uint8_t *__restrict__ cnt,
                                                 const double *__restrict__ contrib, double *acc) {
    const uint64_t nseg = nseg_of(g.H);
    const int gl = threadIdx.x & 7;
    for (uint64_t s = (blockIdx.x * (uint64_t)TPB + threadIdx.x) >> 3; s < nseg; s += (gridDim.x * (uint64_t)TPB) >> 3) {
        uint64_t k[4];
        uint8_t v[4];
        const uint32_t m = load_seg_part(g, cnt, s, 0, ~0ull, gl, k, v);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (((m >> q) & 1u) && !is_sentinel(k[q])) {
                const uint32_t src = (uint32_t)(k[q] >> SRC_SHIFT);
                const uint32_t dst = (uint32_t)((k[q] & DST_MASK) >> DST_SHIFT);
                atomicAdd(&acc[dst], contrib[src]);
            }
        }
    }
}

// rank = (1 - alpha) / V + alpha * (acc + dangling / V); clears acc and
// leaves the dangling sum for the next iteration at zero
__global__ void __launch_bounds__(TPB) k_pr_finish(double *rank, double *acc, uint32_t V, double alpha,
                                                   const double *__restrict__ dangling) {
    const double base = (1.0 - alpha) / (double)V, dv = *dangling / (double)V;
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB) {
        rank[v] = base + alpha * (acc[v] + dv);
        acc[v] = 0.0;
    }
}

__global__ void k_zero_f64(double *p) { *p = 0.0; }

// PageRank of several iterations reads the edges by destination instead.
// The edges are laid out once per call as 32-bit words src << 10 | (dst mod
// 1024), grouped by dst / 1024 (a bin), each bin cut into chunks of up to
// PR_CHUNK edges that are sorted by destination.  An iteration is then a sum
// over runs of equal destinations: one CTA a chunk, 32 consecutive edges a
// thread, a run inside a thread's edges stored once, one that crosses
// threads added in shared memory; a chunk adds at most 1,024 sums to acc.
//
// The push form (k_pr_push) makes one f64 atomic an edge: 276-300 us an
// iteration on a scale-20 graph (16.8M edges).  This form takes 102 (86 of
// them the sums) after 342 for the layout; bound by the random 8-byte reads
// of contrib (one a stored edge, out of L2: 5.5 TB/s of 32-byte sectors) and
// the FP64 adds.  Chunks of 8,192 edges by 256 threads: 97 with 16,384 by
// 512, whose CTAs wait longer for their last warp.
constexpr uint32_t PR_LOW = 10, PR_BIN = 1u << PR_LOW, PR_MAX_BINS = 4096, PR_CHUNK = 8192;
constexpr uint32_t PR_SORT_TPB = 1024, PR_PULL_TPB = 256, PR_EPT = PR_CHUNK / PR_PULL_TPB;
constexpr uint32_t PR_TILE_SEGS = 512;  // segments a CTA counts or places

// the edges of segment s: f(src, dst) on each of the group's lanes
template <typename F>
__device__ __forceinline__ void seg_edges(Geo g, const uint8_t *__restrict__ cnt, uint64_t s, int gl, F f) {
    uint64_t k[4];
    uint8_t v[4];
    const uint32_t m = load_seg_part(g, cnt, s, 0, ~0ull, gl, k, v);
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (((m >> q) & 1u) && !is_sentinel(k[q]))
            f((uint32_t)(k[q] >> SRC_SHIFT), (uint32_t)((k[q] & DST_MASK) >> DST_SHIFT));
}

__global__ void __launch_bounds__(TPB) k_pr_count(Geo g, const uint8_t *__restrict__ cnt, uint32_t nbins,
                                                  uint32_t *bins) {
    __shared__ uint32_t hist[PR_MAX_BINS];
    for (uint32_t b = threadIdx.x; b < nbins; b += TPB) hist[b] = 0;
    __syncthreads();
    const uint64_t nseg = nseg_of(g.H), t0 = (uint64_t)blockIdx.x * PR_TILE_SEGS;
    for (uint32_t r = threadIdx.x >> 3; r < PR_TILE_SEGS; r += TPB / 8)
        if (t0 + r < nseg)
            seg_edges(g, cnt, t0 + r, threadIdx.x & 7,
                      [&](uint32_t, uint32_t dst) { atomicAdd(&hist[dst >> PR_LOW], 1u); });
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nbins; b += TPB)
        if (hist[b]) atomicAdd(&bins[b], hist[b]);
}

// one CTA: bins[b] (counts) -> where each bin starts (multiples of 4 words),
// the cursors of the placing, and the chunks (first word, edges, bin, the
// bin's chunks)
__global__ void __launch_bounds__(1024) k_pr_table(uint32_t nbins, uint32_t *bins, uint4 *chunks,
                                                   uint32_t *n_chunks) {
    constexpr uint32_t PER = PR_MAX_BINS / 1024;
    __shared__ uint64_t ws[32];
    const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    uint32_t c[PER];
    uint64_t sum = 0;  // words in the low half (below 2^32: at most 2^30 keys), chunks in the high
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
        const uint32_t b = threadIdx.x * PER + q;
        c[q] = b < nbins ? bins[b] : 0u;
        sum += (uint64_t)((c[q] + 3) & ~3u) | ((uint64_t)((c[q] + PR_CHUNK - 1) / PR_CHUNK) << 32);
    }
    uint64_t v = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    if (lane == 31) ws[wp] = v;
    __syncthreads();
    uint64_t off = v - sum, tot = 0;
    for (uint32_t k = 0; k < 32; k++) {
        off += k < wp ? ws[k] : 0u;
        tot += ws[k];
    }
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
        const uint32_t b = threadIdx.x * PER + q;
        if (b >= nbins) break;
        const uint32_t nch = (c[q] + PR_CHUNK - 1) / PR_CHUNK;
        bins[b] = (uint32_t)off;
        for (uint32_t k = 0; k < nch; k++)
            chunks[(uint32_t)(off >> 32) + k] =
                make_uint4((uint32_t)off + k * PR_CHUNK, min(PR_CHUNK, c[q] - k * PR_CHUNK), b, nch);
        off += (uint64_t)((c[q] + 3) & ~3u) | ((uint64_t)nch << 32);
    }
    if (threadIdx.x == 0) *n_chunks = (uint32_t)(tot >> 32);
}

// every edge to its bin: a CTA counts its tile's edges per bin, takes its
// places in each bin with one atomic, and writes them
__global__ void __launch_bounds__(TPB) k_pr_place(Geo g, const uint8_t *__restrict__ cnt, uint32_t nbins,
                                                  uint32_t *cursor, uint32_t *edges, uint32_t cap) {
    __shared__ uint32_t at[PR_MAX_BINS];
    for (uint32_t b = threadIdx.x; b < nbins; b += TPB) at[b] = 0;
    __syncthreads();
    const uint64_t nseg = nseg_of(g.H), t0 = (uint64_t)blockIdx.x * PR_TILE_SEGS;
    for (uint32_t r = threadIdx.x >> 3; r < PR_TILE_SEGS; r += TPB / 8)
        if (t0 + r < nseg)
            seg_edges(g, cnt, t0 + r, threadIdx.x & 7,
                      [&](uint32_t, uint32_t dst) { atomicAdd(&at[dst >> PR_LOW], 1u); });
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nbins; b += TPB)
        if (at[b]) at[b] = atomicAdd(&cursor[b], at[b]);
    __syncthreads();
    for (uint32_t r = threadIdx.x >> 3; r < PR_TILE_SEGS; r += TPB / 8)
        if (t0 + r < nseg)
            seg_edges(g, cnt, t0 + r, threadIdx.x & 7, [&](uint32_t src, uint32_t dst) {
                const uint32_t p = atomicAdd(&at[dst >> PR_LOW], 1u);
                if (p < cap) edges[p] = (src << PR_LOW) | (dst & (PR_BIN - 1));
            });
}

// each chunk sorted by destination, in place (a counting sort in shared memory)
__global__ void __launch_bounds__(PR_SORT_TPB) k_pr_sort(const uint4 *__restrict__ chunks,
                                                         const uint32_t *__restrict__ n_chunks, uint32_t *edges) {
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t *e = sm, *o = sm + PR_CHUNK, *at = sm + 2 * PR_CHUNK, *ws = at + PR_BIN;
    static_assert(PR_SORT_TPB == PR_BIN, "a counter a thread");
    if (blockIdx.x >= *n_chunks) return;
    const uint4 c = chunks[blockIdx.x];
    const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    at[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c.y; i += PR_SORT_TPB) {
        e[i] = edges[c.x + i];
        atomicAdd(&at[e[i] & (PR_BIN - 1)], 1u);
    }
    __syncthreads();
    const uint32_t x = at[threadIdx.x];
    uint32_t v = x;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, k);
        if (lane >= (uint32_t)k) v += y;
    }
    if (lane == 31) ws[wp] = v;
    __syncthreads();
    uint32_t off = v - x;
    for (uint32_t k = 0; k < wp; k++) off += ws[k];
    at[threadIdx.x] = off;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c.y; i += PR_SORT_TPB) o[atomicAdd(&at[e[i] & (PR_BIN - 1)], 1u)] = e[i];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c.y; i += PR_SORT_TPB) edges[c.x + i] = o[i];
}

__global__ void __launch_bounds__(PR_PULL_TPB) k_pr_pull(const uint4 *__restrict__ chunks,
                                                         const uint32_t *__restrict__ n_chunks,
                                                         const uint32_t *__restrict__ edges,
                                                         const double *__restrict__ contrib, double *acc, uint32_t V) {
    __shared__ double sum[PR_BIN];
    if (blockIdx.x >= *n_chunks) return;
    const uint4 c = chunks[blockIdx.x];
    for (uint32_t d = threadIdx.x; d < PR_BIN; d += PR_PULL_TPB) sum[d] = 0.0;
    __syncthreads();
    const uint32_t e0 = threadIdx.x * PR_EPT;
    if (e0 < c.y) {
        const uint32_t n = min(PR_EPT, c.y - e0);
        const uint4 *ep = reinterpret_cast<const uint4 *>(edges + c.x + e0);  // chunks start at multiples of 4
        uint32_t cur = 0xFFFFFFFFu;
        double run = 0.0;
        bool shared_run = true;  // the first run may go on from the thread before
        for (uint32_t i = 0; i < n; i += 8) {
            const uint4 a = ep[i / 4], b = i + 4 < n ? ep[i / 4 + 1] : make_uint4(0, 0, 0, 0);
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            double x[8];
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = i + q < n ? contrib[w[q] >> PR_LOW] : 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (i + q >= n) break;
                const uint32_t d = w[q] & (PR_BIN - 1);
                if (d != cur) {
                    if (cur != 0xFFFFFFFFu) {
                        if (shared_run)
                            atomicAdd(&sum[cur], run);
                        else
                            sum[cur] = run;
                        shared_run = false;
                    }
                    cur = d;
                    run = x[q];
                } else {
                    run += x[q];
                }
            }
        }
        atomicAdd(&sum[cur], run);  // the last run may go on in the next thread
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < PR_BIN; d += PR_PULL_TPB) {
        const uint32_t v = c.z * PR_BIN + d;
        if (v >= V) break;
        if (c.w == 1)
            acc[v] = sum[d];
        else if (sum[d] != 0.0)
            atomicAdd(&acc[v], sum[d]);
    }
}

// out-degrees from the slot ranks of the sentinels (P: exclusive prefix of
// the segment counts): their reciprocals, and they themselves
__global__ void __launch_bounds__(TPB) k_pr_deg(const uint32_t *__restrict__ P, const uint32_t *__restrict__ sent,
                                                uint32_t H, uint32_t V, double2 *inv) {
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB) {
        const uint64_t p1 = linear_slot(sent[v], H), p0 = v ? linear_slot(sent[v - 1], H) : 0;
        const uint32_t r1 = P[p1 >> 5] + (uint32_t)(p1 & 31), r0 = v ? P[p0 >> 5] + (uint32_t)(p0 & 31) + 1 : 0u;
        const double n = (double)(r1 - r0);
        inv[v] = r1 > r0 ? make_double2(1.0 / n, n) : make_double2(0.0, 0.0);
    }
}

// rank (1/V when init, else from acc and *dangling), contrib = rank / deg,
// the next dangling sum; clears acc and the dangling word after that
// (base = (1 - alpha) / V, first = 1 / V).
//
// Bound by the FP64 pipes, which take two lanes a clock: five operations a
// vertex, the degree being stored as a double beside its reciprocal.  So no
// thread divides (three quotients a thread took 20 of the 28 us of a step
// over 1M vertices; quotient.h has the same result), and zero sums are not
// added up.
__global__ void __launch_bounds__(TPB) k_pr_step(bool init, double *rank, double *acc, const double2 *__restrict__ inv,
                                                 uint32_t V, double alpha, double base, double first, const double *__restrict__ dangling, double *next,
                                                 double *after, double *contrib) {
    __shared__ double ws[TPB / 32], s_dv;
    if (threadIdx.x == 0) s_dv = init ? 0.0 : *dangling / (double)V;
    __syncthreads();
    const double dv = s_dv;
    double d = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB) {
        const double r = init ? first : base + alpha * (acc[v] + dv);
        rank[v] = r;
        acc[v] = 0.0;
        const double2 i = inv[v];
        if (__double_as_longlong(i.y) == 0) {
            contrib[v] = 0.0;
            d += r;
        } else {
            contrib[v] = quotient(r, i.y, i.x);  // alpha is at most 1: no rank is infinite
        }
    }
    if (__any_sync(0xffffffffu, __double_as_longlong(d) != 0))
#pragma unroll
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int i = 0; i < TPB / 32; i++)
            if (__double_as_longlong(ws[i]) != 0) t += ws[i];
        if (t != 0.0) atomicAdd(next, t);
        if (blockIdx.x == 0) *after = 0.0;
    }
}

__global__ void __launch_bounds__(TPB) k_fill_f64(double *p, uint64_t n, double x) {
    for (uint64_t i = blockIdx.x * (uint64_t)TPB + threadIdx.x; i < n; i += gridDim.x * (uint64_t)TPB) p[i] = x;
}

inline uint32_t grid_for(uint64_t n, uint32_t per_block, uint32_t cap = 152 * 16) {
    const uint64_t b = (n + per_block - 1) / per_block;
    return (uint32_t)(b == 0 ? 1 : (b < cap ? b : cap));
}

}  // namespace

cudaError_t launch_nbr_count(const uint32_t *srcs, const uint64_t *windows, uint32_t n, Geo g, const uint8_t *cnt,
                             const uint32_t *sent, uint32_t V, const NbrScratch &q, uint32_t *offsets,
                             cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(q.done, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    if (n <= NBR_ONE_CTA) {
        ProfScope ps_("nbr_weigh", s);
        k_nbr_weigh_scan<<<1, 1024, 0, s>>>(srcs, n, g, sent, V, q.rounds);
        note_launch();
    } else {
        ProfScope ps_("nbr_weigh", s);
        k_nbr_weigh<<<grid_for(n, TPB, 152 * 8), TPB, 0, s>>>(srcs, n, g, sent, V, q.rounds);
        note_launch();
        if ((e = scan_u32(q.rounds, q.rounds, n, q.rounds + n, q.tmp, s)) != cudaSuccess) return e;
    }
    ProfScope ps_("nbr_count", s);
    k_nbr_count<<<NBR_CTAS, TPB, 0, s>>>(srcs, windows, n, g, cnt, sent, V, q.rounds, q.done, q.at, q.base, offsets);
    note_launch();
    if (n > NBR_ONE_CTA) {
        k_nbr_offsets<<<(n + TPB - 1) / TPB, TPB, 0, s>>>(n, q.at, q.base, offsets);
        note_launch();
    }
    return cudaGetLastError();
}

void launch_nbr_fill(const uint32_t *srcs, const uint64_t *windows, uint32_t n, Geo g, const uint8_t *cnt,
                     const uint32_t *sent, uint32_t V, const NbrScratch &q, uint32_t *nbrs, uint8_t *vals,
                     cudaStream_t s) {
    ProfScope ps_("nbr_fill", s);
    k_nbr_fill<<<NBR_CTAS, TPB, 0, s>>>(srcs, windows, n, g, cnt, sent, V, q.rounds, q.base, nbrs, vals);
    note_launch();
}

size_t nbr_base_words() { return NBR_SHARES; }

void launch_edge_query(const uint64_t *q, uint32_t n, uint32_t window, Geo g, const ulonglong2 *fl,
                       const uint32_t *sent, uint32_t V, uint32_t *res, cudaStream_t s) {
    ProfScope ps_("edge_query", s);
    k_edge_query<<<grid_for(n, TPB, 152 * 16), TPB, 0, s>>>(q, n, window, g, fl, sent, V, res);
    note_launch();
}

void launch_bfs_init(const uint32_t *sources, uint32_t n, uint32_t V, Geo g, const uint32_t *sent, int32_t *dist,
                     uint2 *items, uint32_t cap, uint32_t *n_items, uint32_t *n_found, cudaStream_t s) {
    ProfScope ps_("bfs_init", s);
    k_bfs_init<<<grid_for(V, TPB, 152 * 16), TPB, 0, s>>>(dist, V);
    k_bfs_seed<<<grid_for(n, TPB, 152 * 16), TPB, 0, s>>>(sources, n, V, g, sent, dist, items, cap, n_items, n_found);
    note_launch(2);
}

uint32_t bfs_items_for(uint32_t V, uint32_t H) { return (uint32_t)(V + (nseg_of(H) + V) / BFS_SEGS + 1); }

void launch_bfs_expand(const uint2 *items, const uint32_t *n_items, int32_t level, Geo g, const uint8_t *cnt,
                       const uint32_t *sent, int32_t *dist, uint2 *next, uint32_t cap, uint32_t *n_next,
                       uint32_t *n_found, cudaStream_t s) {
    ProfScope ps_("bfs_expand", s);
    // the list's length is known on the device only: a resident grid that
    // loops (8 CTAs a SM), smaller for a graph that cannot fill it
    k_bfs_expand<<<grid_for(cap, TPB / 8, 152 * 8), TPB, 0, s>>>(items, n_items, level, g, cnt, sent, dist, next, cap,
                                                                 n_next, n_found);
    note_launch();
}

void launch_outdeg(Geo g, const uint8_t *cnt, uint32_t *deg, cudaStream_t s) {
    ProfScope ps_("outdeg", s);
    k_outdeg<<<grid_for(nseg_of(g.H), TPB / 8, 152 * 16), TPB, 0, s>>>(g, cnt, deg);
    note_launch();
}

void launch_fill_f64(double *p, uint64_t n, double x, cudaStream_t s) {
    k_fill_f64<<<grid_for(n, TPB, 152 * 8), TPB, 0, s>>>(p, n, x);
    note_launch();
}

size_t pr_words(uint32_t V, uint64_t edges, PrLayout *l) {
    l->nbins = (V + PR_BIN - 1) >> PR_LOW;
    l->max_chunks = (uint32_t)(edges / PR_CHUNK) + l->nbins;
    l->cap = (uint32_t)(edges + 4ull * l->nbins);
    return 4ull * l->max_chunks + l->cap + l->nbins + 1;
}

cudaError_t launch_pr_layout(Geo g, const uint8_t *cnt, const uint32_t *P, const uint32_t *sent, uint32_t V,
                             const PrLayout &l, uint32_t *words, double2 *inv, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_pr_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((2 * PR_CHUNK + PR_BIN + 32) * 4));
    if (e != cudaSuccess) return e;
    uint4 *chunks = reinterpret_cast<uint4 *>(words);
    uint32_t *edges = words + 4ull * l.max_chunks, *bins = edges + l.cap, *n_chunks = bins + l.nbins;
    ProfScope ps_("pr_layout", s);
    if ((e = cudaMemsetAsync(bins, 0, 4ull * l.nbins, s)) != cudaSuccess) return e;
    const uint32_t tiles = (uint32_t)((nseg_of(g.H) + PR_TILE_SEGS - 1) / PR_TILE_SEGS);
    k_pr_count<<<tiles, TPB, 0, s>>>(g, cnt, l.nbins, bins);
    k_pr_table<<<1, 1024, 0, s>>>(l.nbins, bins, chunks, n_chunks);
    k_pr_place<<<tiles, TPB, 0, s>>>(g, cnt, l.nbins, bins, edges, l.cap);
    k_pr_sort<<<l.max_chunks, PR_SORT_TPB, (2 * PR_CHUNK + PR_BIN + 32) * 4, s>>>(chunks, n_chunks, edges);
    k_pr_deg<<<grid_for(V, TPB, 152 * 8), TPB, 0, s>>>(P, sent, g.H, V, inv);
    note_launch(5);
    return cudaGetLastError();
}

void launch_pr_pull(uint32_t it, const PrLayout &l, const uint32_t *words, uint32_t V, double alpha, const double2 *inv,
                    double *rank, double *contrib, double *acc, double *dangling,
                    cudaStream_t s) {
    ProfScope ps_("pagerank", s);
    const uint4 *chunks = reinterpret_cast<const uint4 *>(words);
    const uint32_t *edges = words + 4ull * l.max_chunks, *n_chunks = edges + l.cap + l.nbins;
    if (it) {
        k_pr_pull<<<l.max_chunks, PR_PULL_TPB, 0, s>>>(chunks, n_chunks, edges, contrib, acc, V);
        note_launch();
    }
    k_pr_step<<<grid_for(V, TPB, 152 * 8), TPB, 0, s>>>(it == 0, rank, acc, inv, V, alpha,
                                                        (1.0 - alpha) / (double)V, 1.0 / (double)V, dangling + it % 3, dangling + (it + 1) % 3,
                                                        dangling + (it + 2) % 3, contrib);
    note_launch();
}

void launch_pr_iteration(Geo g, const uint8_t *cnt, const uint32_t *deg, uint32_t V, double alpha, double *rank,
                         double *contrib, double *acc, double *dangling, cudaStream_t s) {
    ProfScope ps_("pagerank", s);
    k_zero_f64<<<1, 1, 0, s>>>(dangling);
    k_pr_contrib<<<grid_for(V, TPB, 152 * 8), TPB, 0, s>>>(rank, deg, V, contrib, dangling);
    k_pr_push<<<grid_for(nseg_of(g.H), TPB / 8, 152 * 16), TPB, 0, s>>>(g, cnt, contrib, acc);
    k_pr_finish<<<grid_for(V, TPB, 152 * 8), TPB, 0, s>>>(rank, acc, V, alpha, dangling);
    note_launch(4);
}

}  // namespace lpma
