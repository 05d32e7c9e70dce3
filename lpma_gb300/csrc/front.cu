// The partitioned update front: one pass puts the batch's keys into buckets
// that are subtrees of the segment tree, then one CTA a bucket locates its
// keys, orders them by segment, resolves them against the stored keys and
// executes the single-segment windows that pass, all from one read of each
// touched segment.  What is left (segments whose own window fails) becomes
// the update list that the planner goes on with.
//
// It replaces the pack, the batch sort, the locate, the compaction and the
// single-segment executor of the sorted front.  Why that is the same result:
// a window's merge size is live + inserts - deletes of its segments whatever
// ran below it, so a segment whose own window passes may be executed before
// the larger windows are planned, as the reference's level loop does
// (rpma.cuh:1611-1657): the counts then hold its items and the list no
// longer its updates.  A larger window or a rebuild that covers it spreads
// the same items.
//
// What bounds it: the partition, the scatter of 16-byte entries into L2; the
// buckets, instructions (95 a key; 59% of the issue slots, HBM at 24% of its
// rate): the segments are asked of L2 while the CTA orders its keys.  A batch of 1M keys into a scale-21 graph: partition 29 us, buckets
// 139, list 8, and the planner 20 on the 5% of the segments that remain;
// before, pack 17, sort 87, locate 46, compaction 18, planner 51, executor 89.
#include <algorithm>

#include "kernels.cuh"
#include "prims.cuh"

namespace lpma {
namespace {

constexpr int TPB = 256;
constexpr int PT = 512;                      // threads of a partition CTA
constexpr int BT = 256;                      // threads of a bucket's CTA
constexpr uint32_t NWARPS = BT / 32;
constexpr int BUCKET_CTAS = 1024 / BT;
constexpr uint32_t PART_GRID = 152;          // CTAs of the partition, about
constexpr uint32_t PART_WAVE = 7;            // 2^7 buckets: a CTA an SM at most
constexpr uint32_t PART_FEW = 32;            // keys a bucket from which there are more, up to 2^PART_WAVE,
constexpr uint32_t PART_AVG = 128;           // and up to 2^10
constexpr uint64_t PART_LARGE = 400000;      // keys of a batch from which there are 2^11

constexpr uint32_t CROWD = 64;               // keys of one counter from which the bucket is sorted by key
constexpr uint32_t PAY_DEL = 1u << 8, PAY_STOP = 1u << 9, PAY_IDX = 10;  // payload: value, delete, stop, input position
constexpr uint32_t PAY_RANK = 12;  // later: kind at PAY_IDX, and the slots below the key

// ------------------------------------------------------------------ partition
// Validates the batch and puts every key into its bucket.  The buckets are
// the 2^L subtrees at level L: the descent of the locate over the top L
// levels (staged in shared memory), where a key that stops at a top node a
// goes to the leftmost bucket of a's right subtree, so all updates of a
// segment meet in one bucket and a bucket holds a contiguous run of linear
// segments, [b W - 1, b W + W - 1) with W = 2^(H - L + 1).  A CTA counts its
// keys per bucket, takes its places in each bucket with one atomic and
// writes them; the order within a bucket is arbitrary (the bucket kernel
// orders by key and input position).  A bucket that would overflow marks the
// batch (part_ovf), and nothing of this front changes the structure.
__global__ void __launch_bounds__(PT) k_part(PartArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t NB = 1u << a.L, ntop = NB - 1;
    uint64_t *first = reinterpret_cast<uint64_t *>(smem), *last = first + NB;  // the top nodes' bounds
    uint32_t *hist = reinterpret_cast<uint32_t *>(last + NB);
    const uint32_t n = a.n_ins + a.n_del, tile = a.ipt * PT, i0 = blockIdx.x * tile + threadIdx.x;
    uint64_t key[PART_IPT];
    uint32_t pay[PART_IPT], bkt[PART_IPT], at[PART_IPT];
    bool hole = false;
    for (uint32_t t = threadIdx.x; t < ntop; t += PT) {
        const ulonglong2 f = a.fl[t];
        first[t] = f.x;
        last[t] = f.y;
        hole |= f.x == KEY_NONE;
    }
    for (uint32_t t = threadIdx.x; t < NB; t += PT) hist[t] = 0;
    hole = __syncthreads_or(hole);
    uint32_t mint = 0xFFFFFFFFu, bad = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t q = 0; q < PART_IPT; q++) {
        const uint32_t i = i0 + q * PT;
        bkt[q] = ~0u;
        if (q >= a.ipt || i >= n) continue;
        const bool is_del = i >= a.n_ins;
        uint64_t k = is_del ? a.del[i - a.n_ins] : a.ins[i];
        bool ok = true;
        if (a.key_format == 1) {  // src << 32 | dst
            const uint64_t s = k >> 32, d = k & 0xFFFFFFFFull;
            ok = s < a.V && d < a.V;
            k = (s << SRC_SHIFT) | (d << DST_SHIFT);
        }
        const uint64_t src = k >> SRC_SHIFT, dst = (k & DST_MASK) >> DST_SHIFT;
        ok = ok && k != KEY_NONE && src < a.V && dst < a.V;
        uint32_t p;
        if (!is_del) {
            p = a.ins_vals ? a.ins_vals[i] : 1u;
            ok = ok && p != VAL_TOMB && (k & TIME_MASK) >= (uint64_t)a.thres;
            mint = min(mint, (uint32_t)(k & TIME_MASK));
        } else {
            p = PAY_DEL;
        }
        if (!ok) bad = min(bad, i);
        uint32_t j = 0, lvl = 0, b;
        bool stop = false;
        if (!hole) {
            // one compare a level: the key stops at the last node it went
            // right of when it is not behind that node's last key (the nodes
            // it meets below are all behind)
            uint32_t pred = ~0u;
            for (; lvl < a.L; lvl++) {
                const bool right = k >= first[j];
                pred = right ? j : pred;
                j = 2 * j + 1 + (right ? 1u : 0u);
            }
            stop = pred != ~0u && k <= last[pred];
            b = j - (NB - 1);  // already the leftmost bucket right of pred
        } else {
            for (; lvl < a.L && !stop; lvl++) {
                const uint64_t f = first[j];
                if (k < f && f != KEY_NONE)
                    j = 2 * j + 1;
                else if (k > last[j])  // never of an empty node (its last is the largest key)
                    j = 2 * j + 2;
                else
                    stop = true;
            }
            b = j - (NB - 1);
            if (stop) {
                lvl--;  // the level it stopped at
                b = (2 * (j - ((1u << lvl) - 1)) + 1) << (a.L - lvl - 1);
            }
        }
        if (stop) p |= PAY_STOP;
        key[q] = k;
        pay[q] = p | (i << PAY_IDX);
        bkt[q] = b;
        at[q] = atomicAdd(&hist[b], 1u);
    }
    // one set of atomics per block: the status words are single addresses
    mint = __reduce_min_sync(0xffffffffu, mint);
    bad = __reduce_min_sync(0xffffffffu, bad);
    __shared__ uint32_t s_min[PT / 32], s_bad[PT / 32];
    if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5] = mint, s_bad[threadIdx.x >> 5] = bad;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < PT / 32; i++) mint = min(mint, s_min[i]), bad = min(bad, s_bad[i]);
        if (mint != 0xFFFFFFFFu) atomicMin(&a.st->min_t_ins, mint);
        if (bad != 0xFFFFFFFFu) {
            atomicOr(&a.st->error, ERR_KEY);
            atomicMin(&a.st->err_info[0], bad);
        }
    }
    for (uint32_t t = threadIdx.x; t < NB; t += PT) {
        const uint32_t c = hist[t];
        if (c) hist[t] = atomicAdd(&a.fill[t], c);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < PART_IPT; q++) {
        if (bkt[q] == ~0u) continue;
        const uint32_t pos = hist[bkt[q]] + at[q];
        if (pos < a.cap)
            a.ent[(uint64_t)bkt[q] * a.cap + pos] = make_ulonglong2(key[q], pay[q]);
        else
            a.st->part_ovf = 1;
    }
}

// ------------------------------------------------------------------ buckets
// 32-byte accesses (aligned): a lane moves 8 slots as two of them
__device__ __forceinline__ void ld32(const uint64_t *p, uint64_t *k) {
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(k[0]), "=l"(k[1]), "=l"(k[2]), "=l"(k[3])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st32(uint64_t *p, const uint64_t *k) {
    asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(k[0]), "l"(k[1]), "l"(k[2]), "l"(k[3])
                 : "memory");
}

// Shared memory of the bucket kernel for a capacity of cap entries: the
// fixed part, a region used in turn by the staged subtree (locate), the
// segment counters (ordering) and three arrays over the touched segments
// (from then on), and the entries' keys, payloads and index arrays.
struct BucketFixed {
    uint32_t wsum[BT / 32];
    uint32_t crowded;
    uint32_t stat[8];  // noops, upserts, windows, their inserts and deletes
};
__host__ __device__ inline uint32_t staged_levels(uint32_t h) { return h + 1 < 10 ? h + 1 : 10; }
__host__ __device__ inline uint32_t bin_shift(uint32_t h) { return h + 1 > 11 ? h - 10 : 0; }
__host__ __device__ inline uint32_t bucket_region(uint32_t cap, uint32_t h) {
    const uint32_t sub = 16u << staged_levels(h), bins = ((4u * (2u << h) >> bin_shift(h)) + 15u) & ~15u, segs = 8 * cap;
    const uint32_t x = sub > bins ? sub : bins;
    return x > segs ? x : segs;
}

// The slots of a segment held by 4 lanes, 8 each, in order: slot r and all
// above it move up (down) by one; inactive groups pass r >= 64.
__device__ __forceinline__ void seg_insert(uint64_t (&k)[8], uint64_t &v, int r, uint64_t key, uint64_t val, int gl) {
    const uint64_t up = __shfl_up_sync(0xffffffffu, k[7], 1, 4);
    const uint32_t upv = __shfl_up_sync(0xffffffffu, (uint32_t)(v >> 56), 1, 4);
    r -= 8 * gl;
#pragma unroll
    for (int q = 7; q >= 1; q--) k[q] = q > r ? k[q - 1] : k[q];
    if (r < 0) {
        k[0] = up;
        v = (v << 8) | upv;
    } else if (r < 8) {
#pragma unroll
        for (int q = 0; q < 8; q++) k[q] = q == r ? key : k[q];
        const uint64_t low = (1ull << (8 * r)) - 1;
        v = (v & low) | ((v & ~low) << 8) | (val << (8 * r));
    }
}
__device__ __forceinline__ void seg_erase(uint64_t (&k)[8], uint64_t &v, int r, int gl) {
    uint64_t dn = __shfl_down_sync(0xffffffffu, k[0], 1, 4);
    uint64_t dnv = __shfl_down_sync(0xffffffffu, (uint32_t)v & 0xFFu, 1, 4);
    if (gl == 3) dn = KEY_NONE, dnv = 0;
    r -= 8 * gl;
#pragma unroll
    for (int q = 0; q < 7; q++) k[q] = q >= r ? k[q + 1] : k[q];
    if (r < 8) {
        k[7] = dn;
        const uint64_t low = r > 0 ? (1ull << (8 * r)) - 1 : 0ull;
        v = (v & low) | ((v >> 8) & ~low) | (dnv << 56);
    }
}

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t *wsum, uint32_t &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) wsum[w] = v;
    __syncthreads();
    uint32_t off = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < BT / 32; k++) {
        const uint32_t y = wsum[k];
        off += k < w ? y : 0u;
        tot += y;
    }
    __syncthreads();
    total = tot;
    return off + v - x;
}

template <bool TH>
__global__ void __launch_bounds__(BT, BUCKET_CTAS) k_bucket(BucketArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t region = bucket_region(a.cap, a.g.H - a.L);
    uint64_t *K = reinterpret_cast<uint64_t *>(smem + region);
    uint32_t *P = reinterpret_cast<uint32_t *>(K + a.cap);
    uint16_t *lb = reinterpret_cast<uint16_t *>(P + a.cap);  // linear segment - (b W - 1)
    uint16_t *idx = lb + a.cap, *ord = idx + a.cap;
    BucketFixed &F = *reinterpret_cast<BucketFixed *>(ord + a.cap);
    uint32_t *bits = reinterpret_cast<uint32_t *>(&F + 1);  // executed segments, W / 32 words
    ulonglong2 *sub = reinterpret_cast<ulonglong2 *>(smem);
    uint32_t *bin = reinterpret_cast<uint32_t *>(smem);
    uint32_t *sc = reinterpret_cast<uint32_t *>(smem);  // per touched segment: new keys, deletes; then what becomes of it
    uint16_t *sseg = reinterpret_cast<uint16_t *>(sc + a.cap), *el = sseg + a.cap;
    const uint32_t b = blockIdx.x, W = 2u << (a.g.H - a.L);
    const int lane = threadIdx.x & 31;
    // Before the partition is done: the planner's bitmap of this call starts
    // clear, and the top levels of the bucket's subtree come in.  Node (level
    // l, position p) of bucket b's subtree is heap index
    // 2^(L+l) - 1 + (b << l) + p.
    const uint32_t h = a.g.H - a.L;  // its height
    const uint32_t sl = a.stage ? staged_levels(h) : 0;
    for (uint32_t i = b * BT + threadIdx.x; i < a.bitmap_words; i += gridDim.x * BT) a.bitmap[i] = 0;
    for (uint32_t t = threadIdx.x; t + 1 < (1u << sl); t += BT) {
        const uint32_t l = 31 - __clz(t + 1), p = t + 1 - (1u << l);
        sub[t] = a.fl[((1u << (a.L + l)) - 1) + (b << l) + p];
    }
    griddep_wait();
    // a rejected batch, or one whose buckets overflowed, changes nothing
    if (a.st->error | a.st->part_ovf) return;
    const uint32_t thres = TH ? a.st->thres : 0;
    const uint32_t c = min(a.fill[b], a.cap);
    for (uint32_t i = threadIdx.x; i < W / 32; i += BT) bits[i] = 0;
    if (threadIdx.x < 8) F.stat[threadIdx.x] = 0;
    if (threadIdx.x == 0) F.crowded = 0;
    if (c == 0) {
        for (uint32_t i = threadIdx.x; i < W / 32; i += BT) a.absbits[(uint64_t)b * (W / 32) + i] = 0;
        if (threadIdx.x == 0) a.pcnt[b] = 0, a.bwin[b] = 0;
        return;
    }
    const ulonglong2 *ent = a.ent + (uint64_t)b * a.cap;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c; i += BT) {
        const ulonglong2 e = ent[i];
        const uint64_t key = e.x;
        const uint32_t p = (uint32_t)e.y;
        uint32_t l = 0, pos = 0, seg = 0;
        if (!(p & PAY_STOP)) {
            while (l < h) {
                const ulonglong2 f =
                    l < sl ? sub[(1u << l) - 1 + pos] : a.fl[((1u << (a.L + l)) - 1) + (b << l) + pos];
                if (f.x == KEY_NONE) break;
                if (key < f.x)
                    pos = 2 * pos;
                else if (key > f.y)
                    pos = 2 * pos + 1;
                else
                    break;
                l++;
            }
            seg = (2 * pos + 1) << (h - l);
        }
        // DRAM -> L2 while the keys are put in order: the lines that hold keys
        const uint32_t sg = b * W - 1 + seg;
        const uint64_t j = heap_of_linear32(sg, a.g.H);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.g.keys + 32 * j));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.g.vals + 32 * j));
        if (a.cnt[sg] > 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.g.keys + 32 * j + 16));
        K[i] = key;
        P[i] = p & ~PAY_STOP;
        lb[i] = (uint16_t)seg;
    }
    // ---- order by (segment, key, input position): a counting sort over the
    // segments (or runs of 2^shift of them), then ranks within a counter
    const uint32_t shift = bin_shift(h), nbin = W >> shift;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nbin; i += BT) bin[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c; i += BT) atomicAdd(&bin[lb[i] >> shift], 1u);
    __syncthreads();
    {
        // nbin / BT counters a thread (nbin <= 2048)
        const uint32_t per = (nbin + BT - 1) / BT, i0 = per * threadIdx.x;
        uint32_t x[2048 / BT], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < 2048 / BT; q++) {
            x[q] = q < per && i0 + q < nbin ? bin[i0 + q] : 0u;
            if (x[q] > CROWD) F.crowded = 1;
            sum += x[q];
        }
        uint32_t tot, off = block_excl_scan(sum, F.wsum, tot);
#pragma unroll
        for (uint32_t q = 0; q < 2048 / BT; q++) {
            if (q < per && i0 + q < nbin) bin[i0 + q] = off;
            off += x[q];
        }
    }
    __syncthreads();
    const bool crowded = F.crowded != 0;
    if (!crowded) {
        for (uint32_t i = threadIdx.x; i < c; i += BT) idx[atomicAdd(&bin[lb[i] >> shift], 1u)] = (uint16_t)i;
    } else {
        // many keys of few segments: a bitonic sort by (key, input position)
        uint32_t m = 1;
        while (m < c) m <<= 1;
        for (uint32_t p = threadIdx.x; p < c; p += BT) ord[p] = (uint16_t)p;
        __syncthreads();
        // positions past c count as the largest key: only pairs inside c move
        for (uint32_t k = 2; k <= m; k <<= 1)
            for (uint32_t s = k >> 1; s; s >>= 1) {
                for (uint32_t t = threadIdx.x; t < m / 2; t += BT) {
                    // the first step of a merge mirrors, so every run ascends
                    const uint32_t lo = 2 * s * (t / s) + t % s;
                    const uint32_t hi = s == k >> 1 ? (lo | (k - 1)) - (lo & (k - 1)) : lo + s;
                    if (hi < c) {
                        const uint32_t x = ord[lo], y = ord[hi];
                        if (K[y] < K[x] || (K[y] == K[x] && (P[y] >> PAY_IDX) < (P[x] >> PAY_IDX))) {
                            ord[lo] = (uint16_t)y;
                            ord[hi] = (uint16_t)x;
                        }
                    }
                }
                __syncthreads();
            }
        for (uint32_t i = threadIdx.x; i < c; i += BT) {
            atomicAdd(&bin[lb[i] >> shift], 1u);
            idx[i] = ord[i];
        }
    }
    __syncthreads();
    // From here on every warp works alone on its share of the entries: an
    // eighth of them, cut where a counter's run starts (so no segment is
    // cut).  bin[x] is now the end of counter x's run.
    const uint32_t w = threadIdx.x >> 5, lt = lanemask_lt();
    auto run_start = [&](uint32_t p) -> uint32_t {
        if (p == 0 || p >= c) return p;
        const uint32_t x = lb[idx[p]] >> shift;
        return x ? bin[x - 1] : 0u;
    };
    const uint32_t S = run_start(c * w / NWARPS), E = run_start(c * (w + 1) / NWARPS);
    if (!crowded)  // rank within the runs; the array bin goes away after this
        for (uint32_t p = S + lane; p < E; p += 32) {
            const uint32_t i = idx[p], x = lb[i] >> shift;
            const uint32_t s = x ? bin[x - 1] : 0u, e = bin[x];
            uint32_t less = 0;
            const uint64_t key = K[i];
            const uint32_t pi = P[i] >> PAY_IDX;
            for (uint32_t q = s; q < e; q++) {
                const uint32_t o = idx[q];
                const uint64_t ko = K[o];
                less += (ko < key || (ko == key && (P[o] >> PAY_IDX) < pi)) ? 1u : 0u;
            }
            ord[s + less] = (uint16_t)i;
        }
    __syncthreads();
    // ---- the touched segments: segment t of the warp (t from S on) has its
    // entries from idx[t] on and is sseg[t]; an entry keeps its t in place of
    // lb, and learns whether it stands for its key (the last insert of a key
    // does, or, when it is not inserted, its first delete: delete first, last
    // value wins)
    uint32_t nseg = 0;
    {
        uint32_t before = ~0u;  // the segment of the entry before the chunk
        for (uint32_t p0 = S; p0 < E; p0 += 32) {
            const uint32_t p = p0 + lane;
            uint32_t i = 0, l = ~0u;
            if (p < E) {
                i = ord[p];
                l = lb[i];
                const uint64_t key = K[i];
                bool stands = true;
                if (P[i] & PAY_DEL) {
                    stands = p == S || K[ord[p - 1]] != key;
                } else if (p + 1 < E) {
                    const uint32_t o = ord[p + 1];
                    stands = K[o] != key || (P[o] & PAY_DEL);
                }
                if (stands) P[i] |= PAY_STOP;  // the bit's second use
            }
            uint32_t lp = __shfl_up_sync(0xffffffffu, l, 1);
            if (lane == 0) lp = before;
            const bool first = p < E && l != lp;
            const uint32_t fm = __ballot_sync(0xffffffffu, first);
            const uint32_t t = S + nseg + __popc(fm & lt) - (first ? 0u : 1u);
            if (first) {
                idx[t] = (uint16_t)p;
                sseg[t] = (uint16_t)l;
                sc[t] = 0;
            }
            if (p < E) lb[i] = (uint16_t)t;
            nseg += __popc(fm);
            before = __shfl_sync(0xffffffffu, l, 31);
        }
    }
    __syncwarp();
    const uint32_t TE = S + nseg;  // the warp's segments are [S, TE)
    // ---- membership, one thread an entry: upserts and tombstones in place
    uint32_t noop = 0, ups = 0, w_n = 0, w_ins = 0, w_del = 0;
    for (uint32_t p = S + lane; p < E; p += 32) {
        const uint32_t i = ord[p], pay = P[i];
        const uint64_t key = K[i];
        uint32_t kd = KIND_NOP, rank = 0;
        if (pay & PAY_STOP) {
            const uint32_t t = lb[i];
            const uint64_t slot0 = 32ull * heap_of_linear32(b * W - 1 + sseg[t], a.g.H);
            const uint64_t *sk = a.g.keys + slot0;
            // two probes choose a quarter (the slots are sorted, empty ones last)
            rank = sk[15] < key ? 16u : 0u;
            if (sk[rank + 7] < key) rank += 8;
            uint64_t q[8];
            ld32(sk + rank, q);
            ld32(sk + rank + 4, q + 4);
            bool found = false;
            uint32_t below = 0;
#pragma unroll
            for (int x = 0; x < 8; x++) {
                below += q[x] < key ? 1u : 0u;
                found |= q[x] == key;
            }
            rank += below;
            if (!(pay & PAY_DEL)) {
                if (found) {
                    a.g.vals[slot0 + rank] = (uint8_t)pay;  // upsert (handle_del_mod, gpma.cuh:162-175)
                    ups++;
                } else {
                    kd = KIND_INS;
                    atomicAdd(&sc[t], 1u);
                }
            } else if (found && (!TH || (key & TIME_MASK) >= (uint64_t)thres)) {
                a.g.vals[slot0 + rank] = VAL_TOMB;  // until a window executes
                kd = KIND_DEL;
                atomicAdd(&sc[t], 1u << 16);
            } else {
                noop++;
            }
        } else {
            noop++;
        }
        P[i] = (pay & 0x1FFu) | (kd << PAY_IDX) | (rank << PAY_RANK);
    }
    __syncwarp();
    // ---- one thread a touched segment: does its own window pass?  The ones
    // that do are listed by the number of their updates (1, 2, 3, 4, more),
    // so that the groups of a warp have the same work
    constexpr uint32_t NO_EXEC = 0xFFFFFFFFu;
    uint32_t cls[5] = {0, 0, 0, 0, 0};  // segments of each class, then where it goes on
    for (uint32_t t0 = S; t0 < TE; t0 += 32) {
        const uint32_t t = t0 + lane;
        uint32_t ops = 5;
        if (t < TE) {
            const uint32_t x = sc[t], ni = x & 0xFFFFu, nd = x >> 16, s = b * W - 1 + sseg[t];
            const uint32_t held = a.cnt[s], m = (TH ? a.cnt_live[s] : held) + ni - nd;
            if (x && m >= a.lower0 && m <= 32) {
                ops = min(ni + nd, 5u) - 1;
                sc[t] = m | (nd ? 0x100u : 0u) | (ops << 12) | (held << 16);
                atomicOr(&bits[sseg[t] >> 5], 1u << (sseg[t] & 31));
                w_n++;
                w_ins += ni;
                w_del += nd;
            } else {
                sc[t] = NO_EXEC;
            }
        }
#pragma unroll
        for (uint32_t q = 0; q < 5; q++) cls[q] += __popc(__ballot_sync(0xffffffffu, ops == q));
    }
    uint32_t nexec = 0;
#pragma unroll
    for (uint32_t q = 0; q < 5; q++) {
        const uint32_t n = cls[q];
        cls[q] = S + nexec;
        nexec += n;
    }
    __syncwarp();
    for (uint32_t t0 = S; t0 < TE; t0 += 32) {
        const uint32_t t = t0 + lane;
        const uint32_t x = t < TE ? sc[t] : NO_EXEC, ops = x == NO_EXEC ? 5u : (x >> 12) & 7u;
#pragma unroll
        for (uint32_t q = 0; q < 5; q++) {
            const uint32_t bal = __ballot_sync(0xffffffffu, ops == q);
            if (ops == q) el[cls[q] + __popc(bal & lt)] = (uint16_t)t;
            cls[q] += __popc(bal);
        }
    }
    __syncwarp();
    // ---- merge: one 4-lane group a segment, lane gl holds slots 8 gl .. 8 gl + 7
    const int gl = lane & 3;
    for (uint32_t x0 = 0; x0 < nexec; x0 += 8) {  // uniform over the warp
        const uint32_t x = x0 + (lane >> 2);
        const bool active = x < nexec;
        const uint32_t t = active ? el[S + x] : 0u;
        const uint32_t ea = active ? idx[t] : 0u, ee = active ? (t + 1 < TE ? idx[t + 1] : E) : 0u;
        const uint32_t info = active ? sc[t] : 0u, m = info & 0xFFu, held = info >> 16;
        const uint32_t s = b * W - 1 + (active ? sseg[t] : 1u);
        const uint64_t j = heap_of_linear32(s, a.g.H);
        uint64_t *const gk = a.g.keys + 32 * j + 8 * gl;
        uint8_t *const gv = a.g.vals + 32 * j + 8 * gl;
        uint64_t k[8];
        uint64_t v8 = 0;
        // the sectors that hold keys only (a segment is about 18 of 32 full)
#pragma unroll
        for (int q = 0; q < 8; q++) k[q] = KEY_NONE;
        if (8 * (uint32_t)gl < held) {
            ld32(gk, k);
            v8 = *reinterpret_cast<const volatile uint64_t *>(gv);
        }
        if (8 * (uint32_t)gl + 4 < held) ld32(gk + 4, k + 4);
        // slots that go: this batch's tombstones, and expired keys
        uint32_t dm = 0;
        if (__any_sync(0xffffffffu, TH || (info & 0x100u))) {
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const uint8_t v = (uint8_t)(v8 >> (8 * q));
                if (k[q] != KEY_NONE && !(TH ? kept_slot(k[q], v, thres) : v != VAL_TOMB)) dm |= 1u << q;
            }
            dm <<= 8 * gl;
            dm |= __shfl_xor_sync(0xffffffffu, dm, 1, 4);
            dm |= __shfl_xor_sync(0xffffffffu, dm, 2, 4);
            uint32_t left = dm;  // from the last one down, so that the positions below stay
            while (__any_sync(0xffffffffu, left)) {
                const int r = left ? 31 - __clz(left) : 64;
                if (left) left &= ~(1u << r);
                seg_erase(k, v8, r, gl);
            }
        }
        // new keys, the last one first
        int low = dm ? __ffs(dm) - 1 : 64;  // the first slot that changes
        bool end = held && ((dm >> (held - 1)) & 1u);  // the last key goes or a new one is behind it
        const int nk = (int)held - __popc(dm);
        const uint32_t rounds = __reduce_max_sync(0xffffffffu, ee - ea);
        for (uint32_t r = 0; r < rounds; r++) {
            int at = 64;
            uint64_t key = 0, val = 0;
            if (r < ee - ea) {
                const uint32_t i = ord[ee - 1 - r], pay = P[i];
                if (((pay >> PAY_IDX) & 3u) == KIND_INS) {
                    const uint32_t rank = pay >> PAY_RANK;
                    at = (int)(rank - __popc(dm & (rank >= 32 ? ~0u : (1u << rank) - 1)));
                    key = K[i];
                    val = pay & 0xFFu;
                    low = min(low, at);
                    end |= at == nk;
                }
            }
            seg_insert(k, v8, at, key, val, gl);
        }
        if (active) {
            const uint32_t hi = max(m, held);  // slots from here on were and are empty
            uint64_t last = KEY_NONE;
            const int lr = (int)m - 1 - 8 * gl;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (q == lr) last = k[q];
                if ((uint32_t)k[q] == (uint32_t)DST_AND_TIME_END && 8 * gl + q >= low && is_sentinel(k[q])) {
                    const uint32_t row = (uint32_t)(k[q] >> SRC_SHIFT);
                    if (row < a.V) a.sent[row] = (uint32_t)(32 * j + 8 * gl + q);
                }
            }
            if (8 * gl + 4 > low && 8 * (uint32_t)gl < hi) st32(gk, k);
            if (8 * gl + 8 > low && 8 * (uint32_t)gl + 4 < hi) st32(gk + 4, k + 4);
            if (8 * gl + 8 > low && 8 * (uint32_t)gl < hi) *reinterpret_cast<uint64_t *>(gv) = v8;
            uint64_t *fp = reinterpret_cast<uint64_t *>(a.fl + j);
            if (gl == 0) {
                if (m != held) a.cnt[s] = (uint8_t)m;
                if (TH) a.cnt_live[s] = (uint8_t)m;
                if (low == 0) fp[0] = k[0];
                if (m == 0) fp[1] = KEY_NONE;
            }
            if (end && lr >= 0 && lr < 8) fp[1] = last;
        }
    }
    noop = __reduce_add_sync(0xffffffffu, noop);
    ups = __reduce_add_sync(0xffffffffu, ups);
    w_n = __reduce_add_sync(0xffffffffu, w_n);
    w_ins = __reduce_add_sync(0xffffffffu, w_ins);
    w_del = __reduce_add_sync(0xffffffffu, w_del);
    if (lane == 0) {
        if (noop) atomicAdd(&F.stat[0], noop);
        if (ups) atomicAdd(&F.stat[1], ups);
        if (w_n) {
            atomicAdd(&F.stat[2], w_n);
            atomicAdd(&F.stat[3], w_ins);
            atomicAdd(&F.stat[4], w_del);
        }
    }
    // ---- what stays, in order, over the bucket's entries: counted by every
    // warp, then placed behind the warps before it
    ulonglong2 *out = a.ent + (uint64_t)b * a.cap;
    uint32_t mine = 0;  // updates, and inserts among them in the high half
    for (uint32_t p0 = S; p0 < E; p0 += 32) {
        const uint32_t p = p0 + lane;
        uint32_t kd = KIND_NOP;
        if (p < E) {
            const uint32_t i = ord[p];
            if (sc[lb[i]] == NO_EXEC) kd = (P[i] >> PAY_IDX) & 3u;
        }
        mine += __popc(__ballot_sync(0xffffffffu, kd != KIND_NOP)) |
                (__popc(__ballot_sync(0xffffffffu, kd == KIND_INS)) << 16);
    }
    if (lane == 0) F.wsum[w] = mine;
    __syncthreads();
    uint32_t base = 0, total = 0;
#pragma unroll
    for (uint32_t k = 0; k < NWARPS; k++) {
        const uint32_t x = F.wsum[k];
        base += k < w ? x & 0xFFFFu : 0u;
        total += x;
    }
    if (mine)
        for (uint32_t p0 = S; p0 < E; p0 += 32) {
            const uint32_t p = p0 + lane;
            uint32_t i = 0, t = 0, kd = KIND_NOP;
            if (p < E) {
                i = ord[p];
                t = lb[i];
                if (sc[t] == NO_EXEC) kd = (P[i] >> PAY_IDX) & 3u;
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, kd != KIND_NOP);
            if (kd != KIND_NOP)
                out[base + __popc(bal & lt)] =
                    make_ulonglong2(K[i], (uint64_t)(b * W - 1 + sseg[t]) | ((uint64_t)(P[i] & 0xFFu) << 32) | ((uint64_t)kd << 40));
            base += __popc(bal);
        }
    for (uint32_t i = threadIdx.x; i < W / 32; i += BT) a.absbits[(uint64_t)b * (W / 32) + i] = bits[i];
    if (threadIdx.x == 0) {
        a.pcnt[b] = total;
        a.bwin[b] = F.stat[2];
        if (F.stat[0]) atomicAdd(&a.st->n_noop, F.stat[0]);
        if (F.stat[1]) atomicAdd(&a.st->n_upsert, F.stat[1]);
        if (F.stat[2]) {
            atomicAdd(&a.st->abs_win, F.stat[2]);
            atomicAdd(&a.st->abs_ins, F.stat[3]);
            atomicAdd(&a.st->abs_del, F.stat[4]);
            // the stored and live keys that the planner's root test starts from
            const unsigned long long net = (unsigned long long)((long long)F.stat[3] - (long long)F.stat[4]);
            atomicAdd(&a.st->total_items, net);
            if (TH) atomicAdd(&a.st->live_total, net);
        }
    }
}

// ------------------------------------------------------------------ update list
// The buckets' remaining updates end to end (buckets are in segment order),
// a warp a bucket; clears the fill counts for the next call.
__global__ void __launch_bounds__(TPB) k_part_list(BucketArgs a, UpdList u, uint32_t NB) {
    __shared__ uint64_t ws[TPB / 32];
    __shared__ uint32_t own[TPB / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = blockIdx.x * (TPB / 32) + w;
    griddep_wait();
    if (lane == 0 && b < NB) a.fill[b] = 0;
    if (a.st->error | a.st->part_ovf) return;
    uint64_t acc = 0;  // entries in the low half, inserts in the high
    for (uint32_t t = threadIdx.x; t < blockIdx.x * (TPB / 32); t += TPB) {
        const uint32_t x = a.pcnt[t];
        acc += (uint64_t)(x & 0xFFFFu) | ((uint64_t)(x >> 16) << 32);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const uint32_t mine = b < NB ? a.pcnt[b] : 0u;
    if (lane == 0) ws[w] = acc, own[w] = mine;
    __syncthreads();
    uint32_t base = 0, ib = 0;
    for (uint32_t k = 0; k < TPB / 32; k++) {
        base += (uint32_t)ws[k] + (k < w ? own[k] & 0xFFFFu : 0u);
        ib += (uint32_t)(ws[k] >> 32) + (k < w ? own[k] >> 16 : 0u);
    }
    if (b >= NB) return;
    const ulonglong2 *ent = a.ent + (uint64_t)b * a.cap;
    const uint32_t c = mine & 0xFFFFu;
    for (uint32_t i0 = 0; i0 < c; i0 += 32) {
        const uint32_t i = i0 + lane;
        ulonglong2 e = make_ulonglong2(0, 0);
        if (i < c) e = ent[i];
        const uint32_t kd = (uint32_t)(e.y >> 40);
        const uint32_t ins = __ballot_sync(0xffffffffu, i < c && kd == KIND_INS);
        if (i < c) {
            const uint32_t x = base + i;
            u.key[x] = e.x;
            u.val[x] = (uint8_t)(e.y >> 32);
            u.kind[x] = (uint8_t)kd;
            u.seg[x] = (uint32_t)e.y;
            u.ip[x] = ib + __popc(ins & lanemask_lt());
        }
        ib += __popc(ins);
    }
    if (b == NB - 1 && lane == 0) {
        const uint32_t nu = base + c;
        a.st->n_u = nu;
        a.st->n_ins = ib;
        a.st->n_del = nu - ib;
        u.ip[nu] = ib;
    }
}

inline uint32_t bucket_smem(uint32_t cap, uint32_t H, uint32_t L) {
    return bucket_region(cap, H - L) + cap * (8 + 4 + 3 * 2) + (uint32_t)sizeof(BucketFixed) + (2u << (H - L)) / 8;
}
inline uint32_t part_smem(uint32_t L) { return (16u + 4u) << L; }

}  // namespace

const void *part_kernel_fn() { return reinterpret_cast<const void *>(&k_part); }

cudaError_t part_prepare() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_part, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)part_smem(PART_L_MAX))) ||
        (e = cudaFuncSetAttribute(k_bucket<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024)) ||
        (e = cudaFuncSetAttribute(k_bucket<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024)))
        return e;
    return cudaSuccess;
}

// When the partitioned front takes a batch of n keys, and with how many
// buckets of which capacity.
PartPlan part_plan(uint64_t n, uint32_t H) {
    PartPlan p{};
    if (n < PART_MIN || n > PART_MAX || H < 9) return p;
    // Buckets of 32 keys as long as every one has an SM to itself (against
    // 128 keys: calls of 1,000 to 5,000 keys 66-70 us instead of 71-83),
    // then of 128, and more once there are 1,024 (7 for every SM), until
    // their shared memory holds the CTAs back: a batch of 65K keys took 35 us
    // of bucket work with 64 keys a bucket, 29 with 128, 33 with 256; 200K
    // 61 / 48 with 98 / 195; 300K 60 / 53 with 146 / 293; 1M 196 / 139 with
    // 1,024 / 512.  A bucket's segments are whole words of the bitmap of
    // executed segments (H - L >= 4)
    uint32_t L = 0;
    while (L < PART_L_MAX - 1 && (n >> (L + 1)) >= (L < PART_WAVE ? PART_FEW : PART_AVG)) L++;
    if (n > PART_LARGE) L = PART_L_MAX;
    // (and at most 2^15 of them: 16-bit indexes, H - L <= 14)
    L = std::max(L, std::max(3u, H > 14 ? H - 14 : 0u));
    L = std::min(L, H - 4);
    const uint64_t avg = (n + (1u << L) - 1) >> L;
    // 3.5 times the average; where buckets are few their shared memory does
    // not matter, and a batch that aims at one place need not overflow
    const uint64_t least = L <= PART_WAVE ? std::min<uint64_t>(1024, (n + 63) / 64 * 64) : 256;
    const uint64_t cap = std::max(least, (avg * 7 / 2 + 63) / 64 * 64);
    if (cap > 4096) return p;  // a batch that is large against the tree
    p.L = L;
    p.cap = (uint32_t)cap;
    // a bucket of few keys stages its subtree only where that costs others
    // nothing: the descents of 32 keys through 14 levels in L2 took 7 us
    p.stage = L <= PART_WAVE || avg >= 64;
    p.ipt = (uint32_t)std::min<uint64_t>(PART_IPT, std::max<uint64_t>(1, n / (PT * PART_GRID)));
    return p;
}

void launch_part(const PartArgs &a, cudaStream_t s) {
    ProfScope ps_("part", s);
    const uint32_t tile = a.ipt * PT, n = a.n_ins + a.n_del;
    k_part<<<(n + tile - 1) / tile, PT, part_smem(a.L), s>>>(a);
    note_launch();
}

void launch_buckets(const BucketArgs &a, const UpdList &u, cudaStream_t s) {
    const uint32_t NB = 1u << a.L;
    {
        ProfScope ps_("bucket", s);
        launch_pdl(a.cnt_live ? k_bucket<true> : k_bucket<false>, dim3(NB), dim3(BT), bucket_smem(a.cap, a.g.H, a.L), s, a);
    }
    ProfScope ps_("part_list", s);
    launch_pdl(k_part_list, dim3((NB + TPB / 32 - 1) / (TPB / 32)), dim3(TPB), 0, s, a, u, NB);
    note_launch(2);
}

}  // namespace lpma
