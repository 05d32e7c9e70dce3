// CSR view / export kernels and the synthetic workload generator.
#include "kernels.cuh"
#include "prims.cuh"

namespace lpma {
namespace {

constexpr int TPB = 256;

// to_csr_rpma (rpma.cuh:2249-2295): the present keys in linear order,
// compacted.  Tiles of 128 consecutive segments: k_csr_tiles sums each
// tile's counts, its last CTA turns the sums into starts, and one CTA of
// k_csr_fill a tile places the columns and values in shared memory and
// writes them out whole, 16 and 4 bytes a thread.
//
// Bound by HBM (9 bytes a slot read, 5 an item written).  One warp per
// segment and one slot a lane kept too few bytes in flight and wrote 4-byte
// words at odd places: 138 us for 18.9M items in 33.5M slots, and 16 for
// the three kernels of its prefix; now 78 and 14.  5 CTAs a SM: 4 measured
// 82 us, 6 (spills) 101.
constexpr uint32_t CT = 128;                // segments a tile
constexpr uint32_t CT_SLOTS = 32 * CT;
constexpr int CT_TPB = 1024;  // 128 tiles a CTA, so that the last one scans 8,192 starts in one round

__global__ void __launch_bounds__(CT_TPB) k_csr_tiles(const uint8_t *__restrict__ cnt, uint64_t nseg, uint32_t ntiles,
                                                   uint32_t *tiles, uint32_t *row_offset, uint32_t *done) {
    // 8 threads a tile, 16 counts each (the count array is padded past nseg)
    const uint32_t t = (blockIdx.x * CT_TPB + threadIdx.x) >> 3;
    const uint64_t s0 = (uint64_t)t * CT + 16 * (threadIdx.x & 7);
    uint32_t c = 0;
    if (s0 + 16 <= nseg) {
        const uint4 v = *reinterpret_cast<const uint4 *>(cnt + s0);
        c = __dp4a(v.x, 0x01010101u, c);
        c = __dp4a(v.y, 0x01010101u, c);
        c = __dp4a(v.z, 0x01010101u, c);
        c = __dp4a(v.w, 0x01010101u, c);
    } else {
        for (uint64_t s = s0; s < nseg; s++) c += cnt[s];
    }
    c += __shfl_xor_sync(0xffffffffu, c, 1, 8);
    c += __shfl_xor_sync(0xffffffffu, c, 2, 8);
    c += __shfl_xor_sync(0xffffffffu, c, 4, 8);
    if ((threadIdx.x & 7) == 0 && t < ntiles) tiles[t] = c;
    // the last CTA to finish: exclusive starts, 8 tiles a thread and round
    __shared__ uint32_t last, ws[CT_TPB / 32];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1 ? 1u : 0u;  // back to 0 for the next call
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < ntiles; b0 += 8 * CT_TPB) {
        const uint32_t i0 = b0 + 8 * threadIdx.x;
        uint32_t x[8], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) sum += x[q] = i0 + q < ntiles ? __ldcg(tiles + i0 + q) : 0u;
        uint32_t v = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) ws[w] = v;
        __syncthreads();
        uint32_t off = carry + v - sum;
#pragma unroll
        for (int k = 0; k < CT_TPB / 32; k++) {
            const uint32_t y = ws[k];
            off += k < w ? y : 0u;
            carry += y;
        }
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) {
            if (i0 + q < ntiles) tiles[i0 + q] = off;
            off += x[q];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        tiles[ntiles] = carry;
        if (row_offset) row_offset[0] = 0;  // the sentinels write the others
    }
}

__global__ void __launch_bounds__(TPB, 5) k_csr_fill(Geo g, const uint8_t *__restrict__ cnt,
                                                  const uint32_t *__restrict__ tiles, uint32_t *row_offset,
                                                  uint32_t *col_index, uint8_t *values, uint64_t *ek, uint8_t *ev) {
    __shared__ __align__(16) uint32_t col[CT_SLOTS + 4];
    __shared__ __align__(16) uint8_t val[CT_SLOTS + 4];
    __shared__ uint32_t off[CT], ws[CT / 32];
    const uint32_t base = tiles[blockIdx.x], tot = tiles[blockIdx.x + 1] - base;
    if (!tot) return;
    const uint64_t nseg = nseg_of(g.H), t0 = (uint64_t)blockIdx.x * CT;
    const int lane = threadIdx.x & 31, gl = lane & 7, grp = threadIdx.x >> 3;
    // the lane's slots of four segments load together
    uint64_t k[4][4];
    uint32_t v4[4], c[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint64_t s = t0 + 32 * r + grp;
        c[r] = s < nseg ? cnt[s] : 0u;
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
        if (4 * (uint32_t)gl < c[r]) {
            const uint64_t j = heap_of_linear32((uint32_t)(t0 + 32 * r + grp), g.H);
            const ulonglong2 *kp = reinterpret_cast<const ulonglong2 *>(g.keys + 32 * j + 4 * gl);
            const ulonglong2 a = kp[0], b = kp[1];
            k[r][0] = a.x, k[r][1] = a.y, k[r][2] = b.x, k[r][3] = b.y;
            v4[r] = *reinterpret_cast<const uint32_t *>(g.vals + 32 * j + 4 * gl);
        }
    // where each segment's items start in the tile
    uint32_t x = 0, v = 0;
    if (threadIdx.x < CT) {
        v = x = t0 + threadIdx.x < nseg ? cnt[t0 + threadIdx.x] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) ws[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < CT) {
        for (uint32_t q = 0; q < threadIdx.x >> 5; q++) v += ws[q];
        off[threadIdx.x] = v - x;
    }
    __syncthreads();
    const uint32_t sh = base & 3;  // shared position + base - sh = global position
#pragma unroll
    for (int r = 0; r < 4; r++) {
        if (4 * (uint32_t)gl >= c[r]) continue;
        const uint32_t p0 = off[32 * r + grp] + 4 * gl;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (4 * (uint32_t)gl + q >= c[r]) break;
            const uint64_t key = k[r][q];
            const uint32_t pos = p0 + q, src = (uint32_t)(key >> SRC_SHIFT);
            const uint32_t dst = (uint32_t)((key & DST_MASK) >> DST_SHIFT);
            const bool end = dst == NBR_END;
            const uint8_t vq = (uint8_t)(v4[r] >> (8 * q));
            if (col_index) {
                col[sh + pos] = end ? src : dst;
                val[sh + pos] = end ? VAL_TOMB : vq;
                if (end) row_offset[src + 1] = base + pos + 1;
            }
            if (ek) {
                ek[base + pos] = key;
                ev[base + pos] = vq;
            }
        }
    }
    if (!col_index) return;
    __syncthreads();
    // shared words [sh, sh + tot): whole vectors, the ends by element
    const uint32_t e = sh + tot, v0 = (sh + 3) / 4, v1 = e / 4, at = base - sh;
    for (uint32_t i = v0 + threadIdx.x; i < v1; i += TPB) {
        reinterpret_cast<uint4 *>(col_index + at)[i] = reinterpret_cast<const uint4 *>(col)[i];
        reinterpret_cast<uint32_t *>(values + at)[i] = reinterpret_cast<const uint32_t *>(val)[i];
    }
    const uint32_t head = min(4 * v0, e), tail = max(4 * v1, head);
    if (threadIdx.x < 8) {
        const uint32_t i = threadIdx.x < 4 ? sh + threadIdx.x : tail + threadIdx.x - 4;
        if (i < (threadIdx.x < 4 ? head : e)) {
            col_index[at + i] = col[i];
            values[at + i] = val[i];
        }
    }
}

__device__ inline uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// R-MAT: per edge and bit level one 64-bit hash, high 32 bits against the
// quadrant thresholds; self loops become ~0 (dropped by the dedup).
__global__ void __launch_bounds__(TPB) k_rmat(uint64_t s0, uint32_t scale, uint64_t n, uint32_t ta, uint32_t tab,
                                              uint32_t tabc, uint64_t *out) {
    for (uint64_t e = blockIdx.x * (uint64_t)TPB + threadIdx.x; e < n; e += gridDim.x * (uint64_t)TPB) {
        uint64_t src = 0, dst = 0;
        for (uint32_t b = 0; b < scale; b++) {
            const uint32_t r = (uint32_t)(mix64(s0 ^ ((e << 6) | b)) >> 32);
            const uint64_t sb = r >= tab, db = (r >= ta && r < tab) || r >= tabc;
            src = (src << 1) | sb;
            dst = (dst << 1) | db;
        }
        out[e] = src == dst ? KEY_NONE : (src << SRC_SHIFT) | (dst << DST_SHIFT);
    }
}

__global__ void __launch_bounds__(TPB) k_hash_keys(uint64_t seed, const uint64_t *keys, uint64_t *hash, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)TPB + threadIdx.x; i < n; i += gridDim.x * (uint64_t)TPB)
        hash[i] = mix64(seed ^ keys[i]);
}

__global__ void __launch_bounds__(TPB) k_unique_flags(const uint64_t *keys, uint64_t n, uint32_t *flags) {
    for (uint64_t i = blockIdx.x * (uint64_t)TPB + threadIdx.x; i < n; i += gridDim.x * (uint64_t)TPB)
        flags[i] = keys[i] != KEY_NONE && (i == 0 || keys[i - 1] != keys[i]);
}

__global__ void __launch_bounds__(TPB) k_scatter_flags(const uint64_t *keys, const uint32_t *pos,
                                                       const uint32_t *flags, uint64_t n, uint64_t *out) {
    for (uint64_t i = blockIdx.x * (uint64_t)TPB + threadIdx.x; i < n; i += gridDim.x * (uint64_t)TPB)
        if (flags[i]) out[pos[i]] = keys[i];
}

__global__ void __launch_bounds__(TPB) k_sentinels(uint32_t V, uint64_t *keys, uint8_t *vals) {
    for (uint64_t v = blockIdx.x * (uint64_t)TPB + threadIdx.x; v < V; v += gridDim.x * (uint64_t)TPB) {
        keys[v] = (v << SRC_SHIFT) + DST_AND_TIME_END;  // col_idx_none, rpma.cuh:1797-1805
        vals[v] = 0;                                     // rpma.cuh:1814
    }
}

inline uint32_t grid_for(uint64_t n, uint32_t per_block, uint32_t cap = 152 * 16) {
    uint64_t g = (n + per_block - 1) / per_block;
    if (g == 0) g = 1;
    return (uint32_t)(g < cap ? g : cap);
}

}  // namespace

void launch_csr_fill(Geo g, const uint8_t *cnt, uint32_t *tiles, uint32_t *done, uint32_t *row_offset,
                     uint32_t *col_index, uint8_t *values, uint64_t *export_keys, uint8_t *export_vals,
                     cudaStream_t s) {
    const uint64_t nseg = nseg_of(g.H);
    const uint32_t ntiles = (uint32_t)((nseg + CT - 1) / CT);
    {
        ProfScope ps_("csr_tiles", s);
        k_csr_tiles<<<(ntiles + CT_TPB / 8 - 1) / (CT_TPB / 8), CT_TPB, 0, s>>>(cnt, nseg, ntiles, tiles, row_offset, done);
    }
    ProfScope ps_("csr_fill", s);
    k_csr_fill<<<ntiles, TPB, 0, s>>>(g, cnt, tiles, row_offset, col_index, values, export_keys, export_vals);
    note_launch(2);
}

void launch_sentinels(uint32_t V, uint64_t *keys, uint8_t *vals, cudaStream_t s) {
    ProfScope ps_("sentinels", s);
    k_sentinels<<<grid_for(V, TPB), TPB, 0, s>>>(V, keys, vals);
    note_launch();
}

void launch_rmat(uint64_t seed, uint32_t scale, uint64_t n, uint32_t ta, uint32_t tab, uint32_t tabc, uint64_t *out,
                 cudaStream_t s) {
    ProfScope ps_("gen_rmat", s);
    uint64_t s0 = seed;
    // same seeding as the CPU generator: s0 = mix64(seed)
    s0 += 0x9E3779B97F4A7C15ull;
    s0 = (s0 ^ (s0 >> 30)) * 0xBF58476D1CE4E5B9ull;
    s0 = (s0 ^ (s0 >> 27)) * 0x94D049BB133111EBull;
    s0 = s0 ^ (s0 >> 31);
    k_rmat<<<grid_for(n, TPB), TPB, 0, s>>>(s0, scale, n, ta, tab, tabc, out);
    note_launch();
}

void launch_hash_keys(uint64_t seed, const uint64_t *keys, uint64_t *hash, uint64_t n, cudaStream_t s) {
    ProfScope ps_("hash_keys", s);
    k_hash_keys<<<grid_for(n, TPB), TPB, 0, s>>>(seed, keys, hash, n);
    note_launch();
}

void launch_unique_flags(const uint64_t *keys, uint64_t n, uint32_t *flags, cudaStream_t s) {
    ProfScope ps_("unique_flags", s);
    k_unique_flags<<<grid_for(n, TPB), TPB, 0, s>>>(keys, n, flags);
    note_launch();
}

void launch_scatter_flags(const uint64_t *keys, const uint32_t *pos, const uint32_t *flags, uint64_t n, uint64_t *out,
                          cudaStream_t s) {
    ProfScope ps_("scatter_flags", s);
    k_scatter_flags<<<grid_for(n, TPB), TPB, 0, s>>>(keys, pos, flags, n, out);
    note_launch();
}

}  // namespace lpma
