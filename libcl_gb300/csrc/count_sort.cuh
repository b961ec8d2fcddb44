// count_sort.cuh -- the fused step's stable sort of particles by cell, as a counting sort over the
// cells: count (an atomic per particle, which also gives the particle a place among its cell's),
// sums of tiles of cells, scan (a CTA per tile adds up the tiles before it; it also writes the
// cell table), scatter of the particle ids, and a last pass that puts every cell's ids into
// ascending order, gathers the sorted state and sets the counts back to zero. The order inside a
// cell that the atomics leave is of no account, so the result is the stable sort's, and
// deterministic.
//
// Against the radix sort of the keys (three passes at 4M cells) it reads the keys once instead of
// once a pass, needs no histogram and no bounds pass, and the cell table comes with the scan. Its
// cost grows with the cells, though, and the last pass compares each cell's ids with one another,
// which is less than the density pass does with the same cells. count_sort_fits() draws the line.
#pragma once

#include "fluid3d_kernels.cuh"
#include "onesweep.cuh"

namespace gbsph {

// Cells per scan tile: a thread takes 4 (one 16-byte word of counts), or 16 of large tables.
constexpr uint32_t SCAN_THREADS = 256, SCAN_ALIGN = SCAN_THREADS * 16;
inline uint32_t scan_items(uint32_t cells) { return cells <= (1u << 20) ? 4u : 16u; }
inline uint32_t scan_tiles(uint32_t cells) {
    const uint32_t tile = SCAN_THREADS * scan_items(cells);
    return (cells + tile - 1) / tile;
}
// Words of the count table (whole tiles, so that the scan may read and clear 16 bytes at a time).
inline size_t count_words(uint32_t cells) { return ((size_t)cells + SCAN_ALIGN - 1) / SCAN_ALIGN * SCAN_ALIGN; }

// Tables up to this size need no tile sums: a tile's CTA adds up the counts themselves, 60 KB at
// most (10,000 cells: 3 us; 65,536 cells took 9.8 us, with tile sums 2.9 and 3.6).
constexpr uint32_t SCAN_DIRECT = 1u << 14;

// Whether the counting sort serves n particles in `cells` cells. Reading the counts costs 4 bytes
// per cell, about 1.3 us per million, a radix pass 20 us per million particles; so up to 32
// cells per particle the scan stays below one pass (1,048,576 particles in 4M cells: 50 us for
// the whole sort with the table, 100 us by three radix passes; in no spatial order 67 and 110;
// 17.3M particles of 256 scenes in 14M cells: 0.49 against 0.84 ms; 16,384 in 10,000: 16 against
// 33 us). Tables of up to 2^18 cells (the hash's) are a few us at any particle count (256
// particles: 17 against 30 us); 2^25 cells bound the tile sums a CTA reads.
inline bool count_sort_fits(uint32_t cells, uint32_t n) {
    return cells <= (1u << 18) || (cells / 32u <= n && cells <= (1u << 25));
}

// Bytes of the sort scratch that serve either sort of n particles (the tile sums take a word per
// 1,024 or 4,096 cells, at most n / 8 bytes by count_sort_fits()'s second rule, where the radix
// sort's look-back words take 4 n).
inline size_t sort_scratch_bytes(uint32_t n) {
    const size_t small = SORT_HEADER_BYTES + (size_t)scan_tiles(1u << 18) * 4, radix = onesweep_scratch_bytes(n, SORT_MAX_PASSES);
    return radix > small ? radix : small;
}

// Key and place of every particle, ITEMS per thread (their loads and atomics in flight together);
// with CLEAR the table entries of the previous step's occupied cells are reset (its sorted keys
// are still in `prev_keys`). `count` is all zero before. (Adding up the tiles here as well, with
// an atomic per warp and tile, took 280 us for 1M hashed keys, 24 us more than k_tile_sums for
// particles in no spatial order.)
template <bool CLEAR, bool BATCH, int ITEMS>
__global__ void __launch_bounds__(256) k_count(const float4* __restrict__ pos, KParams kp, uint32_t* __restrict__ keys,
                                               uint32_t* __restrict__ places, uint32_t* __restrict__ count,
                                               const uint32_t* __restrict__ prev_keys, uint2* __restrict__ table,
                                               uint32_t* __restrict__ counters) {
    if (blockIdx.x == 0 && threadIdx.x < 4) counters[threadIdx.x] = 0u;  // of the bricks, for the kernels to come
    const uint32_t i0 = blockIdx.x * (256u * ITEMS) + threadIdx.x;
    uint32_t k[ITEMS], pk[ITEMS], before[ITEMS];
    float4 p[ITEMS];
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t i = i0 + q * 256u;
        if (i >= kp.n) continue;
        p[q] = pos[i];
        if (CLEAR) {
            pk[q] = prev_keys[i];
            before[q] = i ? prev_keys[i - 1] : EMPTY;
        }
    }
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t i = i0 + q * 256u;
        if (i >= kp.n) continue;
        k[q] = BATCH ? batch_key(kp, i, p[q]) : particle_key(kp, p[q]);
        keys[i] = k[q];
        if (CLEAR && (i == 0 || before[q] != pk[q]) && pk[q] < kp.table_cells) table[pk[q]] = make_uint2(EMPTY, EMPTY);
    }
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t i = i0 + q * 256u;
        if (i < kp.n) places[i] = atomicAdd(count + k[q], 1u);
    }
}

// The tiles' sums from the counts, a CTA per tile.
template <uint32_t ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_sums(const uint32_t* __restrict__ count, uint32_t* __restrict__ tile_sum) {
    __shared__ uint32_t s_tmp[SORT_WARPS];
    const uint4* w = reinterpret_cast<const uint4*>(count) + (size_t)blockIdx.x * (SCAN_THREADS * ITEMS / 4) + threadIdx.x;
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < ITEMS / 4; ++q) {
        const uint4 x = w[q * SCAN_THREADS];
        sum += x.x + x.y + x.z + x.w;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31u) == 0) s_tmp[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
#pragma unroll
        for (int k = 0; k < SORT_WARPS; ++k) all += s_tmp[k];
        tile_sum[blockIdx.x] = all;
    }
}

// Exclusive scan of the counts: the occupied cells' table entries (FULL: every cell's, EMPTY where
// there is nothing). A CTA per tile adds up the sums of the tiles before its own (at most 8,192
// words, as a rule 4 or 17 KB, out of L2), or with DIRECT the counts before it, and waits for
// nobody; tiles without particles are not read again. 4M cells with 131,072 occupied: 6 us, 18 us
// with a decoupled look-back over all tiles.
template <uint32_t ITEMS, bool FULL, bool DIRECT>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_cells(const uint32_t* __restrict__ count, uint2* __restrict__ table,
                                                             const uint32_t* __restrict__ tile_sum) {
    __shared__ uint32_t s_tmp[SORT_WARPS];
    const uint32_t tile = blockIdx.x, c0 = (tile * SCAN_THREADS + threadIdx.x) * ITEMS;
    uint32_t v[ITEMS], at = 0;
    if (DIRECT || tile_sum[tile]) {
        uint32_t sum = 0, before = 0;
        const uint4* w = reinterpret_cast<const uint4*>(count);
#pragma unroll
        for (uint32_t q = 0; q < ITEMS / 4; ++q) {
            const uint4 x = w[c0 / 4 + q];
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
            sum += x.x + x.y + x.z + x.w;
        }
        if (DIRECT) {
#pragma unroll 4
            for (uint32_t t = threadIdx.x; t < tile * (SCAN_THREADS * ITEMS / 4); t += SCAN_THREADS) {
                const uint4 x = w[t];
                before += x.x + x.y + x.z + x.w;
            }
        } else {
#pragma unroll 4
            for (uint32_t t = threadIdx.x; t < tile; t += SCAN_THREADS) before += tile_sum[t];
        }
        before = __reduce_add_sync(0xffffffffu, before);
        if ((threadIdx.x & 31u) == 0) s_tmp[threadIdx.x >> 5] = before;
        __syncthreads();
        before = 0;
#pragma unroll
        for (int k = 0; k < SORT_WARPS; ++k) before += s_tmp[k];
        __syncthreads();
        at = before + block_exclusive_scan(sum, s_tmp);
    } else {
        if (!FULL) return;
#pragma unroll
        for (uint32_t q = 0; q < ITEMS; ++q) v[q] = 0;
    }
    if (FULL) {
#pragma unroll
        for (uint32_t q = 0; q < ITEMS; q += 2) {  // the table is a whole number of tiles long
            uint4 e;
            e.x = v[q] ? at : EMPTY;
            e.y = v[q] ? at + v[q] : EMPTY;
            at += v[q];
            e.z = v[q + 1] ? at : EMPTY;
            e.w = v[q + 1] ? at + v[q + 1] : EMPTY;
            at += v[q + 1];
            reinterpret_cast<uint4*>(table + c0)[q / 2] = e;
        }
    } else {
#pragma unroll
        for (uint32_t q = 0; q < ITEMS; ++q) {
            if (v[q]) table[c0 + q] = make_uint2(at, at + v[q]);
            at += v[q];
        }
    }
}

// Key and id of every particle to its cell's slots.
static __global__ void __launch_bounds__(256) k_scatter_ids(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ places,
                                                            const uint2* __restrict__ table, uint2* __restrict__ slots,
                                                            uint32_t n, uint32_t* err) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = keys[i], s = table[k].x + places[i];
    if (s >= n) {  // a table that does not fit the keys: never write out of range
        atomicOr(err, DEV_ERR_KEY_RANGE);
        return;
    }
    slots[s] = make_uint2(k, i);
}

// Sorted keys, permutation and state: a slot's particle goes behind those of its cell with smaller
// ids. With BRICKS the ids of the occupied bricks are appended to `bricks`.
template <bool BRICKS, bool VEL, class BrickOf>
__device__ __forceinline__ void order_cells(const uint2* __restrict__ slots, const uint2* __restrict__ table,
                                            const float4* __restrict__ pos, const float4* __restrict__ vel,
                                            uint32_t* __restrict__ keys, uint32_t* __restrict__ index,
                                            float4* __restrict__ spos, float4* __restrict__ svel,
                                            uint32_t* __restrict__ bricks, uint32_t* __restrict__ n_bricks,
                                            uint32_t* __restrict__ count, uint32_t n, uint32_t table_cells, uint32_t* err,
                                            BrickOf brick_of) {
    __shared__ uint32_t s_cnt, s_base;
    if (BRICKS) {
        if (threadIdx.x == 0) s_cnt = 0;
        __syncthreads();
    }
    const uint32_t s = blockIdx.x * 256u + threadIdx.x;
    uint32_t rank = EMPTY, bid = 0;
    if (s < n) {
        const uint2 me = slots[s];
        const uint2 cell = me.x < table_cells ? table[me.x] : make_uint2(0u, 0u);
        if (cell.y > n || s < cell.x || s >= cell.y) {  // as above
            atomicOr(err, DEV_ERR_KEY_RANGE);
        } else {
            const float4 p = pos[me.y];
            float4 v;
            if (VEL) v = vel[me.y];
            uint32_t d = cell.x;
#pragma unroll 4
            for (uint32_t t = cell.x; t < cell.y; ++t) d += slots[t].y < me.y ? 1u : 0u;
            keys[s] = me.x;
            index[d] = me.y;
            spos[d] = p;
            if (VEL) svel[d] = v;
            if (s == cell.x) count[me.x] = 0u;
            if (BRICKS) {
                bid = brick_of(me.x);
                if (s == 0 || bid != brick_of(slots[s - 1].x)) rank = atomicAdd(&s_cnt, 1u);
            }
        }
    }
    if (BRICKS) {
        __syncthreads();
        if (threadIdx.x == 0 && s_cnt) s_base = atomicAdd(n_bricks, s_cnt);
        __syncthreads();
        if (rank != EMPTY) bricks[s_base + rank] = bid;
    }
}

template <bool BRICKS, bool VEL, bool BATCH>
__global__ void __launch_bounds__(256) k_order_cells(const uint2* __restrict__ slots, const uint2* __restrict__ table,
                                                     const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ index,
                                                     float4* __restrict__ spos, float4* __restrict__ svel,
                                                     uint32_t* __restrict__ bricks, uint32_t* __restrict__ n_bricks,
                                                     uint32_t* __restrict__ count, KParams kp, uint32_t* err) {
    const uint32_t nx = (uint32_t)kp.nx, bw = (uint32_t)kp.bw, bxn = (uint32_t)kp.bxn;
    order_cells<BRICKS, VEL>(slots, table, pos, vel, keys, index, spos, svel, bricks, n_bricks, count, kp.n, kp.table_cells, err,
                             [&](uint32_t k) { return BATCH ? batch_brick_of(kp, k) : (k % nx) / bw + bxn * (k / nx); });
}

struct CountSort {
    const float4 *pos, *vel;  // vel may be null: the velocities are gathered elsewhere
    float4 *spos, *svel;
    uint32_t *keys_in, *places;      // per particle
    uint2* slots;                     // per particle
    uint32_t *keys, *index, *bricks;  // sorted keys (the previous step's on entry), permutation, occupied bricks
    uint32_t* count;                  // count_words(cells) zeros
    uint2* table;
    void* scratch;                    // the radix sort's: caller counters; tile sums in place of look-back words
    uint32_t* err;
    bool clear;                       // reset the previous step's table entries
    bool full;  // hashed keys (REF_BUCKETS cells): write every entry of the table, list no bricks
};

// Enqueues the sort. LINEAR_GRID (full = false): `table` is empty but for the runs of `keys` if
// `clear`, and the brick counters are set to zero before the bricks are counted.
template <bool BATCH>
inline cudaError_t count_sort(const CountSort& a, const KParams& kp, cudaStream_t s) {
    const uint32_t tiles = scan_tiles(kp.table_cells);
    uint32_t* counters = (uint32_t*)((char*)a.scratch + SORT_USER_COUNTER_OFFSET);
    uint32_t* sums = (uint32_t*)((char*)a.scratch + SORT_HEADER_BYTES);
    const unsigned g = (kp.n + 255u) / 256u;
    auto count = [&](auto kern, int items) {
        kern<<<(kp.n + 256u * items - 1) / (256u * items), 256, 0, s>>>(a.pos, kp, a.keys_in, a.places, a.count, a.keys, a.table,
                                                                      counters);
    };
    // four particles per thread once there are enough for two CTAs' worth of them on every SM
    if (kp.n >= (1u << 19)) {
        if (a.clear) count(k_count<true, BATCH, 4>, 4);
        else count(k_count<false, BATCH, 4>, 4);
    } else {
        if (a.clear) count(k_count<true, BATCH, 1>, 1);
        else count(k_count<false, BATCH, 1>, 1);
    }
    auto scan = [&](auto kern) { kern<<<tiles, SCAN_THREADS, 0, s>>>(a.count, a.table, sums); };
    if (kp.table_cells <= SCAN_DIRECT) {
        scan(k_scan_cells<4, false, true>);
    } else if (scan_items(kp.table_cells) == 4) {
        k_tile_sums<4><<<tiles, SCAN_THREADS, 0, s>>>(a.count, sums);
        if (a.full) scan(k_scan_cells<4, true, false>);
        else scan(k_scan_cells<4, false, false>);
    } else {
        k_tile_sums<16><<<tiles, SCAN_THREADS, 0, s>>>(a.count, sums);
        scan(k_scan_cells<16, false, false>);
    }
    k_scatter_ids<<<g, 256, 0, s>>>(a.keys_in, a.places, a.table, a.slots, kp.n, a.err);
    auto order = [&](auto kern) {
        kern<<<g, 256, 0, s>>>(a.slots, a.table, a.pos, a.vel, a.keys, a.index, a.spos, a.svel, a.bricks, counters, a.count, kp, a.err);
    };
    if (a.full) {
        if (a.vel) order(k_order_cells<false, true, BATCH>);
        else order(k_order_cells<false, false, BATCH>);
    } else {
        if (a.vel) order(k_order_cells<true, true, BATCH>);
        else order(k_order_cells<true, false, BATCH>);
    }
    return cudaGetLastError();
}

// ---- few particles --------------------------------------------------------------------------

// Up to RANK_MAX particles are sorted without counts: every CTA works out all keys, and a warp a
// particle counts how many come before it, and where its cell begins and ends, among
// key * RANK_MAX + id of all. Two launches where the counting sort has five, each mostly its own
// latency; the comparisons grow with the square of the particles. Us a step, with its copies in
// and out, by the counting sort and by this: hashed keys, 256 particles 33.6 / 29.4, 1,024 33.9 / 31.5,
// 2,048 35.2 / 32.4; a grid 23.6 / 21.5, 25.7 / 23.7, 25.8 / 25.7. (Four lanes a particle: 39.8 and 37.7 at 2,048.)
constexpr uint32_t RANK_MAX = 2048, RANK_CELLS = 1u << 20;  // key * RANK_MAX + id stays below 2^31
constexpr uint32_t RANK_TARGETS = 16, RANK_LANES = 32;       // particles per CTA, lanes per particle

inline bool rank_sort_fits(uint32_t cells, uint32_t n) { return n <= RANK_MAX && cells <= RANK_CELLS; }

// Empties the table entries of the previous step's cells (its sorted keys are in `keys`) if
// `clear`, and the brick counters.
static __global__ void __launch_bounds__(256) k_clear_cells(const uint32_t* __restrict__ keys, uint2* __restrict__ table,
                                                            uint32_t* __restrict__ counters, uint32_t n, uint32_t cells, bool clear) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i < 4) counters[i] = 0u;
    if (!clear || i >= n) return;
    const uint32_t k = keys[i];
    if ((i == 0 || keys[i - 1] != k) && k < cells) table[k] = make_uint2(EMPTY, EMPTY);
}

template <bool BRICKS, bool VEL>
__global__ void __launch_bounds__(RANK_LANES * RANK_TARGETS) k_rank_cells(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ index,
                                                                 float4* __restrict__ spos, float4* __restrict__ svel,
                                                                 uint2* __restrict__ table, uint32_t* __restrict__ bricks,
                                                                 uint32_t* __restrict__ n_bricks, KParams kp) {
    __shared__ __align__(16) uint32_t s_c[RANK_MAX];
    const uint32_t all = (kp.n + 15u) & ~15u;
#pragma unroll 4
    for (uint32_t j = threadIdx.x; j < all; j += RANK_LANES * RANK_TARGETS)
        s_c[j] = j < kp.n ? particle_key(kp, pos[j]) * RANK_MAX + j : 0xFFFFFFFFu;  // the padding is behind everything
    __syncthreads();
    const uint32_t i = blockIdx.x * RANK_TARGETS + threadIdx.x / RANK_LANES, q = threadIdx.x % RANK_LANES;
    const uint32_t mine = s_c[min(i, kp.n - 1u)], key = mine / RANK_MAX, lo = key * RANK_MAX, hi = lo + RANK_MAX;
    uint32_t blo = 0;  // first of the brick's keys
    if (BRICKS) {
        const uint32_t x = key % (uint32_t)kp.nx;
        blo = (key - x % (uint32_t)kp.bw) * RANK_MAX;
    }
    uint32_t d = 0, first = 0, end = 0, bfirst = 0;  // how many come before: me, my cell, the next cell, my brick
#pragma unroll 4
    for (uint32_t j = q; j < all / 4; j += RANK_LANES) {
        const uint4 c = reinterpret_cast<const uint4*>(s_c)[j];
        auto count = [&](uint32_t v) {
            d += v < mine;
            first += v < lo;
            end += v < hi;
            if (BRICKS) bfirst += v < blo;
        };
        count(c.x);
        count(c.y);
        count(c.z);
        count(c.w);
    }
#pragma unroll
    for (uint32_t m = 1; m < RANK_LANES; m <<= 1) {
        d += __shfl_xor_sync(0xffffffffu, d, m);
        first += __shfl_xor_sync(0xffffffffu, first, m);
        end += __shfl_xor_sync(0xffffffffu, end, m);
        if (BRICKS) bfirst += __shfl_xor_sync(0xffffffffu, bfirst, m);
    }
    if (q != 0 || i >= kp.n) return;
    keys[d] = key;
    index[d] = i;
    spos[d] = pos[i];
    if (VEL) svel[d] = vel[i];
    if (d == first) table[key] = make_uint2(first, end);
    if (BRICKS && d == bfirst) bricks[atomicAdd(n_bricks, 1u)] = (key % (uint32_t)kp.nx) / (uint32_t)kp.bw + (uint32_t)kp.bxn * (key / (uint32_t)kp.nx);
}

// Enqueues the sort; arguments as for count_sort(), but hashed keys' table is filled here.
inline cudaError_t rank_sort(const CountSort& a, const KParams& kp, cudaStream_t s) {
    uint32_t* counters = (uint32_t*)((char*)a.scratch + SORT_USER_COUNTER_OFFSET);
    const unsigned g = (kp.n + RANK_TARGETS - 1) / RANK_TARGETS;
    auto rank = [&](auto kern) {
        kern<<<g, RANK_LANES * RANK_TARGETS, 0, s>>>(a.pos, a.vel, a.keys, a.index, a.spos, a.svel, a.table, a.bricks, counters, kp);
    };
    if (a.full) {
        const cudaError_t e = cudaMemsetAsync(a.table, 0xFF, (size_t)REF_BUCKETS * sizeof(uint2), s);
        if (e != cudaSuccess) return e;
        if (a.vel) rank(k_rank_cells<false, true>);
        else rank(k_rank_cells<false, false>);
    } else {
        k_clear_cells<<<(kp.n + 255u) / 256u, 256, 0, s>>>(a.keys, a.table, counters, kp.n, kp.table_cells, a.clear);
        if (a.vel) rank(k_rank_cells<true, true>);
        else rank(k_rank_cells<true, false>);
    }
    return cudaGetLastError();
}

}  // namespace gbsph
