// fluid3d_kernels.cuh -- device code of the 3D (and 2D poly6/spiky) SPH step.
//
// Two families of neighbour kernels:
//   * "exact" kernels (the density by warps of several particles, the forces a thread per particle or by
//     warps) restate clCalculateDensity /
//     clCalculateForces (libCL/phys/oclFluid3D.cl:150-255) operation for operation with
//     round-to-nearest intrinsics (no FMA contraction, IEEE sqrt and division), visiting the
//     27 (or 9) neighbour cells in the reference's z, y, x order. In REFERENCE_HASH mode that
//     includes visiting a bucket twice when two neighbour cells hash to it. They reproduce the
//     FP32 restatement bit for bit and serve the parity modes.
//   * "brick" kernels (LINEAR_GRID only) are the fast path: persistent CTAs stage the particles
//     around W cells along x in shared memory, a producer warp ahead of the others, and each
//     warp takes eight pairs of targets; density leaves neighbour lists for forces. FMA and the
//     approximate reciprocals are used, so results agree with the restatement within FP32
//     tolerance.
#pragma once

#include <type_traits>

#include "device.cuh"
#include "internal.h"

namespace gbsph {

constexpr uint32_t EMPTY = 0xFFFFFFFFu;
constexpr uint32_t REF_BUCKETS = 262144u;  // BUCKETS, libCL/phys/oclFluid3D.cl:32
constexpr int BRICK_THREADS = 256;  // of the batch's persistent step, whose other phases it fits
constexpr int BRICK_WARPS = BRICK_THREADS / 32;
constexpr int BRICK_W_MAX = 16;

// One scene of a batch (LINEAR_GRID): its particles, cells and bricks are consecutive ranges
// of the batch's arrays, and its gas constant, viscosity, box and grid are its own.
struct SceneDev {
    uint32_t part_off, cell_off, brick_off, n;
    int nx, ny, nz, bxn;
    float4 origin, box_min, box_max;
    float stiff, cvisc, pad0, pad1;
};

// Kernel-side parameters, passed by value.
struct KParams {
    float dt, radius, h, mass, p0, rho0, stiff, cvisc, cpress, kconst, vlimit;
    float h2;         // h*h
    float r2_thresh;  // smallest float x with sqrtf(x) >= h, so (sqrtf(r2) < h) == (r2 < r2_thresh)
    float v2_thresh;  // smallest float x with sqrtf(x) > vlimit (NaN: none), so (sqrtf(f2) > vlimit) == (f2 >= v2_thresh)
    float4 gravity, box_min, box_max, origin;
    int nx, ny, nz;
    int key_mode, dims;
    int end_bit;     // sort bits [0, end_bit)
    int digit_bits;  // sort digit width (bits per pass)
    int bw, bxn;  // brick width (cells) and bricks per x row
    uint32_t n;
    uint32_t table_cells;
    const SceneDev* scenes;  // batches only: n_scenes entries, sorted by part/cell/brick offsets
    int n_scenes;
    float4* rec_force;  // when set: receives each particle's force after the clip box, before the clamp
    // When set (brick kernels): slot *rec_slot of rec_nbr (rec_n4 * NBR_CAP words per slot)
    // receives each particle's in-range neighbours (itself included) as sorted indices,
    // NBR_CAP per particle, and slot *rec_slot of rec_cnt (rec_n4 words) their number, or
    // REC_SCAN where the list overflowed or the brick was not staged.
    uint32_t* rec_nbr;
    uint32_t* rec_cnt;
    const uint32_t* rec_slot;
    uint32_t rec_n4;
};

// Index of the scene whose range [off, next off) holds v (binary search over `n` scenes).
template <int FIELD>
__device__ __forceinline__ int scene_of(const SceneDev* __restrict__ sc, int n, uint32_t v) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const uint32_t o = FIELD == 0 ? sc[mid].part_off : (FIELD == 1 ? sc[mid].cell_off : sc[mid].brick_off);
        if (o <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---- keys ---------------------------------------------------------------------------------

// gridPosition (libCL/phys/oclFluid3D.cl:34-42); LINEAR_GRID subtracts the grid origin.
__device__ __forceinline__ void grid_position(const KParams& kp, float4 p, int& gx, int& gy, int& gz) {
    if (kp.key_mode == GBSPH_KEY_LINEAR_GRID) {
        p.x = __fsub_rn(p.x, kp.origin.x);
        p.y = __fsub_rn(p.y, kp.origin.y);
        p.z = __fsub_rn(p.z, kp.origin.z);
    }
    gx = (int)floorf(__fdiv_rn(p.x, kp.h));
    gy = (int)floorf(__fdiv_rn(p.y, kp.h));
    gz = kp.dims == 2 ? 0 : (int)floorf(__fdiv_rn(p.z, kp.h));
}

// hashKey (libCL/phys/oclFluid3D.cl:44-52).
__device__ __forceinline__ uint32_t hash_key(int x, int y, int z) {
    uint32_t n = (73856093u * (uint32_t)x) ^ (19349663u * (uint32_t)y) ^ (83492791u * (uint32_t)z);
    return n % REF_BUCKETS;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

__device__ __forceinline__ uint32_t linear_key(const KParams& kp, int x, int y, int z) {
    x = clampi(x, 0, kp.nx - 1);
    y = clampi(y, 0, kp.ny - 1);
    z = clampi(z, 0, kp.nz - 1);
    return (uint32_t)x + (uint32_t)kp.nx * ((uint32_t)y + (uint32_t)kp.ny * (uint32_t)z);
}

__device__ __forceinline__ uint32_t particle_key(const KParams& kp, float4 p) {
    int gx, gy, gz;
    grid_position(kp, p, gx, gy, gz);
    return kp.key_mode == GBSPH_KEY_LINEAR_GRID ? linear_key(kp, gx, gy, gz) : hash_key(gx, gy, gz);
}

// clHash (libCL/phys/oclFluid3D.cl:57-64) fused with the digit histogram of every sort pass
// (the index is implicit: the first sort pass generates values 0..n-1). With CLEAR, the
// linear cell table entries of the previous step's occupied cells are reset (the previous
// sorted keys are still in `prev_keys`), replacing a full fill of the table.
template <bool CLEAR>
__global__ void __launch_bounds__(256) k_hash(const float4* __restrict__ pos, KParams kp,
                                              uint32_t* __restrict__ keys,
                                              uint32_t* __restrict__ hist,
                                              const uint32_t* __restrict__ prev_keys,
                                              uint2* __restrict__ table) {
    __shared__ uint32_t s_h[SORT_MAX_PASSES * SORT_RADIX];
    for (int i = threadIdx.x; i < SORT_MAX_PASSES * SORT_RADIX; i += blockDim.x) s_h[i] = 0;
    __syncthreads();
    const int passes = sort_passes(0, kp.end_bit, kp.digit_bits);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kp.n; i += gridDim.x * blockDim.x) {
        const uint32_t k = particle_key(kp, pos[i]);
        keys[i] = k;
        for (int p = 0; p < passes; ++p) {
            const int shift = p * kp.digit_bits;
            const int bits = min(kp.digit_bits, kp.end_bit - shift);
            atomicAdd(&s_h[p * SORT_RADIX + ((k >> shift) & ((1u << bits) - 1u))], 1u);
        }
        if (CLEAR) {
            const uint32_t pk = prev_keys[i];
            if ((i == 0 || prev_keys[i - 1] != pk) && pk < kp.table_cells) table[pk] = make_uint2(EMPTY, EMPTY);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * SORT_RADIX; i += blockDim.x)
        if (s_h[i]) atomicAdd(&hist[i], s_h[i]);
}

// clReorder (libCL/phys/oclFluid3D.cl:66-72), used when the gather is not fused into the
// last sort pass.
static __global__ void k_reorder(const uint32_t* __restrict__ index, const float4* __restrict__ pos,
                          const float4* __restrict__ vel, float4* __restrict__ spos,
                          float4* __restrict__ svel, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t s = index[i];
    spos[i] = pos[s];
    svel[i] = vel[s];
}

// Cell bounds into the interleaved LINEAR_GRID table, plus the list of occupied bricks,
// for BOUNDS_TILE consecutive sorted keys per CTA (BOUNDS_ITEMS per thread, strided by the
// block). A key that starts a cell writes the cell's first index, one that ends it the end;
// a key whose brick differs from its predecessor's appends the brick id: the CTA's appends
// take ranks from a shared counter and reserve their slots with one global atomic (one
// counter address, so per-key atomics would queue behind each other).
constexpr uint32_t BOUNDS_ITEMS = 4;
constexpr uint32_t BOUNDS_TILE = 256 * BOUNDS_ITEMS;

// Tile `tile` of the keys; COH: the keys were written earlier in the same launch.
template <bool COH = false, class BrickOf>
__device__ __forceinline__ void bounds_tile(const uint32_t* __restrict__ keys, const KParams& kp,
                                            uint2* __restrict__ table, uint32_t* __restrict__ bricks,
                                            uint32_t* __restrict__ n_bricks, uint32_t* err, BrickOf brick_of,
                                            uint32_t tile) {
    __shared__ uint32_t s_cnt, s_base;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    uint32_t bid[BOUNDS_ITEMS], rank[BOUNDS_ITEMS];
    const uint32_t i0 = tile * BOUNDS_TILE + threadIdx.x;
#pragma unroll
    for (uint32_t it = 0; it < BOUNDS_ITEMS; ++it) {
        const uint32_t i = i0 + it * blockDim.x;
        rank[it] = EMPTY;
        bid[it] = 0;
        if (i >= kp.n) continue;
        const uint32_t k = ld_phase<COH>(keys + i);
        if (k >= kp.table_cells) {
            atomicOr(err, DEV_ERR_KEY_RANGE);
            continue;
        }
        const uint32_t prev = i > 0 ? ld_phase<COH>(keys + i - 1) : EMPTY;
        const uint32_t next = i + 1 < kp.n ? ld_phase<COH>(keys + i + 1) : EMPTY;
        if (k != prev) table[k].x = i;
        if (k != next) table[k].y = i + 1;
        bid[it] = brick_of(k);
        if (prev == EMPTY || bid[it] != brick_of(prev)) rank[it] = atomicAdd(&s_cnt, 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt) s_base = atomicAdd(n_bricks, s_cnt);
    __syncthreads();
#pragma unroll
    for (uint32_t it = 0; it < BOUNDS_ITEMS; ++it)
        if (rank[it] != EMPTY) bricks[s_base + rank[it]] = bid[it];
}

// Single scene: brick id = x/W + bxn*(y + ny*z).
static __global__ void __launch_bounds__(256) k_bounds_linear(const uint32_t* __restrict__ keys, KParams kp,
                                                              uint2* __restrict__ table, uint32_t* __restrict__ bricks,
                                                              uint32_t* __restrict__ n_bricks, uint32_t* err) {
    const uint32_t nx = (uint32_t)kp.nx, bw = (uint32_t)kp.bw, bxn = (uint32_t)kp.bxn;
    bounds_tile(keys, kp, table, bricks, n_bricks, err,
                [=](uint32_t k) { return (k % nx) / bw + bxn * (k / nx); }, blockIdx.x);
}

// A batch's key: the scene's cell offset plus the linear key in the scene's own grid.
__device__ __forceinline__ uint32_t batch_key(const KParams& kp, uint32_t i, float4 p) {
    const SceneDev& d = kp.scenes[scene_of<0>(kp.scenes, kp.n_scenes, i)];
    const int gx = (int)floorf(__fdiv_rn(__fsub_rn(p.x, d.origin.x), kp.h));
    const int gy = (int)floorf(__fdiv_rn(__fsub_rn(p.y, d.origin.y), kp.h));
    const int gz = (int)floorf(__fdiv_rn(__fsub_rn(p.z, d.origin.z), kp.h));
    return d.cell_off + (uint32_t)clampi(gx, 0, d.nx - 1) +
           (uint32_t)d.nx * ((uint32_t)clampi(gy, 0, d.ny - 1) + (uint32_t)d.ny * (uint32_t)clampi(gz, 0, d.nz - 1));
}

// Batch version of k_hash: each particle keys into its own scene's grid. The body takes the block's histogram
// buffer (SORT_MAX_PASSES * SORT_RADIX words of shared memory) from the caller.
template <bool CLEAR>
__device__ __forceinline__ void hash_batch_run(uint32_t* s_h, const float4* __restrict__ pos, const KParams& kp,
                                               uint32_t* __restrict__ keys, uint32_t* __restrict__ hist,
                                               const uint32_t* __restrict__ prev_keys, uint2* __restrict__ table) {
    for (int i = threadIdx.x; i < SORT_MAX_PASSES * SORT_RADIX; i += blockDim.x) s_h[i] = 0;
    __syncthreads();
    const int passes = sort_passes(0, kp.end_bit, kp.digit_bits);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kp.n; i += gridDim.x * blockDim.x) {
        const uint32_t k = batch_key(kp, i, pos[i]);
        keys[i] = k;
        for (int q = 0; q < passes; ++q) {
            const int shift = q * kp.digit_bits;
            const int bits = min(kp.digit_bits, kp.end_bit - shift);
            atomicAdd(&s_h[q * SORT_RADIX + ((k >> shift) & ((1u << bits) - 1u))], 1u);
        }
        if (CLEAR) {
            const uint32_t pk = prev_keys[i];
            if ((i == 0 || prev_keys[i - 1] != pk) && pk < kp.table_cells) table[pk] = make_uint2(EMPTY, EMPTY);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * SORT_RADIX; i += blockDim.x)
        if (s_h[i]) atomicAdd(&hist[i], s_h[i]);
    __syncthreads();  // s_h is free for the caller
}

template <bool CLEAR>
__global__ void __launch_bounds__(256) k_hash_batch(const float4* __restrict__ pos, KParams kp,
                                                    uint32_t* __restrict__ keys, uint32_t* __restrict__ hist,
                                                    const uint32_t* __restrict__ prev_keys, uint2* __restrict__ table) {
    __shared__ uint32_t s_h[SORT_MAX_PASSES * SORT_RADIX];
    hash_batch_run<CLEAR>(s_h, pos, kp, keys, hist, prev_keys, table);
}

__device__ __forceinline__ uint32_t batch_brick_of(const KParams& kp, uint32_t k) {
    const SceneDev& d = kp.scenes[scene_of<1>(kp.scenes, kp.n_scenes, k)];
    const uint32_t local = k - d.cell_off, nx = (uint32_t)d.nx;
    return d.brick_off + (local % nx) / (uint32_t)kp.bw + (uint32_t)d.bxn * (local / nx);
}

// Batch version of k_bounds_linear: brick ids are global (scene brick offset + local id).
static __global__ void __launch_bounds__(256) k_bounds_batch(const uint32_t* __restrict__ keys, KParams kp,
                                                             uint2* __restrict__ table, uint32_t* __restrict__ bricks,
                                                             uint32_t* __restrict__ n_bricks, uint32_t* err) {
    bounds_tile(keys, kp, table, bricks, n_bricks, err, [&](uint32_t k) { return batch_brick_of(kp, k); }, blockIdx.x);
}

// Cell bounds of sorted keys alone (REFERENCE_HASH, per-stage calls): the cells' first index and end.
static __global__ void __launch_bounds__(256) k_bounds_hash(const uint32_t* __restrict__ keys, uint32_t n,
                                                            uint2* __restrict__ table, uint32_t cells, uint32_t* err) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = keys[i];
    if (k >= cells) {
        atomicOr(err, DEV_ERR_KEY_RANGE);
        return;
    }
    if (i == 0 || keys[i - 1] != k) table[k].x = i;
    if (i + 1 == n || keys[i + 1] != k) table[k].y = i + 1;
}

// Splits the interleaved table into two arrays (for inspection through the ABI).
static __global__ void k_table_split(const uint2* __restrict__ table, uint32_t cells,
                              uint32_t* __restrict__ cs, uint32_t* __restrict__ ce) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const uint2 e = table[i];
    cs[i] = e.x;
    ce[i] = e.x == EMPTY ? EMPTY : e.y;
}

// ---- exact (reference-order) neighbour kernels ---------------------------------------------

// The cell a particle's neighbours are counted from.
template <int MODE>
__device__ __forceinline__ void neighbour_centre(const KParams& kp, float4 p, int& gx, int& gy, int& gz) {
    grid_position(kp, p, gx, gy, gz);
    if (MODE == GBSPH_KEY_LINEAR_GRID) {
        gx = clampi(gx, 0, kp.nx - 1);
        gy = clampi(gy, 0, kp.ny - 1);
        gz = kp.dims == 2 ? 0 : clampi(gz, 0, kp.nz - 1);
    }
}

// The table entry of cell (x, y, z); false outside the grid.
template <int MODE>
__device__ __forceinline__ bool neighbour_cell(const KParams& kp, int x, int y, int z, uint32_t& cell) {
    if (MODE == GBSPH_KEY_LINEAR_GRID) {
        if (x < 0 || y < 0 || z < 0 || x >= kp.nx || y >= kp.ny || z >= kp.nz) return false;
        cell = (uint32_t)x + (uint32_t)kp.nx * ((uint32_t)y + (uint32_t)kp.ny * (uint32_t)z);
    } else {
        cell = hash_key(x, y, z);
    }
    return true;
}

// Calls f(start, end) for each non-empty neighbour cell in the reference's visiting order.
template <int MODE, class F>
__device__ __forceinline__ void for_each_neighbour_cell(const KParams& kp, const uint2* __restrict__ tab, float4 p, F&& f) {
    int gx, gy, gz;
    neighbour_centre<MODE>(kp, p, gx, gy, gz);
    const int zr = kp.dims == 2 ? 0 : 1;
    for (int z = -zr; z <= zr; z++)
        for (int y = -1; y <= 1; y++)
            for (int x = -1; x <= 1; x++) {
                uint32_t cell;
                if (!neighbour_cell<MODE>(kp, gx + x, gy + y, gz + z, cell)) continue;
                const uint2 e = tab[cell];
                if (e.x == EMPTY) continue;
                f(e.x, e.y);
            }
}

// fast_length of (a - b) with w = 0 is the correctly rounded sqrt of exact_r2 =
// ((x*x + y*y) + z*z). The correctly rounded sqrt is monotone, so sqrt(r2) < h exactly when
// r2 < kp.r2_thresh (the least float whose sqrt is >= h): the kernels test r2 and take the
// root of in-range candidates only.
__device__ __forceinline__ float exact_r2(float vx, float vy, float vz) {
    return __fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz));
}

// In-range neighbours the exact density kernel records per particle for the exact force
// kernel (sorted indices in visiting order); a particle with more is scanned again.
constexpr uint32_t XL_CAP = 64;
constexpr int EXACT_WARPS = 2;         // per CTA of the density kernel
constexpr uint32_t EXACT_HELD = 128;   // candidates a warp holds before it pairs them, a multiple of 64

// A warp's shared memory in the exact density kernel, for T targets per warp.
template <int T>
struct ExactWarp {
    float4 a[EXACT_HELD / 64][32];  // candidate 64 p + l and candidate 64 p + 32 + l: x, x, y, y
    float4 b[EXACT_HELD / 64][32];  // z, z, sorted index, sorted index
    uint32_t base[32];              // non-empty neighbour cells in visiting order: first index - candidates before
    float list[XL_CAP * (T + 1)];   // r2 of the in-range candidates: entry k of target t at k * (T + 1) + t
};

// clCalculateDensity, libCL/phys/oclFluid3D.cl:150-200. With RECORD, the in-range neighbours
// j (visiting order, repeats of a bucket visited twice included) go to xl[particle * XL_CAP + k]
// and their number to xc[particle].
//
// The sum of a particle runs in the reference's order, so it is one thread's; what leads to
// it need not be. A warp takes T consecutive sorted particles and, for each cell among them,
//  - reads the neighbour cells' ranges at once, a lane each;
//  - goes through the candidates 32 at a time, in visiting order, and holds those within h of
//    the box around the cell's targets. For a target inside the box and each axis,
//    fl(target - candidate) is at least the rounded distance to the box in magnitude
//    (rounding is monotone), and exact_r2 grows with each: none that is left out is in range;
//  - for each target tests the held candidates, two to a lane, and appends r2 of those in
//    range to the target's list, whose terms are added up as often as it is full.
// Then the rest of each list is summed. A thread that scans its 27 buckets by itself (12 of
// the 32 lanes at work, and the root and the sum executed for nearly every candidate because
// some lane is in range) took 522 us for 1,048,576 particles, 324 candidates and 34 in range
// each, and 23.6 us for 256, all of it the chain of table reads; this takes 393 and 7.7 us.
// Bound by instruction issue (78% of cycles). A list that is summed only
// at the end and, beyond XL_CAP, from the buckets again: 377, but 2.6 ms instead of 0.9 at 0.7 x the
// spacing (100 in range). Tried with that: 64 and 192 candidates held (+3 %), 32 targets per
// warp (+13 %), the two candidates of a lane next to each other (+5 %).
template <int MODE, bool RECORD, int T>
__global__ void __launch_bounds__(32 * EXACT_WARPS) k_density_exact(float4* __restrict__ spos, float4* __restrict__ svel,
                                                                    const uint2* __restrict__ tab, KParams kp,
                                                                    uint32_t* __restrict__ xl, uint32_t* __restrict__ xc) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ ExactWarp<T> shared[EXACT_WARPS];
    ExactWarp<T>& S = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, lt = lanemask_lt();
    const uint32_t first = (blockIdx.x * EXACT_WARPS + (threadIdx.x >> 5)) * T, particle = first + lane;
    const bool live = lane < T && particle < kp.n;
    uint32_t left = __ballot_sync(FULL, live);
    if (!left) return;
    const float4 posI = live ? spos[particle] : make_float4(0.f, 0.f, 0.f, 0.f);
    int gx, gy, gz;
    neighbour_centre<MODE>(kp, posI, gx, gy, gz);
    const int l = (int)lane, ox = l % 3 - 1, oy = l / 3 % 3 - 1, oz = kp.dims == 2 ? 0 : l / 9 - 1;  // place in the visiting order
    float density = 0.0f;              // lane t: the sum of target t's first `summed` terms,
    uint32_t count = 0, summed = 0;    // of `count` so far; the others' r2 are in its list
    auto term = [&](float r2) {
        const float vlen = __fsqrt_rn(r2);
        const float u = __fsub_rn(__fmul_rn(kp.h, kp.h), __fmul_rn(vlen, vlen));
        return __fmul_rn(__fmul_rn(u, u), u);
    };
    // d plus the terms of the n entries of target t's list, in order (by the whole warp). Four spacings a
    // cell (some 270 in range): 262,144 particles 536 us, 565 with four loads in flight, 465 a thread per
    // particle; a drain of all lists at once took 508, and 1 % more at the usual spacing.
    auto add_list = [&](int t, uint32_t n, float d) {
        float* list = S.list + t;
        for (uint32_t k = lane; k < n; k += 32) list[k * (T + 1)] = term(list[k * (T + 1)]);
        __syncwarp();
#pragma unroll 8
        for (uint32_t k = 0; k < n; ++k) d = __fadd_rn(d, list[k * (T + 1)]);
        return d;
    };
    while (left) {
        const int lead = __ffs(left) - 1;
        const int cx = __shfl_sync(FULL, gx, lead), cy = __shfl_sync(FULL, gy, lead), cz = __shfl_sync(FULL, gz, lead);
        const uint32_t group = __ballot_sync(FULL, live && gx == cx && gy == cy && gz == cz);
        left &= ~group;

        // the neighbour cells' ranges, lane = place in the visiting order
        uint2 e = make_uint2(EMPTY, EMPTY);
        uint32_t cell;
        if (l < (kp.dims == 2 ? 9 : 27) &&
            neighbour_cell<MODE>(kp, cx + ox, cy + oy, cz + oz, cell))
            e = tab[cell];
        const uint32_t n = e.x == EMPTY ? 0u : e.y - e.x;
        uint32_t off = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(FULL, off, d);
            if (l >= d) off += o;
        }
        const uint32_t total = __shfl_sync(FULL, off, 31);
        off -= n;
        const uint32_t some = __ballot_sync(FULL, n != 0);
        if (n) S.base[__popc(some & lt)] = e.x - off;

        // the box around the group's targets
        const bool in = (group >> lane) & 1u;
        float lo[3], hi[3];
        {
            const float x0 = __shfl_sync(FULL, posI.x, lead), y0 = __shfl_sync(FULL, posI.y, lead), z0 = __shfl_sync(FULL, posI.z, lead);
            const float v[3] = {in ? posI.x : x0, in ? posI.y : y0, in ? posI.z : z0};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = warp_min(v[a]);
                hi[a] = warp_max(v[a]);
            }
        }
        __syncwarp();

        uint32_t seen = 0, held = 0;
        // candidate base + lane: its index (EMPTY beyond the last) and position
        auto fetch = [&](uint32_t base, float4& p) -> uint32_t {
            const uint32_t heads = __reduce_or_sync(FULL, n && off - base < 32u ? 1u << (off - base) : 0u);
            const uint32_t r = seen + (uint32_t)__popc(heads & (lt | 1u << lane)) - 1u;
            seen += (uint32_t)__popc(heads);
            if (base + lane >= total) return EMPTY;
            const uint32_t j = base + lane + S.base[r];
            p = spos[j];
            return j;
        };
        // pairs the held candidates with the group's targets
        auto pair = [&]() {
            for (uint32_t s = held + lane; s < (held + 63u & ~63u); s += 32)  // never in range
                reinterpret_cast<float*>(&S.a[s >> 6][s & 31])[s >> 5 & 1] = INFINITY;
            __syncwarp();
            const uint32_t np = (held + 63u) >> 6;
            for (uint32_t g = group; g; g &= g - 1) {
                const int t = __ffs(g) - 1;
                const float x = __shfl_sync(FULL, posI.x, t), y = __shfl_sync(FULL, posI.y, t), z = __shfl_sync(FULL, posI.z, t);
                const uint64_t x2 = f2_pack(x, x), y2 = f2_pack(y, y), z2 = f2_pack(z, z);
                const uint32_t self = first + (uint32_t)t;
                uint32_t c = __shfl_sync(FULL, count, t), base = __shfl_sync(FULL, summed, t);
                float* list = S.list + t;
                uint32_t* rec = RECORD ? xl + (size_t)self * XL_CAP : nullptr;
                for (uint32_t p = 0; p < np; ++p) {
                    const float4 a = S.a[p][lane], b = S.b[p][lane];
                    const uint64_t vx = f2_sub(x2, f2_pack(a.x, a.y)), vy = f2_sub(y2, f2_pack(a.z, a.w)),
                                   vz = f2_sub(z2, f2_pack(b.x, b.y));
                    // summed one by one: a packed square and a packed sum are joined into an fma, which rounds once
                    float x0, x1, y0, y1, z0, z1;
                    f2_unpack(f2_mul(vx, vx), x0, x1);
                    f2_unpack(f2_mul(vy, vy), y0, y1);
                    f2_unpack(f2_mul(vz, vz), z0, z1);
                    const float r0 = __fadd_rn(__fadd_rn(x0, y0), z0), r1 = __fadd_rn(__fadd_rn(x1, y1), z1);
                    const uint32_t j0 = __float_as_uint(b.z), j1 = __float_as_uint(b.w);
                    const bool in0 = r0 < kp.r2_thresh && j0 != self, in1 = r1 < kp.r2_thresh && j1 != self;  // fast_length < h
                    const uint32_t m0 = __ballot_sync(FULL, in0), m1 = __ballot_sync(FULL, in1);
                    const uint32_t k0 = c + (uint32_t)__popc(m0 & lt), n0 = c + (uint32_t)__popc(m0);
                    const uint32_t k1 = n0 + (uint32_t)__popc(m1 & lt), n1 = n0 + (uint32_t)__popc(m1);
                    if (n1 - base > XL_CAP) {  // the list is full: its terms are added up now
                        __syncwarp();
                        const float d = add_list(t, c - base, __shfl_sync(FULL, density, t));
                        if (l == t) density = d;
                        __syncwarp();
                        base = c;
                    }
                    c = n1;
                    if (in0) {
                        list[(k0 - base) * (T + 1)] = r0;
                        if (RECORD && k0 < XL_CAP) rec[k0] = j0;
                    }
                    if (in1) {
                        list[(k1 - base) * (T + 1)] = r1;
                        if (RECORD && k1 < XL_CAP) rec[k1] = j1;
                    }
                }
                if (l == t) {
                    count = c;
                    summed = base;
                }
            }
            __syncwarp();
            held = 0;
        };
        float4 p, ahead;
        uint32_t j = fetch(0, p), next = EMPTY;
        for (uint32_t base = 0; base < total; base += 32, j = next, p = ahead) {
            if (base + 32 < total) next = fetch(base + 32, ahead);
            bool keep = false;
            if (j != EMPTY)
                keep = exact_r2(fmaxf(fmaxf(__fsub_rn(lo[0], p.x), __fsub_rn(p.x, hi[0])), 0.f),
                                fmaxf(fmaxf(__fsub_rn(lo[1], p.y), __fsub_rn(p.y, hi[1])), 0.f),
                                fmaxf(fmaxf(__fsub_rn(lo[2], p.z), __fsub_rn(p.z, hi[2])), 0.f)) < kp.r2_thresh;
            const uint32_t m = __ballot_sync(FULL, keep);
            if (keep) {
                const uint32_t s = held + (uint32_t)__popc(m & lt), half = s >> 5 & 1;
                float* a = reinterpret_cast<float*>(&S.a[s >> 6][s & 31]) + half;
                float* b = reinterpret_cast<float*>(&S.b[s >> 6][s & 31]) + half;
                a[0] = p.x;
                a[2] = p.y;
                b[0] = p.z;
                b[2] = __uint_as_float(j);
            }
            held += (uint32_t)__popc(m);
            if (held > EXACT_HELD - 32) pair();
        }
        if (held) pair();
    }
    __syncwarp();
    // 32 / T lanes share a target: each computes every (32 / T)-th term, all add them in order
    {
        constexpr uint32_t SHARE = 32 / T;
        const int t = l / (int)SHARE, first_lane = l - l % (int)SHARE;
        const uint32_t mine = __shfl_sync(FULL, count - summed, t), most = warp_max(mine);
        float d = __shfl_sync(FULL, density, t);
        for (uint32_t k = 0; k < most; k += SHARE) {
            const uint32_t at = k + lane % SHARE;
            const float v = at < mine ? term(S.list[at * (T + 1) + (uint32_t)t]) : 0.0f;
#pragma unroll
            for (int i = 0; i < (int)SHARE; ++i) {
                const float o = __shfl_sync(FULL, v, first_lane + i);
                if (k + i < mine) d = __fadd_rn(d, o);
            }
        }
        density = __shfl_sync(FULL, d, (l * (int)SHARE) & 31);
    }
    if (!live) return;
    if (RECORD) xc[particle] = count;
    // The reference writes .w in place while other work-items read .xyz only. Here the
    // candidates' positions are loaded as whole float4s, so a load may race with another
    // thread's write of that particle's .w; the loaded .w is never used (the sums take .xyz
    // only), so the race cannot change a result.
    if (count > 2) {
        density = fmaxf(1.0f, __fmul_rn(__fmul_rn(kp.mass, kp.kconst), density));
        reinterpret_cast<float*>(spos)[4 * (size_t)particle + 3] = density;
        reinterpret_cast<float*>(svel)[4 * (size_t)particle + 3] =
            __fadd_rn(kp.p0, __fmul_rn(kp.stiff, __fsub_rn(density, kp.rho0)));
    } else {
        reinterpret_cast<float*>(spos)[4 * (size_t)particle + 3] = kp.rho0;
        reinterpret_cast<float*>(svel)[4 * (size_t)particle + 3] = kp.p0;
    }
}

// ---- post stages ---------------------------------------------------------------------------

// repulsionForce walls of clClipBox (libCL/phys/oclFluid3D.cl:304-361): EPSILON 1e-5,
// stiffness 2000, damping 256, in the order y-min, y-max, z-min, z-max, x-min, x-max.
__device__ __forceinline__ void add_wall(float& fa, float& fw, float sign, float diff, float vn) {
    if (diff > 0.00001f) {
        const float mag = __fsub_rn(__fmul_rn(2000.0f, diff), __fmul_rn(256.0f, __fmul_rn(sign, vn)));
        fa = __fadd_rn(fa, __fmul_rn(sign, mag));
        fw = __fadd_rn(fw, __fmul_rn(0.0f, mag));
    }
}

__device__ __forceinline__ float4 clip_box_force(const KParams& kp, const float4& box_min, const float4& box_max,
                                                  float4 pos, float4 vel, float4 f) {
    const float r = kp.radius;
    add_wall(f.y, f.w, 1.0f, __fsub_rn(r, __fsub_rn(pos.y, box_min.y)), vel.y);
    add_wall(f.y, f.w, -1.0f, __fsub_rn(r, __fsub_rn(box_max.y, pos.y)), vel.y);
    if (kp.dims != 2) {
        add_wall(f.z, f.w, 1.0f, __fsub_rn(r, __fsub_rn(pos.z, box_min.z)), vel.z);
        add_wall(f.z, f.w, -1.0f, __fsub_rn(r, __fsub_rn(box_max.z, pos.z)), vel.z);
    }
    add_wall(f.x, f.w, 1.0f, __fsub_rn(r, __fsub_rn(pos.x, box_min.x)), vel.x);
    add_wall(f.x, f.w, -1.0f, __fsub_rn(r, __fsub_rn(box_max.x, pos.x)), vel.x);
    return f;
}

__device__ __forceinline__ float4 clip_box_force(const KParams& kp, float4 pos, float4 vel, float4 f) {
    return clip_box_force(kp, kp.box_min, kp.box_max, pos, vel, f);
}

// clIntegrateForce (libCL/phys/oclFluid3D.cl:258-271): clamp |F|, v += F*dt on 4 lanes.
__device__ __forceinline__ float4 integrate_force(const KParams& kp, float4 v, float4 f) {
    const float speed = __fsqrt_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(f.x, f.x), __fmul_rn(f.y, f.y)),
                                                       __fmul_rn(f.z, f.z)), __fmul_rn(f.w, f.w)));
    if (speed > kp.vlimit) {
        const float s = __fdiv_rn(kp.vlimit, speed);
        f.x = __fmul_rn(f.x, s);
        f.y = __fmul_rn(f.y, s);
        f.z = __fmul_rn(f.z, s);
        f.w = __fmul_rn(f.w, s);
    }
    v.x = __fadd_rn(v.x, __fmul_rn(f.x, kp.dt));
    v.y = __fadd_rn(v.y, __fmul_rn(f.y, kp.dt));
    v.z = __fadd_rn(v.z, __fmul_rn(f.z, kp.dt));
    v.w = __fadd_rn(v.w, __fmul_rn(f.w, kp.dt));
    return v;
}

// clIntegrateVelocity (libCL/phys/oclFluid3D.cl:284-291): all four lanes.
__device__ __forceinline__ float4 integrate_velocity(const KParams& kp, float4 p, float4 v) {
    return make_float4(__fadd_rn(p.x, __fmul_rn(v.x, kp.dt)), __fadd_rn(p.y, __fmul_rn(v.y, kp.dt)),
                       __fadd_rn(p.z, __fmul_rn(v.z, kp.dt)), __fadd_rn(p.w, __fmul_rn(v.w, kp.dt)));
}

// The six terms of an in-range pair, in the reference's arithmetic: pressure (x, y, z) and
// viscosity (x, y, z), without their constants.
__device__ __forceinline__ void exact_pair(const KParams& kp, const float4& posI, const float4& velI, const float4& posJ,
                                           const float4& velJ, float t[6]) {
    const float vx = __fsub_rn(posI.x, posJ.x), vy = __fsub_rn(posI.y, posJ.y), vz = __fsub_rn(posI.z, posJ.z);
    const float vlen = __fsqrt_rn(exact_r2(vx, vy, vz));
    const float density2 = __fmul_rn(posI.w, posJ.w);
    const float s = __fdiv_rn(__fadd_rn(velI.w, velJ.w), density2);
    const float hr = __fsub_rn(kp.h, vlen);
    t[0] = __fmul_rn(s, __fmul_rn(__fmul_rn(__fdiv_rn(vx, vlen), hr), hr));
    t[1] = __fmul_rn(s, __fmul_rn(__fmul_rn(__fdiv_rn(vy, vlen), hr), hr));
    t[2] = __fmul_rn(s, __fmul_rn(__fmul_rn(__fdiv_rn(vz, vlen), hr), hr));
    t[3] = __fmul_rn(__fdiv_rn(__fsub_rn(velJ.x, velI.x), density2), hr);
    t[4] = __fmul_rn(__fdiv_rn(__fsub_rn(velJ.y, velI.y), density2), hr);
    t[5] = __fmul_rn(__fdiv_rn(__fsub_rn(velJ.z, velI.z), density2), hr);
}

// The force from the pairs' sums; with POST clip + integrate-force + gravity + integrate-velocity
// as well, as the four reference kernels after this one (index is a permutation).
template <bool POST>
__device__ __forceinline__ void exact_finish(const KParams& kp, uint32_t particle, const float4& posI, const float4& velI, float px,
                                             float py, float pz, float qx, float qy, float qz, float4* __restrict__ force,
                                             const uint32_t* __restrict__ index, float4* __restrict__ pos, float4* __restrict__ vel) {
    const uint32_t o = index[particle];
    float4 f = force[o];
    f.x = __fadd_rn(f.x, __fmul_rn(__fadd_rn(__fmul_rn(kp.cpress, px), __fmul_rn(kp.cvisc, qx)), kp.mass));
    f.y = __fadd_rn(f.y, __fmul_rn(__fadd_rn(__fmul_rn(kp.cpress, py), __fmul_rn(kp.cvisc, qy)), kp.mass));
    f.z = __fadd_rn(f.z, __fmul_rn(__fadd_rn(__fmul_rn(kp.cpress, pz), __fmul_rn(kp.cvisc, qz)), kp.mass));
    f.w = 0.0f;
    if (!POST) {
        force[o] = f;
        return;
    }
    f = clip_box_force(kp, posI, velI, f);
    if (kp.rec_force) kp.rec_force[o] = f;
    const float4 v = integrate_force(kp, vel[o], f);
    vel[o] = v;
    force[o] = kp.gravity;
    pos[o] = integrate_velocity(kp, pos[o], v);
}

constexpr uint32_t XL_BLOCK = 16;  // list entries the exact force kernel stages at once

// clCalculateForces, libCL/phys/oclFluid3D.cl:202-255: force[index[i]] += SPH force, w = 0.
// With LISTED, a particle whose in-range neighbours the density kernel recorded (xc <= XL_CAP)
// takes them from its list, in the same visiting order, instead of scanning the buckets again:
// the same pairs in the same order, so the same sums, but the warp's threads step through
// their pairs together rather than each meeting its in-range candidates at different steps.
// A warp copies its particles' lists through shared memory, XL_BLOCK entries at a time; threads
// that read their own rows took 269 us where this takes 190 (1,048,576 particles), and lists
// laid out entry by entry, which they read in 224, cost the density kernel 43 us in scattered
// stores. With POST (the fused step without a hook) the particle is also clipped and integrated
// here: 217 us for both, and a launch less (224 and 30 in kernels of their own at first). Bound by the
// latency of the gathers. Loading two, four or eight neighbours at once takes more registers
// and is slower (238 / 256 / 322).
template <int MODE, bool LISTED, bool POST>
__global__ void __launch_bounds__(256) k_forces_exact(const float4* __restrict__ spos,
                                                      const float4* __restrict__ svel,
                                                      float4* __restrict__ force,
                                                      const uint32_t* __restrict__ index,
                                                      const uint2* __restrict__ tab, KParams kp, const uint32_t* __restrict__ xl,
                                                      const uint32_t* __restrict__ xc, float4* __restrict__ pos,
                                                      float4* __restrict__ vel) {
    const uint32_t particle = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = particle < kp.n;
    if (!LISTED && !live) return;
    const float4 posI = spos[live ? particle : 0], velI = svel[live ? particle : 0];
    float px = 0.f, py = 0.f, pz = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
    // one pair with the neighbour's position and velocity at hand
    auto pair_at = [&](const float4& posJ, const float4& velJ) {
        // always so for listed ones; with the test the compiler keeps this in 64 registers without spills
        if (!(exact_r2(__fsub_rn(posI.x, posJ.x), __fsub_rn(posI.y, posJ.y), __fsub_rn(posI.z, posJ.z)) < kp.r2_thresh)) return;
        float t[6];
        exact_pair(kp, posI, velI, posJ, velJ, t);
        px = __fadd_rn(px, t[0]);
        py = __fadd_rn(py, t[1]);
        pz = __fadd_rn(pz, t[2]);
        qx = __fadd_rn(qx, t[3]);
        qy = __fadd_rn(qy, t[4]);
        qz = __fadd_rn(qz, t[5]);
    };
    auto pair = [&](uint32_t j) {
        const float4 posJ = spos[j];
        const float vx = __fsub_rn(posI.x, posJ.x), vy = __fsub_rn(posI.y, posJ.y), vz = __fsub_rn(posI.z, posJ.z);
        if (exact_r2(vx, vy, vz) < kp.r2_thresh) pair_at(posJ, svel[j]);
    };
    bool scan = true;
    if (LISTED) {
        __shared__ uint32_t staged[256 / 32][32 * (XL_BLOCK + 1)];
        uint32_t* block = staged[threadIdx.x >> 5];
        const uint32_t lane = threadIdx.x & 31u, all = live ? xc[particle] : 0u;
        scan = all > XL_CAP;
        const uint32_t nl = scan ? 0u : all, most = __reduce_max_sync(0xffffffffu, nl);
        const uint4* rows = reinterpret_cast<const uint4*>(xl) + (size_t)(particle - lane) * (XL_CAP / 4);
        for (uint32_t k0 = 0; k0 < most; k0 += XL_BLOCK) {
            __syncwarp();
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {  // eight rows a load, four lanes to a row
                const uint32_t row = 8 * i + lane / 4, q = lane % 4;
                if (k0 + 4 * q < __shfl_sync(0xffffffffu, nl, (int)row)) {
                    const uint4 v = rows[row * (XL_CAP / 4) + k0 / 4 + q];
                    uint32_t* to = block + row * (XL_BLOCK + 1) + 4 * q;
                    to[0] = v.x;
                    to[1] = v.y;
                    to[2] = v.z;
                    to[3] = v.w;
                }
            }
            __syncwarp();
            // the next neighbour's position and velocity are loaded while the current pair is computed
            const uint32_t* mine = block + lane * (XL_BLOCK + 1);
            const uint32_t m = k0 < nl ? min(nl - k0, XL_BLOCK) : 0u;
            float4 pn = posI, vn = velI;
            if (m) {
                pn = spos[mine[0]];
                vn = svel[mine[0]];
            }
            for (uint32_t k = 0; k < m; ++k) {
                const float4 posJ = pn, velJ = vn;
                if (k + 1 < m) {
                    const uint32_t j = mine[k + 1];
                    pn = spos[j];
                    vn = svel[j];
                }
                pair_at(posJ, velJ);
            }
        }
        if (!live) return;
    }
    if (scan)
        for_each_neighbour_cell<MODE>(kp, tab, posI, [&](uint32_t start, uint32_t end) {
            for (uint32_t j = start; j < end; j++)
                if (j != particle) pair(j);
        });
    exact_finish<POST>(kp, particle, posI, velI, px, py, pz, qx, qy, qz, force, index, pos, vel);
}

constexpr int LISTED_WARPS = 2, LISTED_TARGETS = 4;  // per CTA, per warp

// The same for few particles, by their lists: a warp takes LISTED_TARGETS particles, its lanes compute
// the terms of all their pairs side by side, and a lane per particle and component adds them in the
// lists' order. A thread that goes through its particle's pairs by itself waits for some 34
// gathers one after the other, and few particles leave nothing beside them: 20.5 us for 4,096 or
// 16,384 particles where this takes 10.2 and 12.3. From some 50,000 on its six stores and loads per
// pair cost more than the wait (65,536: 28.7 / 24.6; 1,048,576: 426 / 217). Two particles per warp
// 10.2 and 14.3, five 12.3 and 12.3. Particles with more neighbours than a list holds take the whole
// warp as well: left to a lane each, a step of 32,768 particles at twice the usual density a side
// (four spacings a cell) took 1,251 us, 459 so, 1,008 with a thread per particle.
template <bool POST>
__global__ void __launch_bounds__(32 * LISTED_WARPS) k_forces_listed(const float4* __restrict__ spos, const float4* __restrict__ svel,
                                                                     float4* __restrict__ force, const uint32_t* __restrict__ index,
                                                                     const uint2* __restrict__ tab, KParams kp,
                                                                     const uint32_t* __restrict__ xl, const uint32_t* __restrict__ xc,
                                                                     float4* __restrict__ pos, float4* __restrict__ vel) {
    constexpr uint32_t FULL = 0xffffffffu, T = LISTED_TARGETS;
    __shared__ float s_term[LISTED_WARPS][6 * T][XL_CAP + 1];  // odd rows: a column is read without conflicts
    float(*term)[XL_CAP + 1] = s_term[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, first = (blockIdx.x * LISTED_WARPS + (threadIdx.x >> 5)) * T, particle = first + lane;
    if (first >= kp.n) return;  // whole warps
    const bool live = lane < T && particle < kp.n;
    const uint32_t all = live ? xc[particle] : 0u;
    const bool scan = all > XL_CAP;
    // particles without a list, one after the other: the warp goes through the buckets, 32 candidates at a
    // time, and adds the terms up as often as the particle's rows are full; the sums wait in the rows' last entry
    for (uint32_t left = __ballot_sync(FULL, scan); left; left &= left - 1) {
        const uint32_t t = (uint32_t)__ffs((int)left) - 1u, i = first + t;
        const float4 pi = spos[i], vi = svel[i];
        uint32_t n = 0;
        float part = 0.0f;  // of component `lane`
        auto add = [&]() {
            __syncwarp();
            if (lane < 6) {
#pragma unroll 4
                for (uint32_t k = 0; k < n; ++k) part = __fadd_rn(part, term[lane * T + t][k]);
            }
            __syncwarp();
            n = 0;
        };
        for_each_neighbour_cell<GBSPH_KEY_REFERENCE_HASH>(kp, tab, pi, [&](uint32_t start, uint32_t end) {
            for (uint32_t base = start; base < end; base += 32) {
                const uint32_t j = base + lane;
                float4 pj = pi;
                bool in = j < end && j != i;
                if (in) {
                    pj = spos[j];
                    in = exact_r2(__fsub_rn(pi.x, pj.x), __fsub_rn(pi.y, pj.y), __fsub_rn(pi.z, pj.z)) < kp.r2_thresh;
                }
                const uint32_t m = __ballot_sync(FULL, in), at = (uint32_t)__popc(m & lanemask_lt());
                if (n + (uint32_t)__popc(m) > XL_CAP) add();
                if (in) {
                    float x[6];
                    exact_pair(kp, pi, vi, pj, svel[j], x);
#pragma unroll
                    for (uint32_t c = 0; c < 6; ++c) term[c * T + t][n + at] = x[c];
                }
                n += (uint32_t)__popc(m);
            }
        });
        add();
        if (lane < 6) term[lane * T + t][XL_CAP] = part;
    }
    uint32_t before[T + 1];
    before[0] = 0;
#pragma unroll
    for (uint32_t t = 0; t < T; ++t) before[t + 1] = before[t] + __shfl_sync(FULL, scan ? 0u : all, (int)t);
    for (uint32_t e = lane; e < before[T]; e += 32) {
        uint32_t t = 0, k = e;
#pragma unroll
        for (uint32_t q = 1; q < T; ++q)
            if (e >= before[q]) {
                t = q;
                k = e - before[q];
            }
        const uint32_t i = first + t, j = xl[(size_t)i * XL_CAP + k];
        float v[6];
        exact_pair(kp, spos[i], svel[i], spos[j], svel[j], v);
#pragma unroll
        for (uint32_t c = 0; c < 6; ++c) term[c * T + t][k] = v[c];
    }
    __syncwarp();
    const uint32_t mine = __shfl_sync(FULL, all, (int)(lane % T));
    float sum = 0.0f;
    if (lane < 6 * T && mine > XL_CAP) {
        sum = term[lane][XL_CAP];
    } else if (lane < 6 * T) {
#pragma unroll 4
        for (uint32_t k = 0; k < mine; ++k) sum = __fadd_rn(sum, term[lane][k]);
    }
    float v[6];
#pragma unroll
    for (uint32_t c = 0; c < 6; ++c) v[c] = __shfl_sync(FULL, sum, (int)(c * T + lane % T));
    if (!live) return;
    const float4 posI = spos[particle], velI = svel[particle];
    exact_finish<POST>(kp, particle, posI, velI, v[0], v[1], v[2], v[3], v[4], v[5], force, index, pos, vel);
}

static __global__ void k_clip_box(const float4* __restrict__ spos, const float4* __restrict__ svel,
                           float4* __restrict__ force, const uint32_t* __restrict__ index, KParams kp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    const uint32_t o = index[i];
    const float4 f = clip_box_force(kp, spos[i], svel[i], force[o]);
    force[o] = f;
    if (kp.rec_force) kp.rec_force[o] = f;
}

static __global__ void k_integrate_force(float4* __restrict__ vel, const float4* __restrict__ force, KParams kp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    vel[i] = integrate_force(kp, vel[i], force[i]);
}

static __global__ void k_gravity(float4* __restrict__ force, KParams kp) {  // clGravity, :294-298
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    force[i] = kp.gravity;
}

static __global__ void k_integrate_velocity(float4* __restrict__ pos, const float4* __restrict__ vel, KParams kp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    pos[i] = integrate_velocity(kp, pos[i], vel[i]);
}

// clEmitter (libCL/phys/oclFluid3D.cl:273-282): particles emit+1 .. emit+99 are placed on a
// 10-wide sheet at y = 0.6 (index = emit - particle, negative, with C's truncating / and %)
// and given velocity (0, emit_speed, 0). The z lane `0.6 + index%10*2*radius` adds the float
// product to the double literal 0.6 in double and rounds the sum to float once (OpenCL C on a
// device with doubles, as the reference's kernels compile on the host and GPU OpenCL stacks).
static __global__ void k_emitter(float4* __restrict__ pos, float4* __restrict__ vel, uint32_t n, uint32_t emit,
                                 float emit_speed, float radius) {
    const uint32_t particle = blockIdx.x * blockDim.x + threadIdx.x;
    if (particle >= n) return;
    if (particle > emit && particle < emit + 100u) {
        const int index = (int)(emit - particle);
        const float dz = __fmul_rn((float)(index % 10 * 2), radius);
        pos[particle] = make_float4(__fmul_rn((float)(index / 10 * 2), radius), 0.6f,
                                    __double2float_rn(__dadd_rn(0.6, (double)dz)), 1.0f);
        vel[particle] = make_float4(0.0f, emit_speed, 0.0f, 1.0f);
    }
}

// ---- brick (fast, LINEAR_GRID) neighbour kernels ---------------------------------------------
//
// Both passes run as persistent CTAs over the occupied bricks. The last warp of a CTA produces: it
// takes bricks from a queue, reads the cell ranges of the brick's neighbour rows, cuts the brick
// into units of at most BRICK_UNIT target cells whose candidates fit the staging, and copies
// each unit's candidates into one of two buffers. The other warps consume the units: while they
// compute one, the other buffer is filled, so that the chain queue -> brick -> cell table ->
// particles does not stand in line with the arithmetic. A unit is handed over through two
// mbarriers per buffer (full: filled; empty: every consumer is done).
//
// The candidates are staged by columns: all cells (y, z = -1..1) of column x, then those of
// column x + 1. The 27 (or 9) cells around a target are then one contiguous window of the
// staging, the same for every target of a cell, and a candidate's place in its target's window
// depends neither on the brick nor on the unit; neighbour lists hold such places, so that the
// two passes need not cut the bricks alike. Staged by rows, the window is nine short pieces,
// and the row loop around them cost as many instructions as the candidates themselves.
//
// A consumer waits for copies and for a task at most; the producer waits for whole units, and a unit
// that is not staged may take long (8,000 particles in one cell: 57 ms for both passes; 60,000:
// seconds). So consumers count the cells that they read from global memory in S.progress, and
// the producer gives up only after a second in which nothing moved.
//
// A cell's particles are taken in pairs (two consecutive sorted particles; the last of an odd
// cell alone), numbered through the unit, and both passes give four lanes to a pair and eight
// pairs to a warp whatever cells they are in. A lane holds both targets, so a candidate read
// from shared memory serves two, and the two share one neighbour list: the candidates in range
// of either (about 46 entries where each has 34).
//
// 1,048,576 particles at the start of the block collapse (8 per cell, 216 candidates and 34 in
// range each): density 136 us (213 us with the rows staged by bulk copies, a warp per cell and
// lists appended per candidate), forces 149 us (184 us with two lanes per target and the lists
// staged). Density is bound by instruction issue (77% of cycles; 63 of the 137 us are the
// candidate loop at 21 instructions for 64 pairs, 20 the lists, 16 the staging), forces by issue
// and the LSU pipe's wavefronts (59% and 68%).
// Tried: a bulk copy per cell instead of the 16-byte asynchronous copies (170 / 260 us: the
// small copies queue), two producers, one per buffer (139 / 178), 3 to 7 consumers at 3 to 6
// CTAs per SM (density 133-137, forces 150-172).
constexpr int DENSITY_CONSUMERS = 4, FORCE_CONSUMERS = 5;      // warps beside the producer
constexpr int DENSITY_CTAS = 5, FORCE_CTAS = 4;                // per SM, by shared memory
constexpr int BRICK_UNIT = 8;                     // target cells per unit at most
constexpr int BRICK_CELLS = (BRICK_UNIT + 2) * 9;  // staged cells of a unit
// Staged candidates per unit (8 lattice cells with their neighbours are 720). Both may cut a
// brick differently; a target whose window alone exceeds the cap reads global memory.
constexpr uint32_t DENSITY_CAP = 1024, FORCE_CAP = 768;
constexpr uint32_t NBR_CAP = 64;                  // neighbour list entries per particle (a pair: twice that)
constexpr uint32_t TASK_PAIRS = 8;                // pairs a warp takes at once, four lanes each
constexpr uint32_t LIST_AHEAD = 6;                // 8-entry chunks of a list the force pass loads at once
constexpr uint32_t LIST_STRIDE = 2 * NBR_CAP + 8;  // halves between a warp's lists (16-byte rows)
constexpr uint32_t NBR_SCAN = 0xFFFFFFFFu;        // nbr_meta: no list, the force pass scans
constexpr uint32_t REC_SCAN = 0xFFFFFFFFu;        // rec_cnt: no recorded list for this particle

// One unit.
struct BrickUnit {
    uint32_t off[BRICK_CELLS + 1];  // staged place of cell (column * R + row); the last entry: all candidates
    uint2 cell[BRICK_CELLS];        // the cell's first sorted index; staged place | count << 16 (staged units)
    uint32_t pair[BRICK_UNIT];      // pairs before target cell c (beyond the last cell: npair)
    uint32_t npair;
    int ncell;                      // target cells (columns 1 .. ncell); 0: an end
    int staged;                     // 0: the candidates did not fit, read them from global memory
    int more;                       // at an end: units of the other kind follow
    float stiff, cvisc;             // the scene's parameters (they differ within a batch)
    float4 box_min, box_max;
};

struct BrickShared {
    BrickUnit unit[2];
    uint32_t progress;              // cells that consumers have begun to read from global memory
    unsigned long long full[2], empty[2];
};

// What a lane knows of its pair.
struct PairTask {
    bool live, two;         // a pair of this unit (else a stand-in, nothing of which is stored); it has two targets
    uint32_t gi;            // sorted index of the first target
    uint32_t self;          // its staged place
    uint32_t lo, len;       // the window's first staged place and its candidates
    int c;                  // target cell: column c + 1
};

template <int R, int RC>
__device__ __forceinline__ PairTask pair_task(const BrickUnit& U, uint32_t p) {
    PairTask t;
    t.live = p < U.npair;
    p = min(p, U.npair - 1u);
    t.c = 0;
#pragma unroll
    for (int k = 1; k < BRICK_UNIT; ++k) t.c += p >= U.pair[k] ? 1 : 0;
    const uint32_t k = 2u * (p - U.pair[t.c]), i = (uint32_t)((t.c + 1) * R + RC), o = U.off[i];
    t.two = k + 1u < U.off[i + 1] - o;
    t.gi = U.cell[i].x + k;
    t.self = o + k;
    t.lo = U.off[t.c * R];
    t.len = U.off[(t.c + 3) * R] - t.lo;
    return t;
}

// Dynamic shared memory: two staging buffers, then (density) each consumer's neighbour lists.
constexpr size_t density_smem(int consumers) {
    return 2 * (size_t)DENSITY_CAP * 16 + (size_t)consumers * TASK_PAIRS * LIST_STRIDE * 2;
}
constexpr size_t DENSITY_SMEM = density_smem(DENSITY_CONSUMERS);
constexpr size_t FORCE_SMEM = 2 * (size_t)FORCE_CAP * 32;

__device__ __forceinline__ void brick_init(BrickShared& S) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            // the producer's lanes arrive twice each: once for their own writes, once when their
            // asynchronous copies have landed
            mbar_init(reinterpret_cast<uint64_t*>(&S.full[i]), 64);
            mbar_init(reinterpret_cast<uint64_t*>(&S.empty[i]), blockDim.x / 32u - 1u);
        }
        S.progress = 0u;
        fence_mbar_init();
    }
    __syncthreads();
}

// Ends the barriers' life (after a CTA barrier behind the pass), so that a later phase may
// initialise them again.
__device__ __forceinline__ void brick_fini(BrickShared& S) {
    if (threadIdx.x == 0)
        for (int i = 0; i < 2; ++i) {
            mbar_inval(reinterpret_cast<uint64_t*>(&S.full[i]));
            mbar_inval(reinterpret_cast<uint64_t*>(&S.empty[i]));
        }
}

// The producer warp's loop (see above). `queue` is the pass's brick counter; a0 (and a1 with
// NARR = 2) the sorted arrays to stage: buffer s holds a0's candidates at s_buf + s * NARR * CAP
// and a1's CAP entries behind. With SPLIT a brick that has units of both kinds, staged and not, is gone
// through once for either, and an end is put between units of different kinds, so that consumers have a loop
// for each: with both in one, the staged targets of the force pass took 149 to 153 us where they
// take 147 now. Returns false if a wait gave up.
template <int DIMS, bool BATCH, uint32_t CAP, int NARR, bool SPLIT>
__device__ __forceinline__ bool brick_produce(BrickShared& S, float4* s_buf, const float4* __restrict__ a0,
                                              const float4* __restrict__ a1, const uint2* __restrict__ table,
                                              const uint32_t* __restrict__ bricks, uint32_t n_bricks, uint32_t* queue,
                                              const KParams& kp, uint32_t* err) {
    constexpr int R = DIMS == 3 ? 9 : 3;
    constexpr int RC = DIMS == 3 ? 4 : 1;  // the brick's own row
    const int lane = threadIdx.x & 31;
    uint32_t fill = 0;  // units handed over
    // Waits until the buffer of the next unit is free.
    auto acquire = [&]() -> bool {
        if (fill < 2) return true;
        const bool ok = mbar_wait_progress(reinterpret_cast<uint64_t*>(&S.empty[fill & 1u]), ((fill >> 1) - 1u) & 1u, &S.progress);
        if (!ok) atomicOr(err, DEV_ERR_MBAR_TIMEOUT);
        return __all_sync(0xffffffffu, ok);
    };
    auto hand_over = [&]() {
        uint64_t* full = reinterpret_cast<uint64_t*>(&S.full[fill & 1u]);
        mbar_arrive(full);
        cp_async_mbar_arrive(full);
        ++fill;
    };
    // The first brick goes by the CTA's own number, the queue deals out those behind: a scene of
    // few bricks is spared a trip to the queue, and the brick is read beside their number
    // (`bricks` has a word per particle). 16,384 particles in 2D: a step 29.6 -> 25.5 us.
    uint32_t b = blockIdx.x, bid = ld_relaxed_gpu(bricks + min(b, kp.n - 1u));
    bool slow = false;  // SPLIT: units that are not staged are handed over now
    // Ends the units (of one kind).
    auto end = [&](bool more) -> bool {
        if (!acquire()) {
            cp_async_wait_all();
            return false;
        }
        if (lane == 0) {
            S.unit[fill & 1u].ncell = 0;
            S.unit[fill & 1u].more = more;
        }
        __syncwarp();
        hand_over();
        return true;
    };
    while (b < n_bricks) {
        uint32_t nb = 0;  // the next brick's ticket, asked for early
        if (lane == 0) nb = gridDim.x + atomicAdd(queue, 1u);
        const SceneDev* sc = BATCH ? kp.scenes + scene_of<2>(kp.scenes, kp.n_scenes, bid) : nullptr;
        const int nx = BATCH ? sc->nx : kp.nx, ny = BATCH ? sc->ny : kp.ny, nz = BATCH ? sc->nz : kp.nz;
        const uint32_t bxn = BATCH ? (uint32_t)sc->bxn : (uint32_t)kp.bxn;
        const uint32_t lb = BATCH ? bid - sc->brick_off : bid;
        const uint2* tab = BATCH ? table + sc->cell_off : table;
        const int bx = (int)(lb % bxn);
        const uint32_t yz = lb / bxn;
        const int y = (int)(yz % (uint32_t)ny), z = (int)(yz / (uint32_t)ny);
        const int xb = bx * kp.bw, ncell = min(kp.bw, nx - xb);
        // lane c holds column c (cell xb - 1 + c): start and count of its R cells
        const int cx = xb - 1 + lane;
        const bool col = lane < ncell + 2 && cx >= 0 && cx < nx;
        uint32_t st[R], cn[R], tot = 0;
        bool bad = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int cy = y + (r % 3) - 1, cz = DIMS == 3 ? z + (r / 3) - 1 : 0;
            uint2 e = make_uint2(EMPTY, 0u);
            if (col && cy >= 0 && cy < ny && cz >= 0 && cz < nz)
                e = tab[(uint32_t)cx + (uint32_t)nx * ((uint32_t)cy + (uint32_t)ny * (uint32_t)cz)];
            const bool some = e.x != EMPTY, in = e.x <= e.y && e.y <= kp.n;
            bad |= some && !in;  // inconsistent table: report, use an empty cell
            cn[r] = some && in ? e.y - e.x : 0u;
            st[r] = some && in ? e.x : 0u;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) tot += cn[r];
        if (bad) atomicOr(err, DEV_ERR_KEY_RANGE);
        b = __shfl_sync(0xffffffffu, nb, 0);
        bid = b < n_bricks ? bricks[b] : 0u;
        uint32_t incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t excl = incl - tot, incl_next = __shfl_down_sync(0xffffffffu, incl, 1);
        bool other = false, again = false;  // there are units of the other kind; it is their turn
        for (int c0 = 0; c0 < ncell;) {
            // targets: columns c0 + 1 .. c1, the most that fit the staging with their neighbours
            const uint32_t e0 = __shfl_sync(0xffffffffu, excl, c0);
            const uint32_t fits =
                __ballot_sync(0xffffffffu, lane > c0 && lane <= min(ncell, c0 + BRICK_UNIT) && incl_next - e0 <= CAP);
            const int c1 = fits ? 31 - __clz((int)fits) : c0 + 1;
            const uint32_t mine = lane > c0 && lane <= c1 ? cn[RC] : 0u;
            const uint32_t some = __ballot_sync(0xffffffffu, mine != 0u);
            const bool turn = !SPLIT || (fits == 0u) == slow;
            if (some && !turn) other = true;
            if (some && turn) {
                uint32_t pairs = (mine + 1u) >> 1;  // inclusive count of the pairs up to this column
                const uint32_t own = pairs;
#pragma unroll
                for (int o = 1; o < BRICK_W_MAX + 2; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, pairs, o);
                    if (lane >= o) pairs += v;
                }
                if (!acquire()) {
                    cp_async_wait_all();
                    return false;
                }
                BrickUnit& U = S.unit[fill & 1u];
                const int k = lane - c0;
                if (k >= 0 && k < c1 - c0 + 2) {
                    uint32_t o = excl - e0;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        U.off[k * R + r] = o;
                        U.cell[k * R + r] = make_uint2(st[r], o | (cn[r] << 16));
                        o += cn[r];
                    }
                    if (k == c1 - c0 + 1) U.off[(k + 1) * R] = o;
                }
                // target cells beyond the unit's last have no pairs: their entry is the total
                if (lane > c0 && lane <= c0 + BRICK_UNIT) U.pair[lane - c0 - 1] = pairs - own;
                if (lane == c1) {
                    U.npair = pairs;
                    U.ncell = c1 - c0;
                    U.staged = fits != 0u;
                    U.stiff = BATCH ? sc->stiff : kp.stiff;
                    U.cvisc = BATCH ? sc->cvisc : kp.cvisc;
                    U.box_min = BATCH ? sc->box_min : kp.box_min;
                    U.box_max = BATCH ? sc->box_max : kp.box_max;
                }
                __syncwarp();
                if (fits) {
                    // 8 lanes per cell (a cell of eight particles is one line), 4 x 4 cells at a time
                    const uint32_t e = (uint32_t)lane & 7u;
                    const uint32_t dst = smem_addr(s_buf + (fill & 1u) * NARR * CAP) + e * 16u;
                    const float4* const src0 = a0 + e;
                    const float4* const src1 = NARR > 1 ? a1 + e : nullptr;
                    const int nc = (c1 - c0 + 2) * R;
                    for (int i = lane >> 3; i < nc; i += 16) {
                        uint2 w[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) w[u] = i + u * 4 < nc ? U.cell[i + u * 4] : make_uint2(0u, 0u);
                        bool more = false;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t n = w[u].y >> 16, d = dst + (w[u].y & 0xFFFFu) * 16u;
                            if (e < n) {
                                cp_async16(d, src0 + w[u].x);
                                if (NARR > 1) cp_async16(d + CAP * 16u, src1 + w[u].x);
                            }
                            if (e + 8u < n) {
                                cp_async16(d + 128u, src0 + w[u].x + 8);
                                if (NARR > 1) cp_async16(d + 128u + CAP * 16u, src1 + w[u].x + 8);
                            }
                            more |= n > 16u;
                        }
                        if (more) {
                            for (int u = 0; u < 4; ++u) {
                                const uint32_t n = w[u].y >> 16, d = dst + (w[u].y & 0xFFFFu) * 16u;
                                for (uint32_t p = 16u; e + p < n; p += 8u) {
                                    cp_async16(d + p * 16u, src0 + w[u].x + p);
                                    if (NARR > 1) cp_async16(d + (p + CAP) * 16u, src1 + w[u].x + p);
                                }
                            }
                        }
                    }
                }
                hand_over();
            }
            c0 = c1;
            if (SPLIT && c0 >= ncell && other && !again) {
                if (!end(true)) return false;
                slow = !slow;
                again = true;
                c0 = 0;
            }
        }
    }
    if (!end(false)) return false;
    cp_async_wait_all();
    return true;
}

// A consumer warp's wait for unit number `use`; false if it gave up.
__device__ __forceinline__ bool unit_wait(BrickShared& S, uint32_t use, uint32_t* err) {
    const bool ok = mbar_wait_bounded(reinterpret_cast<uint64_t*>(&S.full[use & 1u]), (use >> 1) & 1u);
    if (!ok) atomicOr(err, DEV_ERR_MBAR_TIMEOUT);
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void unit_release(BrickShared& S, uint32_t use) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(reinterpret_cast<uint64_t*>(&S.empty[use & 1u]));
}

// What ends a consumer's loop over the units of one kind.
constexpr int UNITS_DONE = 0, UNITS_MORE = 1, UNITS_GAVE_UP = 2;
__device__ __forceinline__ int units_end(BrickShared& S, uint32_t& use) {
    const int more = S.unit[use & 1u].more;
    unit_release(S, use++);
    return more ? UNITS_MORE : UNITS_DONE;
}
// The staged units, then those that are not, and so on while there are more. Returns false if a wait gave up.
template <class F>
__device__ __forceinline__ bool both_kinds(F&& units) {
    for (;;) {
        int r = units(std::true_type());
        if (r == UNITS_MORE) r = units(std::false_type());
        if (r != UNITS_MORE) return r == UNITS_DONE;
    }
}

// min(r^2 - h^2, 0) of a candidate: its sign bit says whether the candidate is in range (a NaN
// distance is not), minus its cube is the density term. The x and y differences run as a packed
// pair, which pays for rounding r^2 before h^2 comes off (folding h^2 into the first
// multiply-add saves the subtraction and loses up to 14% in the pressure's accuracy).
template <int DIMS>
__device__ __forceinline__ float density_term(const float4& pi, const float4& pj, float h2) {
    float dx, dy;
    f2_unpack(f2_sub(f2_pack(pi.x, pi.y), f2_pack(pj.x, pj.y)), dx, dy);
    float r2 = fmaf(dy, dy, dx * dx);
    if (DIMS == 3) {
        const float dz = pi.z - pj.z;
        r2 = fmaf(dz, dz, r2);
    }
    return fminf(r2 - h2, 0.0f);
}

// Recording (an adjoint's recomputation): each target's own part of its pair's list, as sorted
// indices, in the list's order, and its length (REC_SCAN where there is none or it is too long).
template <int R>
__device__ __forceinline__ void density_record(const BrickUnit& U, const KParams& kp, const PairTask& t, bool list,
                                               uint32_t nU, const float4& pA, const float4& pB, const float4* buf,
                                               const uint16_t* wlist) {
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u, quad = 0xFu << (lane & 28u);
    const size_t base = (size_t)*kp.rec_slot * kp.rec_n4;
    uint32_t n[2] = {0u, 0u};
    const uint32_t rounds = t.live && list ? (nU + 3u) >> 2 : 0u;
    for (uint32_t k = 0; __any_sync(0xffffffffu, k < rounds); ++k) {
        const uint32_t e = 4u * k + q;
        const bool some = k < rounds && e < nU;
        uint32_t g = 0;
        float4 pj = pA;
        if (some) {
            const uint32_t v = t.lo + (wlist[e] >> 4);
            pj = buf[v];
            int a = t.c * R, z = (t.c + 3) * R;  // the last cell that starts at or before v
            while (z - a > 1) {
                const int m = (a + z) >> 1;
                if (U.off[m] <= v) a = m;
                else z = m;
            }
            g = U.cell[a].x + (v - U.off[a]);
        }
#pragma unroll
        for (uint32_t w = 0; w < 2u; ++w) {
            const bool in = some && (w == 0u || t.two) && density_term<R == 9 ? 3 : 2>(w ? pB : pA, pj, kp.h2) < 0.0f;
            const uint32_t m = __ballot_sync(0xffffffffu, in) & quad, at = n[w] + (uint32_t)__popc(m & lanemask_lt());
            if (in && at < NBR_CAP) kp.rec_nbr[(base + t.gi + w) * NBR_CAP + at] = g;
            n[w] += (uint32_t)__popc(m);
        }
    }
    if (t.live && q < (t.two ? 2u : 1u)) {
        const uint32_t c = q ? n[1] : n[0];
        kp.rec_cnt[base + t.gi + q] = list && c <= NBR_CAP ? c : REC_SCAN;
    }
}

// Density + pressure for every particle of the occupied bricks, and the pairs' neighbour lists.
// Writes sorted position .w = density and sorted velocity .w = pressure, as
// clCalculateDensity does (libCL/phys/oclFluid3D.cl:189-199). A pair's four lanes walk every
// fourth candidate of its window. Whether a candidate is in range is kept as a bit per target
// (one funnel shift of the term's sign), and the lists are written from the bits afterwards.
// Every target meets itself (term h^6, one count); that term is taken off after the sum. A list
// lies in the 128 (a single: 64) entries of nbr that belong to its particles; entries are places
// in the window times 16 (bytes). nbr_meta of the pair's first particle: their number, or
// NBR_SCAN where there are more or the unit was not staged.
// Returns false if a wait gave up.
template <int DIMS, bool BATCH>
__device__ __forceinline__ bool density_brick_run(float4* s_buf, BrickShared& S, float4* __restrict__ spos,
                                                  float4* __restrict__ svel, const uint2* __restrict__ table,
                                                  const uint32_t* __restrict__ bricks, uint32_t* counters,
                                                  const KParams& kp, uint16_t* __restrict__ nbr,
                                                  uint32_t* __restrict__ nbr_meta, uint32_t* err) {
    constexpr int R = DIMS == 3 ? 9 : 3;
    constexpr int RC = DIMS == 3 ? 4 : 1;
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u;
    const int warp = threadIdx.x >> 5, consumers = (int)(blockDim.x >> 5) - 1;
    brick_init(S);
    const uint32_t n_bricks = __ldcg(counters);  // written by the bounds pass (an earlier kernel or phase)
    if (warp == consumers) {
        const bool ok = brick_produce<DIMS, BATCH, DENSITY_CAP, 1, false>(S, s_buf, spos, nullptr, table, bricks, n_bricks,
                                                                   &counters[1], kp, err);
        if (!ok) atomicExch(&counters[3], 1u);
        return ok;
    }
    uint16_t* wlist = reinterpret_cast<uint16_t*>(s_buf + 2 * DENSITY_CAP) + (warp * TASK_PAIRS + (lane >> 2)) * LIST_STRIDE;
    const uint32_t row = smem_addr(wlist);
    const float h2 = kp.h2;
    int turn = warp;  // tasks of eight pairs are dealt to the consumer warps in turn, across units
    for (uint32_t use = 0;; ++use) {
        if (!unit_wait(S, use, err)) {
            atomicExch(&counters[3], 1u);  // no lists for the rest: the force pass leaves them out
            return false;
        }
        const BrickUnit& U = S.unit[use & 1u];
        if (U.ncell == 0) break;
        const float4* buf = s_buf + (use & 1u) * DENSITY_CAP;
        const bool staged = U.staged != 0;
        const int tasks = (int)((U.npair + TASK_PAIRS - 1u) / TASK_PAIRS);
        for (; turn < tasks; turn += consumers) {
            const PairTask t = pair_task<R, RC>(U, (uint32_t)turn * TASK_PAIRS + (lane >> 2));
            const float4 pA = staged ? buf[t.self] : spos[t.gi];
            const float4 pB = staged ? buf[t.self + (t.two ? 1u : 0u)] : spos[t.gi + (t.two ? 1u : 0u)];
            float accA = 0.0f, accB = 0.0f;
            uint32_t cnt = 0;  // this lane's in-range candidates: A low, B high half
            uint32_t nU = 0;   // the pair's list entries so far
            const uint32_t cap = t.two ? 2u * NBR_CAP : NBR_CAP;
            // terms of one candidate; the signs go to the bits
            uint32_t mA = 0, mB = 0;
            auto candidate = [&](const float4& pj) {
                const float uA = density_term<DIMS>(pA, pj, h2), uB = density_term<DIMS>(pB, pj, h2);
                const uint64_t u = f2_pack(uA, uB);  // packed: half the issue slots
                f2_unpack(f2_fma(f2_mul(u, u), u, f2_pack(accA, accB)), accA, accB);
                mA = __funnelshift_l(__float_as_uint(uA), mA, 1);
                mB = __funnelshift_l(__float_as_uint(uB), mB, 1);
            };
            if (staged) {
                const uint32_t total = (t.len + 3u - q) >> 2;  // this lane's candidates
                uint32_t a = smem_addr(buf + t.lo + q), v0 = q * 16u;
                for (uint32_t i0 = 0; __any_sync(0xffffffffu, i0 < total); i0 += 32u) {
                    const uint32_t m = i0 < total ? min(32u, total - i0) : 0u;  // at most a word of bits
                    mA = mB = 0u;
#pragma unroll 4
                    for (uint32_t i = 0; i < m; ++i, a += 64u) candidate(lds_f4(a));
                    if (!t.two) mB = 0u;
                    cnt += (uint32_t)__popc(mA) + ((uint32_t)__popc(mB) << 16);
                    uint32_t either = mA | mB;
                    // places in the list: the counts of the pair's lanes before this one
                    const uint32_t own = (uint32_t)__popc(either);
                    uint32_t inc = own;
                    uint32_t v = __shfl_up_sync(0xffffffffu, inc, 1);
                    if (q >= 1u) inc += v;
                    v = __shfl_up_sync(0xffffffffu, inc, 2);
                    if (q >= 2u) inc += v;
                    uint32_t w = row + 2u * (nU + inc - own);
                    nU += __shfl_sync(0xffffffffu, inc, lane | 3u);
                    if (nU > cap) either = 0u;  // too many: no list
                    const uint32_t vk = v0 + (m - 1u) * 64u;  // the candidate at bit 0
                    while (either) {
                        const uint32_t bit = 31u - (uint32_t)__clz((int)either);
                        either ^= 1u << bit;
                        sts_u16(w, vk - bit * 64u);
                        w += 2u;
                    }
                    v0 += 32u * 64u;
                }
            } else {  // unstaged unit: candidates from global memory, no lists
                for (int i = t.c * R; i < (t.c + 3) * R; ++i) {
                    if (lane == 0u) atomicAdd(&S.progress, 1u);
                    const uint32_t n = U.off[i + 1] - U.off[i], first = U.cell[i].x;
                    for (uint32_t k = q; k < n; k += 4u) {
                        mA = mB = 0u;
                        candidate(spos[first + k]);
                        if ((cnt & 0xFFFFu) < 0x1000u) cnt += mA;  // "many" is all that is asked of the counts
                        if ((cnt >> 16) < 0x1000u) cnt += mB << 16;
                    }
                }
            }
#pragma unroll
            for (uint32_t m = 1; m < 4u; m <<= 1) {
                accA += __shfl_xor_sync(0xffffffffu, accA, m);
                accB += __shfl_xor_sync(0xffffffffu, accB, m);
                cnt += __shfl_xor_sync(0xffffffffu, cnt, m);
            }
            const bool list = staged && nU <= cap;
            // lane 0 of the four finishes target A, lane 1 target B
            if (t.live && (q == 0u || (q == 1u && t.two))) {
                const uint32_t gi = t.gi + q, n = q ? cnt >> 16 : cnt & 0xFFFFu;
                const float sum = -(q ? accB : accA) - kp.h2 * kp.h2 * kp.h2;  // without the target's own term
                const float4 pi = q ? pB : pA;
                float rho = kp.rho0, p = kp.p0;
                if (n > 3u) {  // the reference's count > 2 does not count the target
                    rho = fmaxf(1.0f, kp.mass * kp.kconst * sum);
                    p = kp.p0 + U.stiff * (rho - kp.rho0);
                }
                spos[gi] = make_float4(pi.x, pi.y, pi.z, rho);
                reinterpret_cast<float*>(svel)[4 * (size_t)gi + 3] = p;
                if (q == 0u) nbr_meta[gi] = list ? nU : NBR_SCAN;
            }
            __syncwarp();
            if (list && t.live)
                for (uint32_t ch = q; ch * 8u < nU; ch += 4u)
                    reinterpret_cast<uint4*>(nbr)[(size_t)t.gi * (NBR_CAP / 8) + ch] =
                        *reinterpret_cast<const uint4*>(wlist + ch * 8u);
            if (kp.rec_nbr) density_record<R>(U, kp, t, list, nU, pA, pB, buf, wlist);
            __syncwarp();
        }
        turn -= tasks;
        unit_release(S, use);
    }
    return true;
}

template <int DIMS, bool BATCH>
__global__ void __launch_bounds__(32 * DENSITY_CONSUMERS + 32, DENSITY_CTAS) k_density_brick(float4* __restrict__ spos,
                                                                 float4* __restrict__ svel,
                                                                 const uint2* __restrict__ table,
                                                                 const uint32_t* __restrict__ bricks,
                                                                 uint32_t* counters, KParams kp,
                                                                 uint16_t* __restrict__ nbr,
                                                                 uint32_t* __restrict__ nbr_meta, uint32_t* err) {
    extern __shared__ float4 s_buf[];
    __shared__ BrickShared S;
    density_brick_run<DIMS, BATCH>(s_buf, S, spos, svel, table, bricks, counters, kp, nbr, nbr_meta, err);
}

// Reciprocal and reciprocal square root with the hardware's approximations (1 and 2 ulp).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
constexpr uint32_t MIN_NORMAL = 0x00800000u;  // bits of the smallest normal float

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Pressure + viscosity contribution of one candidate (acc: pressure xyz, viscosity xyz), if it is
// in range. The w lanes hold density (positions) and pressure (velocities); ai = 1 / rho_i, aj =
// 1 / rho_j. The range test is one unsigned compare of r^2's bits, which also leaves out r = 0
// (the target itself, which its list holds, and coincident particles) and NaN.
template <int DIMS>
__device__ __forceinline__ void force_pair(const float4& pi, const float4& vi, float ai, const float4& pj,
                                           const float4& vj, float aj, float h, uint32_t thr, float* acc) {
    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = DIMS == 3 ? pi.z - pj.z : 0.0f;
    float r2 = fmaf(dy, dy, dx * dx);
    if (DIMS == 3) r2 = fmaf(dz, dz, r2);
    const float inv = rsqrt_approx(r2);
    const float hr = fmaf(-r2, inv, h);               // h - r
    const float cv = hr * (ai * aj);                   // (h - r) / (rho_i rho_j)
    const float sp = (vi.w + vj.w) * cv * (hr * inv);  // (p_i + p_j) (h - r)^2 / (rho_i rho_j r)
    if (__float_as_uint(r2) - MIN_NORMAL < thr) {
        acc[0] = fmaf(sp, dx, acc[0]);
        acc[1] = fmaf(sp, dy, acc[1]);
        if (DIMS == 3) acc[2] = fmaf(sp, dz, acc[2]);
        acc[3] = fmaf(vj.x - vi.x, cv, acc[3]);
        acc[4] = fmaf(vj.y - vi.y, cv, acc[4]);
        acc[5] = fmaf(vj.z - vi.z, cv, acc[5]);
    }
}

// clip_box_force with a particle on four lanes, lane l holding component l of its force: the two
// walls of the lane's axis (none for w, nor for z in 2D), and the sum of the walls' w terms
// (0 * magnitude) on lane 3. Whole warps; `live` lanes have a particle.
template <int DIMS>
__device__ __forceinline__ float clip_box_lane(const KParams& kp, const float4& box_min, const float4& box_max,
                                               const float4& pos, const float4& vel, float f, uint32_t l, bool live) {
    const float x = l == 0u ? pos.x : (l == 1u ? pos.y : pos.z);
    const float lo = l == 0u ? box_min.x : (l == 1u ? box_min.y : box_min.z);
    const float hi = l == 0u ? box_max.x : (l == 1u ? box_max.y : box_max.z);
    const float below = __fsub_rn(kp.radius, __fsub_rn(x, lo)), above = __fsub_rn(kp.radius, __fsub_rn(hi, x));
    const bool axis = live && l < (DIMS == 3 ? 3u : 2u);
    if (!__any_sync(0xffffffffu, axis && (below > 0.00001f || above > 0.00001f))) return f;
    const float v = l == 0u ? vel.x : (l == 1u ? vel.y : vel.z);
    float fw = 0.0f;
    if (axis) {
        add_wall(f, fw, 1.0f, below, v);
        add_wall(f, fw, -1.0f, above, v);
    }
    fw += __shfl_xor_sync(0xffffffffu, fw, 1);
    fw += __shfl_xor_sync(0xffffffffu, fw, 2);
    return l == 3u ? __fadd_rn(f, fw) : f;
}

// integrate_force with a particle on four lanes: the lane's component of the new velocity. The
// clamp's test on the length is made on its square (kp.v2_thresh), so that the root and the
// division are left to the particles that are clamped.
__device__ __forceinline__ float integrate_force_lane(const KParams& kp, float v, float f) {
    const float q = __fmul_rn(f, f);
    const int g = threadIdx.x & 28;
    const float f2 = __fadd_rn(__fadd_rn(__fadd_rn(__shfl_sync(0xffffffffu, q, g), __shfl_sync(0xffffffffu, q, g + 1)),
                                         __shfl_sync(0xffffffffu, q, g + 2)), __shfl_sync(0xffffffffu, q, g + 3));
    if (f2 >= kp.v2_thresh) f = __fmul_rn(f, __fdiv_rn(kp.vlimit, __fsqrt_rn(f2)));
    return __fadd_rn(v, __fmul_rn(f, kp.dt));
}

// The lane's part of a pair's state: component l of the two particles' force, velocity and position.
struct PairState {
    uint32_t oA, oB;  // the particles
    float fA, fB, vA, vB, pA, pB;
};

template <bool FUSED, bool COH>
__device__ __forceinline__ PairState pair_state(const PairTask& t, uint32_t l, const uint32_t* __restrict__ index,
                                                const float4* pos, const float4* vel, const float4* force) {
    PairState s{};
    s.oA = ld_phase<COH>(index + t.gi);
    s.oB = ld_phase<COH>(index + t.gi + (t.two ? 1u : 0u));
    s.fA = reinterpret_cast<const float*>(force + s.oA)[l];
    s.fB = reinterpret_cast<const float*>(force + s.oB)[l];
    if (FUSED) {
        s.vA = reinterpret_cast<const float*>(vel + s.oA)[l];
        s.vB = reinterpret_cast<const float*>(vel + s.oB)[l];
        s.pA = reinterpret_cast<const float*>(pos + s.oA)[l];
        s.pB = reinterpret_cast<const float*>(pos + s.oB)[l];
    }
    return s;
}

// Pressure and viscosity terms together, then the sums over the pair's lanes.
__device__ __forceinline__ void pair_sums(const KParams& kp, float cvisc, const float* accA, const float* accB, float (*f)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        f[0][k] = fmaf(kp.cpress, accA[k], cvisc * accA[3 + k]);
        f[1][k] = fmaf(kp.cpress, accB[k], cvisc * accB[3 + k]);
#pragma unroll
        for (uint32_t m = 1; m < 4u; m <<= 1) {
            f[0][k] += __shfl_xor_sync(0xffffffffu, f[0][k], m);
            f[1][k] += __shfl_xor_sync(0xffffffffu, f[1][k], m);
        }
    }
}

// Lane l takes component l of the pair's new state, target A and then target B.
template <int DIMS, bool FUSED>
__device__ __forceinline__ void pair_finish(const KParams& kp, const BrickUnit& U, const PairTask& t, uint32_t l, const PairState& s,
                                            const float (*f)[3], const float4& pA, const float4& pB, const float4& vA,
                                            const float4& vB, float4* __restrict__ pos, float4* __restrict__ vel,
                                            float4* __restrict__ force) {
    const float g = l == 0u ? kp.gravity.x : (l == 1u ? kp.gravity.y : (l == 2u ? kp.gravity.z : kp.gravity.w));
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const bool live = t.live && (w == 0 || t.two);
        const uint32_t o = w ? s.oB : s.oA;
        const float add = l == 0u ? f[w][0] : (l == 1u ? f[w][1] : f[w][2]);
        float F = l == 3u ? 0.0f : __fadd_rn(w ? s.fB : s.fA, __fmul_rn(add, kp.mass));
        if (FUSED) {
            F = clip_box_lane<DIMS>(kp, U.box_min, U.box_max, w ? pB : pA, w ? vB : vA, F, l, live);
            if (kp.rec_force && live) reinterpret_cast<float*>(kp.rec_force + o)[l] = F;
            const float v = integrate_force_lane(kp, w ? s.vB : s.vA, F);
            if (live) {
                reinterpret_cast<float*>(vel + o)[l] = v;
                reinterpret_cast<float*>(force + o)[l] = g;
                reinterpret_cast<float*>(pos + o)[l] = __fadd_rn(w ? s.pB : s.pA, __fmul_rn(v, kp.dt));
            }
        } else if (live) {
            reinterpret_cast<float*>(force + o)[l] = F;
        }
    }
}

// Forces (pressure + viscosity) for every particle of the occupied bricks
// (clCalculateForces, libCL/phys/oclFluid3D.cl:202-255). A pair's lane l evaluates entries 2 l and
// 2 l + 1 of each 8-entry chunk of the pair's list for both targets; the lists' first LIST_AHEAD
// chunks are read straight from global memory before anything else, the candidates lie in the
// staging. Targets without a list in a staged unit are scanned over their window by the whole
// warp; in an unstaged unit the pair's lanes scan the cells in global memory. With FUSED the
// clip-box, integrate-force, gravity and integrate-velocity stages follow in registers, a
// component per lane; otherwise the SPH force is added to force[index[i]] (with w = 0) as
// clCalculateForces does.
// COH: the sorted state and the lists were written earlier in the same launch, so the direct
// loads of them go through L2 only. Returns false if a wait gave up.
template <int DIMS, bool FUSED, bool BATCH, bool COH = false>
__device__ __forceinline__ bool force_brick_run(float4* s_buf, BrickShared& S, const float4* __restrict__ spos,
                                                const float4* __restrict__ svel, const uint32_t* __restrict__ index,
                                                float4* __restrict__ pos, float4* __restrict__ vel,
                                                float4* __restrict__ force, const uint2* __restrict__ table,
                                                const uint32_t* __restrict__ bricks, uint32_t* counters,
                                                const KParams& kp, const uint16_t* __restrict__ nbr,
                                                const uint32_t* __restrict__ nbr_meta, uint32_t* err) {
    constexpr int R = DIMS == 3 ? 9 : 3;
    constexpr int RC = DIMS == 3 ? 4 : 1;
    const uint32_t lane = threadIdx.x & 31u, l = lane & 3u;
    const int warp = threadIdx.x >> 5, consumers = (int)(blockDim.x >> 5) - 1;
    brick_init(S);
    // written by the bounds pass (an earlier kernel or phase); nothing to do where the density
    // pass gave up, which leaves particles without a list
    const uint32_t n_bricks = __ldcg(counters + 3) ? 0u : __ldcg(counters);
    if (warp == consumers)
        return brick_produce<DIMS, BATCH, FORCE_CAP, 2, true>(S, s_buf, spos, svel, table, bricks, n_bricks, &counters[2], kp,
                                                        err);
    const uint32_t thr = max(__float_as_uint(kp.r2_thresh), MIN_NORMAL) - MIN_NORMAL;
    int turn = warp;  // tasks of eight pairs are dealt to the consumer warps in turn, across units
    uint32_t use = 0;
    auto units = [&](auto kind) {
        constexpr bool staged = decltype(kind)::value;
        for (;; ++use) {
            if (!unit_wait(S, use, err)) return UNITS_GAVE_UP;
            const BrickUnit& U = S.unit[use & 1u];
            if (U.ncell == 0) return units_end(S, use);
            const float4* s_pos = s_buf + (use & 1u) * 2u * FORCE_CAP;
            const float4* s_vel = s_pos + FORCE_CAP;
            const float cvisc = U.cvisc;
            const int tasks = (int)((U.npair + TASK_PAIRS - 1u) / TASK_PAIRS);
            for (; turn < tasks; turn += consumers) {
                const PairTask t = pair_task<R, RC>(U, (uint32_t)turn * TASK_PAIRS + (lane >> 2));
                const uint32_t two = t.two ? 1u : 0u;
                if constexpr (staged) {
                    // everything from global memory at once: the list's length and first chunks (whatever
                    // its length), the targets' particles and, with those known, the lane's part of their state
                    const uint32_t meta = ld_phase<COH>(nbr_meta + t.gi);
                    const PairState st = pair_state<FUSED, COH>(t, l, index, pos, vel, force);
                    const uint32_t* list = reinterpret_cast<const uint32_t*>(nbr) + (size_t)t.gi * (NBR_CAP / 2) + l;
                    uint32_t ch[LIST_AHEAD];
#pragma unroll
                    for (uint32_t k = 0; k < LIST_AHEAD; ++k) ch[k] = ld_phase<COH>(list + 4u * k);
                    const float4 pA = s_pos[t.self], pB = s_pos[t.self + two], vA = s_vel[t.self], vB = s_vel[t.self + two];
                    const float aA = rcp_approx(pA.w), aB = rcp_approx(pB.w);
                    float accA[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, accB[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    auto both = [&](const float4& pj, const float4& vj) {
                        const float aj = rcp_approx(pj.w);
                        force_pair<DIMS>(pA, vA, aA, pj, vj, aj, kp.h, thr, accA);
                        force_pair<DIMS>(pB, vB, aB, pj, vj, aj, kp.h, thr, accB);
                    };
                    const bool scan = meta == NBR_SCAN;
                    const uint32_t n = scan ? 0u : meta, win = smem_addr(s_pos + t.lo);
                    auto entry = [&](uint32_t v) { both(lds_f4(win + v), lds_f4(win + v + FORCE_CAP * 16u)); };
                    for (uint32_t k0 = 2u * l; k0 < n; k0 += 8u * LIST_AHEAD) {
                        if (k0 >= 8u * LIST_AHEAD) {
#pragma unroll
                            for (uint32_t k = 0; k < LIST_AHEAD; ++k)
                                if (k0 + 8u * k < n) ch[k] = ld_phase<COH>(list + 4u * k + ((k0 >> 3) << 2));
                        }
#pragma unroll
                        for (uint32_t k = 0; k < LIST_AHEAD; ++k) {
                            if (k0 + 8u * k >= n) break;
                            entry(ch[k] & 0xFFFFu);
                            if (k0 + 8u * k + 1u < n) entry(ch[k] >> 16);
                        }
                    }
                    float f[2][3];
                    pair_sums(kp, cvisc, accA, accB, f);
                    // pairs without a list: the whole warp scans each one's window in turn
                    uint32_t pend = __ballot_sync(0xffffffffu, t.live && scan && l == 0u);
                    while (pend) {
                        const int src = __ffs((int)pend) - 1;
                        pend &= pend - 1u;
                        const uint32_t self = __shfl_sync(0xffffffffu, t.self, src), lo = __shfl_sync(0xffffffffu, t.lo, src),
                                       len = __shfl_sync(0xffffffffu, t.len, src), more = __shfl_sync(0xffffffffu, two, src);
#pragma unroll 1
                        for (uint32_t w = 0; w <= more; ++w) {
                            const float4 ps = s_pos[self + w], vs = s_vel[self + w];
                            const float as = rcp_approx(ps.w);
                            float a[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                            for (uint32_t j = lo + lane; j < lo + len; j += 32u)
                                force_pair<DIMS>(ps, vs, as, s_pos[j], s_vel[j], rcp_approx(s_pos[j].w), kp.h, thr, a);
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                float x = fmaf(kp.cpress, a[k], cvisc * a[3 + k]);
                                for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
                                if ((lane >> 2) == (uint32_t)src >> 2) {
                                    if (w) f[1][k] = x;
                                    else f[0][k] = x;
                                }
                            }
                        }
                    }
                    pair_finish<DIMS, FUSED>(kp, U, t, l, st, f, pA, pB, vA, vB, pos, vel, force);
                } else {
                    // with correctly rounded reciprocals of the densities (the staged targets take the
                    // hardware's, one unit in the last place off for one density in eight)
                    const PairState st = pair_state<FUSED, COH>(t, l, index, pos, vel, force);
                    const float4 pA = ld_phase<COH>(spos + t.gi), pB = ld_phase<COH>(spos + t.gi + two);
                    const float4 vA = ld_phase<COH>(svel + t.gi), vB = ld_phase<COH>(svel + t.gi + two);
                    const float aA = __frcp_rn(pA.w), aB = __frcp_rn(pB.w);
                    float accA[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, accB[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    for (int i = t.c * R; i < (t.c + 3) * R; ++i) {
                        if (lane == 0u) atomicAdd(&S.progress, 1u);
                        const uint32_t cnt = U.off[i + 1] - U.off[i], first = U.cell[i].x;
                        if (l >= cnt) continue;
                        float4 pn = ld_phase<COH>(spos + first + l), vn = ld_phase<COH>(svel + first + l);  // loaded a candidate ahead
                        for (uint32_t j = l; j < cnt; j += 4u) {
                            const float4 pj = pn, vj = vn;
                            if (j + 4u < cnt) {
                                pn = ld_phase<COH>(spos + first + j + 4u);
                                vn = ld_phase<COH>(svel + first + j + 4u);
                            }
                            const float aj = __frcp_rn(pj.w);
                            force_pair<DIMS>(pA, vA, aA, pj, vj, aj, kp.h, thr, accA);
                            force_pair<DIMS>(pB, vB, aB, pj, vj, aj, kp.h, thr, accB);
                        }
                    }
                    __syncwarp();
                    float f[2][3];
                    pair_sums(kp, cvisc, accA, accB, f);
                    pair_finish<DIMS, FUSED>(kp, U, t, l, st, f, pA, pB, vA, vB, pos, vel, force);
                }
            }
            turn -= tasks;
            unit_release(S, use);
        }
    };
    return both_kinds(units);
}

template <int DIMS, bool FUSED, bool BATCH>
__global__ void __launch_bounds__(32 * FORCE_CONSUMERS + 32, FORCE_CTAS) k_force_brick(const float4* __restrict__ spos,
                                                               const float4* __restrict__ svel,
                                                               const uint32_t* __restrict__ index,
                                                               float4* __restrict__ pos,
                                                               float4* __restrict__ vel,
                                                               float4* __restrict__ force,
                                                               const uint2* __restrict__ table,
                                                               const uint32_t* __restrict__ bricks,
                                                               uint32_t* counters, KParams kp,
                                                               const uint16_t* __restrict__ nbr,
                                                               const uint32_t* __restrict__ nbr_meta,
                                                               uint32_t* err) {
    extern __shared__ float4 s_buf[];
    __shared__ BrickShared S;
    force_brick_run<DIMS, FUSED, BATCH>(s_buf, S, spos, svel, index, pos, vel, force, table, bricks, counters, kp, nbr,
                                        nbr_meta, err);
}

}  // namespace gbsph
