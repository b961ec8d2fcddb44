// fluid2d.cu -- the reference's 2D SPH model (double-density relaxation with an image-sampled
// wall field) on sm_103a: the oclFluid2D replacement behind the C ABI.
//
// The reference kernels of libCL/phys/oclFluid2D.cl are evaluated with the same arithmetic in
// the same order (round-to-nearest intrinsics, no FMA contraction, IEEE sqrt and division), so
// results reproduce the FP32 restatement bit for bit. The sort on the linear cell key is the
// counting sort of the 3D steps where it fits (16,384 particles in 40 x 36 cells: 16 us with
// the bounds and the reorder, 24 by two radix passes and four more launches), else the one-sweep
// radix sort. At the scene sizes of this model launches count, so the whole step is
// replayed as a CUDA graph: six kernels, eleven nodes before.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_fp16.h>

#include "count_sort.cuh"

using namespace gbsph;

namespace {

// libCL/phys/oclFluid2D.cl:121-133, the OpenCL C macros evaluated in float.
constexpr float kRestDensity = 82.0f;
constexpr float kStiffness = 0.08f;
constexpr float kNearStiffness = 0.1f;
constexpr float kSurfaceTension = 21.00035f;
constexpr float kPi = 3.1415926535f;
constexpr float kParticleRadius = 0.05f / 5;
constexpr uint32_t EMPTY2 = 0xFFFFFFFFu;

struct P2 {
    float px, py, vx, vy, mass, unused;
};

struct K2 {
    float dT, h, cW, cH, cellSize, m, psize;
    float kNorm, kNearNorm;
    int ncx, ncy;
    uint32_t n, table;
    int W, H;  // wall image size
    float r2_lo, r2_hi;  // len2 > 1e-7 and len2 < h, on the squares
};

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float len2(float x, float y) { return __fsqrt_rn(fa(fm(x, x), fm(y, y))); }
__device__ __forceinline__ float half_round(float x) { return __half2float(__float2half_rn(x)); }

// read_imagef with normalised coordinates, linear filtering and clamp-to-edge (OpenCL C spec).
__device__ __forceinline__ float4 sample(const float4* __restrict__ img, int W, int H, float s, float t) {
    const float u = fs(fm(s, (float)W), 0.5f), v = fs(fm(t, (float)H), 0.5f);
    const float fu = floorf(u), fv = floorf(v);
    const float a = fs(u, fu), b = fs(v, fv);
    int i0 = (int)fu, j0 = (int)fv;
    int i1 = i0 + 1, j1 = j0 + 1;
    i0 = min(max(i0, 0), W - 1);
    i1 = min(max(i1, 0), W - 1);
    j0 = min(max(j0, 0), H - 1);
    j1 = min(max(j1, 0), H - 1);
    const float w00 = fm(fs(1.f, a), fs(1.f, b)), w10 = fm(a, fs(1.f, b)), w01 = fm(fs(1.f, a), b), w11 = fm(a, b);
    const float4 t00 = img[(size_t)j0 * W + i0], t10 = img[(size_t)j0 * W + i1];
    const float4 t01 = img[(size_t)j1 * W + i0], t11 = img[(size_t)j1 * W + i1];
    float4 o;
    o.x = fa(fa(fa(fm(w00, t00.x), fm(w10, t10.x)), fm(w01, t01.x)), fm(w11, t11.x));
    o.y = fa(fa(fa(fm(w00, t00.y), fm(w10, t10.y)), fm(w01, t01.y)), fm(w11, t11.y));
    o.z = fa(fa(fa(fm(w00, t00.z), fm(w10, t10.z)), fm(w01, t01.z)), fm(w11, t11.z));
    o.w = fa(fa(fa(fm(w00, t00.w), fm(w10, t10.w)), fm(w01, t01.w)), fm(w11, t11.w));
    return o;
}

// clAdvanceState (libCL/phys/oclFluid2D.cl:173-182) and clHash (:61-69) of particle i. Cell
// coordinates are clamped to the grid.
__device__ __forceinline__ uint32_t advance_hash(P2* __restrict__ st, float2* __restrict__ prev, const K2& k, uint32_t i) {
    P2 p = st[i];
    prev[i] = make_float2(p.px, p.py);
    p.vx = fa(p.vx, fm(0.0f, k.dT));
    p.vy = fa(p.vy, fm(-9.81f, k.dT));
    p.px = fa(p.px, fm(p.vx, k.dT));
    p.py = fa(p.py, fm(p.vy, k.dT));
    st[i] = p;
    const int gx = min(max((int)floorf(fd(p.px, k.cellSize)), 0), k.ncx - 1);
    const int gy = min(max((int)floorf(fd(p.py, k.cellSize)), 0), k.ncy - 1);
    return (uint32_t)(gy * k.ncx + gx);
}

// Counting sort: key, and a place among the cell's particles (count_sort.cuh).
__global__ void __launch_bounds__(256) k2_advance_count(P2* __restrict__ st, float2* __restrict__ prev, uint32_t* __restrict__ keys,
                                                        uint32_t* __restrict__ places, uint32_t* __restrict__ count, K2 k) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= k.n) return;
    const uint32_t key = advance_hash(st, prev, k, i);
    keys[i] = key;
    places[i] = atomicAdd(count + key, 1u);
}

// Counting sort: sorted keys, permutation and clReorder (libCL/phys/oclFluid2D.cl:71-76), a slot's
// particle behind those of its cell with smaller ids; the counts are zero again afterwards.
__global__ void __launch_bounds__(256) k2_order(const uint2* __restrict__ slots, const uint2* __restrict__ table,
                                                const P2* __restrict__ st, uint32_t* __restrict__ keys, uint32_t* __restrict__ index,
                                                P2* __restrict__ srt, uint32_t* __restrict__ count, K2 k, uint32_t* err) {
    const uint32_t s = blockIdx.x * 256u + threadIdx.x;
    if (s >= k.n) return;
    const uint2 me = slots[s];
    const uint2 cell = me.x < k.table ? table[me.x] : make_uint2(0u, 0u);
    if (cell.y > k.n || s < cell.x || s >= cell.y) {  // a table that does not fit the keys: never write out of range
        atomicOr(err, DEV_ERR_KEY_RANGE);
        return;
    }
    const P2 p = st[me.y];
    uint32_t d = cell.x;
#pragma unroll 4
    for (uint32_t t = cell.x; t < cell.y; ++t) d += slots[t].y < me.y ? 1u : 0u;
    keys[s] = me.x;
    index[d] = me.y;
    srt[d] = p;
    if (s == cell.x) count[me.x] = 0u;
}

// Radix sort (where the counting sort does not fit): keys and the digit histogram of the sort.
__global__ void k2_advance_hash(P2* __restrict__ st, float2* __restrict__ prev, uint32_t* __restrict__ keys,
                                uint32_t* __restrict__ hist, K2 k, int end_bit) {
    __shared__ uint32_t s_h[SORT_MAX_PASSES * SORT_RADIX];
    for (int i = threadIdx.x; i < SORT_MAX_PASSES * SORT_RADIX; i += blockDim.x) s_h[i] = 0;
    __syncthreads();
    const int passes = sort_passes(0, end_bit);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < k.n; i += gridDim.x * blockDim.x) {
        const uint32_t key = advance_hash(st, prev, k, i);
        keys[i] = key;
        for (int q = 0; q < passes; ++q) {
            const int shift = q * SORT_RADIX_BITS;
            const int bits = min(SORT_RADIX_BITS, end_bit - shift);
            atomicAdd(&s_h[q * SORT_RADIX + ((key >> shift) & ((1u << bits) - 1u))], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * SORT_RADIX; i += blockDim.x)
        if (s_h[i]) atomicAdd(&hist[i], s_h[i]);
}

// clReorder (libCL/phys/oclFluid2D.cl:71-76): 24-byte particles.
__global__ void k2_reorder(const uint32_t* __restrict__ index, const P2* __restrict__ st, P2* __restrict__ srt, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) srt[i] = st[index[i]];
}

// clUpdateState (libCL/phys/oclFluid2D.cl:329-339) of particle o, relaxed to (rx, ry).
__device__ __forceinline__ void update_state(P2* __restrict__ st, const float2* __restrict__ prev, uint32_t o, float rx, float ry,
                                             const K2& k) {
    const float2 pr = prev[o];
    float dx = fs(rx, pr.x), dy = fs(ry, pr.y);
    const float l = len2(dx, dy);
    const float cap = fm(4.0f, k.psize);
    const float lim = (cap < l) ? cap : l;  // min(l, 4 * particleSize) with the restatement's NaN rule
    dx = fd(fm(dx, lim), l);
    dy = fd(fm(dy, lim), l);
    P2 p = st[o];
    p.vx = fd(dx, k.dT);
    p.vy = fd(dy, k.dT);
    p.px = fa(pr.x, dx);
    p.py = fa(pr.y, dy);
    st[o] = p;
}

// The neighbour loops of clComputePressure / clComputePosition visit cells x (outer), y (inner)
// of the 3 x 3 around a particle and the particles of each cell in sorted order, summing in
// that order. A warp takes T consecutive sorted particles and
//  - for each cell among them goes through the candidates of the nine cells, 32 at a time in
//    the reference's order, keeps those within h of the box around the cell's targets (no
//    target is nearer to a candidate than the box, in rounded arithmetic as well: every
//    operation of the distance is monotone), tests the kept ones against each target and
//    appends those in range to the target's list;
//  - then computes the terms of all lists, a lane each, and a lane per target adds them in order.
// A target with more in range than its list holds takes the warp to itself, through the candidates
// again, the list as a buffer whose terms are computed side by side whenever it is half full. (With
// the terms computed where they were found and added by shuffles, 1,024 particles at half the
// spacing took 164 us a step, 62 now; 16,384 particles 257 and 206. Adding all lists up whenever
// one was full 124, but 2 to 5 % more for every scene without such targets.)
// At 16,384 particles (the default scene) a warp for every particle, its candidates' terms computed
// wherever one of 32 was in range and added by shuffles, took 33 us for the pressures and 43 for
// the positions; this takes 15 and 18. Bound by latency: 27 warps an SM (issue
// 60% of cycles), each a chain of table, candidates, lists, terms and sums. All nine cells instead of those in reach: 136 us for two
// steps instead of 102.
// T: 4, or 2 or 1 where few particles leave the chip idle and only the length of a warp's chain
// counts. Us a step with 1 / 2 / 4: 2,025 particles 34.5 / 36.9 / 41.6, 4,096 35.4 / 38.6 / 42.4, 5,184 38.0 / 39.5 / 43.5,
// 8,100 47.4 / 41.3 / 44.5, 10,000 50.6 / 43.6 / 46.2, 12,100 57.3 / 48.4 / 46.6; eight at 16,384: 113 for two steps.
constexpr int SEARCH_WARPS = 4;           // per CTA
constexpr uint32_t SEARCH_ONE = 4096, SEARCH_TWO = 8192;  // particles up to which T is 1, 2
constexpr uint32_t LIST2 = 64;            // entries of a target's list
constexpr uint32_t HELD2 = 128;           // candidates held before they are tested, a multiple of 32

template <class TERM, int T>
struct Search2 {
    float2 xy[HELD2];
    uint32_t id[HELD2];
    uint32_t base[32];
    uint32_t j[T][LIST2];
    TERM term[T][LIST2];  // first the neighbour's distance (x, y), then its terms
};

// Whether particle j at distance (dx, dy) is a neighbour of particle i: r > 1e-7 and r < h.
__device__ __forceinline__ bool near2(const K2& k, float dx, float dy) {
    const float r2 = fa(fm(dx, dx), fm(dy, dy));
    return r2 >= k.r2_lo && r2 < k.r2_hi;
}

// The candidates of cell (cx, cy) that may be within h of the box (xl..xh, yl..yh): calls
// f(j, px, py, last) for 32 at a time (j = EMPTY2 beyond the last), in the reference's order, by
// the whole warp. Cells are 2 h wide, so that a box in one cell reaches four to six of the nine;
// the slack is a hundred times what rounding can move a particle against its cell's bounds, and
// the cells at the grid's edges hold what lies beyond as well.
template <class F>
__device__ __forceinline__ void for_candidates2(const K2& k, int cx, int cy, const P2* __restrict__ srt,
                                                const uint2* __restrict__ table, uint32_t* __restrict__ s_base, float xl, float xh, float yl,
                                                float yh, F&& f) {
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, lt = lanemask_lt();
    uint32_t n = 0, first = 0;
    if (lane < 9) {
        const int x = cx - 1 + (int)lane / 3, y = cy - 1 + (int)lane % 3;
        // out of reach beyond cell c of m: the box lies outside [c, c + 1] cells, give or take h
        auto far = [&](int c, int m, float lo, float hi) {
            const float from = (float)c * k.cellSize, to = from + k.cellSize, reach = k.h + 1e-5f * (k.h + to);
            return (c > 0 && from - hi > reach) || (c < m - 1 && lo - to > reach);
        };
        if (x >= 0 && x < k.ncx && y >= 0 && y < k.ncy && !far(x, k.ncx, xl, xh) && !far(y, k.ncy, yl, yh)) {
            const uint2 e = table[y * k.ncx + x];
            if (e.x <= e.y && e.y <= k.n) {  // not empty, and never out of range
                first = e.x;
                n = e.y - e.x;
            }
        }
    }
    uint32_t off = n;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const uint32_t o = __shfl_up_sync(FULL, off, d);
        if ((int)lane >= d) off += o;
    }
    const uint32_t total = __shfl_sync(FULL, off, 8), some = __ballot_sync(FULL, n != 0);
    off -= n;
    __syncwarp();
    if (n) s_base[__popc(some & lt)] = first - off;
    __syncwarp();
    uint32_t seen = 0;
    auto fetch = [&](uint32_t base, float& px, float& py) -> uint32_t {
        const uint32_t heads = __reduce_or_sync(FULL, n && off - base < 32u ? 1u << (off - base) : 0u);
        const uint32_t r = seen + (uint32_t)__popc(heads & (lt | 1u << lane)) - 1u;
        seen += (uint32_t)__popc(heads);
        if (base + lane >= total) return EMPTY2;
        const uint32_t j = base + lane + s_base[r];
        px = srt[j].px;
        py = srt[j].py;
        return j;
    };
    float px = 0.f, py = 0.f, ax = 0.f, ay = 0.f;
    uint32_t j = fetch(0, px, py), next = EMPTY2;
    for (uint32_t base = 0; base < total; base += 32, j = next, px = ax, py = ay) {
        if (base + 32 < total) next = fetch(base + 32, ax, ay);
        f(j, px, py, base + 32 >= total);
    }
}

// Fills the lists of the warp's targets; lane t's `count` is that of target t (may exceed LIST2).
template <class TERM, int T>
__device__ __forceinline__ uint32_t search2(Search2<TERM, T>& S, const K2& k, uint32_t first, bool live, float px, float py,
                                            const P2* __restrict__ srt, const uint2* __restrict__ table) {
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, lt = lanemask_lt();
    const int gx = (int)floorf(fd(px, k.cellSize)), gy = (int)floorf(fd(py, k.cellSize));
    uint32_t count = 0;
    for (uint32_t left = __ballot_sync(FULL, live); left;) {
        const int lead = __ffs(left) - 1;
        const int cx = __shfl_sync(FULL, gx, lead), cy = __shfl_sync(FULL, gy, lead);
        const uint32_t group = __ballot_sync(FULL, live && gx == cx && gy == cy);
        left &= ~group;
        const bool in = (group >> lane) & 1u;
        const float x0 = __shfl_sync(FULL, px, lead), y0 = __shfl_sync(FULL, py, lead);
        const float xl = warp_min(in ? px : x0), xh = warp_max(in ? px : x0), yl = warp_min(in ? py : y0), yh = warp_max(in ? py : y0);
        uint32_t held = 0;
        auto test = [&]() {
            if (held + lane < ((held + 31u) & ~31u)) S.xy[held + lane].x = INFINITY;  // never in range
            __syncwarp();
            for (uint32_t g = group; g; g &= g - 1) {
                const int t = __ffs(g) - 1;
                const float x = __shfl_sync(FULL, px, t), y = __shfl_sync(FULL, py, t);
                const uint32_t self = first + (uint32_t)t;
                uint32_t c = __shfl_sync(FULL, count, t);
                for (uint32_t p = 0; p < held; p += 32) {
                    const float2 q = S.xy[p + lane];
                    const uint32_t j = S.id[p + lane];
                    const float dx = fs(q.x, x), dy = fs(q.y, y);
                    const bool hit = near2(k, dx, dy) && j != self;
                    const uint32_t m = __ballot_sync(FULL, hit), at = c + (uint32_t)__popc(m & lt);
                    c += (uint32_t)__popc(m);
                    if (hit && at < LIST2) {
                        S.j[t][at] = j;
                        S.term[t][at].x = dx;
                        S.term[t][at].y = dy;
                    }
                }
                if ((int)lane == t) count = c;
            }
            __syncwarp();
            held = 0;
        };
        for_candidates2(k, cx, cy, srt, table, S.base, xl, xh, yl, yh, [&](uint32_t j, float qx, float qy, bool) {
            const float dx = fmaxf(fmaxf(fs(xl, qx), fs(qx, xh)), 0.f), dy = fmaxf(fmaxf(fs(yl, qy), fs(qy, yh)), 0.f);
            const bool keep = j != EMPTY2 && fa(fm(dx, dx), fm(dy, dy)) < k.r2_hi;
            const uint32_t m = __ballot_sync(FULL, keep);
            if (keep) {
                const uint32_t at = held + (uint32_t)__popc(m & lt);
                S.xy[at] = make_float2(qx, qy);
                S.id[at] = j;
            }
            held += (uint32_t)__popc(m);
            if (held > HELD2 - 32) test();
        });
        if (held) test();
    }
    __syncwarp();
    return count;
}

// Calls f(t, entry) for every entry of the lists, a lane each (lane t's `n` entries of target t).
template <int T, class F>
__device__ __forceinline__ void for_entries2(uint32_t n, F&& f) {
    uint32_t before[T + 1];
    before[0] = 0;
#pragma unroll
    for (int t = 0; t < T; ++t) before[t + 1] = before[t] + __shfl_sync(0xffffffffu, n, t);
    for (uint32_t e = threadIdx.x & 31u; e < before[T]; e += 32) {
        int t = 0;
        uint32_t at = e;
#pragma unroll
        for (int q = 1; q < T; ++q)
            if (e >= before[q]) {
                t = q;
                at = e - before[q];
            }
        f(t, at);
    }
    __syncwarp();
}

struct Pressure2 {
    // the terms of a neighbour at distance r
    static __device__ __forceinline__ float2 term(const K2& k, float dx, float dy) {
        const float a = fs(1.f, fd(len2(dx, dy), k.h));
        return make_float2(fm(fm(fm(fm(k.m, a), a), a), k.kNorm), fm(fm(fm(fm(fm(k.m, a), a), a), a), k.kNearNorm));
    }
};

// clComputePressure (libCL/phys/oclFluid2D.cl:185-245).
template <int T>
__global__ void __launch_bounds__(32 * SEARCH_WARPS) k2_pressure(const P2* __restrict__ srt, float4* __restrict__ ps,
                                                                 const uint2* __restrict__ table,
                                                                 const float4* __restrict__ bstate, K2 k) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ Search2<float2, T> shared[SEARCH_WARPS];
    Search2<float2, T>& S = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, first = (blockIdx.x * SEARCH_WARPS + (threadIdx.x >> 5)) * T, i = first + lane;
    const bool live = lane < T && i < k.n;
    if (first >= k.n) return;  // whole warps
    const float px = live ? srt[i].px : 0.f, py = live ? srt[i].py : 0.f;
    const uint32_t count = search2<float2, T>(S, k, first, live, px, py, srt, table);
    for_entries2<T>(count <= LIST2 ? count : 0u, [&](int t, uint32_t e) {
        const float2 d = S.term[t][e];
        S.term[t][e] = Pressure2::term(k, d.x, d.y);
    });
    float density = 0.f, nearDensity = 0.f;
    if (live) {
        const float4 wall = sample(bstate, k.W, k.H, fd(px, k.cW), fd(py, k.cH));
        if (wall.x != 0.f) {
            density = fa(density, wall.x);
            nearDensity = fa(nearDensity, wall.y);
        }
        if (count <= LIST2) {
#pragma unroll 4
            for (uint32_t e = 0; e < count; ++e) {
                const float2 v = S.term[lane][e];
                density = fa(density, v.x);
                nearDensity = fa(nearDensity, v.y);
            }
        }
    }
    for (uint32_t more = __ballot_sync(FULL, live && count > LIST2); more; more &= more - 1) {
        const int t = __ffs(more) - 1;
        const uint32_t self = first + (uint32_t)t;
        const float x = __shfl_sync(FULL, px, t), y = __shfl_sync(FULL, py, t);
        uint32_t n = 0;
        for_candidates2(k, (int)floorf(fd(x, k.cellSize)), (int)floorf(fd(y, k.cellSize)), srt, table, S.base, x, x, y, y,
                        [&](uint32_t j, float qx, float qy, bool last) {
                            const float dx = fs(qx, x), dy = fs(qy, y);
                            const bool hit = j != EMPTY2 && j != self && near2(k, dx, dy);
                            const uint32_t m = __ballot_sync(FULL, hit);
                            if (hit) S.term[t][n + (uint32_t)__popc(m & lanemask_lt())] = make_float2(dx, dy);
                            n += (uint32_t)__popc(m);
                            if (n <= LIST2 - 32 && !last) return;
                            __syncwarp();
                            for (uint32_t e = lane; e < n; e += 32) S.term[t][e] = Pressure2::term(k, S.term[t][e].x, S.term[t][e].y);
                            __syncwarp();
                            if ((int)lane == t) {
#pragma unroll 4
                                for (uint32_t e = 0; e < n; ++e) {
                                    density = fa(density, S.term[t][e].x);
                                    nearDensity = fa(nearDensity, S.term[t][e].y);
                                }
                            }
                            __syncwarp();
                            n = 0;
                        });
    }
    if (live)
        ps[i] = make_float4(density, nearDensity, fm(kStiffness, fs(density, fm(k.m, kRestDensity))),
                            fm(kNearStiffness, nearDensity));
}

struct Position2 {
    // displacements (away by pressure: x, y; towards by surface tension: z, w)
    static __device__ __forceinline__ float4 term(const K2& k, float dt2, float tension, const float4& si, const float4& sj, float dx,
                                                  float dy) {
        const float r = len2(dx, dy);
        const float a = fs(1.f, fd(r, k.h));
        const float near = fm(fm(fm(fm(fa(si.w, sj.w), a), a), a), k.kNearNorm);
        const float far = fm(fm(fm(fa(si.z, sj.z), a), a), k.kNorm);
        const float d = fd(fm(dt2, fa(near, far)), 2.f);
        const float rm = fm(r, k.m);
        const float surf = fd(fm(tension, fa(fm(fm(fm(a, a), a), k.kNearNorm), fm(fm(a, a), k.kNorm))), 2.f);
        return make_float4(fd(fm(dx, d), rm), fd(fm(dy, d), rm), fm(surf, dx), fm(surf, dy));
    }
};

// clComputePosition (libCL/phys/oclFluid2D.cl:247-326) and, as it concerns the particle alone,
// clUpdateState. The reference's viscosity term uses vel_j - vel_j (:299), which is zero, so
// it never contributes and is not evaluated here.
template <int T>
__global__ void __launch_bounds__(32 * SEARCH_WARPS) k2_position(const P2* __restrict__ srt, const float4* __restrict__ ps,
                                                                 float2* __restrict__ relaxed, const uint2* __restrict__ table,
                                                                 const float4* __restrict__ bstate,
                                                                 const float4* __restrict__ bvec, P2* __restrict__ st,
                                                                 const float2* __restrict__ prev,
                                                                 const uint32_t* __restrict__ index, K2 k) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ Search2<float4, T> shared[SEARCH_WARPS];
    Search2<float4, T>& S = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, first = (blockIdx.x * SEARCH_WARPS + (threadIdx.x >> 5)) * T, i = first + lane;
    const bool live = lane < T && i < k.n;
    if (first >= k.n) return;  // whole warps
    const float px = live ? srt[i].px : 0.f, py = live ? srt[i].py : 0.f;
    const float dt2 = fm(k.dT, k.dT), tension = fm(fm(dt2, fd(kSurfaceTension, k.m)), k.m);
    const uint32_t count = search2<float4, T>(S, k, first, live, px, py, srt, table);
    for_entries2<T>(count <= LIST2 ? count : 0u, [&](int t, uint32_t e) {
        const float4 d = S.term[t][e];
        S.term[t][e] = Position2::term(k, dt2, tension, ps[first + t], ps[S.j[t][e]], d.x, d.y);
    });
    float rx = px, ry = py;
    if (live && count <= LIST2) {
#pragma unroll 4
        for (uint32_t e = 0; e < count; ++e) {
            const float4 v = S.term[lane][e];
            rx = fa(fs(rx, v.x), v.z);
            ry = fa(fs(ry, v.y), v.w);
        }
    }
    for (uint32_t more = __ballot_sync(FULL, live && count > LIST2); more; more &= more - 1) {
        const int t = __ffs(more) - 1;
        const uint32_t self = first + (uint32_t)t;
        const float x = __shfl_sync(FULL, px, t), y = __shfl_sync(FULL, py, t);
        const float4 si = ps[self];
        uint32_t n = 0;
        for_candidates2(k, (int)floorf(fd(x, k.cellSize)), (int)floorf(fd(y, k.cellSize)), srt, table, S.base, x, x, y, y,
                        [&](uint32_t j, float qx, float qy, bool last) {
                            const float dx = fs(qx, x), dy = fs(qy, y);
                            const bool hit = j != EMPTY2 && j != self && near2(k, dx, dy);
                            const uint32_t m = __ballot_sync(FULL, hit);
                            if (hit) {
                                const uint32_t at = n + (uint32_t)__popc(m & lanemask_lt());
                                S.j[t][at] = j;
                                S.term[t][at].x = dx;
                                S.term[t][at].y = dy;
                            }
                            n += (uint32_t)__popc(m);
                            if (n <= LIST2 - 32 && !last) return;
                            __syncwarp();
                            for (uint32_t e = lane; e < n; e += 32)
                                S.term[t][e] = Position2::term(k, dt2, tension, si, ps[S.j[t][e]], S.term[t][e].x, S.term[t][e].y);
                            __syncwarp();
                            if ((int)lane == t) {
#pragma unroll 4
                                for (uint32_t e = 0; e < n; ++e) {
                                    const float4 v = S.term[t][e];
                                    rx = fa(fs(rx, v.x), v.z);
                                    ry = fa(fs(ry, v.y), v.w);
                                }
                            }
                            __syncwarp();
                            n = 0;
                        });
    }
    if (!live) return;
    const float4 si = ps[i];
    const float4 wall = sample(bstate, k.W, k.H, fd(rx, k.cW), fd(ry, k.cH));
    if (wall.x != 0.f) {
        const float4 normal = sample(bvec, k.W, k.H, fd(rx, k.cW), fd(ry, k.cH));
        const float a = fs(1.f, fd(normal.z, k.h));
        const float near = fm(fm(fm(fm(fa(si.w, wall.w), a), a), a), k.kNearNorm);
        const float far = fm(fm(fm(fa(si.z, wall.z), a), a), k.kNorm);
        const float d = fd(fm(dt2, fa(near, far)), 2.f);
        rx = fa(rx, fd(fm(normal.x, d), k.m));
        ry = fa(ry, fd(fm(normal.y, d), k.m));
    }
    relaxed[i] = make_float2(rx, ry);
    update_state(st, prev, index[i], rx, ry, k);
}

// clComputeBorder (libCL/phys/oclFluid2D.cl:358-443), one thread per pixel.
__global__ void k2_border(const float4* __restrict__ mask, int w, int h, float4* __restrict__ vout,
                          float4* __restrict__ sout, K2 k, float s) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float pw = mask[(size_t)y * w + x].w;
    const int dW = (int)((double)fd(fm((float)w, k.h), k.cW) + 0.5);
    const int dH = (int)((double)fd(fm((float)h, k.h), k.cH) + 0.5);
    const float dX = fd(k.cW, (float)w), dY = fd(k.cH, (float)h);
    float dmin = 10000.f;
    float4 vec = make_float4(0.f, 0.f, 0.f, 0.f);
    float density = 0.f, nearDensity = 0.f;
    if (pw == 1.0f) {
        density = fm(fm(112.f, k.m), k.kNorm);
        nearDensity = fm(fm(112.f, k.m), k.kNearNorm);
        for (int i = max(x - dW, 0); i < min(x + dW, w); i++)
            for (int j = max(y - dH, 0); j < min(y + dH, h); j++) {
                if (mask[(size_t)j * w + i].w != 1.0f) {
                    const float dx = fs(fm((float)i, dX), fm((float)x, dX)), dy = fs(fm((float)j, dY), fm((float)y, dY));
                    const float r = len2(dx, dy);
                    if (r < dmin) {
                        vec.x = fd(dx, r);
                        vec.y = fd(dy, r);
                        vec.z = r;
                        dmin = r;
                    }
                }
            }
    } else {
        for (int i = max(x - dW, 0); i < min(x + dW, w); i++)
            for (int j = max(y - dH, 0); j < min(y + dH, h); j++) {
                if (mask[(size_t)j * w + i].w == 1.0f) {
                    const float dx = fs(fm((float)x, dX), fm((float)i, dX)), dy = fs(fm((float)y, dY), fm((float)j, dY));
                    const float r = len2(dx, dy);
                    if (r < k.h) {
                        const float a = fs(1.f, fd(r, k.h));
                        density = fa(density, fm(fm(fm(fm(fm(s, k.m), a), a), a), k.kNorm));
                        nearDensity = fa(nearDensity, fm(fm(fm(fm(fm(fm(s, k.m), a), a), a), a), k.kNearNorm));
                        if (r < dmin) {
                            vec.x = fd(dx, r);
                            vec.y = fd(dy, r);
                            vec.z = r;
                            dmin = r;
                        }
                    }
                }
            }
    }
    vout[(size_t)y * w + x] = make_float4(half_round(vec.x), half_round(vec.y), half_round(vec.z), half_round(vec.w));
    sout[(size_t)y * w + x] = make_float4(half_round(density), half_round(nearDensity),
                                          half_round(fm(kStiffness, fs(density, fm(k.m, kRestDensity)))),
                                          half_round(fm(kNearStiffness, nearDensity)));
}

int grid1(uint32_t n) { return (int)((n + 255) / 256); }

// clEmitter (libCL/phys/oclFluid2D.cl:342-352): particle emit+1 enters at x = 1 on one of
// four heights, with velocity (25, 1); the sixth field (`age` there) is set to 1.
__global__ void k2_emitter(P2* __restrict__ state, uint32_t n, uint32_t emit, float psize) {
    const uint32_t particle = blockIdx.x * blockDim.x + threadIdx.x;
    if (particle >= n) return;
    if (particle > emit && particle < emit + 2u) {
        P2 q = state[particle];
        q.px = 1.0f;
        q.py = __fadd_rn(14.0f, __fmul_rn((float)(particle % 4u * 12u), psize));
        q.vx = 25.0f;
        q.vy = 1.0f;
        q.unused = 1.0f;
        state[particle] = q;
    }
}

}  // namespace

struct gbsph_fluid2d_s {
    int device = 0;
    gbsph_fluid2d_params params{};
    bool compiled = false;
    size_t n = 128 * 128;
    void* state = nullptr;  // P2[n]
    bool state_owned = true;
    size_t state_count = 0;
    void* block = nullptr;  // internal per-particle arrays
    P2* sorted = nullptr;
    float4* pstate = nullptr;
    float2* relaxed = nullptr;
    float2* prev = nullptr;
    uint32_t *keys_a = nullptr, *keys_b = nullptr, *keys_c = nullptr, *vals_a = nullptr, *vals_b = nullptr, *index = nullptr;
    uint2* cells = nullptr;  // cell start, end: `table` entries (whole scan tiles allocated)
    uint32_t* count = nullptr;  // the counting sort's counts, behind them, zero between steps
    bool count_clean = false;
    uint32_t table = 0;
    float4* bstate = nullptr;  // wall images W x H
    float4* bvec = nullptr;
    int W = 256, Hh = 256;
    void* scratch = nullptr;
    uint32_t* err = nullptr;
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t gexec = nullptr;
    std::vector<char> gkey;
    std::string last_error;
};

namespace {

using H2 = gbsph_fluid2d_s;

void default_params2d(gbsph_fluid2d_params* p) {
    // clInitFluid, libCL/phys/oclFluid2D.cl:136-151 (vmax and B are never set there)
    std::memset(p, 0, sizeof(*p));
    const float kH = (22 * 0.05f / 5);
    p->dT = (float)0.00433333333;
    p->h = kH;
    p->containerW = (float)17.68;
    p->containerH = (float)15.76;
    p->cellSize = 2 * p->h;
    p->cellCountX = (int)((double)(p->containerW / p->cellSize) + 0.5);
    p->cellCountY = (int)((double)(p->containerH / p->cellSize) + 0.5);
    p->particleSize = kParticleRadius;
    p->particleMass = 0.7f;
    p->p0 = kRestDensity;
}

K2 make_k2(const H2* h) {
    const gbsph_fluid2d_params& p = h->params;
    K2 k;
    std::memset(&k, 0, sizeof(k));
    k.dT = p.dT;
    k.h = p.h;
    k.cW = p.containerW;
    k.cH = p.containerH;
    k.cellSize = p.cellSize;
    k.m = p.particleMass;
    k.psize = p.particleSize;
    // kNorm / kNearNorm are macros of the compile-time kH (libCL/phys/oclFluid2D.cl:129-133)
    const float kH = (22 * 0.05f / 5);
    k.kNorm = (20 / (2 * kPi * kH * kH));
    k.kNearNorm = (30 / (2 * kPi * kH * kH));
    k.ncx = p.cellCountX;
    k.ncy = p.cellCountY;
    k.n = (uint32_t)h->n;
    k.table = h->table;
    k.W = h->W;
    k.H = h->Hh;
    k.r2_lo = r2_threshold(std::nextafter(0.0000001f, 1.0f));
    k.r2_hi = r2_threshold(p.h);
    return k;
}

void invalidate2(H2* h) {
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    h->gexec = nullptr;
    h->gkey.clear();
}

int alloc_arrays2(H2* h, size_t n) {
    if (h->block) cudaFree(h->block);
    if (h->scratch) cudaFree(h->scratch);
    h->block = h->scratch = nullptr;
    const size_t n4 = (n + 63) & ~size_t(63);
    const size_t bytes = n4 * (24 + 16 + 8 + 8 + 6 * 4);
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->block, bytes));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->block, 0, bytes));
    char* p = (char*)h->block;
    h->pstate = (float4*)p;
    p += n4 * 16;
    h->sorted = (P2*)p;
    p += n4 * 24;
    h->relaxed = (float2*)p;
    p += n4 * 8;
    h->prev = (float2*)p;
    p += n4 * 8;
    uint32_t** arr[6] = {&h->keys_a, &h->keys_b, &h->keys_c, &h->vals_a, &h->vals_b, &h->index};
    for (auto a : arr) {
        *a = (uint32_t*)p;
        p += n4 * 4;
    }
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->scratch, sort_scratch_bytes((uint32_t)n)));
    return GBSPH_OK;
}

int alloc_state2(H2* h, size_t n) {
    if (h->state_owned && h->state) cudaFree(h->state);
    h->state = nullptr;
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->state, std::max<size_t>(n, 1) * 24));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->state, 0, std::max<size_t>(n, 1) * 24));
    h->state_owned = true;
    h->state_count = n;
    return GBSPH_OK;
}

int alloc_border2(H2* h, int w, int hh) {
    if (h->bstate) cudaFree(h->bstate);
    if (h->bvec) cudaFree(h->bvec);
    h->bstate = h->bvec = nullptr;
    const size_t bytes = (size_t)w * hh * sizeof(float4);
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->bstate, bytes));
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->bvec, bytes));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->bstate, 0, bytes));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->bvec, 0, bytes));
    h->W = w;
    h->Hh = hh;
    invalidate2(h);
    return GBSPH_OK;
}

int alloc_table2(H2* h) {
    const gbsph_fluid2d_params& p = h->params;
    const uint32_t t = (uint32_t)(p.cellCountX * p.cellCountY) / 256 * 256 + 256;
    if (h->cells && t == h->table) return GBSPH_OK;
    if (h->cells) cudaFree(h->cells);
    h->cells = nullptr;
    h->count = nullptr;
    const size_t words = count_words(t);
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->cells, words * 12));
    h->count = (uint32_t*)(h->cells + words);
    GBSPH_CUDA_TRY(&h->last_error, fill_now(h->cells, 0xFF, words * 8));
    GBSPH_CUDA_TRY(&h->last_error, fill_now(h->count, 0, words * 4));
    h->count_clean = true;
    h->table = t;
    invalidate2(h);
    return GBSPH_OK;
}

int bits_for2(uint64_t cells) {
    int b = 0;
    while (b < 32 && (1ull << b) < cells) b++;
    return std::max(b, 1);
}

#define RC2(x)                \
    do {                      \
        int _rc = (x);        \
        if (_rc) return _rc;  \
    } while (0)

int enqueue2(H2* h, const K2& k, cudaStream_t s) {
    const unsigned g = (unsigned)grid1(k.n);
    P2* state = (P2*)h->state;
    if (count_sort_fits(k.table, k.n)) {
        const uint32_t tiles = scan_tiles(k.table);
        uint32_t* sums = (uint32_t*)((char*)h->scratch + SORT_HEADER_BYTES);
        uint2* slots = (uint2*)h->vals_a;  // and vals_b behind it
        k2_advance_count<<<g, 256, 0, s>>>(state, h->prev, h->keys_a, h->keys_b, h->count, k);
        if (k.table <= SCAN_DIRECT) {
            k_scan_cells<4, true, true><<<tiles, SCAN_THREADS, 0, s>>>(h->count, h->cells, sums);
        } else if (scan_items(k.table) == 4) {
            k_tile_sums<4><<<tiles, SCAN_THREADS, 0, s>>>(h->count, sums);
            k_scan_cells<4, true, false><<<tiles, SCAN_THREADS, 0, s>>>(h->count, h->cells, sums);
        } else {
            k_tile_sums<16><<<tiles, SCAN_THREADS, 0, s>>>(h->count, sums);
            k_scan_cells<16, true, false><<<tiles, SCAN_THREADS, 0, s>>>(h->count, h->cells, sums);
        }
        k_scatter_ids<<<g, 256, 0, s>>>(h->keys_a, h->keys_b, h->cells, slots, k.n, h->err);
        k2_order<<<g, 256, 0, s>>>(slots, h->cells, state, h->keys_c, h->index, h->sorted, h->count, k, h->err);
        GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    } else {
        const int end_bit = bits_for2((uint64_t)h->params.cellCountX * h->params.cellCountY);
        const int P = sort_passes(0, end_bit);
        GBSPH_CUDA_TRY(&h->last_error, onesweep_prepare(h->scratch, k.n, P, s));
        const int blocks = std::max(1, std::min(grid1(k.n), num_sms() * 8));
        k2_advance_hash<<<blocks, 256, 0, s>>>(state, h->prev, h->keys_a, (uint32_t*)h->scratch, k, end_bit);
        GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
        OnesweepArgs a;
        a.keys_in = h->keys_a;
        a.keys_out = h->keys_c;
        a.vals_out = h->index;
        a.tmp_keys[0] = h->keys_b;
        a.tmp_vals[0] = h->vals_b;
        a.tmp_keys[1] = h->keys_a;
        a.tmp_vals[1] = h->vals_a;
        a.n = k.n;
        a.start_bit = 0;
        a.end_bit = end_bit;
        a.scratch = h->scratch;
        a.err = h->err;
        GBSPH_CUDA_TRY(&h->last_error, onesweep_passes(a, s));
        k2_reorder<<<g, 256, 0, s>>>(h->index, state, h->sorted, k.n);
        GBSPH_CUDA_TRY(&h->last_error, cudaMemsetAsync(h->cells, 0xFF, (size_t)k.table * 8, s));
        k_bounds_hash<<<g, 256, 0, s>>>(h->keys_c, k.n, h->cells, k.table, h->err);
        GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    }
    auto relax = [&](uint32_t targets, auto pressure, auto position) {
        const uint32_t per = targets * SEARCH_WARPS, blocks = (k.n + per - 1) / per;
        pressure<<<blocks, 32 * SEARCH_WARPS, 0, s>>>(h->sorted, h->pstate, h->cells, h->bstate, k);
        position<<<blocks, 32 * SEARCH_WARPS, 0, s>>>(h->sorted, h->pstate, h->relaxed, h->cells, h->bstate, h->bvec, state, h->prev, h->index,
                                                      k);
    };
    if (k.n <= SEARCH_ONE) relax(1, k2_pressure<1>, k2_position<1>);
    else if (k.n <= SEARCH_TWO) relax(2, k2_pressure<2>, k2_position<2>);
    else relax(4, k2_pressure<4>, k2_position<4>);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    return GBSPH_OK;
}

int validate2(H2* h) {
    const gbsph_fluid2d_params& p = h->params;
    const float v[9] = {p.dT, p.h, p.containerW, p.containerH, p.cellSize, p.particleSize, p.particleMass, p.p0, 0.f};
    for (float x : v)
        if (!std::isfinite(x)) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "parameters hold a NaN or infinity");
    if (!(p.cellSize > 0.f) || !(p.h > 0.f) || !(p.containerW > 0.f) || !(p.containerH > 0.f))
        return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "cellSize, h and the container must be > 0");
    if (p.cellCountX < 1 || p.cellCountY < 1 || (int64_t)p.cellCountX * p.cellCountY > (1 << 24))
        return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "cell counts must be in [1, 2^24] cells");
    return GBSPH_OK;
}

}  // namespace

extern "C" {

GBSPH_API int gbsph_fluid2d_default_params(gbsph_fluid2d_params* p) {
    if (!p) return GBSPH_ERR_ARGUMENT;
    default_params2d(p);
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_create(gbsph_fluid2d_t* out) {
    if (!out) return GBSPH_ERR_ARGUMENT;
    *out = nullptr;
    H2* h = new H2();
    int rc = GBSPH_OK;
    if (cudaGetDevice(&h->device) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    if (!rc && cudaMalloc(&h->err, 256) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    if (!rc && cudaMemset(h->err, 0, 256) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    if (!rc && cudaStreamCreateWithFlags(&h->cap_stream, cudaStreamNonBlocking) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    default_params2d(&h->params);
    if (!rc) rc = alloc_arrays2(h, h->n);
    if (!rc) rc = alloc_state2(h, h->n);
    if (!rc) rc = alloc_border2(h, 256, 256);
    if (!rc) rc = alloc_table2(h);
    if (rc) {
        cudaGetLastError();
        gbsph_fluid2d_destroy(h);
        return rc;
    }
    *out = h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_destroy(gbsph_fluid2d_t h) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    cudaSetDevice(h->device);
    invalidate2(h);
    if (h->state_owned && h->state) cudaFree(h->state);
    void* ptrs[6] = {h->block, h->scratch, h->cells, h->bstate, h->bvec, h->err};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (h->cap_stream) cudaStreamDestroy(h->cap_stream);
    delete h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_compile(gbsph_fluid2d_t h) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    default_params2d(&h->params);
    RC2(alloc_table2(h));
    h->compiled = true;
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_set_particle_count(gbsph_fluid2d_t h, size_t n) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (n == 0 || n > SORT_MAX_KEYS - SORT_TILE) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "bad particle count");
    if (!h->state_owned && h->state_count != n)
        return fail(&h->last_error, GBSPH_ERR_SIZE_MISMATCH, "borrowed state buffer does not hold n particles");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    invalidate2(h);
    h->n = n;
    RC2(alloc_arrays2(h, n));
    if (h->state_owned) RC2(alloc_state2(h, n));
    return GBSPH_OK;
}

GBSPH_API size_t gbsph_fluid2d_get_particle_count(gbsph_fluid2d_t h) { return h ? h->n : 0; }

GBSPH_API int gbsph_fluid2d_set_state_buffer(gbsph_fluid2d_t h, void* device_ptr, size_t count) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!device_ptr || (uintptr_t)device_ptr % 8) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "null or misaligned state buffer");
    if (count != h->n)
        return fail(&h->last_error, GBSPH_ERR_SIZE_MISMATCH,
                    "state buffer holds " + std::to_string(count) + " particles, count is " + std::to_string(h->n));
    if (h->state_owned && h->state) {
        cudaSetDevice(h->device);
        cudaFree(h->state);
    }
    h->state = device_ptr;
    h->state_owned = false;
    h->state_count = count;
    invalidate2(h);
    return GBSPH_OK;
}

GBSPH_API void* gbsph_fluid2d_get_buffer(gbsph_fluid2d_t h, int which, size_t* count) {
    if (!h) return nullptr;
    size_t c = h->n;
    void* p = nullptr;
    switch (which) {
        case GBSPH2D_BUF_STATE: p = h->state; break;
        case GBSPH2D_BUF_SORTED_STATE: p = h->sorted; break;
        case GBSPH2D_BUF_INDEX: p = h->index; break;
        case GBSPH2D_BUF_CELL: p = h->keys_c; break;
        case GBSPH2D_BUF_PRESSURE: p = h->pstate; break;
        case GBSPH2D_BUF_RELAXED: p = h->relaxed; break;
        case GBSPH2D_BUF_PREVIOUS: p = h->prev; break;
        case GBSPH2D_BUF_BORDER_STATE: p = h->bstate; c = (size_t)h->W * h->Hh; break;
        case GBSPH2D_BUF_BORDER_VECTOR: p = h->bvec; c = (size_t)h->W * h->Hh; break;
        default: return nullptr;
    }
    if (count) *count = c;
    return p;
}

GBSPH_API gbsph_fluid2d_params* gbsph_fluid2d_get_params(gbsph_fluid2d_t h) { return h ? &h->params : nullptr; }

GBSPH_API int gbsph_fluid2d_compute_border(gbsph_fluid2d_t h, const float* mask, int width, int height, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!mask || width < 1 || height < 1 || (int64_t)width * height > (1 << 26))
        return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "bad wall mask");
    RC2(validate2(h));
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    if (width != h->W || height != h->Hh) RC2(alloc_border2(h, width, height));
    const K2 k = make_k2(h);
    const gbsph_fluid2d_params& p = h->params;
    const float dX = p.containerW / width, dY = p.containerH / height;
    const float s = (float)((double)(dX * dY) / (2 * M_PI * (double)p.particleSize * (double)p.particleSize));
    const dim3 blk(16, 16), grd((width + 15) / 16, (height + 15) / 16);
    k2_border<<<grd, blk, 0, (cudaStream_t)stream>>>((const float4*)mask, width, height, h->bvec, h->bstate, k, s);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_emit(gbsph_fluid2d_t h, uint32_t emit, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!h->compiled) return fail(&h->last_error, GBSPH_ERR_NOT_COMPILED, "emit before compile()");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    k2_emitter<<<(unsigned)((h->n + 255) / 256), 256, 0, (cudaStream_t)stream>>>((P2*)h->state, (uint32_t)h->n, emit,
                                                                                h->params.particleSize);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_compute(gbsph_fluid2d_t h, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!h->compiled) return fail(&h->last_error, GBSPH_ERR_NOT_COMPILED, "compute() before compile()");
    RC2(validate2(h));
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    RC2(alloc_table2(h));
    const K2 k = make_k2(h);
    std::vector<char> key(sizeof(K2) + 2 * sizeof(void*));
    std::memcpy(key.data(), &k, sizeof(K2));
    std::memcpy(key.data() + sizeof(K2), &h->state, sizeof(void*));
    std::memcpy(key.data() + sizeof(K2) + sizeof(void*), &h->bstate, sizeof(void*));
    if (!h->gexec || key != h->gkey) {
        invalidate2(h);
        GBSPH_CUDA_TRY(&h->last_error, cudaStreamBeginCapture(h->cap_stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue2(h, k, h->cap_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(h->cap_stream, &g);
        if (rc || ce != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return rc ? rc : fail(&h->last_error, GBSPH_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
        }
        const cudaError_t ie = cudaGraphInstantiate(&h->gexec, g, 0);
        cudaGraphDestroy(g);
        if (ie != cudaSuccess) {
            h->gexec = nullptr;
            return fail(&h->last_error, GBSPH_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ie));
        }
        h->gkey = key;
    }
    // the step leaves the counts as it finds them, all zero
    if (!h->count_clean)
        GBSPH_CUDA_TRY(&h->last_error, cudaMemsetAsync(h->count, 0, count_words(h->table) * 4, (cudaStream_t)stream));
    h->count_clean = false;
    GBSPH_CUDA_TRY(&h->last_error, cudaGraphLaunch(h->gexec, (cudaStream_t)stream));
    h->count_clean = true;
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_get_cell_bounds(gbsph_fluid2d_t h, uint32_t* cell_start, uint32_t* cell_end,
                                            size_t n_cells, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!cell_start || !cell_end || n_cells != h->table)
        return fail(&h->last_error, GBSPH_ERR_SIZE_MISMATCH, "n_cells must equal the table size");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    cudaStream_t s = (cudaStream_t)stream;
    k_table_split<<<grid1((uint32_t)n_cells), 256, 0, s>>>(h->cells, (uint32_t)n_cells, cell_start, cell_end);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    return GBSPH_OK;
}

GBSPH_API int gbsph_fluid2d_sync_status(gbsph_fluid2d_t h, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    uint32_t bits = 0;
    GBSPH_CUDA_TRY(&h->last_error, cudaMemcpy(&bits, h->err, 4, cudaMemcpyDeviceToHost));
    if (bits) {
        GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->err, 0, 4));
        h->count_clean = false;  // a step that refused a particle leaves its cell's count
        return fail(&h->last_error, dev_err_to_status(bits), "device error word 0x" + std::to_string(bits));
    }
    return GBSPH_OK;
}

GBSPH_API const char* gbsph_fluid2d_last_error(gbsph_fluid2d_t h) { return h ? h->last_error.c_str() : "null handle"; }

}  // extern "C"
