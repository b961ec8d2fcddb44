// bvh.cu -- linear BVH over a triangle mesh: the oclBvhTrimesh replacement behind the C ABI
// (libCL/geom/oclBvhTrimesh.h:20-84, libCL/geom/oclBvhTrimesh.cpp:56-143,
// libCL/geom/oclBvhTrimesh.cl:33-298), the reference's second user of the radix sort; and its
// 2D sibling over line segments, the oclBvhLines replacement (libCL/geom/oclBvhLines.h:20-77,
// libCL/geom/oclBvhLines.cpp:48-115, libCL/geom/oclBvhLines.cl:27-245), which shares the tree
// kernel (templated on the node type).
//
// One build, in the reference's order:
//   global bounding box (accumulated into the handle's box, which starts at zero and is never
//   reset, as the reference's is) -> 30-bit Morton key of every triangle centroid -> stable
//   sort of (key, triangle) on 32 bits -> internal node i (between sorted leaves i and i+1)
//   gets the highest bit (29..0) where keys i and i+1 differ -> each internal node links to
//   the nearer of its nearest left / right nodes with a higher bit (the one with the lower
//   bit; the root has neither) -> leaves take the free child slots -> boxes bottom-up.
// The reference makes a pass of each of the last three, finds the higher-bit neighbours by a
// linear scan per node and computes the boxes by one root-to-leaf descent per triangle with a
// visit flag per node. Here one kernel (k_bvh_tree) climbs from the leaves: a subtree that
// covers the sorted leaves [a, b] hangs on node a - 1 or node b, whichever has the lower bit, so
// links, boxes and records are written once, without any search; min and max are evaluated with
// the reference's operand order, so every box is bit-identical.
#include <algorithm>
#include <cfloat>
#include <string>

#include "device.cuh"
#include "internal.h"

using namespace gbsph;

namespace {

constexpr int BVH_THREADS = 256;

// OpenCL's min / max of floats: min(x, y) = y < x ? y : x, max(x, y) = x < y ? y : x.
__device__ __forceinline__ float cl_min(float x, float y) { return y < x ? y : x; }
__device__ __forceinline__ float cl_max(float x, float y) { return x < y ? y : x; }
__device__ __forceinline__ float4 cl_min4(float4 a, float4 b) {
    return make_float4(cl_min(a.x, b.x), cl_min(a.y, b.y), cl_min(a.z, b.z), cl_min(a.w, b.w));
}
__device__ __forceinline__ float4 cl_max4(float4 a, float4 b) {
    return make_float4(cl_max(a.x, b.x), cl_max(a.y, b.y), cl_max(a.z, b.z), cl_max(a.w, b.w));
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {  // "code", libCL/geom/oclBvhTrimesh.cl:82-89
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// 16-bit interleave of clMorton, libCL/geom/oclBvhLines.cl:35-52.
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
    x &= 0x0000FFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

// What the tree kernel needs of a node type: its box, its records and its leaves.
struct TriTree {  // oclBvhTrimesh: 48-byte nodes
    using Node = gbsph_bvh_node;
    struct Box {
        float4 lo, hi;
    };
    struct Prims {
        const uint32_t* index;
        const float4* vertex;
        uint32_t nv;
    };
    static constexpr uint32_t MASK = (1u << 30) - 1u;  // key bits that make nodes
    static constexpr uint32_t TRAV = 2;                 // internal nodes' final flag
    // +-MAXFLOAT in the coordinate lanes (clCreateNodes), w = 0
    static __device__ __forceinline__ Box empty() {
        return {make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f), make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f)};
    }
    static __device__ __forceinline__ Box leaf(const Prims& p, uint32_t tri) {
        Box b = empty();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float4 v = p.vertex[min(p.index[3 * tri + k], p.nv - 1)];
            b.lo = cl_min4(b.lo, v);
            b.hi = cl_max4(b.hi, v);
        }
        return b;
    }
    static __device__ __forceinline__ Box merge(const Box& l, const Box& r) {
        return {cl_min4(l.lo, r.lo), cl_max4(l.hi, r.hi)};
    }
    static __device__ __forceinline__ Box load(const Node* n) {  // written by another CTA: through L2
        const float4* f = reinterpret_cast<const float4*>(n);
        return {__ldcg(f), __ldcg(f + 1)};
    }
    static __device__ __forceinline__ void store(Node* n, const Box& b, int left, int right, uint32_t bit, uint32_t trav) {
        float4* f = reinterpret_cast<float4*>(n);
        f[0] = b.lo;
        f[1] = b.hi;
        reinterpret_cast<int4*>(n)[2] = make_int4(left, right, (int)bit, (int)trav);
    }
};
struct SegTree {  // oclBvhLines: 32-byte nodes
    using Node = gbsph_bvh2d_node;
    struct Box {
        float4 b;  // min xy, max xy
    };
    struct Prims {
        const float2* vertex;
    };
    static constexpr uint32_t MASK = 0xFFFFFFFFu;
    // In the reference the first visitor of a node leaves trav = 2 and the second swaps it for 3
    // before computing the box (libCL/geom/oclBvhLines.cl:186-245).
    static constexpr uint32_t TRAV = 3;
    static __device__ __forceinline__ Box empty() { return {make_float4(FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX)}; }
    static __device__ __forceinline__ Box leaf(const Prims& p, uint32_t seg) {
        const float2 v0 = p.vertex[2 * seg], v1 = p.vertex[2 * seg + 1];
        return {make_float4(cl_min(cl_min(FLT_MAX, v0.x), v1.x), cl_min(cl_min(FLT_MAX, v0.y), v1.y),
                            cl_max(cl_max(-FLT_MAX, v0.x), v1.x), cl_max(cl_max(-FLT_MAX, v0.y), v1.y))};
    }
    static __device__ __forceinline__ Box merge(const Box& l, const Box& r) {
        return {make_float4(cl_min(l.b.x, r.b.x), cl_min(l.b.y, r.b.y), cl_max(l.b.z, r.b.z), cl_max(l.b.w, r.b.w))};
    }
    static __device__ __forceinline__ Box load(const Node* n) { return {__ldcg(reinterpret_cast<const float4*>(n))}; }
    static __device__ __forceinline__ void store(Node* n, const Box& b, int left, int right, uint32_t bit, uint32_t trav) {
        reinterpret_cast<float4*>(n)[0] = b.b;
        reinterpret_cast<int4*>(n)[1] = make_int4(left, right, (int)bit, (int)trav);
    }
};

// Per-block min / max of the vertices (all four lanes), combined with the handle's box by the
// last block to finish (clAABB, libCL/geom/oclBvhTrimesh.cl:33-76).
__global__ void __launch_bounds__(BVH_THREADS) k_bvh_box(const float4* __restrict__ vertex, uint32_t nv,
                                                         float4* __restrict__ part, uint32_t* __restrict__ done,
                                                         float4* __restrict__ box) {
    __shared__ float4 smin[BVH_THREADS], smax[BVH_THREADS];
    __shared__ bool last;
    float4 mn = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f), mx = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f);
    for (uint32_t i = blockIdx.x * BVH_THREADS + threadIdx.x; i < nv; i += gridDim.x * BVH_THREADS) {
        const float4 v = vertex[i];
        mn = cl_min4(mn, v);
        mx = cl_max4(mx, v);
    }
    smin[threadIdx.x] = mn;
    smax[threadIdx.x] = mx;
    __syncthreads();
    for (int s = BVH_THREADS / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            smin[threadIdx.x] = cl_min4(smin[threadIdx.x], smin[threadIdx.x + s]);
            smax[threadIdx.x] = cl_max4(smax[threadIdx.x], smax[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = smin[0];
        part[2 * blockIdx.x + 1] = smax[0];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // the partial boxes by all threads of the last block (min and max of numbers do not depend on
    // the order); one thread reading 257 of them in turn took 40 of the kernel's 48 us
    __threadfence();
    mn = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f);
    mx = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f);
    for (uint32_t k = threadIdx.x; k < gridDim.x; k += BVH_THREADS) {  // written by other blocks: past L1
        mn = cl_min4(mn, __ldcg(part + 2 * k));
        mx = cl_max4(mx, __ldcg(part + 2 * k + 1));
    }
    smin[threadIdx.x] = mn;
    smax[threadIdx.x] = mx;
    __syncthreads();
    for (int s = BVH_THREADS / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            smin[threadIdx.x] = cl_min4(smin[threadIdx.x], smin[threadIdx.x + s]);
            smax[threadIdx.x] = cl_max4(smax[threadIdx.x], smax[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        box[0] = cl_min4(box[0], smin[0]);
        box[1] = cl_max4(box[1], smax[0]);
        *done = 0;
    }
}

// clMorton (libCL/geom/oclBvhTrimesh.cl:91-103): key of the triangle's centroid in the box.
__global__ void __launch_bounds__(BVH_THREADS) k_bvh_morton(const uint32_t* __restrict__ index,
                                                            const float4* __restrict__ vertex,
                                                            const float4* __restrict__ box, uint32_t n,
                                                            uint32_t nv, uint32_t* __restrict__ key,
                                                            uint32_t* __restrict__ val, uint32_t* err) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const uint32_t i0 = index[3 * g], i1 = index[3 * g + 1], i2 = index[3 * g + 2];
    if (i0 >= nv || i1 >= nv || i2 >= nv) atomicOr(err, DEV_ERR_KEY_RANGE);
    const float4 v0 = vertex[min(i0, nv - 1)], v1 = vertex[min(i1, nv - 1)], v2 = vertex[min(i2, nv - 1)];
    const float4 lo = box[0], hi = box[1];
    auto axis = [&](float a, float b, float c, float l, float h) {
        const float cen = __fdiv_rn(__fadd_rn(__fadd_rn(a, b), c), 3.0f);
        const float t = __fdiv_rn(__fsub_rn(cen, l), __fsub_rn(h, l));
        return spread10(__float2uint_rz(__fmul_rn(t, 1023.0f)));
    };
    key[g] = axis(v0.x, v1.x, v2.x, lo.x, hi.x) | (axis(v0.y, v1.y, v2.y, lo.y, hi.y) << 1) |
             (axis(v0.z, v1.z, v2.z, lo.z, hi.z) << 2);
    val[g] = g;
}

// clMorton of oclBvhLines (libCL/geom/oclBvhLines.cl:27-55): the segment's midpoint,
// 0.5 * (v0 + v1), truncated to integers, 16 bits per axis interleaved (x in the even bits).
__global__ void __launch_bounds__(BVH_THREADS) k_bvh_morton_lines(const float2* __restrict__ vertex, uint32_t n,
                                                                  uint32_t* __restrict__ key,
                                                                  uint32_t* __restrict__ val) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const float2 v0 = vertex[2 * g], v1 = vertex[2 * g + 1];
    const uint32_t cx = __float2uint_rz(__fmul_rn(0.5f, __fadd_rn(v0.x, v1.x)));
    const uint32_t cy = __float2uint_rz(__fmul_rn(0.5f, __fadd_rn(v0.y, v1.y)));
    key[g] = spread16(cx) | (spread16(cy) << 1);
    val[g] = g;
}

__device__ __forceinline__ unsigned long long exch_acq_rel(unsigned long long* p, unsigned long long v) {
    unsigned long long o;
    asm volatile("atom.acq_rel.gpu.global.exch.b64 %0, [%1], %2;" : "=l"(o) : "l"(p), "l"(v) : "memory");
    return o;
}

// Nodes, links, leaves and boxes (clCreateNodes, clLinkNodes, clCreateLeaves, clComputeAABBs:
// libCL/geom/oclBvhTrimesh.cl:119-298, libCL/geom/oclBvhLines.cl:71-245) in one climb. A thread
// starts with sorted leaf g; a subtree over the leaves [a, b] is the right child of node a - 1 or
// the left child of node b, whichever has the lower bit (node b at equal bits); the first of a
// node's two children to arrive leaves its box, its far end and its id and stops, the second
// writes the node's record and goes on with the two ranges joined. The subtree over all leaves
// is the root.
//
// Bits above 0 cannot tie (between two nodes with the same highest differing bit the keys must
// fall back, which makes a higher one). Bit 0 ties where keys repeat: of a run of nodes with
// bit 0, all of which claim the same slot in the reference, the last one holds it (as in a
// sequential run of the reference's work-items) and the others keep their left leaf, an empty
// box and no parent; the last one's subtree then stands in for the whole run, whose first leaf is
// the first key of the same value above bit 0.
//
// Nodes of the CTA's own range meet in shared memory; a child whose sibling did not come there,
// and subtrees that leave the range, go on through one 64-bit exchange per node in `link` (all
// ones before the launch). 1.05M triangles: 130 us, of which about 40 are the last subtrees'
// climb through the top levels, an exchange and a box at a time (16,640 triangles: 30 us); 64 to
// 256 leaves per CTA are alike, 512 and 1024 slower. Six kernels did this before (node records with
// empty boxes, block maxima, a neighbour search per node, leaves, parent links, a climb with a
// counter, two fences and 24 scalar loads per node): 415 us.
constexpr int TREE_THREADS = 128;

template <class T>
__global__ void __launch_bounds__(TREE_THREADS) k_bvh_tree(const uint32_t* __restrict__ key, const uint32_t* __restrict__ val,
                                                          uint32_t n, typename T::Prims prims, typename T::Node* node,
                                                          unsigned long long* link, uint32_t* __restrict__ root) {
    using Box = typename T::Box;
    __shared__ uint32_t s_key[TREE_THREADS + 2];  // keys base - 1 ... base + TREE_THREADS
    __shared__ Box s_box[2][TREE_THREADS];         // a node's left and right child
    __shared__ uint2 s_end[2][TREE_THREADS];       // their far ends and ids
    __shared__ uint32_t s_came[TREE_THREADS];      // bit 0: left, bit 1: right
    const uint32_t t = threadIdx.x, base = blockIdx.x * TREE_THREADS, g = base + t, ls = n - 1u;
    for (uint32_t k = t; k < TREE_THREADS + 2; k += TREE_THREADS) {
        const uint32_t i = base + k - 1u;  // wraps for the first key of the first CTA
        s_key[k] = i < n ? key[i] : 0u;
    }
    s_came[t] = 0u;
    __syncthreads();
    auto key_at = [&](uint32_t i) -> uint32_t {
        const uint32_t k = i - base + 1u;
        return (k < TREE_THREADS + 2 ? s_key[k] : __ldg(key + i)) & T::MASK;
    };
    // Highest bit in which keys i and i + 1 differ; NO_NODE before the first and after the last leaf.
    constexpr uint32_t NO_NODE = 64u;
    auto bit_of = [&](uint32_t i) -> uint32_t {
        if (i >= ls) return NO_NODE;
        const uint32_t d = key_at(i) ^ key_at(i + 1u);
        return d ? 31u - (uint32_t)__clz((int)d) : 0u;
    };
    // A subtree: its leaves [a, b], its node c, the bits of the nodes a - 1 and b beside it.
    uint32_t a = g, b = g, c = ls + g, bl = NO_NODE, br = NO_NODE;
    Box box{};
    // Joins this thread's subtree with its sibling (node oc, far end oe, box ob) under node p; side:
    // the thread's is the right child. Writes p's record; false: p is the root.
    auto join = [&](uint32_t p, uint32_t side, uint32_t oc, uint32_t oe, const Box& ob) -> bool {
        const uint32_t bit = side ? bl : br;
        const uint32_t far = bit_of(side ? oe - 1u : oe);
        box = side ? T::merge(ob, box) : T::merge(box, ob);
        T::store(node + p, box, (int)(side ? oc : c), (int)(side ? c : oc), bit, T::TRAV);
        c = p;
        if (side) {
            a = oe;
            bl = far;
        } else {
            b = oe;
            br = far;
        }
        if (bit == 0u && bl == 0u) {  // a run of repeated keys: its first leaf
            const uint32_t k = key_at(p) >> 1;
            uint32_t lo = 0u, hi = a - 1u;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (key_at(mid) >> 1 < k) lo = mid + 1u;
                else hi = mid;
            }
            a = lo;
            bl = bit_of(a - 1u);
        }
        if (bl == NO_NODE && br == NO_NODE) {
            *root = p;
            return false;
        }
        return true;
    };

    bool carry = g < n;
    if (carry) {
        const uint32_t prim = val[g];
        bl = bit_of(g - 1u);
        br = bit_of(g);
        box = T::leaf(prims, prim);
        T::store(node + c, box, 0, 0, prim, 0u);
        // a node that lost its slot to the last of its run
        if (br == 0u && bit_of(g + 1u) == 0u) T::store(node + g, T::empty(), (int)c, -1, 0u, 0u);
        for (;;) {
            const uint32_t side = bl < br ? 1u : 0u, p = side ? a - 1u : b, i = p - base;
            if (i >= TREE_THREADS) break;  // not a node of this CTA
            s_box[side][i] = box;
            s_end[side][i] = make_uint2(side ? b : a, c);
            __threadfence_block();
            carry = atomicOr(&s_came[i], 1u << side) != 0u;
            if (!carry) break;
            __threadfence_block();
            const uint2 o = s_end[side ^ 1u][i];
            carry = join(p, side, o.y, o.x, s_box[side ^ 1u][i]);
            if (!carry) break;
        }
    }
    __syncthreads();
    // Subtrees go on through global memory: this thread's own, then the lone child of its node.
    const uint32_t lone = s_came[t];
    for (int round = 0; round < 2; ++round) {
        if (round == 1) {
            carry = lone == 1u || lone == 2u;
            if (carry) {
                const uint32_t side = lone >> 1;
                const uint2 e = s_end[side][t];
                box = s_box[side][t];
                c = e.y;
                a = side ? g + 1u : e.x;
                b = side ? e.x : g;
                bl = bit_of(a - 1u);
                br = bit_of(b);
            }
        }
        while (carry) {
            const uint32_t side = bl < br ? 1u : 0u, p = side ? a - 1u : b;
            // the exchange releases the subtree's records (also those that other threads of the CTA
            // wrote before the barrier) and acquires its sibling's
            const unsigned long long o = exch_acq_rel(link + p, (unsigned long long)(side ? b : a) << 32 | c);
            if (o == ~0ull) break;  // the sibling is not there yet
            carry = join(p, side, (uint32_t)o, (uint32_t)(o >> 32), T::load(node + (uint32_t)o));
        }
    }
}

int grid(uint32_t n) { return (int)((n + BVH_THREADS - 1) / BVH_THREADS); }

}  // namespace

struct gbsph_bvh_s {
    int device = 0;
    gbsph_radix_sort_t sort = nullptr;
    uint32_t cap = 0;  // triangles the buffers hold
    uint32_t n = 0;    // triangles of the last build
    void* block = nullptr;
    gbsph_bvh_node* node = nullptr;
    uint32_t *key = nullptr, *val = nullptr, *root = nullptr, *err = nullptr, *done = nullptr;
    unsigned long long* link = nullptr;  // per internal node: the first child to arrive
    float4* box = nullptr;   // [min, max], persists across builds
    float4* part = nullptr;  // per-block partial boxes
    std::string last_error;
};

namespace {

constexpr int BOX_BLOCKS = 1024;

int ensure(gbsph_bvh_s* h, uint32_t n) {
    if (n <= h->cap && h->block) return GBSPH_OK;
    if (h->block) cudaFree(h->block);
    h->block = nullptr;
    const size_t nn = 2 * (size_t)n, m = n;
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t bytes = al(nn * sizeof(gbsph_bvh_node)) + 2 * al(m * 4) + al(m * 8);
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->block, bytes));
    char* p = (char*)h->block;
    h->node = (gbsph_bvh_node*)p;
    p += al(nn * sizeof(gbsph_bvh_node));
    h->key = (uint32_t*)p;
    p += al(m * 4);
    h->val = (uint32_t*)p;
    p += al(m * 4);
    h->link = (unsigned long long*)p;
    h->cap = n;
    return GBSPH_OK;
}

}  // namespace

extern "C" {

GBSPH_API int gbsph_bvh_create(gbsph_bvh_t* out) {
    if (!out) return GBSPH_ERR_ARGUMENT;
    *out = nullptr;
    gbsph_bvh_s* h = new gbsph_bvh_s();
    int rc = cudaGetDevice(&h->device) == cudaSuccess ? GBSPH_OK : GBSPH_ERR_CUDA;
    if (!rc) rc = gbsph_radix_sort_create(&h->sort);
    // small state: the persistent box (zero, as the reference's freshly allocated one), the
    // partial boxes, root, error word and the box kernel's block counter
    const size_t small = 2 * 16 + BOX_BLOCKS * 32 + 16;
    void* s = nullptr;
    if (!rc && cudaMalloc(&s, small) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    if (!rc && cudaMemset(s, 0, small) != cudaSuccess) rc = GBSPH_ERR_CUDA;
    if (rc) {
        cudaGetLastError();
        if (s) cudaFree(s);
        if (h->sort) gbsph_radix_sort_destroy(h->sort);
        delete h;
        return rc;
    }
    h->box = (float4*)s;
    h->part = h->box + 2;
    h->root = (uint32_t*)(h->part + 2 * BOX_BLOCKS);
    h->err = h->root + 1;
    h->done = h->root + 2;
    *out = h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_destroy(gbsph_bvh_t h) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    cudaSetDevice(h->device);
    if (h->block) cudaFree(h->block);
    if (h->box) cudaFree(h->box);
    if (h->sort) gbsph_radix_sort_destroy(h->sort);
    delete h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_compute(gbsph_bvh_t h, const float* vertex, size_t n_vertices, const uint32_t* index,
                                size_t n_indices, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!vertex || !index) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "null buffer");
    if (n_indices % 3 != 0) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "index count is not a multiple of 3");
    const size_t nt = n_indices / 3;
    if (nt < 2) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "a BVH needs at least 2 triangles");
    if (n_vertices == 0) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "no vertices");
    if (nt > SORT_MAX_KEYS - SORT_TILE || n_vertices > 0xFFFFFFFFull)
        return fail(&h->last_error, GBSPH_ERR_TOO_LARGE, "too many triangles or vertices");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    const uint32_t n = (uint32_t)nt, m = n - 1, nv = (uint32_t)n_vertices;
    int rc = ensure(h, n);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const float4* v4 = reinterpret_cast<const float4*>(vertex);
    const int bb = std::min(BOX_BLOCKS, std::max(1, (int)((nv + BVH_THREADS * 8 - 1) / (BVH_THREADS * 8))));
    k_bvh_box<<<bb, BVH_THREADS, 0, s>>>(v4, nv, h->part, h->done, h->box);
    k_bvh_morton<<<grid(n), BVH_THREADS, 0, s>>>(index, v4, h->box, n, nv, h->key, h->val, h->err);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    rc = gbsph_radix_sort_compute(h->sort, h->key, h->val, n, n, 0, 32, stream);
    if (rc) return fail(&h->last_error, rc, std::string("sort: ") + gbsph_radix_sort_last_error(h->sort));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemsetAsync(h->link, 0xFF, (size_t)m * 8, s));
    k_bvh_tree<TriTree><<<(n + TREE_THREADS - 1) / TREE_THREADS, TREE_THREADS, 0, s>>>(h->key, h->val, n, TriTree::Prims{index, v4, nv}, h->node, h->link, h->root);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    h->n = n;
    return GBSPH_OK;
}

GBSPH_API gbsph_bvh_node* gbsph_bvh_get_node_buffer(gbsph_bvh_t h, size_t* count) {
    if (!h) return nullptr;
    if (count) *count = h->n ? 2 * (size_t)h->n - 1 : 0;
    return h->node;
}

GBSPH_API size_t gbsph_bvh_get_node_count(gbsph_bvh_t h) { return h && h->n ? 2 * (size_t)h->n - 1 : 0; }

GBSPH_API int gbsph_bvh_get_root_node(gbsph_bvh_t h, uint32_t* root, void* stream) {
    if (!h || !root) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemcpy(root, h->root, 4, cudaMemcpyDeviceToHost));
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_get_bounds(gbsph_bvh_t h, float* box8, void* stream) {
    if (!h || !box8) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemcpy(box8, h->box, 32, cudaMemcpyDeviceToHost));
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_sync_status(gbsph_bvh_t h, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    const int src = gbsph_radix_sort_sync_status(h->sort, stream);
    if (src) return fail(&h->last_error, src, std::string("sort: ") + gbsph_radix_sort_last_error(h->sort));
    uint32_t bits = 0;
    GBSPH_CUDA_TRY(&h->last_error, cudaMemcpy(&bits, h->err, 4, cudaMemcpyDeviceToHost));
    if (bits) {
        GBSPH_CUDA_TRY(&h->last_error, cudaMemset(h->err, 0, 4));
        return fail(&h->last_error, dev_err_to_status(bits), "a triangle index is outside the vertex buffer, or collide() met a root or tree that is not the build's");
    }
    return GBSPH_OK;
}

GBSPH_API const char* gbsph_bvh_last_error(gbsph_bvh_t h) { return h ? h->last_error.c_str() : "null handle"; }

}  // extern "C"

// ---- particle-vs-mesh collision -------------------------------------------------------------
// clCollideBVH (libCL/phys/oclFluid3D.cl:365-550), one work-item per particle, restated with
// round-to-nearest intrinsics (no contraction) so that it matches the CPU restatement bit for
// bit. OpenCL's implementation-defined helpers are fixed as: dot(a, b) = ((ax bx + ay by) +
// az bz) + aw bw; length / fast_length(a) = sqrt(dot(a, a)); normalize(a) = a / length(a)
// per lane; cross() of float4 has w = 0. The traversal keeps the reference's breadth-first
// order with its 256-entry circular queue, so the first colliding triangle is the same.

namespace {

struct F4 {
    float x, y, z, w;
};
__device__ __forceinline__ F4 f4(float4 a) { return {a.x, a.y, a.z, a.w}; }
__device__ __forceinline__ F4 add(F4 a, F4 b) {
    return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w)};
}
__device__ __forceinline__ F4 sub(F4 a, F4 b) {
    return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z), __fsub_rn(a.w, b.w)};
}
__device__ __forceinline__ F4 mul(F4 a, float s) {
    return {__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s), __fmul_rn(a.w, s)};
}
__device__ __forceinline__ F4 divs(F4 a, float s) {
    return {__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s), __fdiv_rn(a.w, s)};
}
__device__ __forceinline__ float dot(F4 a, F4 b) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z)),
                     __fmul_rn(a.w, b.w));
}
__device__ __forceinline__ float len(F4 a) { return __fsqrt_rn(dot(a, a)); }
__device__ __forceinline__ F4 normalize(F4 a) { return divs(a, len(a)); }
__device__ __forceinline__ F4 cross(F4 p, F4 q) {
    return {__fsub_rn(__fmul_rn(p.y, q.z), __fmul_rn(p.z, q.y)), __fsub_rn(__fmul_rn(p.z, q.x), __fmul_rn(p.x, q.z)),
            __fsub_rn(__fmul_rn(p.x, q.y), __fmul_rn(p.y, q.x)), 0.0f};
}

struct CollideParams {
    float dt, radius, pconst, density, h, mass;
};

// collideTriangle (libCL/phys/oclFluid3D.cl:380-459); `tri` is the first index slot.
__device__ bool collide_triangle(uint32_t tri, const uint32_t* __restrict__ index, const float4* __restrict__ vertex,
                                 uint32_t nv, F4& pos, F4& vel, F4& force, const CollideParams& P) {
    F4 V0 = f4(vertex[min(index[tri], nv - 1)]), V1 = f4(vertex[min(index[tri + 1], nv - 1)]),
       V2 = f4(vertex[min(index[tri + 2], nv - 1)]);
    V0.w = V1.w = V2.w = 0.0f;
    pos.w = 0.0f;
    const F4 u = sub(V1, V0), v = sub(V2, V0);
    F4 n = cross(u, v);
    if (dot(n, n) == 0.0f) return false;
    const F4 w0 = sub(pos, V0);
    const F4 disp = mul(vel, P.dt);
    const float a = dot(n, w0);
    if (a < 0.0f) return false;
    const float b = dot(n, disp);
    if (fabsf(b) < 0.000001f) return false;
    const float r = __fdiv_rn(-a, b);
    if (r < 0.0f) return false;
    const F4 I = add(pos, mul(disp, r));
    const float uu = dot(u, u), uv = dot(u, v), vv = dot(v, v);
    const F4 w = sub(I, V0);
    const float wu = dot(w, u), wv = dot(w, v);
    const float D = __fsub_rn(__fmul_rn(uv, uv), __fmul_rn(uu, vv));
    const float s = __fdiv_rn(__fsub_rn(__fmul_rn(uv, wv), __fmul_rn(vv, wu)), D);
    if (s < 0.0f || s > 1.0f) return false;
    const float t = __fdiv_rn(__fsub_rn(__fmul_rn(uv, wu), __fmul_rn(uu, wv)), D);
    if (t < 0.0f || __fadd_rn(s, t) > 1.0f) return false;
    n = normalize(n);
    const F4 Vc = sub(add(pos, disp), V0);
    const float dist = dot(Vc, n);
    const float depth = __fsub_rn(P.radius, dist);
    if (depth > 0.0f) {
        const F4 dPos = mul(mul(normalize(disp), dot(n, disp)), depth);
        const F4 dTan = sub(vel, mul(n, dot(n, vel)));
        force = add(force, divs(dTan, P.dt));
        const float hd = __fsub_rn(P.h, dist);
        force = add(force, mul(mul(mul(mul(n, hd), hd), __fdiv_rn(P.pconst, P.density)), P.mass));
        pos = add(pos, dPos);
        vel = {0.0f, 0.0f, 0.0f, 0.0f};
        return true;
    }
    return false;
}

// intersectBox + collideAABB (libCL/phys/oclFluid3D.cl:462-498) for a particle's ray: inv = 1 /
// normalize(vel) per lane and reach = max(radius, |vel|) stay what they are until the particle
// hits, so they are computed once instead of at each box. OpenCL's min and max (a compare and a
// select each) differ from the hardware's only for NaN, and for the sign of a zero, which no
// compare below sees; a ray of finite inverse direction (each at least 1 in size) from a finite
// position makes no NaN with any box, so `tame` rays take the hardware's.
template <bool TAME>
__device__ __forceinline__ bool collide_box(const float4& lo, const float4& hi, const F4& pos, const F4& inv, float reach) {
    const float bx = __fmul_rn(inv.x, __fsub_rn(lo.x, pos.x)), tx = __fmul_rn(inv.x, __fsub_rn(hi.x, pos.x));
    const float by = __fmul_rn(inv.y, __fsub_rn(lo.y, pos.y)), ty = __fmul_rn(inv.y, __fsub_rn(hi.y, pos.y));
    const float bz = __fmul_rn(inv.z, __fsub_rn(lo.z, pos.z)), tz = __fmul_rn(inv.z, __fsub_rn(hi.z, pos.z));
    float tnear, tfar;
    if (TAME) {
        tnear = fmaxf(fmaxf(fminf(tx, bx), fminf(ty, by)), fminf(tz, bz));
        tfar = fminf(fminf(fmaxf(tx, bx), fmaxf(ty, by)), fmaxf(tz, bz));
    } else {
        const float tminx = cl_min(tx, bx), tminy = cl_min(ty, by), tminz = cl_min(tz, bz);
        const float tmaxx = cl_max(tx, bx), tmaxy = cl_max(ty, by), tmaxz = cl_max(tz, bz);
        tnear = cl_max(cl_max(tminx, tminy), cl_max(tminx, tminz));
        tfar = cl_min(cl_min(tmaxx, tmaxy), cl_min(tmaxx, tmaxz));
    }
    return tfar > tnear && tnear < reach;
}

constexpr uint32_t QUEUE_SIZE = 256;
constexpr uint32_t COLLIDE_THREADS = 128;

// LANES lanes take a particle: they pop that many queue entries at a time (a triangle
// test or two box tests each) and push the hit children at the places a sequential run gives
// them, so the order of the tests, and with it the first triangle hit, is the reference's. Where
// a batch could fill the 256-entry ring, which then counts as empty, entries go one by one, as
// in the reference. The queue lies in shared memory.
// Popped triangles wait until a warp has a full batch of them (or nothing else to do), still in
// queue order: tested as they come they held the box tests up in most rounds.
// 1.05M triangles, 262,144 particles in no order: 425 us. With a thread per particle (queue in
// local memory) every pop waited for its node and its children in turn: 1,120 us, 640 us with
// the ray's constants taken out of the box tests, and more resident threads were slower
// (720-900 us, L1 thrashing). 8 lanes: 590 us; three-operand min / max for tame rays: 475 us; the
// triangles in batches: 425 us. 4 lanes 640 us, 16 lanes 650 us. Bound by the latency of
// the nodes (the longest of its stalls; issue 56% of cycles, the LSU pipe 61%).
// A tree of few nodes does not fill eight lanes, nor the ring: its nodes all fit a smaller one, which
// then never wraps. Us for 1,000,000 particles with 1 / 4 / 8 lanes and by a thread per particle with its
// queue in local memory: 2 triangles 45 / 97 / 163 / 50, 8 127 / 167 / 295 / 154, 33 - / 290 / 463 / 360, 63 - / 432 / 524 / 604; for 256 and
// 4 to 8 triangles one lane takes 22 to 24, four or eight 18 to 20.
template <uint32_t LANES, uint32_t RING>
__global__ void __launch_bounds__(COLLIDE_THREADS, 8) k_collide_bvh(float4* __restrict__ force, float4* __restrict__ position,
                                                             float4* __restrict__ velocity, uint32_t np,
                                                             CollideParams P, const gbsph_bvh_node* __restrict__ bvh,
                                                             const uint32_t* __restrict__ root, uint32_t n_nodes,
                                                             const uint32_t* __restrict__ index,
                                                             const float4* __restrict__ vertex, uint32_t nv,
                                                             uint32_t* err) {
    __shared__ uint32_t s_queue[COLLIDE_THREADS / LANES][RING];
    __shared__ uint32_t s_leaf[COLLIDE_THREADS / LANES][2 * LANES];
    const uint32_t lane = threadIdx.x & 31u, gl = lane % LANES;
    const uint32_t group = ((1u << LANES) - 1u) << (lane - gl), before = group & lanemask_lt();
    uint32_t* queue = s_queue[threadIdx.x / LANES];
    uint32_t* leaf = s_leaf[threadIdx.x / LANES];
    uint32_t leaves = 0;  // triangles popped and not tested yet
    const uint32_t p = blockIdx.x * (COLLIDE_THREADS / LANES) + threadIdx.x / LANES;
    bool active = p < np;
    F4 pos{}, vel{};
    if (active) {
        pos = f4(position[p]);
        vel = f4(velocity[p]);
    }
    const float speed = len(vel);
    const F4 nr = divs(vel, speed);  // normalize(vel)
    const F4 inv = {__fdiv_rn(1.0f, nr.x), __fdiv_rn(1.0f, nr.y), __fdiv_rn(1.0f, nr.z), 0.0f};
    const float reach = cl_max(P.radius, speed);
    const bool tame = isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z) && isfinite(pos.x) && isfinite(pos.y) && isfinite(pos.z);
    const float4* const nodes = reinterpret_cast<const float4*>(bvh);  // three per node
    uint32_t head = 0, tail = 1, steps = 0;
    const uint32_t rt = *root;
    if (rt >= n_nodes) {
        if (active) atomicOr(err, DEV_ERR_KEY_RANGE);
        active = false;
    }
    if (gl == 0) queue[0] = rt;
    __syncwarp();
    for (;;) {
        const bool going = __any_sync(0xffffffffu, active);
        if (!going || __any_sync(0xffffffffu, leaves >= LANES)) {
            // the triangles that wait, a lane each, in the order they were popped
            const uint32_t n = min(leaves, LANES), tri = leaf[gl], next = leaf[LANES + gl];
            bool hit = false;
            if (gl < n) {
                F4 x = pos, v = vel, f{};
                hit = collide_triangle(tri * 3u, index, vertex, nv, x, v, f, P);
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, hit) & group;
            if (hit && (hits & before) == 0u) {  // the first of them: once more, for its result
                F4 x = pos, v = vel, f = f4(force[p]);
                collide_triangle(tri * 3u, index, vertex, nv, x, v, f, P);
                position[p] = make_float4(x.x, x.y, x.z, x.w);
                velocity[p] = make_float4(v.x, v.y, v.z, v.w);
                force[p] = make_float4(f.x, f.y, f.z, f.w);
            }
            leaves -= n;
            if (hits) {
                active = false;
                leaves = 0;
            }
            __syncwarp();
            if (gl < leaves) leaf[gl] = next;
            __syncwarp();
            if (!going && !__any_sync(0xffffffffu, leaves != 0u)) break;
            if (!going) continue;
        }
        const uint32_t waiting = (tail - head) % RING;
        uint32_t k = active ? min(LANES, waiting) : 0u;
        if (waiting + k >= RING) k = min(k, 1u);
        const uint32_t it = queue[(head + gl) % RING];
        __syncwarp();
        bool hl = false, hr = false, tri = false;
        int4 w = make_int4(0, 0, 0, 0);
        if (gl < k) {
            w = *reinterpret_cast<const int4*>(nodes + 3 * (size_t)it + 2);
            tri = w.x == w.y;
            hl = !tri && (uint32_t)w.x < n_nodes;
            hr = !tri && (uint32_t)w.y < n_nodes;
            const float4 *l = nodes + 3 * (size_t)(hl ? w.x : 0), *r = nodes + 3 * (size_t)(hr ? w.y : 0);
            const float4 llo = l[0], lhi = l[1], rlo = r[0], rhi = r[1];
            if (tame) {
                hl = hl && collide_box<true>(llo, lhi, pos, inv, reach);
                hr = hr && collide_box<true>(rlo, rhi, pos, inv, reach);
            } else {
                hl = hl && collide_box<false>(llo, lhi, pos, inv, reach);
                hr = hr && collide_box<false>(rlo, rhi, pos, inv, reach);
            }
        }
        const uint32_t bl = __ballot_sync(0xffffffffu, hl) & group, br = __ballot_sync(0xffffffffu, hr) & group;
        const uint32_t bt = __ballot_sync(0xffffffffu, tri) & group;
        if (tri) leaf[leaves + (uint32_t)__popc(bt & before)] = (uint32_t)w.z;
        leaves += (uint32_t)__popc(bt);
        const uint32_t at = tail + (uint32_t)__popc(bl & before) + (uint32_t)__popc(br & before);
        if (hl) queue[at % RING] = (uint32_t)w.x;
        if (hr) queue[(at + (hl ? 1u : 0u)) % RING] = (uint32_t)w.y;
        head = (head + k) % RING;
        tail = (tail + (uint32_t)__popc(bl) + (uint32_t)__popc(br)) % RING;
        steps += k;
        if (active && steps > 4u * n_nodes + 4u) {  // not a tree: report and stop
            if (gl == 0) atomicOr(err, DEV_ERR_KEY_RANGE);
            active = false;
        }
        if (head == tail) active = false;
        __syncwarp();
    }
}

}  // namespace

extern "C" GBSPH_API int gbsph_bvh_collide(gbsph_bvh_t h, const gbsph_fluid3d_params* params, float* position,
                                           float* velocity, float* force, size_t n_particles, const float* vertex,
                                           size_t n_vertices, const uint32_t* index, void* stream) {
    if (!h || !params) return GBSPH_ERR_ARGUMENT;
    if (!position || !velocity || !force || !vertex || !index)
        return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "null buffer");
    if (h->n == 0) return fail(&h->last_error, GBSPH_ERR_STATE, "collide before a BVH was built");
    if (n_particles == 0) return GBSPH_OK;
    if (n_particles > 0xFFFFFFFFull || n_vertices == 0 || n_vertices > 0xFFFFFFFFull)
        return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "bad particle or vertex count");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    cudaStream_t s = (cudaStream_t)stream;
    CollideParams P;
    P.dt = params->deltaTime;
    P.radius = params->particleRadius;
    P.pconst = params->pressureConstant;
    P.density = params->density;
    P.h = params->cellSize;
    P.mass = params->mass;
    const uint32_t np = (uint32_t)n_particles;
    auto collide = [&](auto kern, uint32_t lanes) {
        const uint32_t per = COLLIDE_THREADS / lanes;
        kern<<<(np + per - 1u) / per, COLLIDE_THREADS, 0, s>>>(reinterpret_cast<float4*>(force), reinterpret_cast<float4*>(position),
                                                               reinterpret_cast<float4*>(velocity), np, P, h->node, h->root, 2 * h->n - 1,
                                                               index, reinterpret_cast<const float4*>(vertex), (uint32_t)n_vertices, h->err);
    };
    const uint32_t nodes = 2 * h->n - 1;
    if (nodes < 16 && np >= 1u << 16) collide(k_collide_bvh<1, 16>, 1);
    else if (nodes < 128) collide(k_collide_bvh<4, 128>, 4);
    else collide(k_collide_bvh<8, QUEUE_SIZE>, 8);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    return GBSPH_OK;
}

// ------------------------------------------------------------------------------------------
// oclBvhLines replacement.
// ------------------------------------------------------------------------------------------
struct gbsph_bvh_lines_s {
    int device = 0;
    gbsph_radix_sort_t sort = nullptr;
    uint32_t cap = 0;  // segments the buffers hold
    uint32_t n = 0;    // segments of the last build
    void* block = nullptr;
    gbsph_bvh2d_node* node = nullptr;
    uint32_t *key = nullptr, *val = nullptr, *root = nullptr;
    unsigned long long* link = nullptr;
    std::string last_error;
};

namespace {

int ensure_lines(gbsph_bvh_lines_s* h, uint32_t n) {
    if (n <= h->cap && h->block) return GBSPH_OK;
    if (h->block) cudaFree(h->block);
    h->block = nullptr;
    h->cap = 0;
    const size_t nn = 2 * (size_t)n, m = n;
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t bytes = al(nn * sizeof(gbsph_bvh2d_node)) + 2 * al(m * 4) + al(m * 8) + 256;
    GBSPH_CUDA_TRY(&h->last_error, cudaMalloc(&h->block, bytes));
    char* p = (char*)h->block;
    h->node = (gbsph_bvh2d_node*)p;
    p += al(nn * sizeof(gbsph_bvh2d_node));
    h->key = (uint32_t*)p;
    p += al(m * 4);
    h->val = (uint32_t*)p;
    p += al(m * 4);
    h->link = (unsigned long long*)p;
    p += al(m * 8);
    h->root = (uint32_t*)p;
    h->cap = n;
    return GBSPH_OK;
}

}  // namespace

extern "C" {

GBSPH_API int gbsph_bvh_lines_create(gbsph_bvh_lines_t* out) {
    if (!out) return GBSPH_ERR_ARGUMENT;
    *out = nullptr;
    gbsph_bvh_lines_s* h = new gbsph_bvh_lines_s();
    int rc = cudaGetDevice(&h->device) == cudaSuccess ? GBSPH_OK : GBSPH_ERR_CUDA;
    if (!rc) rc = gbsph_radix_sort_create(&h->sort);
    if (rc) {
        cudaGetLastError();
        if (h->sort) gbsph_radix_sort_destroy(h->sort);
        delete h;
        return rc;
    }
    *out = h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_lines_destroy(gbsph_bvh_lines_t h) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    cudaSetDevice(h->device);
    if (h->block) cudaFree(h->block);
    if (h->sort) gbsph_radix_sort_destroy(h->sort);
    delete h;
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_lines_compute(gbsph_bvh_lines_t h, const float* vertex, size_t n_vertices, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    if (!vertex) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "null buffer");
    const size_t nl = n_vertices / 2;
    if (nl < 2) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "a BVH needs at least 2 segments");
    if (nl > SORT_MAX_KEYS - SORT_TILE) return fail(&h->last_error, GBSPH_ERR_TOO_LARGE, "too many segments");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    const uint32_t n = (uint32_t)nl, m = n - 1;
    int rc = ensure_lines(h, n);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const float2* v2 = reinterpret_cast<const float2*>(vertex);
    k_bvh_morton_lines<<<grid(n), BVH_THREADS, 0, s>>>(v2, n, h->key, h->val);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    rc = gbsph_radix_sort_compute(h->sort, h->key, h->val, n, n, 0, 32, stream);
    if (rc) return fail(&h->last_error, rc, std::string("sort: ") + gbsph_radix_sort_last_error(h->sort));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemsetAsync(h->link, 0xFF, (size_t)m * 8, s));
    k_bvh_tree<SegTree><<<(n + TREE_THREADS - 1) / TREE_THREADS, TREE_THREADS, 0, s>>>(h->key, h->val, n, SegTree::Prims{v2}, h->node, h->link, h->root);
    GBSPH_CUDA_TRY(&h->last_error, cudaGetLastError());
    h->n = n;
    return GBSPH_OK;
}

GBSPH_API gbsph_bvh2d_node* gbsph_bvh_lines_get_node_buffer(gbsph_bvh_lines_t h, size_t* count) {
    if (!h) return nullptr;
    if (count) *count = h->n ? 2 * (size_t)h->n - 1 : 0;
    return h->node;
}

GBSPH_API size_t gbsph_bvh_lines_get_node_count(gbsph_bvh_lines_t h) { return h && h->n ? 2 * (size_t)h->n - 1 : 0; }

GBSPH_API int gbsph_bvh_lines_get_root_node(gbsph_bvh_lines_t h, uint32_t* root, void* stream) {
    if (!h || !root) return GBSPH_ERR_ARGUMENT;
    if (!h->root) return fail(&h->last_error, GBSPH_ERR_ARGUMENT, "no build yet");
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    GBSPH_CUDA_TRY(&h->last_error, cudaMemcpy(root, h->root, 4, cudaMemcpyDeviceToHost));
    return GBSPH_OK;
}

GBSPH_API int gbsph_bvh_lines_sync_status(gbsph_bvh_lines_t h, void* stream) {
    if (!h) return GBSPH_ERR_ARGUMENT;
    GBSPH_CUDA_TRY(&h->last_error, cudaSetDevice(h->device));
    GBSPH_CUDA_TRY(&h->last_error, cudaStreamSynchronize((cudaStream_t)stream));
    const int src = gbsph_radix_sort_sync_status(h->sort, stream);
    if (src) return fail(&h->last_error, src, std::string("sort: ") + gbsph_radix_sort_last_error(h->sort));
    return GBSPH_OK;
}

GBSPH_API const char* gbsph_bvh_lines_last_error(gbsph_bvh_lines_t h) { return h ? h->last_error.c_str() : "null handle"; }

}  // extern "C"
