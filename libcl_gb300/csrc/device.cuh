// device.cuh -- device-side helpers: relaxed global loads/stores for look-back words,
// mbarrier and asynchronous-copy wrappers with bounded waits, small vector ops.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gbsph {

// Bounded waits: a kernel that has polled for WAIT_LIMIT_NS of wall-clock time (read from
// %globaltimer every 32 polls) gives up, sets an error bit and moves on.
constexpr uint64_t WAIT_LIMIT_NS = 1000000000ull;

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Poll-loop guard: call once per poll; returns true once the wait has lasted too long.
struct WaitBudget {
    uint64_t start = 0;
    uint32_t polls = 0;
    __device__ __forceinline__ bool expired() {
        if ((++polls & 31u) != 0u) return false;
        const uint64_t now = globaltimer_ns();
        if (start == 0) {
            start = now;
            return false;
        }
        return now - start > WAIT_LIMIT_NS;
    }
};

__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_gpu(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Load of data that another CTA of the same launch wrote before a grid-wide barrier: through
// L2 only (ld.global.cg), never from a copy an earlier phase left in this SM's L1 or
// read-only cache. COH = false is an ordinary load.
template <bool COH, class T>
__device__ __forceinline__ T ld_phase(const T* p) {
    if constexpr (COH) return __ldcg(p);
    else return *p;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory load / store by 32-bit shared-window address (volatile: they stay in program
// order with each other and with the barriers around them; the store also orders the
// compiler's own shared-memory accesses around it).
__device__ __forceinline__ float4 lds_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_u16(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}

// ---- mbarrier + cp.async (global -> shared) -------------------------------------------

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}

// Ends the object's life, so that its shared memory may be used for something else.
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(bar)) : "memory");
}

// One 16-byte asynchronous copy (through L2 only; generic proxy), and this thread's arrival on
// `bar` once all its copies so far have landed (one of the barrier's expected arrivals).
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src_gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src_gmem) : "memory");
}
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\t"
        "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_addr(bar)),
        "r"(bytes)
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(10000u)  // suspended for up to 10 us a poll
        : "memory");
    return ok != 0;
}

// Bounded wait on phase `parity`. Returns false if the limit was reached.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    WaitBudget budget;
    while (!mbar_try_wait(bar, parity)) {
        if (budget.expired()) return false;
    }
    return true;
}

// A wait for threads that may be at work for long: the limit begins again whenever `progress`, a word
// of shared memory that they count on, has changed.
__device__ __forceinline__ bool mbar_wait_progress(uint64_t* bar, uint32_t parity, const volatile uint32_t* progress) {
    uint32_t polls = 0, seen = 0;
    uint64_t start = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++polls & 31u) != 0u) continue;
        const uint64_t now = globaltimer_ns();
        const uint32_t p = *progress;
        if (start == 0 || p != seen) {
            start = now;
            seen = p;
        } else if (now - start > WAIT_LIMIT_NS) {
            return false;
        }
    }
    return true;
}

// Least and greatest value over the warp's 32 lanes (NaNs are left out while another lane has a number).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ uint32_t warp_max(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }

// ---- packed FP32 (f32x2, sm_100 and later): two lanes of FP32 per 64-bit register ----------
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// ---- float4 helpers ---------------------------------------------------------------------
__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

}  // namespace gbsph
