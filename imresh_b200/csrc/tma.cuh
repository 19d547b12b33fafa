// Asynchronous bulk copies (TMA) and mbarriers for sm_100a, as inline PTX.
//
// Only CTA-local loads are used: cp.async.bulk (1D, contiguous rows) and
// cp.async.bulk.tensor.2d (column tiles through a CUtensorMap), each
// completing on an mbarrier with a transaction byte count.  No cluster
// multicast is used anywhere.  Every wait is bounded by %globaltimer: a wait
// that runs past its limit returns false, the caller records an error in the
// job state and returns, so a copy that never lands cannot hang the GPU.  The
// limit of a job's waits is JobDev::wait_ns (0: kWaitNs).  A CTA that gave up
// first waits, bounded by kWaitNs, for every copy it still has in flight
// (kDrainNs), so no copy can land in the shared memory of an exited CTA even
// when a short limit made it give up early.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace imr {

constexpr uint64_t kWaitNs = 500000000ull;   // default: give up on a copy after 0.5 s
constexpr uint64_t kDrainNs = kWaitNs;       // bound of the in-flight drain after giving up

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// make the initialised barriers visible to the async proxy
__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// order this thread's generic-proxy shared-memory accesses before later
// async-proxy (TMA) accesses of the same memory
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for the phase with the given parity; false once limit_ns
// have passed without it (limit_ns == 0: kWaitNs).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint64_t limit_ns = kWaitNs)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t lim = limit_ns ? limit_ns : kWaitNs;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > lim) return false;
    return true;
}

__device__ __forceinline__ void mbar_inval(uint64_t *bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// contiguous global -> shared copy; dst, src 16-byte aligned, bytes % 16 == 0
__device__ __forceinline__ void tma_load_1d(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// 2D tile of a tensor map at element coordinates (x inner, y outer);
// x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// 2D tile of shared memory -> global through a tensor map (bulk async group);
// coordinates must be non-negative, x * element size a multiple of 16 bytes.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int x, int y, const void *src)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x),
                 "r"(y), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// wait until the committed bulk stores have read their shared-memory source
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// wait until the committed bulk stores are complete
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }


// ---- programmatic dependent launch ------------------------------------------------
// A pass launched with the attribute may start before the pass ahead of it has
// ended: once all of that pass's CTAs have called pdl_trigger or exited.  What
// it does before pdl_wait may touch only what no pass writes (work lists, job
// descriptions, tables); pdl_wait returns when the passes ahead are complete
// and their writes visible to ordinary loads.  What a pass writes is never read
// with __ldg or through a const __restrict__ pointer: a non-coherent load wants
// memory that stays unwritten for the whole life of the kernel, and that life now
// overlaps the writing pass's.  A pass triggers half-way through its last item,
// after its own pdl_wait, so no pass runs beside the one before the last.  Both
// are no-ops in a launch without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- per-thread asynchronous copies (no alignment beyond the element's) --------
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

}  // namespace imr
