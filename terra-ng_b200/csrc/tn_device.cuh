// Shared device helpers for the sm_100a kernels: layout arithmetic, TMA bulk
// copies with bounded mbarrier waits, and the error flag every bounded wait
// reports to.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace tn {


// Device-side error codes written to the per-context error word.
enum DeviceError : int {
    kDevOk             = 0,
    kDevMbarrierTimeout = 1,
    kDevBadLaunch      = 2,
};

// Nodal index (diamond, x, y, r), r fastest (grid/grid_types.hpp:12-30).
__host__ __device__ __forceinline__ int64_t node_index(int nl, int nr, int d, int x, int y, int r)
{
    return ((static_cast<int64_t>(d) * nl + x) * nl + y) * nr + r;
}

// ---------------------------------------------------------------------------
// mbarrier + bulk copy (cp.async.bulk, no multicast).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// One try, suspended by the hardware for a short while at most. No time hint: with one the wait sleeps on a coarse timer.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_timer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Wait for phase `parity` of `bar`, giving up after ~`limit_ns`. Returns false
// on timeout; the caller records the error and stops using the buffer.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns = 1000000000ull)
{
    for (int i = 0; i < 32; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    while (true) {
        for (int i = 0; i < 16; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_timer_ns() - t0 > limit_ns) return false;
    }
}

// 1-D bulk copy global -> this CTA's shared memory, completing on `bar`.
// dst and src must be 16-byte aligned and bytes a multiple of 16.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void report_error(int* err, int code)
{
    if (err) atomicCAS(err, 0, code);
}

// Chained launches (programmatic dependent launch). A kernel launched with launch_chained may start while the kernel
// before it in its stream drains, so every thread of it calls chain_enter() before it touches memory that another kernel
// writes: it waits until that kernel has completed and its writes are visible (and that kernel has waited for the one
// before it), and then lets the next one start early. Such kernels read mutable memory through pointers without
// __restrict__, so that no load counts as invariant and moves above the wait.
// What it gives: about 1 to 2 us a launch, which is most of what the operators, sums and updates of the small levels take.
// Level-4 velocity solve 15.8 -> 12.6 ms, level-6 mixed preconditioner 2.97 -> 2.64 ms, level-3 apply 14.1 -> 12.7 us.
__device__ __forceinline__ void chain_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim            = grid;
    cfg.blockDim           = block;
    cfg.dynamicSmemBytes   = smem;
    cfg.stream             = st;
    cfg.attrs              = at;
    cfg.numAttrs           = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename T>
__device__ __forceinline__ T shfl_up(T v, int delta)
{
    return __shfl_up_sync(0xffffffffu, v, delta);
}
template <typename T>
__device__ __forceinline__ T shfl_down(T v, int delta)
{
    return __shfl_down_sync(0xffffffffu, v, delta);
}

}  // namespace tn
