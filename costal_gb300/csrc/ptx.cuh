// mbarrier and TMA helpers shared by the coarse kernels, and the tensor map encoder's entry point.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace costal {

constexpr long long WAIT_LIMIT = 1ll << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier --------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false (and the flag raised) if the phase never completes. Every 1024 polls the wait
// also checks the global flag, so once any thread of any CTA has given up, every later wait of the
// launch returns at once and the kernel drains in microseconds.
// Roles that are not the bottleneck (TMA, MMA issue) sleep between polls so that they do not take
// issue slots from the epilogue warps that share their schedulers.
// One more poll of a wait (polls counts them): false once the wait has to give up.
__device__ __forceinline__ bool wait_budget(unsigned long long* timeout_flag, long long& polls) {
    if ((++polls & 1023) == 0) {
        if (*reinterpret_cast<volatile unsigned long long*>(timeout_flag)) return false;
        if (polls >= WAIT_LIMIT) {
            atomicExch(timeout_flag, 1ull);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ bool mbar_wait_long(uint64_t* bar, uint32_t parity, unsigned long long* timeout_flag, bool sleep) {
    long long polls = 0;
    while (wait_budget(timeout_flag, polls)) {
        if (mbar_try_wait(bar, parity)) return true;
        if (sleep) __nanosleep(64);
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned long long* timeout_flag,
                                          bool sleep) {
    return mbar_try_wait(bar, parity) || mbar_wait_long(bar, parity, timeout_flag, sleep);
}

// The wait of a role that has given up for copies or MMAs of its own that are still in flight, which must not
// outlive the CTA's shared memory: bounded too (65,536 polls of 64 ns and more, where they take microseconds).
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    for (int polls = 0; polls < 65536 && !mbar_try_wait(bar, parity); ++polls) __nanosleep(64);
}
// The loads of a ring whose next stage is s with producer parity ph (full[q] of an unused stage passes at once).
__device__ __forceinline__ void drain_ring(uint64_t* full, int stages, int s, uint32_t ph) {
    for (int q = 0; q < stages; ++q) mbar_drain(&full[q], q < s ? ph ^ 1u : ph);
}

// ---- TMA ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

}  // namespace costal
