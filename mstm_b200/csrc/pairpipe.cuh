// pairpipe.cuh -- mbarrier waits and bulk copies (cp.async.bulk) of the pair
// translation kernel.
#pragma once
#include "common.cuh"

namespace pairpipe {

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(uint64_t* bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_expect(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(su32(dst)),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mb_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(su32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
constexpr int WAIT_POLLS = 1 << 22;
// bounded wait: gives up after `limit` polls (the kernels then record
// MSTMG_ERR_CUDA and return instead of hanging)
__device__ __forceinline__ bool mb_wait(uint64_t* bar, uint32_t parity, int limit = WAIT_POLLS)
{
    for (int it = 0; it < limit; ++it)
        if (mb_try(bar, parity)) return true;
    return false;
}

}  // namespace pairpipe
