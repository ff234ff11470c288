// Definitions shared by the tcgen05 attention kernels (attn_fwd_tc.cu, attn_bwd.cu).
#pragma once
#include "attn_walk.cuh"
#include "tc_common.cuh"

namespace natsl {

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Cluster launch control: ask for a block of this grid that has not started; the 16-byte answer lands in shared memory.
__device__ __forceinline__ void request_block(uint32_t dst, uint32_t bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(dst), "r"(bar) : "memory");
}
__device__ __forceinline__ bool taken_block(uint32_t src, int& x) {
    uint32_t ok, rx;
    asm volatile(
        "{\n .reg .pred p;\n .reg .b128 r;\n .reg .b32 y, z, w;\n ld.shared.b128 r, [%2];\n"
        " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n selp.u32 %0, 1, 0, p;\n mov.u32 %1, 0;\n"
        " @p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, y, z, w}, r;\n}\n"
        : "=&r"(ok), "=&r"(rx)
        : "r"(src)
        : "memory");
    x = (int)rx;
    return ok != 0;
}

}  // namespace natsl
