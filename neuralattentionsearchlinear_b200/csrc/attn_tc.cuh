// Definitions shared by the tcgen05 attention kernels (attn_fwd_tc.cu, attn_bwd.cu).
#pragma once
#include "attn_walk.cuh"
#include "tc_common.cuh"

namespace natsl {

constexpr int TC_THREADS = 320;             // backward: TMA producer, MMA issuer, 8 softmax warps
constexpr uint32_t TC_TMEM_COLS = 256;      // backward: tensor-memory columns of a CTA (two CTAs per SM)

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

}  // namespace natsl
