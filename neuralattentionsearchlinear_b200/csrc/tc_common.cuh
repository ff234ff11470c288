// Blackwell (sm_100a) building blocks used by the tensor-core kernels: mbarrier waits with an
// iteration limit, TMA tiled loads, tcgen05 MMA / commit / TMEM load-store, shared-memory matrix
// descriptors for 128-byte-swizzled tiles, and host-side tensor-map encoding.
//
// Shared-memory operand tiles are [rows][64 bf16] sub-tiles with 128-byte rows, 1024-byte aligned,
// 16-byte chunk index XOR (row & 7): exactly what a TMA box of 64 bf16 x rows with SWIZZLE_128B
// writes, and what swz<128>() of common.cuh addresses.
//   K-major operand (row = M or N index, 64 elements of K per sub-tile):  SBO = 1024 B,
//       one MMA K-step (16 elements) = +32 B on the start address.
//   MN-major operand (row = K index, 64 elements of N per sub-tile): SBO = 1024 B (8 K rows),
//       LBO = distance between 64-column sub-tiles, one K-step (16 rows) = +2048 B.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace natsl {

// ------------------------------------------------------------------ device status word
// Set by kernels whose bounded waits gave up; read (and cleared) by natsl_device_status().
// (2 = misaligned shared memory in a tensor-core kernel, 3 = a caller-given capacity was too small.)
enum : int { NATSL_DEV_OK = 0, NATSL_DEV_WAIT_TIMEOUT = 1, NATSL_DEV_CAPACITY = 3 };
// Host: device address of the status word on the current device (looked up once per device).
int status_word_ptr(int** out);

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait with an iteration limit.  On expiry the status word is set and false is returned; callers
// then skip their remaining work and fall through to the common teardown (never spin forever).
constexpr int kWaitLimit = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status) {
    for (int i = 0; i < kWaitLimit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    return false;
}
// The same as a loop that the compiler does not unroll: less code, which pays where a kernel is larger than the instruction
// cache and costs where the chain of waits is what bounds it (K = 192, V = 384 walk: 222 us unrolled, 242 us so).
__device__ __forceinline__ bool mbar_wait_small(uint32_t bar, uint32_t parity, int* status) {
#pragma unroll 1
    for (int i = 0; i < kWaitLimit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    return false;
}

// The same for kernels with many waits: a whole warp waits, and the caller records the status once, at its end.  A few
// instructions per wait where the one above takes two dozen: code that no longer fits the instruction cache costs more than
// the waits do.  (A try suspends the warp for some 25 us, so the limit is a few seconds.)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
    bool done = false;
#pragma unroll 1
    for (int i = 0; i < (1 << 18) && !done; ++i) done = mbar_try_wait(bar, parity);
    return __all_sync(0xffffffffu, done);
}

// ------------------------------------------------------------------ TMA
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
// Tiled store of one box from shared memory (bulk async-group; rows past the tensor's extent are clipped).  The
// writers of the shared-memory tile fence (fence_async_smem) and synchronise with the issuing thread first; that
// thread commits and, before the tile is reused or the CTA exits, waits for the reads with tma_store_wait_read.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// L2 prefetch of one box (no shared-memory destination, no completion tracking)
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];"
                 ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ------------------------------------------------------------------ tcgen05
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 64-bit shared-memory matrix descriptor, SWIZZLE_128B, sm_100 version bit set.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// 32-bit instruction descriptor: bf16 x bf16 -> fp32, A K-major, B K-major or MN-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
// The ones below are called by a whole converged warp and issued by one elected lane (always the same one).  The control
// flow stays uniform, so the descriptors are formed on the uniform datapath; behind a branch on the lane every operand of
// every product is moved there one by one.
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum), "r"(0u)
        : "memory");
}
// Four K-steps (64 elements of K) in one go, descriptors given by their low words (umma_desc_lo; the high word is that of
// umma_desc(., ., 1024)): one election for the four, and the steps differ by constants, which the uniform datapath adds.
// Descriptors formed anew for every product cost the issuing warp about a hundred cycles each.
// (With it, alone in a graph: the Mamba2 walk of that time over 64 x 1024 tokens, H = 32 29 % less; gated delta rule, B = 8, T = 4096, H = 16,
// 128/128, preparation and walk together 357 -> 346 us.  Under the power limit, where the clock gives what the cycles save, the
// latter do not change: 177 - 195 and 176 - 198 us at 1.74 - 1.96 GHz.)
constexpr uint32_t UMMA_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr, uint32_t lbo_bytes) {
    return ((saddr >> 4) & 0x3FFF) | ((lbo_bytes >> 4) << 16);
}
// A and B from shared memory; STEP_A / STEP_B: 16-byte units between K-steps (2 for a K-major operand, 128 for an MN-major one)
template <int STEP_A, int STEP_B>
__device__ __forceinline__ void umma_ss_x4(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n .reg .pred p, t, e;\n .reg .b64 a, b;\n .reg .b32 x, y;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.u32 t, 0, 0;\n elect.sync _|e, 0xffffffff;\n"
        " mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n"
        " add.u32 x, %1, %6;\n add.u32 y, %2, %7;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n"
        " add.u32 x, x, %6;\n add.u32 y, y, %7;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n"
        " add.u32 x, x, %6;\n add.u32 y, y, %7;\n mov.b64 a, {x, %5};\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n}\n"
        ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accum), "n"(UMMA_DESC_HI), "n"(STEP_A), "n"(STEP_B)
        : "memory");
}
// A from tensor memory (8 columns per K-step)
template <int STEP_B>
__device__ __forceinline__ void umma_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n .reg .pred p, t, e;\n .reg .b64 b;\n .reg .b32 x, y;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.u32 t, 0, 0;\n elect.sync _|e, 0xffffffff;\n"
        " mov.b64 b, {%2, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n"
        " add.u32 x, %1, 8;\n add.u32 y, %2, %6;\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, t;\n"
        " add.u32 x, x, 8;\n add.u32 y, y, %6;\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, t;\n"
        " add.u32 x, x, 8;\n add.u32 y, y, %6;\n mov.b64 b, {y, %5};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, t;\n}\n"
        ::"r"(d_tmem), "r"(a_tmem), "r"(blo), "r"(idesc), "r"(accum), "n"(UMMA_DESC_HI), "n"(STEP_B)
        : "memory");
}
// mbarrier arrives once every tcgen05 operation issued so far by the elected lane has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile(
        "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}

// 32 lanes x 32 columns of 32-bit: thread `lane` of the warp gets 32 consecutive columns of its TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16 lanes x 64 columns of 32-bit in the accumulator-fragment layout: thread t of the warp gets, for each group
// of 8 columns k = 0..7, r[4k], r[4k+1] = (lane t/4, columns 8k + 2(t%4), +1) and r[4k+2], r[4k+3] = the same
// columns of lane t/4 + 8.  The lane field of taddr is the first of the 16 lanes (a multiple of 16 inside the
// warp's own quarter of 32 lanes).
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// ------------------------------------------------------------------ host: tensor maps
// bf16 tensor [B][T][H][D] (token-major, contiguous) viewed as a 4-D TMA tensor (D, H, T, B) with
// boxes of `box_cols` (64 or 32) elements x `box_rows` tokens of one head, swizzle over the box row (128 or 64 bytes: the
// layout of swz<128> / swz<64>), zero fill out of range.
int encode_bthd_map(CUtensorMap* out, const void* base, int B, int T, int H, int D, int box_rows, const char* who,
                    int box_cols = 64);
// bf16 rows [B][T][D] (contiguous, D any multiple of 8) in boxes of 64 elements x `box_rows` rows, 128-byte swizzle, zero fill out
// of range.
int encode_rows_map(CUtensorMap* out, const void* base, int B, int T, int D, int box_rows, const char* who);

}  // namespace natsl
