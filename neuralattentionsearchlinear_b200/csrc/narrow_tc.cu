// Narrow projections of a layer: y[t, n] = x[t, :] . W[n, :] for a few rows n (2 H decays and betas, or 2 HQ mixing logits) with
// the pointwise steps behind them (src/nats/layers/natsl_attn_gdn.py:461-480, 590-600, src/nats/layers/natsl_attn_mamba2.py:402-440).
// Bound by reading x once.  One CTA = 128 tokens of a sequence x up to 64 rows of W: TMA brings x and W in steps of 64 features
// through a ring of stages, tcgen05 adds the products up in tensor memory, two threads per token then work on a half of its row of
// results each.  (On mma.sync, fragments straight from global memory, the registers left one CTA on an SM: 16 x 4096 tokens of 1024
// features, 32 rows took 72 us, here 33 us; the traffic needs 21 us.  What a small call is bound by is the issue of a step: a
// commit as long as its products, and every further TMA box, so W comes in one box per matrix and stages are given back in pairs:
// 4 x 1030 tokens of 2048 features 32 -> 21 us.)
//   warp 8 TMA producer, warp 9 MMA issuer, warps 0-7 two threads per TMEM lane, half of the columns each.
// Columns are padded to groups of eight: a group comes from w0 or from w1, and rows past a matrix' end read as zeros.
#include "layer_fwd.cuh"
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

using bf16 = __nv_bfloat16;
constexpr int NW_BACK = 2;                                   // stages given back together: a commit costs as much as a step's products
constexpr int NW_MAX_STAGES = 8, NW_EPI = 256, NW_THREADS = NW_EPI + 64, NW_TOK = 128;

struct NarrowPlan {
    int n0p;                                                 // columns of w0, padded to groups of eight
    int rows;                                                // rows of a box of W
    int steps, stages;
};
template <int NT>
struct NwSmem {                                              // the ring of stages lies behind the rest
    static constexpr int stage = NW_TOK * 128 + NT * 128;    // x tile, then the rows of W
    static constexpr int vec = 0;                            // A, dt_bias: 64 floats each; the scan's carries [2][64]
    static constexpr int bars = vec + 4 * 64 * 4;
    static constexpr int slot = bars + (2 * NW_MAX_STAGES + 1) * 8;
    static constexpr int ring = 2048;
    static constexpr uint32_t tmem = NT < 32 ? 32 : NT;
    static_assert(stage % 1024 == 0 && slot + 4 <= ring, "swizzled tiles start on 1024 bytes");
};

__device__ __forceinline__ float rb(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ float ldw(const void* p, int f32, int i) {
    return f32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}

// 32 lanes x N columns of 32-bit, N = 8, 16 or 32
template <int N>
__device__ __forceinline__ void tmem_row(uint32_t taddr, uint32_t (&r)[N]) {
    if constexpr (N == 32) tmem_ld32(taddr, r);
    else if constexpr (N == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                       "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    tmem_ld_wait();
}

template <int NT>
__global__ void __launch_bounds__(NW_THREADS, NT == 64 ? 3 : 4)
narrow_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
                 const __grid_constant__ CUtensorMap map_w1, const NarrowArgs a, const NarrowPlan p, int* status) {
    using L = NwSmem<NT>;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int t0 = blockIdx.x * NW_TOK, b = blockIdx.y, z0 = blockIdx.z * NT, n0p = p.n0p;          // z0: first column (padded)
    float* s_a = reinterpret_cast<float*>(smem + L::vec);
    float* s_bias = s_a + 64;
    float* s_carry = s_bias + 64;
    const uint32_t bar_full = sbase + L::bars, bar_empty = bar_full + 8 * NW_MAX_STAGES, bar_done = bar_empty + 8 * NW_MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::slot);
    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 1);
        }
        mbar_init(bar_done, 1);
        mbar_fence_init();
    }
    if (warp == 8) tmem_alloc(smem_u32(tmem_slot), L::tmem);
    if (a.mode == 0 && tid < NT && z0 + tid < a.n0) {
        s_a[tid] = -expf(ldw(a.A_log, a.alog_f32, z0 + tid));
        s_bias[tid] = ldw(a.dt_bias, a.dt_f32, z0 + tid);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 8) {
        if (lane == 0) {
            int boxes = 0;
            for (int j = 0; j < NT; j += p.rows) boxes += z0 + j < n0p + a.n1;
#pragma unroll 1
            for (int k = 0, s = 0, turn = 0; k < p.steps; ++k) {
                const uint32_t st = sbase + L::ring + s * L::stage, full = bar_full + 8 * s;
                if (turn && (s & (NW_BACK - 1)) == 0) mbar_wait_small(bar_empty + 8 * s, (turn - 1) & 1, status);
                mbar_expect_tx(full, (NW_TOK + boxes * p.rows) * 128);
                tma_load_4d(st, &map_x, k * 64, 0, t0, b, full);
#pragma unroll 1
                for (int j = 0; j < boxes; ++j) {
                    const int n = z0 + j * p.rows;
                    tma_load_4d(st + NW_TOK * 128 + j * p.rows * 128, n < n0p ? &map_w0 : &map_w1, k * 64, 0, n < n0p ? n : n - n0p, 0, full);
                }
                if (++s == p.stages) { s = 0; ++turn; }
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        constexpr uint32_t id = umma_idesc_bf16(128, NT, false);
#pragma unroll 1
        for (int k = 0, s = 0, turn = 0; k < p.steps; ++k) {
            const uint32_t st = sbase + L::ring + s * L::stage;
            mbar_wait_small(bar_full + 8 * s, turn & 1, status);
            __syncwarp();
            tc_fence_after();
            umma_ss_x4<2, 2>(tmem, umma_desc_lo(st, 16), umma_desc_lo(st + NW_TOK * 128, 16), id, k > 0);
            if ((s & (NW_BACK - 1)) == NW_BACK - 1) umma_commit(bar_empty + 8 * (s - NW_BACK + 1));
            if (++s == p.stages) { s = 0; ++turn; }
        }
        umma_commit(bar_done);
        __syncwarp();
    } else {
        // two warps per quarter of the lanes, half of the columns each
        constexpr int NC = NT / 2;
        const int row = tid & 127, c0 = (tid >> 7) * NC, n_first = z0 + c0;
        const int t = t0 + row;
        const bool ok = t < a.T;
        const long tok = (long)b * a.T + t;
        mbar_wait_small(bar_done, 0, status);
        __syncwarp();
        tc_fence_after();
        uint32_t r[NC];
        tmem_row<NC>(tmem + ((uint32_t)(warp & 3) << 21) + c0, r);
        if (a.mode == 1) {
#pragma unroll
            for (int i = 0; i < NC; i += 8) {
                const int n = n_first + i;
                if (n >= a.n0) break;
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {                  // softmax over a pair (a larger logit of +inf: NaN, by m - m)
                    const float l0 = rb(__uint_as_float(r[i + 2 * e])), l1 = rb(__uint_as_float(r[i + 2 * e + 1]));
                    const float d = l0 - l1, m = fmaxf(l0, l1);
                    const float ex = expf(-fabsf(d)) + (m - m), hi = rcp_newton(1.f + ex), lo = ex * hi;
                    o[e] = d < 0.f ? pack_bf16(lo, hi) : pack_bf16(hi, lo);
                }
                if (!ok) continue;
                bf16* out = a.out + tok * a.n0 + n;
                if (n + 8 <= a.n0 && a.wide) *reinterpret_cast<uint4*>(out) = make_uint4(o[0], o[1], o[2], o[3]);
                else
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + 2 * e < a.n0) *reinterpret_cast<uint32_t*>(out + 2 * e) = o[e];
            }
        } else {
#pragma unroll
            for (int i = 0; i < NC; i += 4) {
                const int n = n_first + i, nb = n - n0p;     // column of w0; of w1
                if (n < a.n0) {
                    float g[4], d[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        g[e] = d[e] = 0.f;
                        if (ok && n + e < a.n0) {
                            const float zz = rb(__uint_as_float(r[i + e])) + s_bias[c0 + i + e];
                            d[e] = zz > 20.f ? zz : log1pf(expf(zz));
                            g[e] = s_a[c0 + i + e] * d[e];
                        }
                        r[i + e] = __float_as_uint(g[e]);
                    }
                    if (!ok) continue;
                    float *pg = a.g + tok * a.n0 + n, *pd = a.dt ? a.dt + tok * a.n0 + n : nullptr;
                    if ((a.n0 & 3) == 0) {
                        *reinterpret_cast<float4*>(pg) = make_float4(g[0], g[1], g[2], g[3]);
                        if (pd) *reinterpret_cast<float4*>(pd) = make_float4(d[0], d[1], d[2], d[3]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (n + e < a.n0) {
                                pg[e] = g[e];
                                if (pd) pd[e] = d[e];
                            }
                    }
                } else if (nb >= 0 && nb < a.n1 && ok) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float y = rb(__uint_as_float(r[i + e])), ex = expf(-fabsf(y)), hi = rcp_newton(1.f + ex);
                        v[e] = rb(y < 0.f ? ex * hi : hi);
                        if (a.neg_eigval) v[e] *= 2.f;
                    }
                    bf16* out = a.out + tok * a.n1 + nb;
                    if ((a.n1 & 3) == 0) *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
                    else
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (nb + e < a.n1) out[e] = __float2bfloat16(v[e]);
                }
            }
            if (a.gcs) {                                     // chunk-local cumsum: two warps are a chunk
                float* carry = s_carry + ((warp >> 1) & 1) * 64 + c0;
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    float x = n_first + i < a.n0 ? __uint_as_float(r[i]) : 0.f;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float u = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += u;
                    }
                    r[i] = __float_as_uint(x);
                    if (!(warp & 1) && lane == 31) carry[i] = x;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(NW_EPI) : "memory");
                if (ok) {
                    float* pc = a.gcs + tok * a.n0 + n_first;
#pragma unroll
                    for (int i = 0; i < NC; i += 4) {
                        float v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[e] = __uint_as_float(r[i + e]) + ((warp & 1) ? carry[i + e] : 0.f);
                        if ((a.n0 & 3) == 0) {
                            if (n_first + i < a.n0) *reinterpret_cast<float4*>(pc + i) = make_float4(v[0], v[1], v[2], v[3]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (n_first + i + e < a.n0) pc[i + e] = v[e];
                        }
                    }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, L::tmem);
}

template <int NT>
int launch(const NarrowArgs& a, int n0p, int B, cudaStream_t st) {
    using L = NwSmem<NT>;
    const long cols = (n0p + a.n1 + NT - 1) / NT;
    NarrowPlan p = {};
    p.n0p = n0p;
    const dim3 grid((a.T + NW_TOK - 1) / NW_TOK, B, (unsigned)cols);
    const long ctas = (long)grid.x * B * cols;
    p.steps = (a.Kdim + 63) / 64;
    // Two CTAs share an SM, so that the first loads and the pointwise work of one lie beside the loads of the other.  Where few CTAs
    // have the GPU to themselves (the decays; the mixing weights run beside the walk, and a CTA that takes more of an SM is in its
    // way: layer of 2 x 2048 tokens, 16 x 128 heads 329 us, 358 to 370 us with eight stages) the ring is twice as deep: 4 x 1030
    // tokens of 2048 features, 32 rows 21 us against 24 us.
    p.stages = a.mode == 0 && ctas <= 148 ? NW_MAX_STAGES : 4;
    while (p.stages > NW_BACK && p.stages - NW_BACK >= p.steps) p.stages -= NW_BACK;          // no more than the contraction fills
    p.rows = NT;                                             // a box of W lies in one matrix
    while (a.n1 && n0p % p.rows) p.rows /= 2;
    CUtensorMap mx, m0, m1;
    int* status = nullptr;
    int rc = encode_rows_map(&mx, a.x, B, a.T, a.Kdim, NW_TOK, "natsl_layer_forward(x)");
    if (rc == NATSL_OK) rc = encode_rows_map(&m0, a.w0, 1, a.n0, a.Kdim, p.rows, "natsl_layer_forward(narrow weights)");
    m1 = m0;
    if (rc == NATSL_OK && a.n1) rc = encode_rows_map(&m1, a.w1, 1, a.n1, a.Kdim, p.rows, "natsl_layer_forward(narrow weights)");
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    auto kern = narrow_tc_kernel<NT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::ring + NW_MAX_STAGES * L::stage);
    if (e != cudaSuccess) {
        set_error("natsl_layer_forward: cannot reserve %d B of shared memory (%s)", L::ring + NW_MAX_STAGES * L::stage, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    kern<<<grid, NW_THREADS, L::ring + p.stages * L::stage, st>>>(mx, m0, m1, a, p, status);
    return check_launch("natsl_layer_forward (narrow projection)");
}

}  // namespace

int launch_narrow(const NarrowArgs& args, int B, cudaStream_t st) {
    NarrowArgs a = args;
    a.wide = aligned_to(16, a.out) && a.n0 % 8 == 0;
    const int n0p = (a.n0 + 7) / 8 * 8, n = n0p + a.n1;
    return n <= 16 ? launch<16>(a, n0p, B, st) : n <= 32 ? launch<32>(a, n0p, B, st) : launch<64>(a, n0p, B, st);
}

}  // namespace natsl
