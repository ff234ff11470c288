// Gated-delta-rule chunk preparation on the 5th-generation tensor cores (head dims D = K = V = 128 and 64).
// Same inputs, outputs and conventions as gdn_prep.cu (the mma.sync kernel, kept for the other head dims):
//   k_rstd, q_rstd, gcs, A = strictLower(beta_i (kn_i . kn_j) e^{gcs_i - gcs_j}),
//   [u | w] = (I + A)^-1 [v beta | kn beta e^{gcs}],  P = tril(qn kn^T e^{gcs_i - gcs_j})
// (src/nats/ops/common/chunk_scaled_dot_kkt.py:105-126, src/nats/ops/utils/solve_tril.py:350-447,
//  src/nats/ops/gated_delta_rule/wy_fast.py:123-153, src/nats/ops/common/chunk_o.py:166,188,202-203).
//
// One CTA per (batch, head, 64-token chunk), 160 threads; D = 128: 128 TMEM columns, 52 KB of shared memory, four CTAs per SM;
// D = 64: 64 columns, 37 KB, six CTAs:
//   warp 4      TMA producer (k, q tiles at the start, the v tile once A is no longer needed; 128-byte swizzle)
//               and single-thread MMA issuer;
//   warps 0-3   one thread per TMEM lane.
// Steps:
//   1. D1 = [k ; q] k^T            one stacked 128 x 64 x D product into TMEM (rows 0-63: K K^T, rows 64-127: Q K^T);
//   2. row norms of k from the diagonal of D1, A (fp32, shared memory) from rows 0-63, P (bf16, global memory,
//      one 128-byte row per thread) from rows 64-127;
//   3. Ai = (I + A)^-1 like the reference does it: the four 16 x 16 diagonal blocks by forward substitution in fp32,
//      the blocks below by the block recursion Ai_ij = -X_ii sum_{j<=m<i} A_im Ai_mj, evaluated per panel of eight
//      columns (the columns of an inverse are independent of one another) with tf32 mma.sync products, fp32
//      accumulation; Ai diag(beta) and Ai diag(beta rstd e^{gcs}) are written as two bf16 operand tiles, so the
//      right-hand sides never have to be scaled in shared memory (D = 64 has room for the first one only: the rows of k are
//      scaled by rstd e^{gcs} while the diagonal blocks are inverted, and the tile leaves the unit diagonal out);
//   4. D2 = [v^T (Ai diag beta)^T | k^T (Ai diag(..))^T]: the raw v and k tiles are the (MN-major) A operands,
//      features in the TMEM lanes, tokens in the columns: no accumulator row is wasted (D = 64: both in one product, and the
//      diagonal's share, beta v and beta rstd e^{gcs} k of the raw tiles, is added in fp32: it makes up most of u and w, and as part
//      of the product it would be rounded with both operands before the result is, w's error 1.66e-3 -> 2.3e-3 with a bf16 beta and
//      2.8e-3 with an fp32 one; on mma.sync it was 1.9e-3);
//   5. w, then u, go from TMEM through a [token][feature] staging tile (transposed by stmatrix) to global memory with TMA
//      stores; P leaves the same way.
// Chains of short phases: what counts is the instructions of a chunk and how many chunks an SM has in flight.  L2 flushed:
// 8 x 4096 tokens, 16 heads, D = 128: 180 us one element at a time and one feature per store, 152 us with the entries of A and P
// in pairs, stmatrix and two diagonal blocks per warp (same bits; traffic 113 us); 16 x 4096 tokens, 16 heads, D = 64: 355 us on
// mma.sync (shared memory 75 % busy), 226 us here (traffic 126 us; 208 us with the diagonal in the product; with k's scaled rows in
// a tile of their own instead of a second load of k, five CTAs per SM, 240 us).
// The decay carried over skipped blocks multiplies w by one scalar per chunk and is applied by the consumers.
// Every mbarrier wait is bounded: on expiry the status word is set and the CTA runs on to its teardown.
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr int PT_THREADS = 160;
constexpr int PT_EPI = 128;
constexpr int PT_A_LD = 68;                  // fp32 row pitch of A: conflict-free 16-byte row stores and fragment loads

template <int D>
struct PtSmem {
    static constexpr int SUB = D / 64;                       // sub-tiles of 64 features, [64 tokens][64 features] = 8 KB each
    // [k sub-tile 0][q sub-tile 0][k sub-tile 1][q sub-tile 1]: the stacked [k ; q] operand of the first product.  The q sub-tiles
    // are reused: first sub-tile 0 for staging P, then for the Ai operand tiles (one where D = 64, two where D = 128).
    static constexpr int kq = 0;
    // fp32 A [64][68] (diagonal blocks replaced by their inverses); once Ai is formed the v tile is loaded over it -- it is
    // needed by the last product only, and this is what lets four CTAs (D = 64: six) share an SM
    static constexpr int As = SUB * 16384;
    static constexpr int v = As;
    static constexpr int kraw = As + 8192;                   // D = 64: k as it came, beside v
    static constexpr int scr = As + 64 * PT_A_LD * 4;        // per warp [16][8] fp32: accumulator -> B-fragment exchange
    static constexpr int vec = scr + 4 * 512;                // gcs, beta, k rstd, w scale, q rstd: 5 x 64 floats
    static constexpr int bars = vec + 5 * 64 * 4;
    static constexpr int total = bars + 64;
    static constexpr int aiu = kq + 8192, aiw = kq + 24576;  // Ai diag(beta), Ai diag(beta rstd e^{gcs}) (D = 128): [64][64] bf16
    static constexpr int pst = kq + 8192;                    // P staging [64][64] bf16
    static constexpr int ctas = D == 64 ? 6 : 4;             // per SM
    static constexpr uint32_t tmem = 64 * SUB;               // columns: with D = 64 the last product lies over the first
    static_assert(As % 1024 == 0 && 64 * PT_A_LD * 4 >= 16384, "v (D = 64: v and k) must fit over A, 1024-byte aligned");
    static_assert(ctas * (total + 1024) <= 233472 && ctas * tmem <= 512, "CTAs per SM");
};

__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
// D (16 x 8, fp32) += A (16 x 8, tf32, row) * B (8 x 8, tf32, col)
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// A fragments (two k-steps of 8) of the 16 x 16 block at (row0, col0) of the fp32 matrix As
__device__ __forceinline__ void load_a_tf32(const float* As, int row0, int col0, int lane, uint32_t (&a)[2][4]) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const float* p = As + (row0 + g) * PT_A_LD + col0 + 8 * s + q;
        a[s][0] = to_tf32(p[0]);
        a[s][1] = to_tf32(p[8 * PT_A_LD]);
        a[s][2] = to_tf32(p[4]);
        a[s][3] = to_tf32(p[8 * PT_A_LD + 4]);
    }
}
// A 16 x 8 accumulator (rows g, g+8; columns 2q, 2q+1) -> the B fragments of the same matrix used as a right factor
__device__ __forceinline__ void acc_to_b(float* scr, const float (&c)[4], int lane, uint32_t (&b)[2][2]) {
    const int g = lane >> 2, q = lane & 3;
    *reinterpret_cast<float2*>(scr + g * 8 + 2 * q) = make_float2(c[0], c[1]);
    *reinterpret_cast<float2*>(scr + (g + 8) * 8 + 2 * q) = make_float2(c[2], c[3]);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        b[s][0] = to_tf32(scr[(8 * s + q) * 8 + g]);
        b[s][1] = to_tf32(scr[(8 * s + q + 4) * 8 + g]);
    }
    __syncwarp();
}

// One panel of eight columns [c0, c0+8) of Ai (c0 = 16 j + 8 half), by one warp: zero above block row j, X_jj's half,
// then block rows j+1..3 by the recursion; every 16 x 8 block is written, scaled per column, into the operand tiles, or (one tile)
// without the unit diagonal, whose products are added up in fp32 at the end.
template <bool TWO>
__device__ __forceinline__ void inverse_panel(const float* As, float* scr, unsigned char* aiu, unsigned char* aiw,
                                              const float* s_beta, const float* s_wsc, int j, int half, int lane) {
    const int g = lane >> 2, q = lane & 3;
    const int c0 = 16 * j + 8 * half;
    const int chunk = c0 >> 3;
    const int ca = c0 + 2 * q;
    const float bu0 = s_beta[ca], bu1 = s_beta[ca + 1], bw0 = TWO ? s_wsc[ca] : 0.f, bw1 = TWO ? s_wsc[ca + 1] : 0.f;
    for (int r = lane; r < 16 * j; r += 32) {
        *reinterpret_cast<uint4*>(aiu + swz<128>(r, chunk)) = make_uint4(0, 0, 0, 0);
        if (TWO) *reinterpret_cast<uint4*>(aiw + swz<128>(r, chunk)) = make_uint4(0, 0, 0, 0);
    }
    auto put = [&](int blk, const float (&y)[4]) {
        const int ra = 16 * blk + g, rb = ra + 8;
        const bool unit = !TWO;
        *reinterpret_cast<uint32_t*>(aiu + swz<128>(ra, chunk) + q * 4) =
            pack_bf16(unit && ra == ca ? 0.f : y[0] * bu0, unit && ra == ca + 1 ? 0.f : y[1] * bu1);
        *reinterpret_cast<uint32_t*>(aiu + swz<128>(rb, chunk) + q * 4) =
            pack_bf16(unit && rb == ca ? 0.f : y[2] * bu0, unit && rb == ca + 1 ? 0.f : y[3] * bu1);
        if (TWO) {
            *reinterpret_cast<uint32_t*>(aiw + swz<128>(ra, chunk) + q * 4) = pack_bf16(y[0] * bw0, y[1] * bw1);
            *reinterpret_cast<uint32_t*>(aiw + swz<128>(rb, chunk) + q * 4) = pack_bf16(y[2] * bw0, y[3] * bw1);
        }
    };
    uint32_t yb[4][2][2];                        // B fragments of the panel's blocks, by block row
    {
        float y[4];
        const float* p = As + (16 * j + g) * PT_A_LD + c0 + 2 * q;
        y[0] = p[0]; y[1] = p[1]; y[2] = p[8 * PT_A_LD]; y[3] = p[8 * PT_A_LD + 1];
        put(j, y);
#pragma unroll
        for (int m = 0; m < 3; ++m)
            if (m == j) acc_to_b(scr, y, lane, yb[m]);
    }
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        if (i > j) {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                if (m >= j && m < i) {
                    uint32_t a[2][4];
                    load_a_tf32(As, 16 * i, 16 * m, lane, a);
                    mma_tf32(t, a[0], yb[m][0][0], yb[m][0][1]);
                    mma_tf32(t, a[1], yb[m][1][0], yb[m][1][1]);
                }
            }
            uint32_t tb[2][2];
            acc_to_b(scr, t, lane, tb);
            uint32_t x[2][4];
            load_a_tf32(As, 16 * i, 16 * i, lane, x);
            float y[4] = {0.f, 0.f, 0.f, 0.f};
            mma_tf32(y, x[0], tb[0][0], tb[0][1]);
            mma_tf32(y, x[1], tb[1][0], tb[1][1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = -y[e];
            put(i, y);
            if (i < 3) acc_to_b(scr, y, lane, yb[i]);
        }
    }
}

// Four entries x r of a row of A or P: (left * right_j) r_j e^{gi - gj}, columns from `first` on (first > 3: none) left out.
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float4 decayed4(const float* gcs, const float* right, const uint32_t* r, uint64_t gi, uint64_t left, int first) {
    const uint64_t neg = pack2(-1.f, -1.f), l2e = pack2(1.44269504f, 1.44269504f);
    const ulonglong2 gj = *reinterpret_cast<const ulonglong2*>(gcs), rj = *reinterpret_cast<const ulonglong2*>(right);
    float a, b, c, d;
    unpack2(mul2(fma2(gj.x, neg, gi), l2e), a, b);
    unpack2(mul2(fma2(gj.y, neg, gi), l2e), c, d);
    const uint64_t x = mul2(mul2(mul2(rj.x, left), pack2(__uint_as_float(r[0]), __uint_as_float(r[1]))), pack2(ex2(a), ex2(b)));
    const uint64_t y = mul2(mul2(mul2(rj.y, left), pack2(__uint_as_float(r[2]), __uint_as_float(r[3]))), pack2(ex2(c), ex2(d)));
    float4 o;
    unpack2(x, o.x, o.y);
    unpack2(y, o.z, o.w);
    o.x = first > 0 ? o.x : 0.f;                               // (a select, not a factor: the exponential may have overflowed)
    o.y = first > 1 ? o.y : 0.f;
    o.z = first > 2 ? o.z : 0.f;
    o.w = first > 3 ? o.w : 0.f;
    return o;
}
// Four 8 x 8 bf16 matrices in the accumulator-fragment layout, stored transposed, each thread giving the address of one row.
__device__ __forceinline__ void stsm_x4_t(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
                 : "memory");
}

template <int D>
__global__ void __launch_bounds__(PT_THREADS, PtSmem<D>::ctas)
gdn_prep_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_p, int has_q,
                   const float* __restrict__ g, const void* __restrict__ beta, int beta_dtype,
                   float* __restrict__ gcs_out, float* __restrict__ krstd_out, float* __restrict__ qrstd_out, int T,
                   int H, int use_l2norm, int* status) {
    using L = PtSmem<D>;
    constexpr int SUB = L::SUB;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int t0 = c * 64;
    const int valid = min(64, T - t0);
    const long tok0 = (long)b * T + t0;

    float* As = reinterpret_cast<float*>(smem + L::As);
    float* s_gcs = reinterpret_cast<float*>(smem + L::vec);
    float* s_beta = s_gcs + 64;
    float* s_rstd = s_beta + 64;
    float* s_wsc = s_rstd + 64;
    float* s_qr = s_wsc + 64;
    const uint32_t bar_load = sbase + L::bars, bar_d1 = bar_load + 8, bar_ai = bar_load + 16, bar_d2w = bar_load + 24,
                   bar_v = bar_load + 32, bar_d2u = bar_load + 40;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 48);

    if (tid == 0) {
        mbar_init(bar_load, 1);
        mbar_init(bar_d1, 1);
        mbar_init(bar_ai, PT_EPI);
        mbar_init(bar_d2w, 1);
        mbar_init(bar_v, 1);
        mbar_init(bar_d2u, 1);
        mbar_fence_init();
    }
    if (warp == 4) tmem_alloc(smem_u32(tmem_slot), L::tmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 4) {
        // ------------------------------------------------------------ TMA producer + MMA issuer
        if (lane == 0) {
            mbar_expect_tx(bar_load, (has_q ? 16384 : 8192) * SUB);
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub) {
                tma_load_4d(sbase + L::kq + sub * 16384, &map_k, sub * 64, h, t0, b, bar_load);
                if (has_q) tma_load_4d(sbase + L::kq + sub * 16384 + 8192, &map_q, sub * 64, h, t0, b, bar_load);
            }
            // v is only needed at the very end: warm L2 now, load it when A is dead
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub) tma_prefetch_4d(&map_v, sub * 64, h, t0, b);
        }
        __syncwarp();
        mbar_wait_small(bar_load, 0, status);
        __syncwarp();
        {
            constexpr uint32_t id_1 = umma_idesc_bf16(128, 64, false);
            tc_fence_after();
            const uint32_t l = umma_desc_lo(sbase + L::kq, 16);
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub) umma_ss_x4<2, 2>(tmem, l + sub * 1024, l + sub * 1024, id_1, sub > 0);
            umma_commit(bar_d1);
        }
        __syncwarp();
        mbar_wait_small(bar_ai, 0, status);
        __syncwarp();
        constexpr uint32_t id_2 = umma_idesc_bf16(128, 64, false) | (1u << 15);      // A MN-major (features x tokens)
        // every thread has finished with A (and fenced): the v tile may land on it
        if (lane == 0) {
            mbar_expect_tx(bar_v, 16384);
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub) tma_load_4d(sbase + L::v + sub * 8192, &map_v, sub * 64, h, t0, b, bar_v);
            if (D == 64) tma_load_4d(sbase + L::kraw, &map_k, 0, h, t0, b, bar_v);      // (from L2: its tile here has been scaled)
        }
        __syncwarp();
        if constexpr (D == 128) {
            tc_fence_after();
            umma_ss_x4<128, 2>(tmem + 64, umma_desc_lo(sbase + L::kq, 16384), umma_desc_lo(sbase + L::aiw, 16), id_2, 0u);
            umma_commit(bar_d2w);
        }
        __syncwarp();
        mbar_wait_small(bar_v, 0, status);
        __syncwarp();
        tc_fence_after();
        if constexpr (D == 128) umma_ss_x4<128, 2>(tmem, umma_desc_lo(sbase + L::v, 8192), umma_desc_lo(sbase + L::aiu, 16), id_2, 0u);
        else umma_ss_x4<128, 2>(tmem, umma_desc_lo(sbase + L::kq, L::v - L::kq), umma_desc_lo(sbase + L::aiu, 16), id_2, 0u);
        umma_commit(bar_d2u);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ one thread per TMEM lane
        const int row = tid;                                   // D1: k row (0-63) or q row (64-127); D2: feature
        const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16);
        if (warp == 0) {
            // gcs = inclusive cumsum of g over the chunk (two elements per lane), beta
            float x0 = 0.f, x1 = 0.f, b0 = 0.f, b1 = 0.f;
            const long g0 = (tok0 + lane) * H + h, g1 = (tok0 + lane + 32) * H + h;
            if (lane < valid) {
                x0 = g[g0];
                b0 = beta_dtype == NATSL_DT_F32 ? reinterpret_cast<const float*>(beta)[g0]
                                                : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(beta)[g0]);
            }
            if (lane + 32 < valid) {
                x1 = g[g1];
                b1 = beta_dtype == NATSL_DT_F32 ? reinterpret_cast<const float*>(beta)[g1]
                                                : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(beta)[g1]);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float a0 = __shfl_up_sync(0xffffffffu, x0, o), a1 = __shfl_up_sync(0xffffffffu, x1, o);
                if (lane >= o) {
                    x0 += a0;
                    x1 += a1;
                }
            }
            x1 += __shfl_sync(0xffffffffu, x0, 31);
            s_gcs[lane] = x0;
            s_gcs[lane + 32] = x1;
            s_beta[lane] = b0;
            s_beta[lane + 32] = b1;
            if (lane < valid) gcs_out[g0] = x0;
            if (lane + 32 < valid) gcs_out[g1] = x1;
        }
        mbar_wait_small(bar_load, 0, status);
        if (warp >= 2 && has_q) {
            // q row norms (one row per thread; the swizzle makes the 16-byte reads of eight rows conflict-free)
            const int r = row - 64;
            float ss = 0.f;
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub)
#pragma unroll
                for (int cc = 0; cc < 8; ++cc) {
                    const uint4 xv = *reinterpret_cast<const uint4*>(smem + L::kq + sub * 16384 + 8192 + swz<128>(r, cc));
                    const uint32_t* xw = reinterpret_cast<const uint32_t*>(&xv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = unpack_bf16(xw[e]);
                        ss += f.x * f.x + f.y * f.y;
                    }
                }
            const float rs = use_l2norm ? rsqrtf(ss + 1e-6f) : 1.0f;
            s_qr[r] = rs;
            if (r < valid && qrstd_out) qrstd_out[(tok0 + r) * H + h] = rs;
        }
        mbar_wait_small(bar_d1, 0, status);
        tc_fence_after();
        if (warp < 2) {
            // k row norms from the diagonal of K K^T: row i of warp w has its diagonal in columns [32 w, 32 w + 32)
            uint32_t r[32];
            tmem_ld32(t_lane + 32 * warp, r);
            tmem_ld_wait();
            float d = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (i == lane) d = __uint_as_float(r[i]);
            const float rs = use_l2norm ? rsqrtf(d + 1e-6f) : 1.0f;
            s_rstd[row] = rs;
            if (row < valid) krstd_out[(tok0 + row) * H + h] = rs;
        }
        epi_barrier();                      // gcs, beta, both row norms are known; the q tile has been read for the last time
        if (warp < 2) {
            const float gi = s_gcs[row];
            const float bi = s_beta[row] * s_rstd[row];
            s_wsc[row] = (D == 64 ? s_rstd[row] : bi) * __expf(gi);
            const uint64_t gi2 = pack2(gi, gi), bi2 = pack2(bi, bi);
#pragma unroll 1
            for (int hh = 0; hh <= warp; ++hh) {           // columns above the row's 32-column group are never read
                uint32_t r[32];
                tmem_ld32(t_lane + 32 * hh, r);
                tmem_ld_wait();
                const int below = row - 32 * hh;           // entries left of the diagonal
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(As + row * PT_A_LD + 32 * hh + j) =
                        decayed4(s_gcs + 32 * hh + j, s_rstd + 32 * hh + j, r + j, gi2, bi2, below - j);
            }
        } else if (has_q) {
            // P = tril(qn kn^T e^{gcs_i - gcs_j}): one row per thread into the staging tile (the q sub-tile is free);
            // one TMA store writes the tile after the next barrier
            const int i = row - 64;
            const uint64_t gi2 = pack2(s_gcs[i], s_gcs[i]), qi2 = pack2(s_qr[i], s_qr[i]);
            unsigned char* pst = smem + L::pst;
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
                if (hh > warp - 2) {                       // above the diagonal
#pragma unroll
                    for (int j = 4; j < 8; ++j) *reinterpret_cast<uint4*>(pst + swz<128>(i, j)) = make_uint4(0, 0, 0, 0);
                    break;
                }
                uint32_t r[32];
                tmem_ld32(t_lane + 32 * hh, r);
                tmem_ld_wait();
                const int upto = i + 1 - 32 * hh;          // entries up to the diagonal
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    const float4 x = decayed4(s_gcs + 32 * hh + j, s_rstd + 32 * hh + j, r + j, gi2, qi2, upto - j);
                    const float4 y = decayed4(s_gcs + 32 * hh + j + 4, s_rstd + 32 * hh + j + 4, r + j + 4, gi2, qi2, upto - j - 4);
                    *reinterpret_cast<uint4*>(pst + swz<128>(i, 4 * hh + (j >> 3))) =
                        make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
                }
            }
            fence_async_smem();
        }
        epi_barrier();                      // A complete, the w scale known, D1 read for the last time, P staged
        if (tid == 64 && has_q) {
            tma_store_4d(&map_p, sbase + L::pst, 0, h, t0, b);
            tma_store_commit();
        }
        if (warp < 2) {
            // X_dd = (I + A_dd)^-1 by forward substitution, two blocks per warp, lane = column; written over A_dd
            const int d0 = warp * 32 + (lane & 16), cidx = lane & 15;
            float xcol[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float arow[16];
#pragma unroll
                for (int j4 = 0; j4 < 16; j4 += 4)
                    if (j4 < i)
                        *reinterpret_cast<float4*>(&arow[j4]) =
                            *reinterpret_cast<const float4*>(&As[(d0 + i) * PT_A_LD + d0 + j4]);
                float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
                for (int j = 0; j < i; ++j) {
                    const float t = arow[j] * xcol[j];
                    if ((j & 3) == 0) p0 += t; else if ((j & 3) == 1) p1 += t; else if ((j & 3) == 2) p2 += t; else p3 += t;
                }
                xcol[i] = ((i == cidx) ? 1.f : 0.f) - ((p0 + p1) + (p2 + p3));
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 16; ++i) As[(d0 + i) * PT_A_LD + d0 + cidx] = xcol[i];
        } else if constexpr (D == 64) {
            // meanwhile: the rows of k, the operand of w, scaled by rstd e^{gcs} (beta comes with Ai); q's factors are done with
            s_qr[row - 64] = s_beta[row - 64] * s_wsc[row - 64];
#pragma unroll
            for (int rr = 0; rr < 8; ++rr) {
                const int r = rr * 8 + (row - 64) / 8, cc = row % 8;
                uint4* ptr = reinterpret_cast<uint4*>(smem + L::kq + swz<128>(r, cc));
                const float sc = s_wsc[r];
                const uint64_t s2 = pack2(sc, sc);
                uint64_t x[4];
                open8(*ptr, x);
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = mul2(x[e], s2);
                *ptr = close8(x);
            }
        }
        if (tid == 64 && has_q) tma_store_wait_read();      // the P tile has been read: its place becomes Ai diag(beta)
        epi_barrier();
        {
            float* scr = reinterpret_cast<float*>(smem + L::scr) + warp * 128;
            unsigned char* aiu = smem + L::aiu;
            unsigned char* aiw = smem + L::aiw;
            if (warp < 2) {
                inverse_panel<D == 128>(As, scr, aiu, aiw, s_beta, s_wsc, 0, warp, lane);
            } else {
#pragma unroll
                for (int j = 1; j < 4; ++j) inverse_panel<D == 128>(As, scr, aiu, aiw, s_beta, s_wsc, j, warp - 2, lane);
            }
        }
        fence_async_smem();
        tc_fence_before();
        mbar_arrive(bar_ai);
        // ---- w and u: lane = feature, column = token.  A warp takes sixteen features at a time in the fragment layout, and
        // stmatrix lays them transposed into a [token][feature] staging tile (conflict-free); one thread stores the tiles with TMA.
        // D = 128: w (columns 64-127, its product does not wait for the v tile) then u (columns 0-63), staged over the k sub-tiles
        // (dead once w's product is done) and over the two Ai tiles.  D = 64: lanes 0-63 are w, the others u, staged over the tiles
        // that they were computed from.
#pragma unroll 1
        for (int arr = D == 128 ? 0 : 1; arr < 2; ++arr) {     // 0: w, 1: u (D = 64: both)
            mbar_wait_small(arr == 0 ? bar_d2w : bar_d2u, 0, status);
            if (D == 64) mbar_wait_small(bar_v, 0, status);
            tc_fence_after();
            const int sub = row >> 6;
            const uint32_t stg = sbase + (D == 64 ? (sub ? L::v : L::kq) : L::kq + sub * 16384 + (arr == 0 ? 0 : 8192));
            // this thread's row of the four matrices: token (lane & 7) of the lower or upper eight, features of its half
            const int tok = (lane & 7) + ((lane & 16) >> 1), half = (lane >> 3) & 1;
            const float* s_unit = (sub ? s_beta : s_qr) + 2 * (lane & 3);
            const uint32_t unit = sbase + (sub ? L::v : L::kraw) - stg;      // D = 64: from an output's place to its raw input's
#pragma unroll 1
            for (int f = 0; f < 2; ++f) {                      // sixteen features
                uint32_t r[32];
                tmem_ld_16x256b_x8(t_lane + ((uint32_t)(16 * f) << 16) + (arr == 0 ? 64 : 0), r);
                tmem_ld_wait();
                const int chunk = (((row & 32) + 16 * f) >> 3) + half;
                const uint32_t at = stg + tok * 128 + ((chunk ^ (tok & 7)) << 4);
#pragma unroll
                for (int k = 0; k < 4; ++k) {                  // sixteen tokens
                    uint32_t p[4];
                    if constexpr (D == 64) {                   // the inverse's diagonal: beta v, or beta rstd e^{gcs} k, in fp32
                        ldsm_x4_t(at + unit + k * 16 * 128, p[0], p[1], p[2], p[3]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint64_t s = *reinterpret_cast<const uint64_t*>(s_unit + 16 * k + 8 * (e >> 1));
                            p[e] = close2(fma2(open2(p[e]), s, pack2(__uint_as_float(r[8 * k + 2 * e]), __uint_as_float(r[8 * k + 2 * e + 1]))));
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            p[e] = pack_bf16(__uint_as_float(r[8 * k + 2 * e]), __uint_as_float(r[8 * k + 2 * e + 1]));
                    }
                    stsm_x4_t(at + k * 16 * 128, p[0], p[1], p[2], p[3]);
                }
            }
            fence_async_smem();
            epi_barrier();
            if (tid == 0) {
                if constexpr (D == 64) {
                    tma_store_4d(&map_w, sbase + L::kq, 0, h, t0, b);
                    tma_store_4d(&map_u, sbase + L::v, 0, h, t0, b);
                } else {
                    const CUtensorMap* mp = arr == 0 ? &map_w : &map_u;
                    tma_store_4d(mp, sbase + L::kq + (arr == 0 ? 0 : 8192), 0, h, t0, b);
                    tma_store_4d(mp, sbase + L::kq + 16384 + (arr == 0 ? 0 : 8192), 64, h, t0, b);
                }
                tma_store_commit();
            }
        }
        if (tid == 0) tma_store_wait_read();
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 4) tmem_dealloc(tmem, L::tmem);
}

template <int D>
static int launch_prep_tc(const void* q, const void* k, const void* v, const float* g, const void* beta, int beta_dtype, void* w, void* u,
                          float* gcs, float* k_rstd, float* q_rstd, void* pmat, int B, int T, int H, int use_l2norm, cudaStream_t st) {
    using L = PtSmem<D>;
    auto kern = gdn_prep_tc_kernel<D>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total);
    if (e != cudaSuccess) {
        set_error("natsl_gdn_chunk_prep: cannot reserve %d B of shared memory (%s)", L::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mw, mu, mp;
    int rc = encode_bthd_map(&mk, k, B, T, H, D, 64, "natsl_gdn_chunk_prep(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T, H, D, 64, "natsl_gdn_chunk_prep(v)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mq, q ? q : k, B, T, H, D, 64, "natsl_gdn_chunk_prep(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mw, w, B, T, H, D, 64, "natsl_gdn_chunk_prep(w)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mu, u, B, T, H, D, 64, "natsl_gdn_chunk_prep(u)");
    if (rc == NATSL_OK) rc = pmat ? encode_bthd_map(&mp, pmat, B, T, H, 64, 64, "natsl_gdn_chunk_prep(P)") : NATSL_OK;
    if (!pmat) mp = mk;
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    const int NT = (T + 63) / 64;
    kern<<<dim3(NT, H, B), PT_THREADS, L::total, st>>>(mq, mk, mv, mw, mu, mp, q ? 1 : 0, g, beta, beta_dtype, gcs, k_rstd, q_rstd, T, H,
                                                       use_l2norm, status);
    return check_launch("natsl_gdn_chunk_prep");
}
int prep_tc64(const void* q, const void* k, const void* v, const float* g, const void* beta, int beta_dtype, void* w, void* u, float* gcs,
              float* k_rstd, float* q_rstd, void* pmat, int B, int T, int H, int use_l2norm, cudaStream_t st) {
    return launch_prep_tc<64>(q, k, v, g, beta, beta_dtype, w, u, gcs, k_rstd, q_rstd, pmat, B, T, H, use_l2norm, st);
}

}  // namespace natsl

extern "C" int natsl_gdn_chunk_prep_tc(const void* q, const void* k, const void* v, const float* g, const void* beta,
                                       int beta_dtype, void* w, void* u, float* gcs, float* k_rstd, float* q_rstd,
                                       void* pmat, int B, int T, int H, int K, int V, int use_l2norm, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(k && v && g && beta && w && u && gcs && k_rstd, NATSL_ERR_NULL, "natsl_gdn_chunk_prep_tc: null pointer");
    NATSL_REQUIRE((q == nullptr) == (pmat == nullptr), NATSL_ERR_NULL,
                  "natsl_gdn_chunk_prep_tc: q and the score-matrix output go together");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0, NATSL_ERR_BAD_SHAPE, "natsl_gdn_chunk_prep_tc: empty shape");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_gdn_chunk_prep_tc: B and H must be <= 65535");
    NATSL_REQUIRE(beta_dtype == NATSL_DT_BF16 || beta_dtype == NATSL_DT_F32, NATSL_ERR_UNSUPPORTED,
                  "natsl_gdn_chunk_prep_tc: beta must be bf16 or f32");
    NATSL_REQUIRE(K == 128 && V == 128, NATSL_ERR_UNSUPPORTED,
                  "natsl_gdn_chunk_prep_tc: built for K = V = 128 (got K=%d V=%d); use natsl_gdn_chunk_prep_ex", K, V);
    return launch_prep_tc<128>(q, k, v, g, beta, beta_dtype, w, u, gcs, k_rstd, q_rstd, pmat, B, T, H, use_l2norm,
                               reinterpret_cast<cudaStream_t>(stream));
}
