// The state that every chunk of the gated delta rule reads, on the 5th-generation tensor cores (head dims K = V = 128,
// nats_block_size = 64): the walk of gdn_walk_tc.cu without its outputs, for the backward pass, which forms the rest chunk by chunk.
// One CTA per (batch, head).  Only chunks of selected blocks update the state S (src/nats/ops/common/chunk_delta_h.py:189-324):
//     v' = u - e^{carry} w S;   S <- e^{g_last+carry} S + k^T (v' rstd_k e^{g_last-g})
// so only they are walked; the others' states are the copies in front of the next update.  Per update: MMA 1 (w S against the bf16
// copy of S in shared memory; the operand's rows 64-127 are whatever lies behind w, their results are never read), v'' by the warps
// of rows 0-63, MMA 3 (accumulates onto S in TMEM), the new copy by all rows.  The two copies take turns: one leaves for global memory
// by TMA, once per chunk that reads it, while the next is written.
// Warp roles as in gdn_walk_tc.cu: warp 0 loads w, k and u (two stages), warp 1 issues the products, warps 2-17 the rows (32 columns
// each), warp 18 stores the copies.  All mbarrier waits are bounded (status word + clean teardown on expiry).
//
// What bounds it: the chain w S -> v'' -> k^T v'' -> copy of an update, one CTA per SM, and HBM: at B = 8, T = 4096, H = 16 it writes 268 MB
// of copies and reads the updating chunks' 48 KB.  Alone (us; before: linear_scan.cu, mma.sync, four CTAs of 32 columns per pair): that
// size with 75 % of the chunks updating 194 -> 116 (4.9 TB/s), 25 % 112 -> 75; B = 16, T = 2048, 50 % 149 -> 97; 64 heads, T = 4096, 75 %
// 135 -> 110.  The states are the same bits (tests/test_gpu_states.py): roundings and sums lie where the scan has them.  linear_scan.cu
// says where the line to it lies.
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr int GS_THREADS = 608;
constexpr int GS_ROW_WARPS = 16;
constexpr uint32_t GS_TMEM_COLS = 512;
constexpr uint32_t GS_S = 0, GS_D1 = 128;                     // TMEM columns: S; w S (two, by update)
constexpr int GS_MAX_NT = 1024;

struct GsSmem {
    // stage: w, k, u, 2 sub-tiles [64][64] each (16 KB)
    static constexpr int w = 0, k = 16384, u = 32768, stage = 49152;
    static constexpr int sbf = 2 * stage;                     // 2 x S bf16: 2 sub-tiles [128 k-rows][64 v-cols]  64 KB
    static constexpr int vs = sbf + 65536;                    // v'': 2 sub-tiles [64 tok][64]
    static constexpr int carry = vs + 16384;                  // per chunk: decay of the skipped blocks in front of it;
    static constexpr int mul = carry + 4 * GS_MAX_NT;         // the next update's decay, sign bit set where the chunk updates the state
    static constexpr int bars = mul + 4 * GS_MAX_NT;
    static constexpr int total = bars + 256;
    static_assert(total <= 232448, "shared memory of one SM");
};

__global__ void __launch_bounds__(GS_THREADS, 1)
gdn_states_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_h, const float* __restrict__ gcs,
                     const float* __restrict__ krstd, const int* __restrict__ types_i, const int* __restrict__ indices,
                     const int* __restrict__ n_blocks, const float* __restrict__ h0, float* __restrict__ carry_out, int T, int H, int HN,
                     int decay, int trailing_quirk, int* status) {
    using L = GsSmem;
    constexpr int K = 128, V = 128;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int h = blockIdx.x, b = blockIdx.y;
    const int hn = h / (H / HN);
    const int NT = (T + 63) / 64;
    float* m_carry = reinterpret_cast<float*>(smem + L::carry);
    uint32_t* m_mul = reinterpret_cast<uint32_t*>(smem + L::mul);
    const uint32_t bar0 = sbase + L::bars;
    // barriers, all counted in updates: full / empty of the two stages of w and of k, u; d1, s3 (MMA 1, 3 done); pv (v'' written and
    // the state written back); sready[2] (copy published); sfree[2] (copy stored)
    const uint32_t bar_w = bar0, bar_w_free = bar0 + 16, bar_ku = bar0 + 32, bar_ku_free = bar0 + 48, bar_d1 = bar0 + 64,
                   bar_pv = bar0 + 72, bar_s3 = bar0 + 80, bar_sready = bar0 + 88, bar_sfree = bar0 + 104;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 192);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_w + 8 * i, 1);
            mbar_init(bar_w_free + 8 * i, 1);
            mbar_init(bar_ku + 8 * i, 1);
            mbar_init(bar_ku_free + 8 * i, GS_ROW_WARPS / 2);
            mbar_init(bar_sready + 8 * i, GS_ROW_WARPS);
            mbar_init(bar_sfree + 8 * i, 1);
        }
        mbar_init(bar_d1, 1);
        mbar_init(bar_pv, GS_ROW_WARPS);
        mbar_init(bar_s3, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), GS_TMEM_COLS);
    // ---- per-chunk scalars, as in gdn_walk_tc.cu
    {
        float* gl = reinterpret_cast<float*>(smem + L::sbf);          // (overwritten by the initial state)
        int* sel = reinterpret_cast<int*>(smem + L::sbf) + GS_MAX_NT;
        for (int c = tid; c < NT; c += GS_THREADS) {
            sel[c] = types_i[(((long)b * NT + c) * HN + hn) * 2 + 1] != 0;
            gl[c] = gcs[((long)b * T + min(c * 64 + 63, T - 1)) * H + h];
        }
        const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
        const int last_sel = nsel > 0 ? indices[(((long)b * NT + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
        __syncthreads();
        for (int c = tid; c < NT; c += GS_THREADS) {
            float carry = 0.f;
            if (decay) {
                int j = c;
                while (j > 0 && !sel[j - 1]) --j;
                for (; j < c; ++j)
                    if (!trailing_quirk || j < last_sel) carry += gl[j];
            }
            m_carry[c] = carry;
            carry_out[((long)b * NT + c) * H + h] = carry;
        }
        __syncthreads();
        for (int c = tid; c < NT; c += GS_THREADS) {
            int j = c + 1;
            while (j < NT && !sel[j]) ++j;
            const float mul = j < NT ? __expf(gl[j] + m_carry[j]) : 1.f;
            m_mul[c] = (__float_as_uint(mul) & 0x7fffffffu) | (sel[c] ? 0x80000000u : 0u);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    auto updates = [&](int c) -> bool { return (m_mul[c] >> 31) != 0; };

    if (warp == 0) {
        // ------------------------------------------------------------ loads
        int nw = 0, nku = 0;                                  // updates asked for
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            if (!updates(c)) continue;
            const int stg = nw & 1, t0 = c * 64;
            const uint32_t par = ((nw >> 1) - 1) & 1, base = sbase + stg * L::stage;
            if (nw >= 2) ok = warp_wait(bar_w_free + stg * 8, par);
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar_w + stg * 8, 16384);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) tma_load_4d(base + L::w + sub * 8192, &map_w, sub * 64, h, t0, b, bar_w + stg * 8);
            }
            __syncwarp();
            ++nw;
            if (nku >= 2) ok = warp_wait(bar_ku_free + stg * 8, par);
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar_ku + stg * 8, 32768);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    tma_load_4d(base + L::u + sub * 8192, &map_u, sub * 64, h, t0, b, bar_ku + stg * 8);
                    tma_load_4d(base + L::k + sub * 8192, &map_k, sub * 64, h, t0, b, bar_ku + stg * 8);
                }
            }
            __syncwarp();
            ++nku;
        }
        if (!ok) {                                            // nothing may still be on its way into shared memory
            for (int i = max(0, nw - 2); i < nw; ++i) warp_wait(bar_w + (i & 1) * 8, (i >> 1) & 1);
            for (int i = max(0, nku - 2); i < nku; ++i) warp_wait(bar_ku + (i & 1) * 8, (i >> 1) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t id = umma_idesc_bf16(128, 128, true);                         // w S
        constexpr uint32_t id_3 = id | (1u << 15);                                       // k^T v'' (A MN-major)
        int i = 0;                                            // updates
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            if (!updates(c)) continue;
            const uint32_t base = sbase + (i & 1) * L::stage, par = (i >> 1) & 1;
            ok = warp_wait(bar_w + (i & 1) * 8, par);
            if (ok) ok = warp_wait(bar_sready + (i & 1) * 8, par);
            if (!ok) break;
            tc_fence_after();
            {
                const uint32_t al = umma_desc_lo(base + L::w, 16), bl = umma_desc_lo(sbase + L::sbf + (i & 1) * 32768, 16384);
#pragma unroll
                for (int e = 0; e < 2; ++e) umma_ss_x4<2, 128>(tmem + GS_D1 + (i & 1) * 128, al + e * 512, bl + e * 512, id, e > 0);
                umma_commit(bar_d1);
            }
            ok = warp_wait(bar_ku + (i & 1) * 8, par);
            if (ok) ok = warp_wait(bar_pv, i & 1);
            if (!ok) break;
            tc_fence_after();
            umma_ss_x4<128, 128>(tmem + GS_S, umma_desc_lo(base + L::k, 8192), umma_desc_lo(sbase + L::vs, 8192), id_3, 1u);
            umma_commit(bar_s3);
            ++i;
        }
    } else if (warp == GS_ROW_WARPS + 2) {
        // ------------------------------------------------------------ stores of the copies
        int i = 0;                                            // updates in front of the chunk: its copy
        bool known = false;                                   // and it has been waited for
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            if (!known) ok = warp_wait(bar_sready + (i & 1) * 8, (i >> 1) & 1);
            if (!ok) break;
            known = true;
            const bool last = updates(c);                     // the copy's last reader
            if (lane == 0) {
                const int at = (b * NT + c) * H + h;
                const uint32_t src = sbase + L::sbf + (i & 1) * 32768;
                tma_store_4d(&map_h, src, 0, 0, 0, at);
                tma_store_4d(&map_h, src + 16384, 64, 0, 0, at);
                tma_store_commit();
                if (last) {
                    tma_store_wait_read();
                    mbar_arrive(bar_sfree + (i & 1) * 8);
                }
            }
            __syncwarp();
            if (last) {
                ++i;
                known = false;
            }
        }
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
    } else {
        // ------------------------------------------------------------ four threads per TMEM lane (32 columns each)
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                     // TMEM lane: S row (k index); w row (0-63)
        const int cb = ((warp - 2) >> 2) * 32;                // this thread's first column
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + cb;
        const bool has_w = quad < 2;
        const uint32_t tile_row = (cb >> 6) * 8192 + (row & 63) * 128, copy_row = (cb >> 6) * 16384 + row * 128;
        auto piece = [&](int i) -> uint32_t { return (uint32_t)((((cb & 63) >> 3) + i) ^ (lane & 7)) << 4; };
        auto arrive = [&](uint32_t bar) {                     // behind the writes and TMEM accesses of the whole warp
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        // the state's row as bf16 into copy i (announced), then S * mul into TMEM
        auto publish = [&](uint32_t (&r)[32], int i, float mul, bool always) {
            unsigned char* dst = smem + L::sbf + (i & 1) * 32768 + copy_row;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                uint32_t w4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w4[e] = pack_bf16(__uint_as_float(r[p * 8 + 2 * e]), __uint_as_float(r[p * 8 + 2 * e + 1]));
                *reinterpret_cast<uint4*>(dst + piece(p)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            fence_async_smem();
            tc_fence_before();
            arrive(bar_sready + (i & 1) * 8);
            if (mul != 1.f || always) {
#pragma unroll
                for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * mul);
                tmem_st32(t_lane + GS_S, r);
                tmem_st_wait();
            }
            tc_fence_before();
        };
        {   // initial state; the rows without w have nothing else to add to the first update
            uint32_t r[32];
            const float* init = h0 ? h0 + (((long)b * H + h) * K + row) * V + cb : nullptr;
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = init ? __float_as_uint(init[e]) : 0u;
            float mul = 1.f;
            if (init) {
                int j = 0;
                while (j < NT && !updates(j)) ++j;
                if (j < NT) mul = __expf(gcs[((long)b * T + min(j * 64 + 63, T - 1)) * H + h] + m_carry[j]);
            }
            publish(r, 0, mul, true);
            if (!has_w) arrive(bar_pv);
        }
        // cumsum g of the row and of the chunk's last token, l2 norm factor of the row of k
        auto load_scalars = [&](int c, float& gg, float& rr, float& gl) {
            const int valid = min(64, T - c * 64), tr = row & 63;
            const long tok0 = (long)b * T + (long)c * 64;
            gg = gcs[(tok0 + min(tr, valid - 1)) * H + h];
            gl = gcs[(tok0 + valid - 1) * H + h];
            rr = tr < valid ? krstd[(tok0 + tr) * H + h] : 0.f;
        };
        auto next_update = [&](int c) -> int {
            while (c < NT && !updates(c)) ++c;
            return c;
        };
        float g_cur = 0.f, r_cur = 0.f, gl_cur = 0.f, g_nxt = 0.f, r_nxt = 0.f, gl_nxt = 0.f;
        int c = next_update(0);
        if (has_w && c < NT) load_scalars(c, g_cur, r_cur, gl_cur);
#pragma unroll 1
        for (int i = 0; ok && c < NT; ++i) {
            const int cn = next_update(c + 1), stg = i & 1;
            const uint32_t par = (i >> 1) & 1;
            if (has_w && cn < NT) load_scalars(cn, g_nxt, r_nxt, gl_nxt);      // consumed in the next update
            uint32_t r[32];
            if (has_w) {
                // ---- v'' = (u - e^{carry} w S) rstd_k e^{g_last - g}
                const unsigned char* stage = smem + stg * L::stage;
                const float ec = __expf(m_carry[c]), f2 = r_cur * __expf(fminf(gl_cur - g_cur, 80.f));
                ok = warp_wait(bar_ku + stg * 8, par);
                if (!ok) break;
                uint4 ux[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) ux[p] = *reinterpret_cast<const uint4*>(stage + L::u + tile_row + piece(p));
                ok = warp_wait(bar_d1, i & 1);
                if (!ok) break;
                tc_fence_after();
                tmem_ld32(t_lane + GS_D1 + stg * 128, r);
                tmem_ld_wait();
                if (warp == 4 && lane == 0) mbar_arrive(bar_w_free + stg * 8);           // MMA 1 has read the stage
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const uint32_t* uw = reinterpret_cast<const uint32_t*>(&ux[p]);
                    uint32_t b4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 uf = unpack_bf16(uw[e]);
                        b4[e] = pack_bf16((uf.x - ec * __uint_as_float(r[p * 8 + 2 * e])) * f2,
                                          (uf.y - ec * __uint_as_float(r[p * 8 + 2 * e + 1])) * f2);
                    }
                    *reinterpret_cast<uint4*>(smem + L::vs + tile_row + piece(p)) = make_uint4(b4[0], b4[1], b4[2], b4[3]);
                }
                fence_async_smem();
                tc_fence_before();
                arrive(bar_pv);
            }
            // ---- every lane: the new state's copy (the one before the last has left), and the next update's decay
            if (i >= 1) ok = warp_wait(bar_sfree + (stg ^ 1) * 8, ((i - 1) >> 1) & 1);
            if (ok) ok = warp_wait(bar_s3, i & 1);
            if (!ok) break;
            tc_fence_after();
            tmem_ld32(t_lane + GS_S, r);
            tmem_ld_wait();
            publish(r, i + 1, __uint_as_float(m_mul[c] & 0x7fffffffu), false);
            if (has_w) {
                if (lane == 0) mbar_arrive(bar_ku_free + stg * 8);               // (u is in registers, MMA 3 has read k)
            } else if (cn < NT) {
                arrive(bar_pv);                               // MMA 3 of the next update may add to the state
            }
            c = cn;
            g_cur = g_nxt;
            r_cur = r_nxt;
            gl_cur = gl_nxt;
        }
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, GS_TMEM_COLS);
}

int gdn_states_tc(const void* k, const void* w, const void* u, const float* gcs, const float* k_rstd, const int32_t* types_i,
                  const int32_t* indices, const int32_t* n_blocks, const float* h0, void* h, float* carry, int B, int T, int H, int HN,
                  int decay, int trailing_quirk, cudaStream_t st) {
    const char* who = "natsl_linear_fwd_h";
    const cudaError_t e = cudaFuncSetAttribute(gdn_states_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GsSmem::total);
    if (e != cudaSuccess) {
        set_error("%s: cannot reserve %d B of shared memory (%s)", who, GsSmem::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mw, mk, mu, mh;
    int rc = encode_bthd_map(&mw, w, B, T, H, 128, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, H, 128, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mu, u, B, T, H, 128, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mh, h, B * ((T + 63) / 64) * H, 128, 1, 128, 128, who);
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    gdn_states_tc_kernel<<<dim3(H, B), GS_THREADS, GsSmem::total, st>>>(mw, mk, mu, mh, gcs, k_rstd, types_i, indices, n_blocks, h0, carry, T, H,
                                                                       HN, decay, trailing_quirk, status);
    return check_launch(who);
}

}  // namespace natsl
