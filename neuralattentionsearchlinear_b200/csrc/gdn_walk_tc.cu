// Gated-delta-rule recurrence AND chunk output in one walk on the 5th-generation tensor cores
// (head dims K = V = 128, nats_block_size = 64).  One CTA per (batch, head) walks the 64-token chunks in
// order; the K x V state lives in TMEM (fp32) and is never written to global memory.  Per chunk c
// (S = state the chunk reads, carry = decay of the skipped blocks before it):
//     [w S ; q S]       one stacked 128-row A operand [w ; q] against S (bf16 copy in shared memory)   (MMA 1)
//     v' = u - e^{carry} w S                                                                           (warps, from TMEM)
//     o  = scale (rstd_q e^{g+carry} q S + P v')      P = tril(qn kn^T e^{g_i-g_j}) from the prep kernel   (MMA 2 + warps)
//     S <- e^{g_last+carry} S + k^T (v' rstd_k e^{g_last-g})       only if the block is selected        (MMA 3)
// which is src/nats/ops/common/chunk_delta_h.py:189-324 (recurrence) fused with
// src/nats/ops/common/chunk_o.py:124-215 (output) and the carry of src/nats/ops/utils/cumsum.py:85-133.
// The decay of the state is applied when the state is copied to shared memory for the next chunk
// (one TMEM pass per update: bf16 copy out, multiply by the next update's decay, write back), so the
// accumulating MMA 3 needs no separate rescale.  P is padded to 128 rows (rows 0-63 zero) so that
// P v' lands in the TMEM lanes of the q rows.
// Warp roles: warp 0 TMA producer (w, q, k, u tiles in two stages, P single-buffered), warp 1 MMA issuer,
// warps 2-9 two threads per TMEM lane (64 columns each).  All mbarrier waits are bounded (status word +
// clean teardown on expiry).
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr int WK_THREADS = 320;
constexpr int WK_EPI = 256;
constexpr uint32_t WK_TMEM_COLS = 512;
constexpr uint32_t WK_S = 0, WK_D1 = 128, WK_D2 = 256, WK_D1B = 384;     // TMEM column offsets (D1 double-buffered)
constexpr int WK_MAX_NT = 1024;

struct WkSmem {
    // stage: [w;q] 2 sub-tiles [128][64] (32 KB), k 2 x [64][64] (16 KB), u 2 x [64][64] (16 KB)
    static constexpr int wq = 0, k = 32768, u = 49152, stage = 65536;
    static constexpr int sbf = 2 * stage;                 // S bf16: 2 sub-tiles [128 k-rows][64 v-cols]   32 KB
    static constexpr int vp = sbf + 32768;                // v'  : 2 sub-tiles [64 tok][64]                16 KB
    static constexpr int vs = vp + 16384;                 // v'' : same layout                              16 KB
    static constexpr int pp = vs + 16384;                 // P padded to 128 rows: [128][64 tok]            16 KB
    static constexpr int meta = pp + 16384;               // per chunk: carry, dec, g_last (float), sel (int)
    static constexpr int bars = meta + 4 * 4 * WK_MAX_NT;
    static constexpr int total = bars + 256;
};

template <bool kDummy>
__global__ void __launch_bounds__(WK_THREADS, 1)
gdn_walk_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_q,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_u,
                   const __grid_constant__ CUtensorMap map_p, const float* __restrict__ gcs,
                   const float* __restrict__ krstd, const float* __restrict__ qrstd, const int* __restrict__ types_i,
                   const int* __restrict__ indices, const int* __restrict__ n_blocks, const float* __restrict__ h0,
                   __nv_bfloat16* __restrict__ o, float* __restrict__ ht, float* hstart, const void* __restrict__ last_types,
                   int last_f32, int last_stride, int T, int H, int HN, int TN, float scale, int decay, int trailing_quirk, int* status) {
    using L = WkSmem;
    constexpr int K = 128, V = 128;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int h = blockIdx.x, b = blockIdx.y;
    const int hn = h / (H / HN);
    const int NT = (T + 63) / 64;
    float* m_carry = reinterpret_cast<float*>(smem + L::meta);
    float* m_dec = m_carry + WK_MAX_NT;
    float* m_gl = m_dec + WK_MAX_NT;
    int* m_sel = reinterpret_cast<int*>(m_gl + WK_MAX_NT);
    const uint32_t bar0 = sbase + L::bars;
    // barriers: full[2] / empty[2] tile stages; pfull / pfree the P tile; d1 (MMA 1 done); pv (v', v'' written by the
    // w lanes); d2 (MMA 2 done); s3 (MMA 3 done); sready (state copy published); odone (output rows read from TMEM)
    const uint32_t bar_full = bar0, bar_empty = bar0 + 16, bar_pfull = bar0 + 32, bar_pfree = bar0 + 40, bar_d1 = bar0 + 48,
                   bar_pv = bar0 + 56, bar_d2 = bar0 + 64, bar_s3 = bar0 + 72, bar_sready = bar0 + 80, bar_odone = bar0 + 88;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 128);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 1);
        }
        mbar_init(bar_pfull, 1);
        mbar_init(bar_pfree, 1);
        mbar_init(bar_d1, 1);
        mbar_init(bar_pv, WK_EPI / 2);
        mbar_init(bar_d2, 1);
        mbar_init(bar_s3, 1);
        mbar_init(bar_sready, WK_EPI);
        mbar_init(bar_odone, WK_EPI / 2);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), WK_TMEM_COLS);
    // ---- per-chunk metadata: selection, carry before the chunk, decay factor of the chunk's update
    for (int c = tid; c < NT; c += WK_THREADS) {
        m_sel[c] = types_i[(((long)b * TN + c) * HN + hn) * 2 + 1] != 0;
        m_gl[c] = gcs[((long)b * T + min(c * 64 + 63, T - 1)) * H + h];
    }
    // the P operand is padded to 128 rows; rows 0-63 stay zero
    for (int i = tid; i < 8192 / 16; i += WK_THREADS) reinterpret_cast<uint4*>(smem + L::pp)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (tid == 0) {
        const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
        const int last_sel = nsel > 0 ? indices[(((long)b * TN + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
        float carry = 0.f;
        for (int c = 0; c < NT; ++c) {
            const float gl = m_gl[c];
            m_carry[c] = carry;
            if (m_sel[c]) {
                m_dec[c] = __expf(gl + carry);
                carry = 0.f;
            } else {
                m_dec[c] = 1.f;
                if (decay && (!trailing_quirk || c < last_sel)) carry += gl;
            }
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            prefetch_tensormap(&map_w); prefetch_tensormap(&map_q); prefetch_tensormap(&map_k);
            prefetch_tensormap(&map_u); prefetch_tensormap(&map_p);
        }
        for (int c = 0; c < NT; ++c) {
            const int stg = c & 1;
            const int t0 = c * 64;
            if (c >= 2) {
                bool ok = mbar_wait_small(bar_empty + stg * 8, ((c >> 1) - 1) & 1, status);
                if (!__all_sync(0xffffffffu, ok)) break;
            }
            if (lane == 0) {
                const uint32_t full = bar_full + stg * 8, base = sbase + stg * L::stage;
                mbar_expect_tx(full, 65536);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    tma_load_4d(base + L::wq + sub * 16384, &map_w, sub * 64, h, t0, b, full);          // rows 0-63
                    tma_load_4d(base + L::wq + sub * 16384 + 8192, &map_q, sub * 64, h, t0, b, full);   // rows 64-127
                    tma_load_4d(base + L::k + sub * 8192, &map_k, sub * 64, h, t0, b, full);
                    tma_load_4d(base + L::u + sub * 8192, &map_u, sub * 64, h, t0, b, full);
                }
            }
            if (c >= 1) {
                bool ok = mbar_wait_small(bar_pfree, (c - 1) & 1, status);       // P of the previous chunk consumed
                if (!__all_sync(0xffffffffu, ok)) break;
            }
            if (lane == 0) {
                mbar_expect_tx(bar_pfull, 8192);
                tma_load_4d(sbase + L::pp + 8192, &map_p, 0, h, t0, b, bar_pfull);                      // rows 64-127
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t id_1 = umma_idesc_bf16(128, 128, true);                       // [w;q] S
        constexpr uint32_t id_2 = umma_idesc_bf16(128, 128, true);                       // P v'
        constexpr uint32_t id_3 = umma_idesc_bf16(128, 128, true) | (1u << 15);          // k^T v'' (A MN-major)
        bool ok = true;
        for (int c = 0; ok && c < NT; ++c) {
            const int stg = c & 1;
            const uint32_t base = sbase + stg * L::stage;
            ok = __all_sync(0xffffffffu, mbar_wait_small(bar_full + stg * 8, (c >> 1) & 1, status));
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait_small(bar_sready, c & 1, status));
            if (!ok) break;
            const uint32_t d1 = tmem + ((c & 1) ? WK_D1B : WK_D1);
            {
                tc_fence_after();
                const uint32_t al = umma_desc_lo(base + L::wq, 16), bl = umma_desc_lo(sbase + L::sbf, 16384);
#pragma unroll
                for (int h = 0; h < 2; ++h) umma_ss_x4<2, 128>(d1, al + h * 1024, bl + h * 512, id_1, h > 0);
                umma_commit(bar_d1);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait_small(bar_pv, c & 1, status));
            if (!ok) break;
            {
                // the state update first: the next chunk's products wait for it, the output does not
                tc_fence_after();
                if (m_sel[c]) {
                    umma_ss_x4<128, 128>(tmem + WK_S, umma_desc_lo(base + L::k, 8192), umma_desc_lo(sbase + L::vs, 8192), id_3, 1u);
                }
                umma_commit(bar_s3);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait_small(bar_pfull, c & 1, status));
            if (ok && c > 0) ok = __all_sync(0xffffffffu, mbar_wait_small(bar_odone, (c - 1) & 1, status));   // D2 is free
            if (!ok) break;
            {
                tc_fence_after();
                umma_ss_x4<2, 128>(tmem + WK_D2, umma_desc_lo(sbase + L::pp, 16), umma_desc_lo(sbase + L::vp, 8192), id_2, 0u);
                umma_commit(bar_d2);
                umma_commit(bar_pfree);
                umma_commit(bar_empty + stg * 8);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------ two threads per TMEM lane (64 columns each)
        const int quad = warp & 3;
        const int half = (warp - 2) >> 2;
        const int row = quad * 32 + lane;                 // TMEM lane: S row (k index); w row (0-63) or q row (64-127)
        const int cb = half * 64;                         // this thread's first column
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16);
        const bool is_q = row >= 64;
        const int tr = row & 63;                          // token row inside the chunk
        bool ok = true;

        // the state in front of the last chunk (with its carried decay), for a decoder that continues the sequence: it is
        // the one published when no chunk from `c` up to the last one updates the state
        float* hs_row = hstart ? hstart + (((long)b * H + h) * K + row) * V : nullptr;
        auto starts_last = [&](int c) -> bool {
            if (!hs_row) return false;
            for (int j = c; j < NT - 1; ++j)
                if (m_sel[j]) return false;
            return true;
        };
        auto store_row = [&](float* dst, int c0, const uint32_t (&r)[32], float f) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(dst + c0 + i) = make_float4(__uint_as_float(r[i]) * f, __uint_as_float(r[i + 1]) * f,
                                                                      __uint_as_float(r[i + 2]) * f, __uint_as_float(r[i + 3]) * f);
        };
        // copies columns [cb, cb+64) of this lane's S row as bf16 into the shared copy and leaves S * mul in TMEM
        auto publish_state = [&](float mul, const float* init_row, bool hs) {
#pragma unroll 1
            for (int c0 = cb; c0 < cb + 64; c0 += 32) {
                uint32_t r[32];
                if (init_row) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(init_row[c0 + i]);
                } else {
                    tmem_ld32(t_lane + WK_S + c0, r);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    uint32_t w4[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        w4[i] = pack_bf16(__uint_as_float(r[cc * 8 + 2 * i]), __uint_as_float(r[cc * 8 + 2 * i + 1]));
                    const int col = c0 + cc * 8;          // v column of this 16-byte chunk
                    *reinterpret_cast<uint4*>(smem + L::sbf + (col >> 6) * 16384 + swz<128>(row, (col & 63) >> 3)) =
                        make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                if (hs) store_row(hs_row, c0, r, __expf(m_carry[NT - 1]));
                if (mul != 1.f || init_row) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * mul);
                    tmem_st32(t_lane + WK_S + c0, r);
                }
            }
            tmem_st_wait();
        };
        // decay factor of the next update at or after chunk c
        auto next_dec = [&](int c) -> float {
            for (int j = c; j < NT; ++j)
                if (m_sel[j]) return m_dec[j];
            return 1.f;
        };
        {   // initial state
            const float* init = h0 ? h0 + (((long)b * H + h) * K + row) * V : nullptr;
            if (init) {
                publish_state(next_dec(0), init, starts_last(0));
            } else {
                const bool hs = starts_last(0);
#pragma unroll 1
                for (int c0 = cb; c0 < cb + 64; c0 += 32) {
                    uint32_t r[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = 0u;
                    tmem_st32(t_lane + WK_S + c0, r);
                    if (hs) store_row(hs_row, c0, r, 1.f);
                }
                tmem_st_wait();
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<uint4*>(smem + L::sbf + half * 16384 + swz<128>(row, i)) = make_uint4(0, 0, 0, 0);
            }
            fence_async_smem();
            tc_fence_before();
            mbar_arrive(bar_sready);
        }
        // per-row scalars of the chunk: cumsum g and the l2 norm factor (k rows for w lanes, q rows for q lanes)
        auto load_scalars = [&](int c, float& gg, float& rr) {
            const int valid = min(64, T - c * 64);
            const long tok0 = (long)b * T + (long)c * 64;
            gg = gcs[(tok0 + min(tr, valid - 1)) * H + h];
            const float* rs = is_q ? qrstd : krstd;
            rr = (tr < valid) ? rs[(tok0 + tr) * H + h] : 0.f;
        };
        float g_cur, r_cur, g_nxt = 0.f, r_nxt = 0.f;
        load_scalars(0, g_cur, r_cur);

        for (int c = 0; c < NT; ++c) {
            const int stg = c & 1;
            const int valid = min(64, T - c * 64);
            const long tok0 = (long)b * T + (long)c * 64;
            unsigned char* stage = smem + stg * L::stage;
            if (c + 1 < NT) load_scalars(c + 1, g_nxt, r_nxt);          // prefetch; consumed next iteration
            const float carry = m_carry[c];
            const float gl = m_gl[c];
            const bool sel = m_sel[c] != 0;
            const uint32_t t_d1 = t_lane + ((c & 1) ? WK_D1B : WK_D1);
            // After a failed (bounded) wait the remaining work is skipped; the loop still runs to its end.
            // Every lane first sees MMA 1 of this chunk complete: it was issued behind the previous phase of the
            // "state published" barrier, so no thread can arrive on that barrier twice within one phase.
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait_small(bar_d1, c & 1, status));
            if (!is_q) {
                // ---- w lanes: v' = u - e^{carry} w S ; v'' = v' rstd_k e^{g_last - g}   (the u tile arrived with the stage)
                if (ok) {
                    tc_fence_after();
                    const float ec = __expf(carry);
                    const float f2 = r_cur * __expf(fminf(gl - g_cur, 80.f));
#pragma unroll 1
                    for (int c0 = cb; c0 < cb + 64; c0 += 32) {
                        uint32_t r[32];
                        tmem_ld32(t_d1 + c0, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc) {
                            const int col = c0 + cc * 8;
                            const uint32_t off = (col >> 6) * 8192 + swz<128>(tr, (col & 63) >> 3);
                            const uint4 ux = *reinterpret_cast<const uint4*>(stage + L::u + off);
                            const uint32_t* uw = reinterpret_cast<const uint32_t*>(&ux);
                            uint32_t a4[4], b4[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float2 uf = unpack_bf16(uw[i]);
                                const float v0 = uf.x - ec * __uint_as_float(r[cc * 8 + 2 * i]);
                                const float v1 = uf.y - ec * __uint_as_float(r[cc * 8 + 2 * i + 1]);
                                a4[i] = pack_bf16(v0, v1);
                                b4[i] = pack_bf16(v0 * f2, v1 * f2);
                            }
                            *reinterpret_cast<uint4*>(smem + L::vp + off) = make_uint4(a4[0], a4[1], a4[2], a4[3]);
                            *reinterpret_cast<uint4*>(smem + L::vs + off) = make_uint4(b4[0], b4[1], b4[2], b4[3]);
                        }
                    }
                    fence_async_smem();
                    tc_fence_before();
                    mbar_arrive(bar_pv);
                }
            }
            // ---- every lane: publish the updated state for the next chunk (and pre-apply the next update's decay).
            // This is the serial chain of the walk; the output rows below are read after it.
            if (ok && sel) {
                ok = __all_sync(0xffffffffu, mbar_wait_small(bar_s3, c & 1, status));
                if (ok) {
                    tc_fence_after();
                    publish_state(next_dec(c + 1), nullptr, c < NT - 1 && starts_last(c + 1));
                    fence_async_smem();
                }
            }
            if (ok) {
                tc_fence_before();
                mbar_arrive(bar_sready);
            }
            if (is_q) {
                // ---- q lanes: o = scale (rstd_q e^{g+carry} q S + P v'), off the chain (D1 is double-buffered, D2 is
                // released by the arrival below)
                if (ok) ok = __all_sync(0xffffffffu, mbar_wait_small(bar_d2, c & 1, status));
                if (ok) {
                    tc_fence_after();
                    const float fq = r_cur * __expf(g_cur + carry);
                    __nv_bfloat16* orow = o + ((tok0 + tr) * H + h) * V;
#pragma unroll 1
                    for (int c0 = cb; c0 < cb + 64; c0 += 32) {
                        uint32_t r1[32], r2[32];
                        tmem_ld32(t_d1 + c0, r1);
                        tmem_ld32(t_lane + WK_D2 + c0, r2);
                        tmem_ld_wait();
                        if (tr < valid) {
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc) {
                                uint32_t w4[4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const int e = cc * 8 + 2 * i;
                                    w4[i] = pack_bf16(scale * (fq * __uint_as_float(r1[e]) + __uint_as_float(r2[e])),
                                                      scale * (fq * __uint_as_float(r1[e + 1]) + __uint_as_float(r2[e + 1])));
                                }
                                *reinterpret_cast<uint4*>(orow + c0 + cc * 8) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                            }
                        }
                    }
                    tc_fence_before();
                    mbar_arrive(bar_odone);
                }
            }
            g_cur = g_nxt;
            r_cur = r_nxt;
        }
        // every update's decay was pre-applied except after the last one: TMEM holds the final state.  A complete last
        // block: the decoder continues from it if that block's own type is linear, else from the state in front of the
        // block, decayed over it.
        bool last_lin = false, last_roll = false;
        if (hs_row && T % 64 == 0) {
            const long li = (long)b * last_stride + hn * 2 + 1;
            last_lin = (last_f32 ? reinterpret_cast<const float*>(last_types)[li]
                                 : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(last_types)[li])) > 0.f;
            last_roll = !last_lin && decay;
        }
        if (ok && (ht || last_lin || last_roll)) {
            tc_fence_after();
            float* hrow = ht ? ht + (((long)b * H + h) * K + row) * V : nullptr;
            const float f = last_roll ? __expf(m_gl[NT - 1]) : 1.f;
#pragma unroll 1
            for (int c0 = cb; c0 < cb + 64; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(t_lane + WK_S + c0, r);
                tmem_ld_wait();
                if (hrow) store_row(hrow, c0, r, 1.f);
                if (last_lin) store_row(hs_row, c0, r, 1.f);
                if (last_roll) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(hs_row[c0 + i]);
                    store_row(hs_row, c0, r, f);
                }
            }
        }
    }
    // ---------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, WK_TMEM_COLS);
}

}  // namespace natsl

extern "C" int natsl_gdn_walk_fused_ex(const void* q, const void* k, const void* w, const void* u, const void* pmat,
                                    const float* gcs, const float* k_rstd, const float* q_rstd, const int32_t* types_i,
                                    const int32_t* indices, const int32_t* n_blocks, const float* h0, void* o, float* ht,
                                    float* hstart, const void* last_types, int last_dtype, int last_stride, int B, int T, int H, int HN, int K,
                                    int V, int nbs, float scale, int flags, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && w && u && pmat && gcs && k_rstd && q_rstd && types_i && indices && n_blocks && o, NATSL_ERR_NULL,
                  "natsl_gdn_walk_fused: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0, NATSL_ERR_BAD_SHAPE, "natsl_gdn_walk_fused: bad shape");
    NATSL_REQUIRE(K == 128 && V == 128 && nbs == 64, NATSL_ERR_UNSUPPORTED,
                  "natsl_gdn_walk_fused: built for K = V = 128 and nats_block_size = 64 (got K=%d V=%d nbs=%d); use "
                  "natsl_linear_fwd_h + natsl_linear_fwd_o", K, V, nbs);
    NATSL_REQUIRE((T + 63) / 64 <= WK_MAX_NT, NATSL_ERR_TOO_LARGE, "natsl_gdn_walk_fused: T <= 65536");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_gdn_walk_fused: B, H <= 65535");
    NATSL_REQUIRE(!hstart || T % nbs != 0 || (last_types && (last_dtype == NATSL_DT_F32 || last_dtype == NATSL_DT_BF16)),
                  NATSL_ERR_NULL, "natsl_gdn_walk_fused: the block-start state of a complete last block needs that block's types");
    auto kern = gdn_walk_tc_kernel<true>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WkSmem::total);
    if (e != cudaSuccess) {
        set_error("natsl_gdn_walk_fused: cannot reserve %d B of shared memory (%s)", WkSmem::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mw, mq, mk, mu, mp;
    int rc = encode_bthd_map(&mw, w, B, T, H, K, 64, "natsl_gdn_walk_fused(w)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mq, q, B, T, H, K, 64, "natsl_gdn_walk_fused(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, H, K, 64, "natsl_gdn_walk_fused(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mu, u, B, T, H, V, 64, "natsl_gdn_walk_fused(u)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mp, pmat, B, T, H, 64, 64, "natsl_gdn_walk_fused(P)");
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    const int TN = (T + nbs - 1) / nbs;
    dim3 grid(H, B);
    kern<<<grid, WK_THREADS, WkSmem::total, reinterpret_cast<cudaStream_t>(stream)>>>(
        mw, mq, mk, mu, mp, gcs, k_rstd, q_rstd, types_i, indices, n_blocks, h0, reinterpret_cast<__nv_bfloat16*>(o), ht, hstart,
        last_types, last_dtype == NATSL_DT_F32, last_stride, T, H, HN, TN, scale, (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0, (flags & NATSL_FLAG_NO_TRAILING_QUIRK) ? 0 : 1, status);
    return check_launch("natsl_gdn_walk_fused");
}

extern "C" int natsl_gdn_walk_fused(const void* q, const void* k, const void* w, const void* u, const void* pmat,
                                    const float* gcs, const float* k_rstd, const float* q_rstd, const int32_t* types_i,
                                    const int32_t* indices, const int32_t* n_blocks, const float* h0, void* o, float* ht,
                                    int B, int T, int H, int HN, int K, int V, int nbs, float scale, int flags,
                                    void* stream) {
    return natsl_gdn_walk_fused_ex(q, k, w, u, pmat, gcs, k_rstd, q_rstd, types_i, indices, n_blocks, h0, o, ht, nullptr, nullptr,
                                   0, 0, B, T, H, HN, K, V, nbs, scale, flags, stream);
}
