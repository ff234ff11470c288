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
// accumulating MMA 3 needs no separate rescale.  The product P v' has 128 rows: P in the rows of q, whatever lies in front of the
// tile in the others, whose results nobody reads.
//
// What bounds it: the chain w S -> v' -> k^T v'' -> copy of the state, chunk after chunk, one CTA per SM.  Hence sixteen warps
// with 32 columns of a TMEM lane each (loads, products and stores of a step in one go, not in a loop), one arrival per warp on a
// barrier, everything that does not depend on the step's product read or computed in front of the wait for it, the multiplied
// state written back behind the announcement of its copy, and outputs that leave through shared memory by TMA: rows of 16 bytes
// per lane kept the load/store unit busy for half of a chunk, and the next chunk's v' waited behind them.
// Alone (us; before: eight warps of 64 columns each, outputs stored row by row): B = 8, T = 4096, H = 16, 75 % of the chunks
// selected 173 -> 130 (738 MB: 5.7 TB/s), 50 % 168 -> 127; 32 CTAs, T = 8192 333 -> 234, 1.8 us a chunk.  Of 4.6 k cycles per chunk the
// old form spent 2.1 k on v' and 1.7 k of the output warps on their stores.
// Warp roles: warp 0 loads w, q and k, u (two stages, each half of a stage given back on its own), warp 1 issues the products,
// warps 2-17 the rows, warp 18 loads P (one buffer) and stores the outputs.  All mbarrier waits are bounded (status word + clean
// teardown on expiry).
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr int WK_THREADS = 608;
constexpr int WK_ROW_WARPS = 16;
constexpr uint32_t WK_TMEM_COLS = 512;
constexpr uint32_t WK_S = 0, WK_D1 = 128, WK_D2 = 256, WK_D1B = 384;     // TMEM column offsets (D1 double-buffered)
constexpr int WK_MAX_NT = 1024;

struct WkSmem {
    // stage: [w;q] 2 sub-tiles [128][64] (32 KB), k 2 x [64][64] (16 KB), u 2 x [64][64] (16 KB)
    static constexpr int wq = 0, k = 32768, u = 49152, stage = 65536;
    static constexpr int sbf = 2 * stage;                 // S bf16: 2 sub-tiles [128 k-rows][64 v-cols]   32 KB
    static constexpr int vp = sbf + 32768;                // v'  : 2 sub-tiles [64 tok][64]                16 KB
    static constexpr int vs = vp + 16384;                 // v'' : same layout                              16 KB
    static constexpr int pp = vs + 16384;                 // P : [64][64 tok]; the operand begins 8 KB in front of it
    static constexpr int out = pp + 8192;                 // outputs on their way: 2 sub-tiles [64 tok][64] 16 KB
    static constexpr int carry = out + 16384;             // per chunk: decay of the skipped blocks in front of it;
    static constexpr int mul = carry + 4 * WK_MAX_NT;     // the next update's decay, sign bit set where the chunk updates the state
    static constexpr int bars = mul + 4 * WK_MAX_NT;
    static constexpr int total = bars + 256;
    static_assert(total <= 232448, "shared memory of one SM");
};

__global__ void __launch_bounds__(WK_THREADS, 1)
gdn_walk_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_q,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_u,
                   const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_o,
                   const float* __restrict__ gcs, const float* __restrict__ krstd, const float* __restrict__ qrstd,
                   const int* __restrict__ types_i, const int* __restrict__ indices, const int* __restrict__ n_blocks,
                   const float* __restrict__ h0, float* __restrict__ ht, float* hstart, const void* __restrict__ last_types,
                   int last_f32, int last_stride, int T, int H, int HN, int TN, float scale, int decay, int trailing_quirk, int* status) {
    using L = WkSmem;
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
    // barriers: full / empty of the two stages of [w;q] and of k, u; pfull (P has landed); d1, s3, d2 (MMA 1, 3, 2 done);
    // pv (v', v'' written and the state written back); sready (state copy published); odone (output rows read from TMEM);
    // ofull / ofree (output rows written to shared memory / stored)
    const uint32_t bar_wq = bar0, bar_wq_free = bar0 + 16, bar_ku = bar0 + 32, bar_ku_free = bar0 + 48, bar_p = bar0 + 64,
                   bar_d1 = bar0 + 72, bar_pv = bar0 + 80, bar_d2 = bar0 + 88, bar_s3 = bar0 + 96, bar_sready = bar0 + 104,
                   bar_odone = bar0 + 112, bar_ofull = bar0 + 120, bar_ofree = bar0 + 128;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 192);
    int* hs_slot = reinterpret_cast<int*>(smem + L::bars + 196);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_wq + 8 * i, 1);
            mbar_init(bar_wq_free + 8 * i, 1);
            mbar_init(bar_ku + 8 * i, 1);
            mbar_init(bar_ku_free + 8 * i, WK_ROW_WARPS / 2);
        }
        mbar_init(bar_p, 1);
        mbar_init(bar_d1, 1);
        mbar_init(bar_pv, WK_ROW_WARPS);
        mbar_init(bar_d2, 1);
        mbar_init(bar_s3, 1);
        mbar_init(bar_sready, WK_ROW_WARPS);
        mbar_init(bar_odone, WK_ROW_WARPS / 2);
        mbar_init(bar_ofull, WK_ROW_WARPS / 2);
        mbar_init(bar_ofree, 1);
        mbar_fence_init();
        *hs_slot = -1;
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), WK_TMEM_COLS);
    // ---- per-chunk scalars.  Every chunk adds up its own run of skipped chunks, first to last, as one thread would do for all.
    {
        float* gl = reinterpret_cast<float*>(smem + L::sbf);          // (overwritten by the initial state)
        int* sel = reinterpret_cast<int*>(smem + L::sbf) + WK_MAX_NT;
        for (int c = tid; c < NT; c += WK_THREADS) {
            sel[c] = types_i[(((long)b * TN + c) * HN + hn) * 2 + 1] != 0;
            gl[c] = gcs[((long)b * T + min(c * 64 + 63, T - 1)) * H + h];
        }
        const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
        const int last_sel = nsel > 0 ? indices[(((long)b * TN + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
        __syncthreads();
        for (int c = tid; c < NT; c += WK_THREADS) {
            float carry = 0.f;
            if (decay) {
                int j = c;
                while (j > 0 && !sel[j - 1]) --j;
                for (; j < c; ++j)
                    if (!trailing_quirk || j < last_sel) carry += gl[j];
            }
            m_carry[c] = carry;
        }
        __syncthreads();
        for (int c = tid; c < NT; c += WK_THREADS) {
            int j = c + 1;
            while (j < NT && !sel[j]) ++j;
            const float mul = j < NT ? __expf(gl[j] + m_carry[j]) : 1.f;
            m_mul[c] = (__float_as_uint(mul) & 0x7fffffffu) | (sel[c] ? 0x80000000u : 0u);
            if (sel[c] && c < NT - 1 && j >= NT - 1) *hs_slot = c;     // the last update in front of the last chunk
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------ loads of w, q and of k, u
        if (lane == 0) {
            prefetch_tensormap(&map_w); prefetch_tensormap(&map_q); prefetch_tensormap(&map_k);
            prefetch_tensormap(&map_u);
        }
        int n_wq = 0, n_ku = 0;                           // chunks asked for
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            const int stg = c & 1, t0 = c * 64;
            const uint32_t par = ((c >> 1) - 1) & 1, base = sbase + stg * L::stage;
            if (c >= 2) ok = warp_wait(bar_wq_free + stg * 8, par);
            if (!ok) break;
            if (lane == 0) {
                const uint32_t full = bar_wq + stg * 8;
                mbar_expect_tx(full, 32768);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    tma_load_4d(base + L::wq + sub * 16384, &map_w, sub * 64, h, t0, b, full);          // rows 0-63
                    tma_load_4d(base + L::wq + sub * 16384 + 8192, &map_q, sub * 64, h, t0, b, full);   // rows 64-127
                }
            }
            __syncwarp();
            ++n_wq;
            if (c >= 2) ok = warp_wait(bar_ku_free + stg * 8, par);
            if (!ok) break;
            if (lane == 0) {
                const uint32_t full = bar_ku + stg * 8;
                mbar_expect_tx(full, 32768);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    tma_load_4d(base + L::u + sub * 8192, &map_u, sub * 64, h, t0, b, full);
                    tma_load_4d(base + L::k + sub * 8192, &map_k, sub * 64, h, t0, b, full);
                }
            }
            __syncwarp();
            ++n_ku;
        }
        if (!ok) {                                        // nothing may still be on its way into shared memory
            for (int c = max(0, n_wq - 2); c < n_wq; ++c) warp_wait(bar_wq + (c & 1) * 8, (c >> 1) & 1);
            for (int c = max(0, n_ku - 2); c < n_ku; ++c) warp_wait(bar_ku + (c & 1) * 8, (c >> 1) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t id = umma_idesc_bf16(128, 128, true);                         // [w;q] S, P v'
        constexpr uint32_t id_3 = id | (1u << 15);                                       // k^T v'' (A MN-major)
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            const int stg = c & 1;
            const uint32_t base = sbase + stg * L::stage, par = (c >> 1) & 1;
            const bool sel = (m_mul[c] >> 31) != 0;
            ok = warp_wait(bar_wq + stg * 8, par);
            if (ok) ok = warp_wait(bar_sready, c & 1);
            if (!ok) break;
            tc_fence_after();
            {
                const uint32_t d1 = tmem + ((c & 1) ? WK_D1B : WK_D1);
                const uint32_t al = umma_desc_lo(base + L::wq, 16), bl = umma_desc_lo(sbase + L::sbf, 16384);
#pragma unroll
                for (int e = 0; e < 2; ++e) umma_ss_x4<2, 128>(d1, al + e * 1024, bl + e * 512, id, e > 0);
                umma_commit(bar_d1);
            }
            // (k: the phase of its barrier stands still only while the chunk's update, which gives the stage back, is to come)
            if (sel) ok = warp_wait(bar_ku + stg * 8, par);
            if (ok) ok = warp_wait(bar_pv, c & 1);
            if (!ok) break;
            tc_fence_after();
            // the state update first: the next chunk's products wait for it, the output does not
            if (sel) {
                umma_ss_x4<128, 128>(tmem + WK_S, umma_desc_lo(base + L::k, 8192), umma_desc_lo(sbase + L::vs, 8192), id_3, 1u);
                umma_commit(bar_s3);
            }
            ok = warp_wait(bar_p, c & 1);
            if (ok && c > 0) ok = warp_wait(bar_odone, (c - 1) & 1);                     // D2 is free
            if (!ok) break;
            tc_fence_after();
            umma_ss_x4<2, 128>(tmem + WK_D2, umma_desc_lo(sbase + L::pp - 8192, 16), umma_desc_lo(sbase + L::vp, 8192), id, 0u);
            umma_commit(bar_d2);
        }
    } else if (warp == WK_ROW_WARPS + 2) {
        // ------------------------------------------------------------ loads of P, stores of the outputs
        int n_p = 0;                                      // tiles asked for
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            if (c > 0) ok = warp_wait(bar_d2, (c - 1) & 1);              // P of the chunk before is used up
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar_p, 8192);
                tma_load_4d(sbase + L::pp, &map_p, 0, h, c * 64, b, bar_p);
            }
            __syncwarp();
            ++n_p;
            if (c > 0) ok = warp_wait(bar_ofull, (c - 1) & 1);
            if (!ok) break;
            if (c > 0 && lane == 0) {
                tma_store_4d(&map_o, sbase + L::out, 0, h, (c - 1) * 64, b);
                tma_store_4d(&map_o, sbase + L::out + 8192, 64, h, (c - 1) * 64, b);
                tma_store_commit();
                tma_store_wait_read();
                mbar_arrive(bar_ofree);
            }
            __syncwarp();
        }
        if (!ok && n_p > 0) warp_wait(bar_p, (n_p - 1) & 1);
        if (ok) ok = warp_wait(bar_ofull, (NT - 1) & 1);
        if (ok && lane == 0) {
            tma_store_4d(&map_o, sbase + L::out, 0, h, (NT - 1) * 64, b);
            tma_store_4d(&map_o, sbase + L::out + 8192, 64, h, (NT - 1) * 64, b);
            tma_store_commit();
            tma_store_wait_read();
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ four threads per TMEM lane (32 columns each)
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                 // TMEM lane: S row (k index); w row (0-63) or q row (64-127)
        const int cb = ((warp - 2) >> 2) * 32;            // this thread's first column
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + cb;
        const bool is_q = quad >= 2;
        const int tr = row & 63;                          // token row inside the chunk
        const int hs_at = *hs_slot;
        // 16-byte pieces of this thread's columns: row `tr` of a [64][64] tile, row `row` of the state's copy
        const uint32_t tile_row = (cb >> 6) * 8192 + tr * 128, copy_row = (cb >> 6) * 16384 + row * 128;
        auto piece = [&](int i) -> uint32_t { return (uint32_t)((((cb & 63) >> 3) + i) ^ (lane & 7)) << 4; };
        auto arrive = [&](uint32_t bar) {                 // behind the writes and TMEM accesses of the whole warp
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };

        // the state in front of the last chunk (with its carried decay), for a decoder that continues the sequence
        float* hs_row = hstart ? hstart + (((long)b * H + h) * K + row) * V + cb : nullptr;
        auto store_row = [&](float* dst, const uint32_t (&r)[32], float f) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(r[i]) * f, __uint_as_float(r[i + 1]) * f,
                                                                 __uint_as_float(r[i + 2]) * f, __uint_as_float(r[i + 3]) * f);
        };
        // the state's row as bf16 into the shared copy (announced), then S * mul into TMEM
        auto publish_state = [&](uint32_t (&r)[32], float mul, bool always, bool hs, float hs_decay) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t w4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w4[e] = pack_bf16(__uint_as_float(r[i * 8 + 2 * e]), __uint_as_float(r[i * 8 + 2 * e + 1]));
                *reinterpret_cast<uint4*>(smem + L::sbf + copy_row + piece(i)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            fence_async_smem();
            tc_fence_before();
            arrive(bar_sready);
            if (hs_row && hs) store_row(hs_row, r, hs_decay);
            if (mul != 1.f || always) {
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * mul);
                tmem_st32(t_lane + WK_S, r);
                tmem_st_wait();
            }
            tc_fence_before();
        };
        {   // initial state; the rows of q have nothing else to add to the first chunk's update
            uint32_t r[32];
            const float* init = h0 ? h0 + (((long)b * H + h) * K + row) * V + cb : nullptr;
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = init ? __float_as_uint(init[i]) : 0u;
            float mul = 1.f;
            if (init) {
                int j = 0;
                while (j < NT && !(m_mul[j] >> 31)) ++j;
                if (j < NT) mul = __expf(gcs[((long)b * T + min(j * 64 + 63, T - 1)) * H + h] + m_carry[j]);
            }
            publish_state(r, mul, true, hs_at < 0, init ? __expf(m_carry[NT - 1]) : 1.f);
            if (is_q) arrive(bar_pv);
        }
        // per-row scalars of the chunk: cumsum g (of the row and of the chunk's last token) and the l2 norm factor (k rows for w
        // lanes, q rows for q lanes)
        auto load_scalars = [&](int c, float& gg, float& rr, float& gl) {
            const int valid = min(64, T - c * 64);
            const long tok0 = (long)b * T + (long)c * 64;
            gg = gcs[(tok0 + min(tr, valid - 1)) * H + h];
            gl = gcs[(tok0 + valid - 1) * H + h];
            const float* rs = is_q ? qrstd : krstd;
            rr = (tr < valid) ? rs[(tok0 + tr) * H + h] : 0.f;
        };
        int n_upd = 0;                                    // updates so far: phases of bar_s3
        float g_cur, r_cur, gl_cur, g_nxt = 0.f, r_nxt = 0.f, gl_nxt = 0.f;
        load_scalars(0, g_cur, r_cur, gl_cur);

#pragma unroll 1
        for (int c = 0; ok && c < NT; ++c) {
            const int stg = c & 1;
            const unsigned char* stage = smem + stg * L::stage;
            if (c + 1 < NT) load_scalars(c + 1, g_nxt, r_nxt, gl_nxt);  // prefetch; consumed next iteration
            const float carry = m_carry[c];
            const uint32_t mulw = m_mul[c];
            const bool sel = (mulw >> 31) != 0;
            const uint32_t t_d1 = t_lane + ((c & 1) ? WK_D1B : WK_D1);
            uint32_t r[32];
            if (!is_q) {
                // ---- w lanes: v' = u - e^{carry} w S ; v'' = v' rstd_k e^{g_last - g}
                const float ec = __expf(carry);
                const float f2 = r_cur * __expf(fminf(gl_cur - g_cur, 80.f));
                ok = warp_wait(bar_ku + stg * 8, (c >> 1) & 1);
                if (!ok) break;
                uint4 ux[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) ux[i] = *reinterpret_cast<const uint4*>(stage + L::u + tile_row + piece(i));
                ok = warp_wait(bar_d1, c & 1);
                if (!ok) break;
                tc_fence_after();
                tmem_ld32(t_d1, r);
                tmem_ld_wait();
                if (warp == 4 && lane == 0) mbar_arrive(bar_wq_free + stg * 8);          // MMA 1 has read the stage
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t* uw = reinterpret_cast<const uint32_t*>(&ux[i]);
                    uint32_t a4[4], b4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 uf = unpack_bf16(uw[e]);
                        const float v0 = uf.x - ec * __uint_as_float(r[i * 8 + 2 * e]);
                        const float v1 = uf.y - ec * __uint_as_float(r[i * 8 + 2 * e + 1]);
                        a4[e] = pack_bf16(v0, v1);
                        b4[e] = pack_bf16(v0 * f2, v1 * f2);
                    }
                    *reinterpret_cast<uint4*>(smem + L::vs + tile_row + piece(i)) = make_uint4(b4[0], b4[1], b4[2], b4[3]);
                    *reinterpret_cast<uint4*>(smem + L::vp + tile_row + piece(i)) = make_uint4(a4[0], a4[1], a4[2], a4[3]);
                }
                fence_async_smem();
                tc_fence_before();
                arrive(bar_pv);
            } else {
                ok = warp_wait(bar_d1, c & 1);
                if (!ok) break;
            }
            // ---- every lane: publish the updated state for the next chunk (and pre-apply the next update's decay).  This is the
            // serial chain of the walk; the output rows are read after it.  (Every lane has seen MMA 1 of this chunk complete: it
            // was issued behind the previous phase of the "state published" barrier, so no warp arrives on that barrier twice
            // within one phase.)
            if (sel) {
                ok = warp_wait(bar_s3, n_upd & 1);
                ++n_upd;
                if (!ok) break;
                tc_fence_after();
                tmem_ld32(t_lane + WK_S, r);
                tmem_ld_wait();
                publish_state(r, __uint_as_float(mulw & 0x7fffffffu), false, c == hs_at, c == hs_at ? __expf(m_carry[NT - 1]) : 0.f);
            } else {
                tc_fence_before();
                arrive(bar_sready);
            }
            if (!is_q) {
                if (lane == 0) mbar_arrive(bar_ku_free + stg * 8);       // (u is in registers, MMA 3 has read k)
            } else {
                // ---- q lanes: o = scale (rstd_q e^{g+carry} q S + P v'), off the chain (D1 is double-buffered).  MMA 3 of the next
                // chunk may add to the state once it is written back: with an update that has just happened; without one the
                // arrival has to wait until the barrier's phase of this chunk is over, which MMA 2 tells.
                if (sel && c + 1 < NT) arrive(bar_pv);
                const float fq = r_cur * __expf(g_cur + carry);
                ok = warp_wait(bar_d2, c & 1);
                if (!ok) break;
                if (!sel && c + 1 < NT) arrive(bar_pv);
                tc_fence_after();
                uint32_t r2[32];
                tmem_ld32(t_d1, r);
                tmem_ld32(t_lane + WK_D2, r2);
                tmem_ld_wait();
                tc_fence_before();
                arrive(bar_odone);
                if (c > 0) ok = warp_wait(bar_ofree, (c - 1) & 1);
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int x = i * 8 + 2 * e;
                        w4[e] = pack_bf16(scale * (fq * __uint_as_float(r[x]) + __uint_as_float(r2[x])),
                                          scale * (fq * __uint_as_float(r[x + 1]) + __uint_as_float(r2[x + 1])));
                    }
                    *reinterpret_cast<uint4*>(smem + L::out + tile_row + piece(i)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                fence_async_smem();
                arrive(bar_ofull);
            }
            g_cur = g_nxt;
            r_cur = r_nxt;
            gl_cur = gl_nxt;
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
            float* hrow = ht ? ht + (((long)b * H + h) * K + row) * V + cb : nullptr;
            uint32_t r[32];
            tmem_ld32(t_lane + WK_S, r);
            tmem_ld_wait();
            if (hrow) store_row(hrow, r, 1.f);
            if (last_lin) store_row(hs_row, r, 1.f);
            if (last_roll) {
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(hs_row[i]);
                store_row(hs_row, r, __expf(gcs[((long)b * T + T - 1) * H + h]));
            }
        }
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
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
    NATSL_REQUIRE(aligned_to(16, ht, hstart), NATSL_ERR_UNSUPPORTED, "natsl_gdn_walk_fused: ht and hstart must start on 16 bytes");
    NATSL_REQUIRE(!hstart || T % nbs != 0 || (last_types && (last_dtype == NATSL_DT_F32 || last_dtype == NATSL_DT_BF16)),
                  NATSL_ERR_NULL, "natsl_gdn_walk_fused: the block-start state of a complete last block needs that block's types");
    auto kern = gdn_walk_tc_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WkSmem::total);
    if (e != cudaSuccess) {
        set_error("natsl_gdn_walk_fused: cannot reserve %d B of shared memory (%s)", WkSmem::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mw, mq, mk, mu, mp, mo;
    int rc = encode_bthd_map(&mw, w, B, T, H, K, 64, "natsl_gdn_walk_fused(w)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mq, q, B, T, H, K, 64, "natsl_gdn_walk_fused(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, H, K, 64, "natsl_gdn_walk_fused(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mu, u, B, T, H, V, 64, "natsl_gdn_walk_fused(u)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mp, pmat, B, T, H, 64, 64, "natsl_gdn_walk_fused(P)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mo, o, B, T, H, V, 64, "natsl_gdn_walk_fused(o)");
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    const int TN = (T + nbs - 1) / nbs;
    dim3 grid(H, B);
    kern<<<grid, WK_THREADS, WkSmem::total, reinterpret_cast<cudaStream_t>(stream)>>>(
        mw, mq, mk, mu, mp, mo, gcs, k_rstd, q_rstd, types_i, indices, n_blocks, h0, ht, hstart, last_types,
        last_dtype == NATSL_DT_F32, last_stride, T, H, HN, TN, scale, (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0,
        (flags & NATSL_FLAG_NO_TRAILING_QUIRK) ? 0 : 1, status);
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
