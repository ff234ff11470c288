// Mamba2 / SSD recurrence AND chunk output in one walk on the 5th-generation tensor cores
// (state dim K = 128, head dim V = 64, any nats_block_size that is a multiple of 64).  One CTA per (batch, head)
// walks the 64-token chunks in order; the K x V state lives in TMEM (fp32) and is never written to global memory.
// Per chunk c (S = state the chunk reads, carry = decay of the skipped blocks before it, g = chunk-local cumsum):
//     DP = q k^T                      128-row A operand [k ; q]: rows 64-127 are the q rows             (MMA 0)
//     P  = tril(DP e^{g_i - g_j})     q warps, from TMEM into shared memory (bf16)
//     o  = scale (e^{g+carry} q S + P v)                                                         (MMA 1, MMA 2 + q warps)
//     S <- e^{g_last+carry} S + k^T (v e^{min(g_last-g, 0)})                                       (MMA 3)
// which is src/nats/ops/mamba/chunk_h.py:139-218 (recurrence) fused with src/nats/ops/mamba/chunk_o.py:137-198
// (output) and the carry of src/nats/ops/utils/cumsum.py:85-133.  Only chunks of selected blocks keep their update:
// with nats_block_size > 64 the chunks of an unselected block update the state as well (their outputs read it), and
// the state saved at the start of the block (a second TMEM region) comes back at its end -- the token recurrence of
// the reference's decode kernel, src/nats/ops/mamba/fused_recurrent.py:28-322.
// The decay of an update is applied when the state is copied to shared memory for the next chunk (one TMEM pass per
// update: bf16 copy out, multiply by the next update's decay, write back), so the accumulating MMA 3 needs no
// separate rescale.  The serial chain of a chunk is MMA 3 -> that pass; it has warps of its own:
//   warp 0      TMA producer (k, q, v tiles in three stages);
//   warp 1      issuer of MMA 3 (the chain); warp 16 issuer of the output products: per chunk MMA 1 (reads the bf16
//               copy the chunk started from; the copy is double-buffered with a full / empty barrier pair, so that the
//               chain runs ahead of the output by one copy) K-step by K-step in turn with MMA 0 of the next chunk, then
//               MMA 2 with P straight from TMEM.  Two issuing threads because one thread issues a 128 x 64 x 16 product only every
//               ~70 to 130 cycles;
//   warps 2-5   state warps, one per quarter of the TMEM lanes: wait for MMA 3, publish the state;
//   warps 8, 9, 12, 13   token warps (rows 0-63, half a row each): the scaled v tile of the next chunk;
//   warps 6, 7, 10, 11 and 14, 15, 18, 19   q warps (rows 64-127, 32 columns each), one set for the even chunks, one for the odd:
//               P of the chunk, then its output rows, which warp 17 stores by TMA.
// With o == NULL only the recurrence runs (final state only): ten warps, no copies of the state, half an SM.
//
// What bounded it: the load/store unit.  Every thread's own arrival on nine barriers (960 a chunk) and output rows stored 16 bytes per
// lane cost more than the chunk's products; the waits of all the other warps' shared loads and stores were the sum.  Now a warp
// arrives once, outputs leave as tiles, the scalars of a chunk are worked out by all threads at the start, and what a step needs is
// read in front of its wait.  Alone in a graph (us, outputs / state only), H = 32, 10 % of the blocks softmax: 64 sub-segments of 1024 tokens
// 563 / 303 -> 381 / 198; 32 of 2048 491 / 266 -> 334 / 170 (4.8 / 4.7 TB/s); 4 of 16384, what one sequence of 65536 is cut into, 486 / 255 ->
// 313 / 186 (5.1 / 4.3 TB/s); B = 8, T = 4096, H = 16 132 / 70 -> 86 / 54.
// Tried and not kept: four stages, the first loads in front of the tables, no L2 prefetch (all +- 3 %, three loads at once at the start
// 5 to 10 % slower).
// All mbarrier waits are bounded (status word + clean teardown on expiry); every barrier is waited for in every one
// of its phases by each of its waiters, and no phase can complete before every waiter has seen the one before it.
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {


constexpr int mw_threads(bool out) { return out ? 640 : 320; }       // 20 or 10 warps
constexpr uint32_t mw_tmem_cols(bool out) { return out ? 512 : 128; }
// TMEM column offsets: state, saved state, q S (double-buffered), P v, q k^T (double-buffered),
// and P (double-buffered, bf16 pairs)
constexpr uint32_t MW_S = 0, MW_BK = 64, MW_D1 = 128, MW_D1B = 192, MW_D2 = 256, MW_DP = 320, MW_DPB = 384, MW_P = 448;
constexpr int MW_MAX_NT = 1024;
constexpr int MW_ACTIVE = 1, MW_RESTORE = 2, MW_SAVE = 4, MW_SEL = 8;     // per-chunk flags

template <bool OUT> struct MwSmem {
    // stage: 2 tiles (one per half of the K dimension), then v [64][64] (8 KB).  With outputs a tile is [128][64], rows 0-63 the k
    // tile, rows 64-127 the q tile: the A operand of the q products (its first 64 result rows, k k^T and k S, are never read); its
    // first half alone is the k operand.  Without them it is the k tile [64][64].
    static constexpr int sub = OUT ? 16384 : 8192, v = 2 * sub, stage = v + 8192, nstage = 3;
    static constexpr int sbf = nstage * stage;            // 2 x S bf16 [128 k-rows][64 v-cols]              32 KB
    static constexpr int vs = sbf + (OUT ? 32768 : 0);    // 2 x scaled v [64 tok][64]                       16 KB
    static constexpr int out = vs + 16384;                // 2 x outputs on their way: [64 tok][64]          16 KB
    static constexpr int gs = out + (OUT ? 16384 : 0);    // per q warp: g of its 32 columns' tokens (float)
    static constexpr int meta = gs + (OUT ? 1024 : 0);    // per chunk: carry, the next update's decay, g_last (float), flags (int)
    static constexpr int bars = meta + 4 * 4 * MW_MAX_NT;
    static constexpr int total = bars + 256;
    static_assert(total <= (OUT ? 232448 : 115712), "shared memory of one SM, of half an SM");
};

// WIDE: the initial state starts on 16 bytes.  A caller's that does not is read word by word, which costs 3.6 us of 13 to 90, in an
// instance of its own (a branch in this one costs 0.3 us in every call).
template <bool OUT, bool WIDE>
__global__ void __launch_bounds__(mw_threads(OUT), OUT ? 1 : 2)
mamba_walk_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                     const float* __restrict__ gcs, const int* __restrict__ types_i, const int* __restrict__ indices,
                     const int* __restrict__ n_blocks, const float* __restrict__ h0, float* __restrict__ ht, float* hstart,
                     const void* __restrict__ last_types, int last_f32, int last_stride, int T, int H, int HN, int TN, int nbs, float scale,
                     int decay, int trailing_quirk, int* status) {
    using L = MwSmem<OUT>;
    constexpr int MW_THREADS = mw_threads(OUT);
    constexpr int K = 128, V = 64;
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
    const int cpb = nbs / 64;
    float* m_carry = reinterpret_cast<float*>(smem + L::meta);
    float* m_mul = m_carry + MW_MAX_NT;
    float* m_gl = m_mul + MW_MAX_NT;
    int* m_fl = reinterpret_cast<int*>(m_gl + MW_MAX_NT);
    const uint32_t bar0 = sbase + L::bars;
    // barriers: full / empty of the tile stages; dp (MMA 0 done); pfull (P written by the q warps); pv (scaled v of a
    // chunk written by the token warps); d2[2] (MMA 2, and with it MMA 1, of an even / odd chunk done); s3 (MMA 3 done); sready
    // (state published); odone (output rows read from TMEM)
    // cfull[2] / cempty[2]: the two bf16 copies of the state (written by the state warps, read by MMA 1)
    // dp[2], pfull[2]: one per q k^T buffer / P tile.  A tile stage is released by the warps that see its last readers complete (the
    // state warps MMA 3, the q warps MMA 2) and so is a state copy (the q warps): a tcgen05.commit costs the issuing
    // thread about as much as two products.
    // ofull[2], ofree[2]: the output rows of a chunk are in shared memory / on their way to global memory.
    // One arrival per warp: arrivals are work of the load/store unit, one lane after another.
    const uint32_t bar_full = bar0, bar_empty = bar0 + 24, bar_dp = bar0 + 48, bar_pfull = bar0 + 64, bar_pv = bar0 + 80,
                   bar_s3 = bar0 + 96, bar_sready = bar0 + 104, bar_odone = bar0 + 112,
                   bar_cfull = bar0 + 120, bar_cempty = bar0 + 136, bar_ofull = bar0 + 152, bar_ofree = bar0 + 168, bar_d2 = bar0 + 184;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 208);
    int* hs_slot = reinterpret_cast<int*>(smem + L::bars + 212);
    auto arrive = [&](uint32_t bar) {                     // behind what the whole warp has done so far
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };

    if (tid == 0) {
        for (int i = 0; i < L::nstage; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, OUT ? 8 : 4);           // state warps (+ q warps)
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_cfull + 8 * i, 4);
            mbar_init(bar_cempty + 8 * i, 4);
            mbar_init(bar_dp + 8 * i, 1);
            mbar_init(bar_pfull + 8 * i, 4);
            mbar_init(bar_ofull + 8 * i, 4);
            mbar_init(bar_ofree + 8 * i, 1);
            mbar_init(bar_d2 + 8 * i, 1);
        }
        mbar_init(bar_pv, 4);
        mbar_init(bar_s3, 1);
        mbar_init(bar_sready, 4);
        mbar_init(bar_odone, 4);
        mbar_fence_init();
        *hs_slot = -1;
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), mw_tmem_cols(OUT));
    // ---- per-chunk metadata
    for (int c = tid; c < NT; c += MW_THREADS) {
        m_fl[c] = types_i[(((long)b * TN + c / cpb) * HN + hn) * 2 + 1] != 0 ? MW_SEL : 0;
        m_gl[c] = gcs[((long)b * T + min(c * 64 + 63, T - 1)) * H + h];
    }
    const int c_last = (TN - 1) * cpb;                    // first chunk of the last block
    {
        const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
        const int last_sel = nsel > 0 ? indices[(((long)b * TN + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
        __syncthreads();
        // decay of the skipped blocks in front of block `blk`: every chunk adds up its own run of them, first to last, as one
        // thread would do for all
        auto skipped = [&](int blk) -> float {
            float carry = 0.f;
            if (!decay) return carry;
            int j = blk;
            while (j > 0 && !(m_fl[(j - 1) * cpb] & MW_SEL)) --j;
            for (; j < blk; ++j) {
                if (trailing_quirk && j >= last_sel) continue;
                float g = 0.f;
                for (int i = j * cpb; i < (j + 1) * cpb; ++i) g += m_gl[i];
                carry += g;
            }
            return carry;
        };
        for (int c = tid; c < NT; c += MW_THREADS) {
            // with blocks of several chunks every chunk updates the state: only a block's first one has skipped ones in front
            m_carry[c] = c % cpb == 0 ? skipped(c / cpb) : 0.f;
        }
        __syncthreads();
        for (int c = tid; c < NT; c += MW_THREADS) {
            const bool sel = (m_fl[c] & MW_SEL) != 0;
            int j = c + 1;
            if (cpb == 1)
                while (j < NT && !(m_fl[j] & MW_SEL)) ++j;
            m_mul[c] = j < NT ? __expf(m_gl[j] + m_carry[j]) : 1.f;
            // the last update in front of the last block
            if ((cpb > 1 || sel) && c < c_last && j >= c_last) *hs_slot = c;
        }
        __syncthreads();
        for (int c = tid; c < NT; c += MW_THREADS) {
            const bool sel = (m_fl[c] & MW_SEL) != 0;
            const int sub = c % cpb;
            int fl = sel ? MW_SEL : 0;
            if (cpb > 1 || sel) fl |= MW_ACTIVE;
            if (cpb > 1 && !sel && sub == 0) fl |= MW_SAVE;
            if (cpb > 1 && !sel && (sub == cpb - 1 || c == NT - 1)) fl |= MW_RESTORE;
            m_fl[c] = fl;
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    // chunk-local cumsum of token `tok` of chunk c (clamped to the last valid token of a ragged chunk)
    auto load_g = [&](int c, int tok) -> float {
        const int valid = min(64, T - c * 64);
        return gcs[((long)b * T + (long)c * 64 + min(tok, valid - 1)) * H + h];
    };

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            prefetch_tensormap(&map_q);
            prefetch_tensormap(&map_k);
            prefetch_tensormap(&map_v);
        }
        int n_loads = 0;                                  // chunks asked for
#pragma unroll 1
        for (int c = 0; c < NT; ++c) {
            const int stg = c % L::nstage;
            const int t0 = c * 64;
            if (c >= L::nstage) {
                ok = warp_wait(bar_empty + stg * 8, ((c / L::nstage) - 1) & 1);
                if (!ok) break;
            }
            if (lane == 0) {
                const uint32_t full = bar_full + stg * 8, base = sbase + stg * L::stage;
                mbar_expect_tx(full, (OUT ? 16384 : 0) + 16384 + 8192);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    tma_load_4d(base + sub * L::sub, &map_k, sub * 64, h, t0, b, full);                       // rows 0-63
                    if (OUT) tma_load_4d(base + sub * L::sub + 8192, &map_q, sub * 64, h, t0, b, full);   // rows 64-127
                }
                tma_load_4d(base + L::v, &map_v, 0, h, t0, b, full);
                if (c + L::nstage < NT) {                           // warm L2 for the tiles this stage receives next
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub) {
                        if (OUT) tma_prefetch_4d(&map_q, sub * 64, h, t0 + 64 * L::nstage, b);
                        tma_prefetch_4d(&map_k, sub * 64, h, t0 + 64 * L::nstage, b);
                    }
                    tma_prefetch_4d(&map_v, 0, h, t0 + 64 * L::nstage, b);
                }
            }
            __syncwarp();
            ++n_loads;
        }
        if (!ok)                                          // nothing may still be on its way into shared memory
            for (int c = max(0, n_loads - L::nstage); c < n_loads; ++c) warp_wait(bar_full + (c % L::nstage) * 8, (c / L::nstage) & 1);
    } else if (warp == 1) {
        // ------------------------------------------------------------ issuer of the state update (the serial chain)
        constexpr uint32_t id_3 = umma_idesc_bf16(128, 64, true) | (1u << 15);          // k^T v~ (A MN-major)
#pragma unroll 1
        for (int c = 0; ok && c < NT; ++c) {
            const int stg = c % L::nstage;
            const uint32_t base = sbase + stg * L::stage;
            const int fl = m_fl[c];
            ok = warp_wait(bar_full + stg * 8, (c / L::nstage) & 1);
            if (ok) ok = warp_wait(bar_sready, c & 1);
            if (ok) ok = warp_wait(bar_pv, c & 1);
            if (!ok) break;
            {
                // the update of the last chunk of an unselected block would be thrown away: it is not issued
                tc_fence_after();
                if ((fl & MW_ACTIVE) && !(fl & MW_RESTORE)) {
                    umma_ss_x4<128, 128>(tmem + MW_S, umma_desc_lo(base, L::sub),
                                         umma_desc_lo(sbase + L::vs + (c & 1) * 8192, 8192), id_3, 1u);
                }
                umma_commit(bar_s3);
            }
            __syncwarp();
        }
    } else if (OUT && warp == 16) {
        // ------------------------------------------------------------ issuer of the output products
        {
            constexpr uint32_t id_0 = umma_idesc_bf16(128, 64, false);                  // [0;q] k^T
            constexpr uint32_t id_1 = umma_idesc_bf16(128, 64, true);                   // [0;q] S
            constexpr uint32_t id_2 = umma_idesc_bf16(128, 64, true);                   // P v
            ok = warp_wait(bar_full, 0);
            if (ok) {                     // q k^T of chunk 0
                tc_fence_after();
                const uint32_t al = umma_desc_lo(sbase, 16);          // the k operand is the first half of the same tile
#pragma unroll
                for (int h = 0; h < 2; ++h) umma_ss_x4<2, 2>(tmem + MW_DP, al + h * 1024, al + h * 1024, id_0, h > 0);
                umma_commit(bar_dp);
            }
            __syncwarp();
            int ncopy = 0;                             // copy of the state that the current chunk reads: ncopy & 1
            bool fresh = true;                         // ... and it has not been waited for yet
#pragma unroll 1
            for (int c = 0; ok && c < NT; ++c) {
                const int stg = c % L::nstage, nstg = (c + 1) % L::nstage;
                const uint32_t base = sbase + stg * L::stage;
                const int fl = m_fl[c];
                const int cp = ncopy & 1;
                if (fresh) ok = warp_wait(bar_cfull + cp * 8, (ncopy >> 1) & 1);
                fresh = false;
                // q k^T of the next chunk goes to the other buffer: its last reader was P of chunk c - 1, waited for
                // before MMA 2 of that chunk
                const bool ahead = c + 1 < NT;
                if (ok && ahead) ok = warp_wait(bar_full + nstg * 8, ((c + 1) / L::nstage) & 1);
                if (ok) {
                    // q S of this chunk and q k^T of the next one, half by half in turn
                    tc_fence_after();
                    const uint32_t d1 = tmem + ((c & 1) ? MW_D1B : MW_D1);
                    const uint32_t nbase = sbase + nstg * L::stage;
                    const uint32_t al = umma_desc_lo(base, 16), bl = umma_desc_lo(sbase + L::sbf + cp * 16384, 16384),
                                   nl = umma_desc_lo(nbase, 16);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        umma_ss_x4<2, 128>(d1, al + h * 1024, bl + h * 512, id_1, h > 0);
                        if (ahead) umma_ss_x4<2, 2>(tmem + (((c + 1) & 1) ? MW_DPB : MW_DP), nl + h * 1024, nl + h * 1024, id_0, h > 0);
                    }
                    if (ahead) umma_commit(bar_dp + ((c + 1) & 1) * 8);
                }
                __syncwarp();
                if (fl & MW_ACTIVE) {
                    ++ncopy;
                    fresh = true;
                }
                if (ok) ok = warp_wait(bar_pfull + (c & 1) * 8, (c >> 1) & 1);   // P of this chunk
                if (ok && c > 0) ok = warp_wait(bar_odone, (c - 1) & 1);   // D2 is free
                if (!ok) break;
                {
                    tc_fence_after();
                    umma_ts_x4<128>(tmem + MW_D2, tmem + MW_P + (c & 1) * 32, umma_desc_lo(base + L::v, 8192), id_2, 0u);
                    umma_commit(bar_d2 + (c & 1) * 8);
                }
                __syncwarp();
            }
        }
    } else if (warp < 6) {
        // ------------------------------------------------------------ state warps: one thread per TMEM lane (= S row)
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16);
        int pubs = 0;                                  // copies published so far; the next one goes to copy pubs & 1
        const int hs_at = *hs_slot;
        // With hs a published value is also what the last block starts from: it goes to hstart with that block's carried decay.
        float* hs_row = hstart ? hstart + (((long)b * H + h) * K + row) * V : nullptr;
        auto store_row = [&](float* dst, int c0, const uint32_t (&r)[32], float f) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(dst + c0 + i) = make_float4(__uint_as_float(r[i]) * f, __uint_as_float(r[i + 1]) * f,
                                                                      __uint_as_float(r[i + 2]) * f, __uint_as_float(r[i + 3]) * f);
        };
        // Publishes this thread's state row (r0, r1: its two halves): bf16 copy into shared memory, announced at once, optionally a
        // raw copy into the saved-state region, and `value * mul` as the state in TMEM.
        auto publish_state = [&](uint32_t (&r0)[32], uint32_t (&r1)[32], float mul, bool write, bool save, bool hs) {
            if (OUT) {
                unsigned char* dst = smem + L::sbf + (pubs & 1) * 16384 + row * 128;
#pragma unroll
                for (int cc = 0; cc < 8; ++cc) {
                    const uint32_t* r = cc < 4 ? r0 + cc * 8 : r1 + (cc - 4) * 8;
                    uint32_t w4[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) w4[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                    *reinterpret_cast<uint4*>(dst + ((cc ^ (row & 7)) << 4)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                fence_async_smem();
                arrive(bar_cfull + (pubs & 1) * 8);
            }
            ++pubs;
            if (save) {
                tmem_st32(t_lane + MW_BK, r0);
                tmem_st32(t_lane + MW_BK + 32, r1);
            }
            if (hs_row && hs) {
                const float f = __expf(m_carry[c_last]);
                store_row(hs_row, 0, r0, f);
                store_row(hs_row, 32, r1, f);
            }
            if (mul != 1.f || write) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    r0[i] = __float_as_uint(__uint_as_float(r0[i]) * mul);
                    r1[i] = __float_as_uint(__uint_as_float(r1[i]) * mul);
                }
                tmem_st32(t_lane + MW_S, r0);
                tmem_st32(t_lane + MW_S + 32, r1);
            }
            tmem_st_wait();
            tc_fence_before();
            arrive(bar_sready);
        };
        {   // initial state
            const float* init = h0 ? h0 + (((long)b * H + h) * K + row) * V : nullptr;
            uint32_t r0[32], r1[32];
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                auto load = [&](const float* p) { return WIDE ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]); };
                const float4 x = init ? load(init + i) : z, y = init ? load(init + 32 + i) : z;
                r0[i] = __float_as_uint(x.x), r0[i + 1] = __float_as_uint(x.y), r0[i + 2] = __float_as_uint(x.z), r0[i + 3] = __float_as_uint(x.w);
                r1[i] = __float_as_uint(y.x), r1[i + 1] = __float_as_uint(y.y), r1[i + 2] = __float_as_uint(y.z), r1[i + 3] = __float_as_uint(y.w);
            }
            float mul = 1.f;
            if (init) {                                   // decay of the first update
                int j = 0;
                while (j < NT && !(m_fl[j] & MW_ACTIVE)) ++j;
                if (j < NT) mul = __expf(m_gl[j] + m_carry[j]);
            }
            publish_state(r0, r1, mul, true, (m_fl[0] & MW_SAVE) != 0, hs_at < 0);
        }
#pragma unroll 1
        for (int c = 0; ok && c < NT; ++c) {
            const int fl = m_fl[c];
            const float mul = m_mul[c];
            const bool restore = (fl & MW_RESTORE) != 0, save = !restore && c + 1 < NT && (m_fl[c + 1] & MW_SAVE) != 0;
            // copy pubs & 1: MMA 1 of the chunks that read its previous content must be complete
            if (OUT && (fl & MW_ACTIVE) && pubs >= 2) ok = warp_wait(bar_cempty + (pubs & 1) * 8, ((pubs >> 1) - 1) & 1);
            // once the update of this chunk is complete, publish the state for the next chunk (and pre-apply the next
            // update's decay); after a failed (bounded) wait the remaining work is skipped
            if (ok) ok = warp_wait(bar_s3, c & 1);
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) mbar_arrive(bar_empty + (c % L::nstage) * 8);       // MMA 3 is done with the k tile
            if (fl & MW_ACTIVE) {
                uint32_t r0[32], r1[32];
                tmem_ld32(t_lane + (restore ? MW_BK : MW_S), r0);
                tmem_ld32(t_lane + (restore ? MW_BK : MW_S) + 32, r1);
                tmem_ld_wait();
                publish_state(r0, r1, mul, restore, save, c == hs_at);
            } else {
                tc_fence_before();
                arrive(bar_sready);
            }
        }
        // every update's decay was pre-applied except after the last one: TMEM holds the final state.  A complete last
        // block: the decoder continues from it if that block's own type is linear, else from the state in front of the
        // block, decayed over it.
        bool last_lin = false, last_roll = false;
        if (hs_row && T % nbs == 0) {
            const long li = (long)b * last_stride + hn * 2 + 1;
            last_lin = (last_f32 ? reinterpret_cast<const float*>(last_types)[li]
                                 : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(last_types)[li])) > 0.f;
            last_roll = !last_lin && decay;
        }
        if (ok && (ht || last_lin || last_roll)) {
            tc_fence_after();
            float* hrow = ht ? ht + (((long)b * H + h) * K + row) * V : nullptr;
            float blk_g = 0.f;
            for (int c = c_last; c < NT; ++c) blk_g += m_gl[c];
            const float f = __expf(blk_g);
#pragma unroll 1
            for (int c0 = 0; c0 < 64; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(t_lane + MW_S + c0, r);
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
    } else if (OUT ? warp == 8 || warp == 9 || warp == 12 || warp == 13 : true) {
        // ------------------------------------------------------------ token warps: v~ = v e^{min(g_last - g, 0)}
        const int tr = (warp & 1) * 32 + lane, half = warp >= (OUT ? 12 : 8);         // token row inside the chunk, half of its columns
        auto stage_v = [&](int c, float gg) {             // chunk c into buffer c & 1 (the arrival follows separately)
            const int stg = c % L::nstage;
            ok = warp_wait(bar_full + stg * 8, (c / L::nstage) & 1);
            if (!ok) return;
            const float f2 = __expf(fminf(m_gl[c] - gg, 0.f));
            const unsigned char* vt = smem + stg * L::stage + L::v;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const uint32_t off = swz<128>(tr, half * 4 + cc);
                const uint4 vx = *reinterpret_cast<const uint4*>(vt + off);
                const uint32_t* vw = reinterpret_cast<const uint32_t*>(&vx);
                uint32_t b4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 vf = unpack_bf16(vw[i]);
                    b4[i] = pack_bf16(vf.x * f2, vf.y * f2);
                }
                *reinterpret_cast<uint4*>(smem + L::vs + (c & 1) * 8192 + off) = make_uint4(b4[0], b4[1], b4[2], b4[3]);
            }
            fence_async_smem();
        };
        float g_n1 = load_g(0, tr), g_n2 = NT > 1 ? load_g(1, tr) : 0.f;
        stage_v(0, g_n1);
        if (ok) arrive(bar_pv);
#pragma unroll 1
        for (int c = 0; ok && c < NT; ++c) {
            g_n1 = g_n2;                                                  // g of chunk c + 1
            if (c + 2 < NT) g_n2 = load_g(c + 2, tr);                     // consumed in the next iteration
            // The tile of the NEXT chunk, off the serial chain.  Its arrival waits until the update of this chunk is
            // complete: the MMA warp has then consumed this chunk's phase of the barrier.
            if (ok && c + 1 < NT) stage_v(c + 1, g_n1);
            if (ok) ok = warp_wait(bar_s3, c & 1);
            if (ok && c + 1 < NT) arrive(bar_pv);
        }
    } else if (warp == 17) {
        // ------------------------------------------------------------ stores of the outputs
#pragma unroll 1
        for (int c = 0; ok && c < NT; ++c) {
            ok = warp_wait(bar_ofull + (c & 1) * 8, (c >> 1) & 1);
            if (ok && lane == 0) {
                tma_store_4d(&map_o, sbase + L::out + (c & 1) * 8192, 0, h, c * 64, b);
                tma_store_commit();
                tma_store_wait_read();
                mbar_arrive(bar_ofree + (c & 1) * 8);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------ q warps: rows 64-127, 32 columns each
        const int quad = warp & 3;                        // 2 or 3
        const int cb = (warp & 4) ? 0 : 32, set = warp >= 14;             // warps 6, 7, 14, 15: the first columns
        const int row = quad * 32 + lane, tr = row - 64;
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + cb;
        float* sg = reinterpret_cast<float*>(smem + L::gs) + (set * 4 + (cb >> 4) + (quad & 1)) * 32;
        auto piece = [&](int i) -> uint32_t { return tr * 128 + ((((cb >> 3) + i) ^ (tr & 7)) << 4); };
        // P = tril(q k^T e^{g_i - g_j}) of chunk c as the bf16 A operand of P v, from TMEM to TMEM; gg: g of the row's token, gk: of
        // key cb + lane, which the warp hands around through shared memory.
        auto build_p = [&](int c, float gg, float gk) {
            __syncwarp();
            sg[lane] = gk;
            __syncwarp();
            ok = warp_wait(bar_dp + (c & 1) * 8, (c >> 1) & 1);
            if (!ok) return;
            tc_fence_after();
            uint32_t w[16];
            if (quad == 2 && cb == 32) {                  // rows 0-31, keys 32-63
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = 0;
            } else {
                uint32_t r[32];
                tmem_ld32(t_lane + ((c & 1) ? MW_DPB : MW_DP), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 gj = *reinterpret_cast<const float4*>(sg + 4 * i);
                    const float gs[4] = {gj.x, gj.y, gj.z, gj.w};
                    float p[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // no branches: the exponent is clamped (it is <= 0 wherever the mask keeps the product)
                        p[e] = __uint_as_float(r[4 * i + e]) * __expf(fminf(gg - gs[e], 0.f));
                        p[e] *= cb + 4 * i + e <= tr ? 1.f : 0.f;
                    }
                    w[2 * i] = pack_bf16(p[0], p[1]);
                    w[2 * i + 1] = pack_bf16(p[2], p[3]);
                }
            }
            tmem_st16(t_lane - cb + MW_P + (c & 1) * 32 + (cb >> 1), w);
            tmem_st_wait();
            tc_fence_before();
            arrive(bar_pfull + (c & 1) * 8);
        };
        // one set of warps takes the even chunks, one the odd ones
        float g_cur = set < NT ? load_g(set, tr) : 0.f, k_cur = set < NT ? load_g(set, cb + lane) : 0.f, g_n = 0.f, k_n = 0.f;
        int ncopy = set == 1 && (m_fl[0] & MW_ACTIVE) ? 1 : 0;            // copy of the state that the chunk reads: ncopy & 1
#pragma unroll 1
        for (int c = set; ok && c < NT; c += 2) {
            if (c + 2 < NT) {                                             // consumed in the next iteration
                g_n = load_g(c + 2, tr);
                k_n = load_g(c + 2, cb + lane);
            }
            build_p(c, g_cur, k_cur);
            const float fq = __expf(g_cur + m_carry[c]);
            const bool active = (m_fl[c] & MW_ACTIVE) != 0;
            // o = scale (e^{g+carry} q S + P v): MMA 2 complete means MMA 1 of the chunk is complete as well
            if (ok) ok = warp_wait(bar_d2 + (c & 1) * 8, (c >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t r1[32], r2[32];
            tmem_ld32(t_lane + ((c & 1) ? MW_D1B : MW_D1), r1);
            tmem_ld32(t_lane + MW_D2, r2);
            if (lane == 0) {
                // every product that read the tile stage of this chunk, or (if an update follows) this copy of the
                // state, is complete
                mbar_arrive(bar_empty + (c % L::nstage) * 8);
                if (active) mbar_arrive(bar_cempty + (ncopy & 1) * 8);
            }
            tmem_ld_wait();
            tc_fence_before();
            arrive(bar_odone);
            if (c >= 2) ok = warp_wait(bar_ofree + (c & 1) * 8, ((c >> 1) - 1) & 1);
            if (!ok) break;
            unsigned char* dst = smem + L::out + (c & 1) * 8192;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                uint32_t w4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int e = cc * 8 + 2 * i;
                    w4[i] = pack_bf16(scale * (fq * __uint_as_float(r1[e]) + __uint_as_float(r2[e])),
                                      scale * (fq * __uint_as_float(r1[e + 1]) + __uint_as_float(r2[e + 1])));
                }
                *reinterpret_cast<uint4*>(dst + piece(cc)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            fence_async_smem();
            arrive(bar_ofull + (c & 1) * 8);
            if (active) ++ncopy;
            if (c + 1 < NT && (m_fl[c + 1] & MW_ACTIVE)) ++ncopy;
            g_cur = g_n;
            k_cur = k_n;
        }
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, mw_tmem_cols(OUT));
}

}  // namespace natsl


extern "C" int natsl_mamba_walk_fused_ex(const void* q, const void* k, const void* v, const float* gcs,
                                      const int32_t* types_i, const int32_t* indices, const int32_t* n_blocks,
                                      const float* h0, void* o, float* ht, float* hstart, const void* last_types,
                                      int last_dtype, int last_stride, int B, int T, int H, int HN, int K, int V, int nbs, float scale, int flags,
                                      void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(k && v && gcs && types_i && indices && n_blocks, NATSL_ERR_NULL, "natsl_mamba_walk_fused: null pointer");
    NATSL_REQUIRE((o && q) || (!o && ht), NATSL_ERR_NULL,
                  "natsl_mamba_walk_fused: o needs q; without o the final state ht must be asked for");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0, NATSL_ERR_BAD_SHAPE, "natsl_mamba_walk_fused: bad shape");
    NATSL_REQUIRE(K == 128 && V == 64 && nbs >= 64 && nbs % 64 == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_mamba_walk_fused: built for K = 128, V = 64 and nats_block_size a multiple of 64 (got K=%d V=%d "
                  "nbs=%d); use natsl_linear_fwd_h + natsl_linear_fwd_o", K, V, nbs);
    NATSL_REQUIRE((T + 63) / 64 <= MW_MAX_NT, NATSL_ERR_TOO_LARGE, "natsl_mamba_walk_fused: T <= 65536");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_mamba_walk_fused: B, H <= 65535");
    NATSL_REQUIRE(aligned_to(16, ht, hstart), NATSL_ERR_UNSUPPORTED, "natsl_mamba_walk_fused: ht and hstart must start on 16 bytes");
    NATSL_REQUIRE(!hstart || T % nbs != 0 || (last_types && (last_dtype == NATSL_DT_F32 || last_dtype == NATSL_DT_BF16)),
                  NATSL_ERR_NULL, "natsl_mamba_walk_fused: the block-start state of a complete last block needs that block's types");
    const bool wide = aligned_to(16, h0);
    auto kern = o ? (wide ? mamba_walk_tc_kernel<true, true> : mamba_walk_tc_kernel<true, false>)
                  : (wide ? mamba_walk_tc_kernel<false, true> : mamba_walk_tc_kernel<false, false>);
    const int bytes = o ? MwSmem<true>::total : MwSmem<false>::total;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) {
        set_error("natsl_mamba_walk_fused: cannot reserve %d B of shared memory (%s)", bytes, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mo;
    int rc = encode_bthd_map(&mk, k, B, T, H, K, 64, "natsl_mamba_walk_fused(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T, H, V, 64, "natsl_mamba_walk_fused(v)");
    if (rc == NATSL_OK && o) rc = encode_bthd_map(&mq, q, B, T, H, K, 64, "natsl_mamba_walk_fused(q)");
    if (rc == NATSL_OK && o) rc = encode_bthd_map(&mo, o, B, T, H, V, 64, "natsl_mamba_walk_fused(o)");
    if (!o) {
        mq = mk;
        mo = mv;
    }
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    const int TN = (T + nbs - 1) / nbs;
    dim3 grid(H, B);
    kern<<<grid, mw_threads(o != nullptr), bytes, reinterpret_cast<cudaStream_t>(stream)>>>(
        mq, mk, mv, mo, gcs, types_i, indices, n_blocks, h0, ht, hstart, last_types,
        last_dtype == NATSL_DT_F32, last_stride, T, H, HN, TN, nbs, scale,
        (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0, (flags & NATSL_FLAG_NO_TRAILING_QUIRK) ? 0 : 1, status);
    return check_launch("natsl_mamba_walk_fused");
}

extern "C" int natsl_mamba_walk_fused(const void* q, const void* k, const void* v, const float* gcs,
                                      const int32_t* types_i, const int32_t* indices, const int32_t* n_blocks,
                                      const float* h0, void* o, float* ht, int B, int T, int H, int HN, int K, int V,
                                      int nbs, float scale, int flags, void* stream) {
    return natsl_mamba_walk_fused_ex(q, k, v, gcs, types_i, indices, n_blocks, h0, o, ht, nullptr, nullptr, 0, 0, B, T, H, HN, K, V,
                                     nbs, scale, flags, stream);
}
