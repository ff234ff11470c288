// Backward of the chunk-masked softmax branch (src/nats/ops/attns/attns.py:1562-1759; preprocess :357-372,
// dq :383-708, dk/dv :719-982).  Key s is visible to query t when its block is softmax-selected and lies
// entirely before t, or when both are in the same block and s <= t (the forward's mask).  With
//     p = exp2(scale*log2(e) * q.k - lse),   delta = rowsum(o * do),   ds = p * (do.v - delta)
// the gradients are dq = scale * ds k, dk = scale * ds^T q, dv = p^T do.
//
// Two kernels on the 5th-generation tensor cores, both deterministic (no atomics; every reduction has a fixed order).
//   attn_bwd_dq_kernel    128 queries of a head against pairs of the 64-key tiles that they see, queries in the TMEM lanes: q k^T
//                         and do v^T (128 x 128), ds back into TMEM (over do.v) as the A operand of dq += ds k, dq stays in TMEM.
//                         It also writes delta (the preprocess kernel of the reference folded in).
//   attn_bwd_dkdv_kernel  pairs of 64-key tiles (two of selected blocks, or what is unselected of two neighbours) against the
//                         128-query tiles that see either, keys in the TMEM lanes: k q^T and v do^T (128 x 128), p and ds back
//                         into TMEM as the A operands of dv += p do and dk += ds q.  It also sums ds over the later blocks'
//                         queries: the reference's `dnats` column for the softmax branch (attns.py:922, 975-978), per (64-key
//                         tile, query head).
// `compat` reproduces the reference's default backward, which drops every own-block entry of ds and p
// (attns.py:590-591, 631-633, 842, 884 with the flag passed at mixed_attn_gdn.py:237) while lse and delta still
// come from the full forward.
// Every mbarrier wait has an iteration limit; on expiry the CTA records a status, stops issuing work, still frees its
// TMEM and returns.
#include <type_traits>

#include "attn_tc.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr float kLog2e = 1.4426950408889634f;

// ------------------------------------------------------------------------------------------------- dq
// 128 queries against pairs of visible key tiles: all three products are 128 x 128 (x head dim), whose operands are read half as often
// as by 128 x 64 ones, and p never leaves the registers.  One persistent CTA per SM takes blocks of the grid over (cluster launch
// control).  Roles: warp 0 loads, warp 1 issues the products, warp 2 plans the steps, warps 4-11 p and ds (a query and 64 keys per
// thread; half the warps per key tile).  o and do of the next block's rows, whose product is delta, are on their way to registers while
// dq of the block before leaves.
// Registers: 384 threads get 168 each, of which the first four warps give back what the others need to hold 64 scores and 64 values of
// do.v, or a block's o and do.  Nothing may spill: the shared memory leaves so little of the first-level cache that a spilled word
// comes back from L2, some 400 cycles in a chain in which nothing else hides them.
// What bounds it: the chain scores -> p -> ds -> dq product of a step, 2.7 k cycles (1.45 k of them p, whose exponentials alone take the
// special function units 1.0 k) against 1.5 k of the tensor core, and 4.4 k cycles between two blocks (delta, dq on its way out).
// Alone (us; before: 128 x 64 score tiles, two CTAs per SM, one block each), block 64:
//   128/128, B = 8, T = 4096, H = 16: 25 % selected 323 -> 265, 50 % 508 -> 410, 2 % 175 -> 141;  64/64, 30 %: 286 -> 239
//   128/64, B = 4, T = 1000, H = 16, 50 %: 38 -> 30;  128/128, B = 1, T = 2048, H = 16, 30 %: 25.6 -> 23.5
//   64/128, B = 2, T = 2048, 12 heads over 6, block 128, 40 %: 36 -> 30;  the smallest, 64/64, B = 2, T = 64, H = 4: 5.3 -> 5.6
// Of that the rows asked into L2 ahead are 8 us at 25 % and 9 us at 2 %.  Eight threads per row for delta, in whole lines: 275 us.
constexpr int BDQ_THREADS = 384;                              // TMA, MMA, planner, (no work), 8 softmax warps
constexpr int BDQ_STEPS = 2;                                  // steps that the planner is ahead
constexpr int BWD_REGS_LOW = 88, BWD_REGS_HIGH = 208;         // a thread: 128 x 88 + 256 x 208 = 384 x 168
// Heads whose blocks are interleaved, heaviest first: the last blocks to start are then light ones, and k and v of that many heads
// (2 MB each at 4096 x 128) stay in L2.
constexpr int BDQ_HEADS = 32;

template <int DK, int DV>
struct DqSmem {
    static constexpr int q = 0;                               // DK/64 sub-tiles [128][64]
    static constexpr int dos = q + 128 * DK * 2;              // DV/64 sub-tiles
    static constexpr int k = dos + 128 * DV * 2;              // 2 stages x DK/64 sub-tiles [128 keys][64]
    static constexpr int v = k + 2 * 128 * DK * 2;            // 2 stages x DV/64 sub-tiles
    static constexpr int out = v + 2 * 128 * DV * 2;          // per softmax warp: 32 rows x 64 columns on their way out
    static constexpr int delta = out + 8 * 4096;              // delta of the rows, of an even / odd block
    static constexpr int desc = delta + 2 * 512;              // steps, 32 bytes each
    static constexpr int clc = desc + BDQ_STEPS * 32;         // answer of the take-over request
    static constexpr int bars = clc + 16;
    static constexpr int total = bars + 240;
    static_assert(total <= 227 * 1024, "one CTA per SM");
};

// What a CTA does in a step: first key tile, flags, second key tile (-1: none); first query, query head, batch.
enum : int {
    BDQ_FIRST = 1, BDQ_LAST = 2,                              // first / last step of the block
    BDQ_STOP = 4,                                             // no block is left
    BDQ_OWN0 = 8, BDQ_OWN1 = 16,                              // the key tile is of the own span: masked per element
    BDQ_SEL0 = 32, BDQ_SEL1 = 64                              // its block is selected
};

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <int DK, int DV>
__global__ void __launch_bounds__(BDQ_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_dq, const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ o,
                   const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse, const int* __restrict__ types_i,
                   float* __restrict__ delta_out, int T, int HQ, int HKV, int HN, int TN, int nbs, float scale, int own, int heads, int* status) {
    using L = DqSmem<DK, DV>;
    constexpr uint32_t C_S = 0, C_DP = 128, C_DQ = 256;       // TMEM: scores; do.v, then ds over each half's first columns; dq
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int NT = (T + 63) / 64, NTq = (T + ATT_BM - 1) / ATT_BM, cpb = nbs / 64;
    float* s_delta = reinterpret_cast<float*>(smem + L::delta);
    int4* s_desc = reinterpret_cast<int4*>(smem + L::desc);
    const uint32_t bar0 = sbase + L::bars;
    // barriers: desc_full / desc_empty (steps); q_full / q_empty, do_full / do_empty (the block's); k_full / k_empty, v_full / v_empty
    // (stages); s, dp (scores, do.v complete); s_free (scores read); ds (written); acc (dq complete); acc_free (read); delta (of all rows)
    const uint32_t desc_full = bar0, desc_empty = bar0 + 16, k_full = bar0 + 32, k_empty = bar0 + 48, v_full = bar0 + 64,
                   v_empty = bar0 + 80, q_full = bar0 + 96, q_empty = bar0 + 104, do_full = bar0 + 112, do_empty = bar0 + 120,
                   bar_s = bar0 + 128, bar_s_free = bar0 + 136, bar_dp = bar0 + 144, bar_ds = bar0 + 152, bar_acc = bar0 + 160,
                   bar_acc_free = bar0 + 168, bar_delta = bar0 + 176, bar_clc = bar0 + 184;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 192);
    auto arrive = [&](uint32_t bar) {                         // behind what the whole warp has done so far
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(desc_full + 8 * i, 1);
            mbar_init(desc_empty + 8 * i, 10);                // eight softmax warps, TMA, MMA
            mbar_init(k_full + 8 * i, 1);
            mbar_init(k_empty + 8 * i, 1);
            mbar_init(v_full + 8 * i, 1);
            mbar_init(v_empty + 8 * i, 1);
        }
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        mbar_init(do_full, 1);
        mbar_init(do_empty, 1);
        mbar_init(bar_s, 1);
        mbar_init(bar_s_free, 8);
        mbar_init(bar_dp, 1);
        mbar_init(bar_ds, 8);
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, 8);
        mbar_init(bar_delta, 8);
        mbar_init(bar_clc, 1);
        mbar_fence_init();
    }
    // the planner's block: first query, query head, batch; its first 32 flags, under way while the rest is set up
    int4 where = make_int4(0, 0, 0, 0);
    bool sel_n = false;
    auto place = [&](int block) {
        const int hbase = block / (BDQ_HEADS * NTq) * BDQ_HEADS, hcount = min(BDQ_HEADS, heads - hbase);
        const int within = block - hbase * NTq, item = within / hcount, head = hbase + (within - item * hcount);
        where = make_int4((NTq - 1 - item) * ATT_BM, head % HQ, head / HQ, 0);
    };
    auto selected = [&](int kt) -> bool {                     // key tile kt's block, for the queries there (column 0)
        return kt < min((where.x + ATT_BM + 63) / 64, NT) && types_i[(((long)where.z * TN + kt / cpb) * HN + where.y / (HQ / HN)) * 2] != 0;
    };
    if (warp == 2) {
        place(blockIdx.x);
        sel_n = selected(lane);
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int n_step = 0;
    int4 d, loc;                                              // the step's words
    auto next_step = [&]() -> int {                           // its flags
        const int slot = n_step & (BDQ_STEPS - 1);
        ok = warp_wait(desc_full + slot * 8, (n_step / BDQ_STEPS) & 1);
        d = s_desc[2 * slot];
        loc = s_desc[2 * slot + 1];
        d.y = ok ? __shfl_sync(0xffffffffu, d.y, 0) : BDQ_STOP;
        return d.y;
    };
    auto release_step = [&]() { arrive(desc_empty + (n_step++ & (BDQ_STEPS - 1)) * 8); };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(BWD_REGS_LOW));
        if (warp == 0) {
            // -------------------------------------------------------- TMA producer
            int n = 0, nq = 0, ndo = 0, nk = 0, nv = 0;       // steps; loads under way or done
#pragma unroll 1
            while (true) {
                next_step();
                release_step();
                if (d.y & BDQ_STOP) break;
                const int q0 = loc.x, hq = loc.y, b = loc.z, hkv = hq / (HQ / HKV);
                const int st = n & 1, par = ((n >> 1) - 1) & 1, tiles = d.z < 0 ? 1 : 2;
                auto rows = [&](int u) -> int { return (u ? d.z : d.x) * 64; };
                if (lane == 0 && n >= 2) {                    // into L2 while the stages are still read
                    for (int u = 0; u < tiles; ++u) {
#pragma unroll
                        for (int sub = 0; sub < DK / 64; ++sub) tma_prefetch_4d(&map_k, sub * 64, hkv, rows(u), b);
#pragma unroll
                        for (int sub = 0; sub < DV / 64; ++sub) tma_prefetch_4d(&map_v, sub * 64, hkv, rows(u), b);
                    }
                }
                __syncwarp();
                if (d.y & BDQ_FIRST) {
                    if (nq > 0) ok = warp_wait(q_empty, (nq - 1) & 1);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(q_full, 128 * DK * 2);
#pragma unroll
                        for (int sub = 0; sub < DK / 64; ++sub) tma_load_4d(sbase + L::q + sub * 16384, &map_q, sub * 64, hq, q0, b, q_full);
                    }
                    __syncwarp();
                    ++nq;
                }
                if (n >= 2) ok = warp_wait(k_empty + st * 8, par);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(k_full + st * 8, tiles * 64 * DK * 2);
                    for (int u = 0; u < tiles; ++u)
#pragma unroll
                        for (int sub = 0; sub < DK / 64; ++sub)
                            tma_load_4d(sbase + L::k + st * (128 * DK * 2) + sub * 16384 + u * 8192, &map_k, sub * 64, hkv, rows(u), b,
                                        k_full + st * 8);
                }
                __syncwarp();
                ++nk;
                if (d.y & BDQ_FIRST) {
                    if (ndo > 0) ok = warp_wait(do_empty, (ndo - 1) & 1);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(do_full, 128 * DV * 2);
#pragma unroll
                        for (int sub = 0; sub < DV / 64; ++sub) tma_load_4d(sbase + L::dos + sub * 16384, &map_do, sub * 64, hq, q0, b, do_full);
                    }
                    __syncwarp();
                    ++ndo;
                }
                if (n >= 2) ok = warp_wait(v_empty + st * 8, par);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(v_full + st * 8, tiles * 64 * DV * 2);
                    for (int u = 0; u < tiles; ++u)
#pragma unroll
                        for (int sub = 0; sub < DV / 64; ++sub)
                            tma_load_4d(sbase + L::v + st * (128 * DV * 2) + sub * 16384 + u * 8192, &map_v, sub * 64, hkv, rows(u), b,
                                        v_full + st * 8);
                }
                __syncwarp();
                ++nv;
                ++n;
            }
            if (!ok) {                                        // nothing may still be on its way into shared memory
                if (nq > 0) warp_wait(q_full, (nq - 1) & 1);
                if (ndo > 0) warp_wait(do_full, (ndo - 1) & 1);
                for (int i = max(0, nk - 2); i < nk; ++i) warp_wait(k_full + (i & 1) * 8, (i >> 1) & 1);
                for (int i = max(0, nv - 2); i < nv; ++i) warp_wait(v_full + (i & 1) * 8, (i >> 1) & 1);
            }
        } else if (warp == 1) {
            // -------------------------------------------------------- MMA issuer
            constexpr uint32_t id_s = umma_idesc_bf16(128, 128, false), id_dq = umma_idesc_bf16(128, DK, true);
            const uint32_t ql = umma_desc_lo(sbase + L::q, 16), dl = umma_desc_lo(sbase + L::dos, 16);
            int n = 0, nq = 0, ndo = 0, done = 0;             // steps; blocks begun (scores, do.v) and complete
            auto scores = [&](int i, int f) {                 // Q K^T of step i
                ok = warp_wait(k_full + (i & 1) * 8, (i >> 1) & 1);
                if (ok && (f & BDQ_FIRST)) ok = warp_wait(q_full, nq++ & 1);
                if (!ok) return;
                tc_fence_after();
                const uint32_t kl = umma_desc_lo(sbase + L::k + (i & 1) * (128 * DK * 2), 16);
#pragma unroll
                for (int h = 0; h < DK / 64; ++h) umma_ss_x4<2, 2>(tmem + C_S, ql + h * 1024, kl + h * 1024, id_s, h > 0);
                umma_commit(bar_s);
                if (f & BDQ_LAST) umma_commit(q_empty);
            };
            auto products = [&](int i, int f) {               // dO V^T
                ok = warp_wait(v_full + (i & 1) * 8, (i >> 1) & 1);
                if (ok && (f & BDQ_FIRST)) ok = warp_wait(do_full, ndo++ & 1);
                if (!ok) return;
                tc_fence_after();
                const uint32_t vl = umma_desc_lo(sbase + L::v + (i & 1) * (128 * DV * 2), 16);
#pragma unroll
                for (int h = 0; h < DV / 64; ++h) umma_ss_x4<2, 2>(tmem + C_DP, dl + h * 1024, vl + h * 1024, id_s, h > 0);
                umma_commit(bar_dp);
                umma_commit(v_empty + (i & 1) * 8);
                if (f & BDQ_LAST) umma_commit(do_empty);
            };
            int f = next_step();
            bool two = d.z >= 0;
            release_step();
            if (!(f & BDQ_STOP)) {
                scores(0, f);
                if (ok) products(0, f);
            }
#pragma unroll 1
            while (ok && !(f & BDQ_STOP)) {
                const int fn = next_step();                   // the next scores as soon as these have been read
                const bool two_n = d.z >= 0;
                release_step();
                const bool more = !(fn & BDQ_STOP);
                if (ok && more) {
                    ok = warp_wait(bar_s_free, n & 1);
                    if (ok) {
                        tc_fence_after();
                        scores(n + 1, fn);
                    }
                }
                if (ok) ok = warp_wait(bar_ds, n & 1);
                if (ok && (f & BDQ_FIRST) && done > 0) ok = warp_wait(bar_acc_free, (done - 1) & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t kl = umma_desc_lo(sbase + L::k + (n & 1) * (128 * DK * 2), 16384);
                umma_ts_x4<128>(tmem + C_DQ, tmem + C_DP, kl, id_dq, !(f & BDQ_FIRST));
                if (two) umma_ts_x4<128>(tmem + C_DQ, tmem + C_DP + 64, kl + 512, id_dq, 1u);
                umma_commit(k_empty + (n & 1) * 8);
                if (f & BDQ_LAST) {
                    umma_commit(bar_acc);
                    ++done;
                }
                if (more) products(n + 1, fn);                // behind ds k in the tensor pipe: ds may be overwritten
                f = fn;
                two = two_n;
                ++n;
            }
        } else if (warp == 2) {
            // -------------------------------------------------------- planner: blocks and their steps
            int n = 0, answers = 0, block;                    // steps, take-over requests
            auto put = [&](int4 x, int4 y) {
                const int slot = n & (BDQ_STEPS - 1);
                if (n >= BDQ_STEPS) ok = warp_wait(desc_empty + slot * 8, (n / BDQ_STEPS - 1) & 1);
                if (!ok) return;
                if (lane == 0) {
                    s_desc[2 * slot] = x;
                    s_desc[2 * slot + 1] = y;
                }
                arrive(desc_full + slot * 8);
                ++n;
            };
#pragma unroll 1
            while (ok) {
                if (lane == 0) {                              // ask for the next block: heavy ones come first, so one ahead does no harm
                    fence_async_smem();
                    mbar_expect_tx(bar_clc, 16);
                    request_block(sbase + L::clc, bar_clc);
                }
                __syncwarp();
                const int q0 = where.x, hq = where.y, b = where.z;
                const int span0 = (q0 / nbs) * cpb;           // first key tile of the own span
                const int n_cand = min((q0 + ATT_BM + 63) / 64, NT);
                for (int i = n > 0 ? lane : 128; i < 128; i += 32) {       // its rows into L2 while the block before is worked on
                    const long t = ((long)b * T + min(q0 + i, T - 1)) * HQ + hq;
#pragma unroll
                    for (int c = 0; c < DK; c += 64) prefetch_l2(q + t * DK + c);
#pragma unroll
                    for (int c = 0; c < DV; c += 64) {
                        prefetch_l2(o + t * DV + c);
                        prefetch_l2(d_o + t * DV + c);
                    }
                }
                // visible key tiles in ascending order, two to a step: those of selected blocks in front of the own span, then the
                // own span.  A step is announced once it is known whether another follows.
                int held0 = -1, held1 = -1, flags = BDQ_FIRST;
#pragma unroll 1
                for (int base = 0; ok && base < n_cand; base += 32) {
                    const bool sel = sel_n;
                    if (base + 32 < n_cand) sel_n = selected(base + 32 + lane);
                    const unsigned ms = __ballot_sync(0xffffffffu, sel);
                    unsigned m = __ballot_sync(0xffffffffu, base + lane < n_cand && (base + lane >= span0 || sel));
                    while (ok && m) {
                        const int i = __ffs(m) - 1, kt = base + i;
                        m &= m - 1;
                        const int mine = (kt >= span0 ? BDQ_OWN0 : 0) | ((ms >> i) & 1 ? BDQ_SEL0 : 0);
                        if (held0 >= 0 && held1 < 0) {
                            held1 = kt;
                            flags |= mine << 1;
                            continue;
                        }
                        if (held0 >= 0) {
                            put(make_int4(held0, flags, held1, 0), where);
                            flags = 0;
                        }
                        held0 = kt;
                        held1 = -1;
                        flags |= mine;
                    }
                }
                if (ok) put(make_int4(held0, flags | BDQ_LAST, held1, 0), where);    // (the own span is never empty)
                const bool came = warp_wait(bar_clc, answers & 1);                   // (also after a failed wait: the answer is on its way)
                ++answers;
                ok = ok && came;
                if (!ok || !taken_block(sbase + L::clc, block)) break;
                __syncwarp();
                place(block);
                sel_n = selected(lane);
            }
            if (ok) put(make_int4(0, BDQ_STOP, -1, 0), make_int4(0, 0, 0, 0));
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(BWD_REGS_HIGH));
        // ------------------------------------------------------------ softmax: one query per thread and half, 64 keys each
        const int quad = warp & 3, half = (warp - 4) >> 2, row = quad * 32 + lane;
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t t_s = t_lane + C_S + half * 64, t_dp = t_lane + C_DP + half * 64;
        const float sl2 = scale * kLog2e;
        unsigned char* const out = smem + L::out + (warp - 4) * 4096;
        // delta = rowsum(o * do): this warp's 16 rows, four threads per row and eight rows at a time
        constexpr int NC = DV / 32;
        const int drow = (warp - 4) * 16 + (lane >> 2);
        uint4 xo[2][NC], xd[2][NC];
        float nlse = 0.f;
        auto load_rows = [&]() {                              // of the block in `loc`
            const int q0 = loc.x, hq = loc.y, b = loc.z;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = q0 + drow + 8 * i;
                const long off = (((long)b * T + t) * HQ + hq) * DV + (lane & 3) * 8;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    xo[i][c] = t < T ? *reinterpret_cast<const uint4*>(o + off + c * 32) : make_uint4(0, 0, 0, 0);
                    xd[i][c] = t < T ? *reinterpret_cast<const uint4*>(d_o + off + c * 32) : make_uint4(0, 0, 0, 0);
                }
            }
            nlse = q0 + row < T ? -lse[((long)b * T + q0 + row) * HQ + hq] : 0.f;
        };
        auto make_delta = [&](int block) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint64_t s2 = 0;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const uint32_t* xw = reinterpret_cast<const uint32_t*>(&xo[i][c]);
                    const uint32_t* yw = reinterpret_cast<const uint32_t*>(&xd[i][c]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 u = unpack_bf16(xw[e]), w = unpack_bf16(yw[e]);
                        s2 = fma2(pack2(u.x, u.y), pack2(w.x, w.y), s2);
                    }
                }
                float s = hsum2(s2);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                const int r = drow + 8 * i, t = loc.x + r;
                if ((lane & 3) == 0) {
                    s_delta[(block & 1) * 128 + r] = s;
                    if (t < T) delta_out[((long)loc.z * T + t) * HQ + loc.y] = s;
                }
            }
            arrive(bar_delta);
        };
        // this warp's rows of dq: 64 columns at a time through its own 4 KB
        auto finish = [&](int q0, int hq, int b, int block) {
            if (!ok) return;
            ok = warp_wait(bar_acc, block & 1);
            if (!ok) return;
            tc_fence_after();
            if (half < DK / 64) {
                if (lane == 0) tma_store_wait_read();         // the block before has left
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 64; c += 32) {            // (in halves: o and do of the next block are held as well)
                    uint32_t x[32];
                    tmem_ld32(t_lane + C_DQ + half * 64 + c, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = pack_bf16(__uint_as_float(x[8 * i + 2 * e]) * scale, __uint_as_float(x[8 * i + 2 * e + 1]) * scale);
                        *reinterpret_cast<uint4*>(out + lane * 128 + (((c / 8 + i) ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            tc_fence_before();
            arrive(bar_acc_free);
            if (half >= DK / 64) return;
            fence_async_smem();
            __syncwarp();
            if (lane == 0 && q0 + quad * 32 < T) {
                tma_store_4d(&map_dq, smem_u32(out), half * 64, hq, q0 + quad * 32, b);
                tma_store_commit();
            }
        };
        int n = 0, blocks = 0;                                // steps, blocks begun
        float ndel = 0.f;
        int f = next_step();
        if (!(f & BDQ_STOP)) load_rows();
#pragma unroll 1
        while (ok && !(f & BDQ_STOP)) {
            if (f & BDQ_FIRST) make_delta(blocks++);
            const int kt = half ? d.z : d.x;
            const bool act = kt >= 0;
            ok = warp_wait(bar_s, n & 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t r[64];
            if (act) {
                uint32_t(&r0)[32] = *reinterpret_cast<uint32_t(*)[32]>(r);
                uint32_t(&r1)[32] = *reinterpret_cast<uint32_t(*)[32]>(r + 32);
                tmem_ld32(t_s, r0);
                tmem_ld32(t_s + 32, r1);
                tmem_ld_wait();
            }
            tc_fence_before();
            arrive(bar_s_free);
            if (act) {
                if (f & (BDQ_OWN0 << half)) {
                    // own-span tile: the row's visible keys are columns [0, lim] (attn_walk.cuh: visible()); an invisible score
                    // becomes -inf, its p zero
                    const int s0 = kt * 64, blk_end = (kt / cpb + 1) * nbs, t = loc.x + row;
                    int lim = T - 1 - s0;
                    if (t < blk_end) lim = own ? min(lim, t - s0) : -1;
                    else if (!(f & (BDQ_SEL0 << half))) lim = -1;
#pragma unroll
                    for (int e = 0; e < 64; ++e)
                        if (e > lim) r[e] = 0xff800000u;
                }
                const uint64_t sc2 = pack2(sl2, sl2), l2 = pack2(nlse, nlse);
#pragma unroll
                for (int e = 0; e < 64; e += 2) {
                    float x0, x1;
                    unpack2(fma2(pack2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), sc2, l2), x0, x1);
                    r[e] = __float_as_uint(ex2(x0));
                    r[e + 1] = __float_as_uint(ex2(x1));
                }
            }
            if (f & BDQ_FIRST) {
                ok = warp_wait(bar_delta, (blocks - 1) & 1);
                if (!ok) break;
                ndel = -s_delta[((blocks - 1) & 1) * 128 + row];
            }
            ok = warp_wait(bar_dp, n & 1);
            if (!ok) break;
            tc_fence_after();
            if (act) {
                const uint64_t d2 = pack2(ndel, ndel);
                uint32_t x0[32], x1[32];
                tmem_ld32(t_dp, x0);
                tmem_ld32(t_dp + 32, x1);
                tmem_ld_wait();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t pk[16];
                    uint32_t(&x)[32] = h ? x1 : x0;
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        pk[e] = close2(mul2(pack2(__uint_as_float(r[h * 32 + 2 * e]), __uint_as_float(r[h * 32 + 2 * e + 1])),
                                            add2(pack2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1])), d2)));
                    tmem_st16(t_dp + h * 16, pk);
                }
                tmem_st_wait();
            }
            tc_fence_before();
            arrive(bar_ds);
            ++n;
            const int4 was = loc;
            release_step();
            const int fn = next_step();
            if (f & BDQ_LAST) {
                const bool had = ok;                          // (the block is complete also if no next one is known)
                if (!(fn & BDQ_STOP)) load_rows();
                ok = true;
                finish(was.x, was.y, was.z, blocks - 1);
                ok = ok && had;
            }
            f = fn;
        }
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------------- dk, dv
// With the keys in the lanes all four products are 128 x 128 (x head dim): their operands are read half as often as by 128 x 64 ones
// with p and ds in shared memory, p and ds need no shared memory at all, and a query tile is loaded once for two key tiles.
// Results of a tile that the queries at hand do not see are kept out by the products' lane mask, whatever the queries hold.
// One persistent CTA per SM takes blocks of the grid over (cluster launch control); a planning warp works out their steps, and
// lse and delta of the queries, while the others are at the steps before.  Roles: warp 0 loads, warp 1 issues the products, warp 2
// plans, warps 4-11 p and ds (a key and 64 queries per thread).
// Registers as above: 168 for all threads and 56 bytes of spills took 389 us where the figures below have 355.
// What bounds it: the chain scores -> p -> dv product and do.v -> ds -> dk product of a step, 3 k cycles against 2 k of the tensor
// core (tensor memory holds one step: 128 columns each of scores, do.v, dk and dv), and 64 KB of q and do from L2 a step.
// Alone (us; before: 128 x 64 score tiles, p and ds through shared memory, one CTA per pair of tiles), block 64:
//   128/128, B = 8, T = 4096, H = 16: 25 % selected 678 -> 355, 50 % 1069 -> 545, 2 % 338 -> 182;  64/64, 30 %: 630 -> 336
//   128/64, B = 4, T = 1000, H = 16, 50 %: 72 -> 41;  128/128, B = 1, T = 2048, H = 16, 30 %: 65 -> 36
//   64/128, B = 2, T = 2048, 12 heads over 6, block 128, 40 %: 113 -> 56;  the smallest, 64/64, B = 2, T = 64, H = 4: 7.5 -> 7.9, and at T = 100 7.5 -> 8.6: one step per CTA, of which the 64 keys
//   of a single tile fill half of the lanes
constexpr int BKV_THREADS = 384;                              // TMA, MMA, planner, (no work), 8 softmax warps
constexpr int BKV_MAXG = 16;
constexpr int BKV_DESCS = 2;                                  // steps that the planner is ahead
template <int DK, int DV>
struct DkvSmem {
    static constexpr int kv = 0;                              // k: DK/64 sub-tiles [128 keys][64], then v the same way
    static constexpr int q = kv + 128 * (DK + DV) * 2;        // 2 stages x DK/64 sub-tiles [128 queries][64]
    static constexpr int dos = q + 2 * 128 * DK * 2;          // 2 stages x DV/64 sub-tiles
    static constexpr int out = dos + 2 * 128 * DV * 2;        // per softmax warp: 32 rows x 64 columns on their way out
    static constexpr int stat = out + 8 * 4096;               // per step (-lse, -delta) of 128 queries
    static constexpr int dn = stat + BKV_DESCS * 1024;        // dnats parts [2 tiles][16 heads][4 warps]
    static constexpr int desc = dn + 2 * BKV_MAXG * 4 * 4;    // steps, 32 bytes each
    static constexpr int last = desc + BKV_DESCS * 32;        // last query tile [2 tiles][16 heads] of a selected pair
    static constexpr int clc = last + 2 * BKV_MAXG * 2;       // answer of the take-over request
    static constexpr int bars = clc + 16;
    static constexpr int total = bars + 240;
    static_assert(total <= 227 * 1024, "one CTA per SM");
};

// What a CTA does in a step, worked out by the planner: first query, flags, query head of the group, head whose sums of ds are
// complete (BKV_FLUSH); the two key tiles (-1: none), key head, batch.
enum : int {
    BKV_ACT0 = 1, BKV_ACT1 = 2,                               // the queries see the first / second key tile of the pair
    BKV_SEL0 = 4, BKV_SEL1 = 8,                               // the head selected the tile's block
    BKV_FIRST = 16, BKV_LAST = 32,                            // first / last step of the pair
    BKV_EMPTY = 64, BKV_STOP = 128,                           // no query sees either tile; no pair is left
    BKV_FLUSH = 256, BKV_ANY0 = 512, BKV_ANY1 = 1024,         // some query sees the first / second tile
    BKV_SUMS = 2048                                           // a pair of selected tiles: sums of ds for it
};

// Heads whose CTAs are interleaved, heaviest first: the last CTAs to start are then light ones, and q and do of that many
// heads (2 MB each at 4096 x 128) stay in L2 for the CTAs of a head that run at the same time.
constexpr int BKV_HEADS = 32;
// A grid of no more blocks than the 148 SMs takes the form SMALL, whose blocks are half as long: a block's pair of selected tiles and
// what is unselected of its neighbours are blocks of their own, which in one block would be one behind the other while SMs are idle
// (us, one block for both / halves: 16 query heads over one, T = 100 64/64 75 / 43, T = 256 76 / 43; 12 over 6, B = 2, T = 100
// 128/128 17.5 / 12.4; 4 heads, B = 2, T = 256 12.6 / 9.5).  Where the halves fit the SMs at once nothing is taken over; otherwise they are
// taken over like the others (B = 4, T = 256, H = 16 13.1 / 12.7; a CTA for each of the 256 halves 16.1).  Blocks of larger grids stay
// whole (16 heads, B = 16, T = 100 64/64 18.9, halves 21.8), in a form of their own: its code is what it was, and these kernels
// lose 5 % to the way that code lies in the instruction cache.  A sequence of one key tile has nothing to halve.
constexpr int BKV_SMALL = 148;

// Four K-steps, A from tensor memory, results added in the lanes whose bit is not set: m01 for lanes 0-63, m23 for lanes 64-127.
template <int STEP_B>
__device__ __forceinline__ void umma_ts_x4_lanes(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t idesc, uint32_t m01, uint32_t m23) {
    asm volatile(
        "{\n .reg .pred t, e;\n .reg .b64 b;\n .reg .b32 x, y;\n"
        " setp.eq.u32 t, 0, 0;\n elect.sync _|e, 0xffffffff;\n"
        " mov.b64 b, {%2, %4};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, {%6, %6, %7, %7}, t;\n"
        " add.u32 x, %1, 8;\n add.u32 y, %2, %5;\n mov.b64 b, {y, %4};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, {%6, %6, %7, %7}, t;\n"
        " add.u32 x, x, 8;\n add.u32 y, y, %5;\n mov.b64 b, {y, %4};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, {%6, %6, %7, %7}, t;\n"
        " add.u32 x, x, 8;\n add.u32 y, y, %5;\n mov.b64 b, {y, %4};\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, {%6, %6, %7, %7}, t;\n}\n"
        ::"r"(d_tmem), "r"(a_tmem), "r"(blo), "r"(idesc), "n"(UMMA_DESC_HI), "n"(STEP_B), "r"(m01), "r"(m23)
        : "memory");
}

template <int DK, int DV, bool SMALL>
__global__ void __launch_bounds__(BKV_THREADS, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                     const __grid_constant__ CUtensorMap map_dk, const __grid_constant__ CUtensorMap map_dv,
                     const float* __restrict__ lse, const float* __restrict__ delta, const int* __restrict__ types_i,
                     float* __restrict__ dnats_part, int T, int HQ, int HKV, int HN, int TN, int nbs, float scale, int own, int heads,
                     int ctas_per_head, int halves, int* status) {
    using L = DkvSmem<DK, DV>;
    // TMEM: scores [128 keys][128 queries], then p over each half's first columns; do.v, then ds; dv; dk
    constexpr uint32_t C_S = 0, C_DP = 128, C_DV = 256, C_DK = 384;
    constexpr int NB = (DK + DV) / 64;                        // 64-column blocks of results: dv, then dk
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int G = HQ / HKV, cpb = nbs / 64;
    const int NT = (T + 63) / 64, NTq = (T + ATT_BM - 1) / ATT_BM;
    float* s_dn = reinterpret_cast<float*>(smem + L::dn);
    int4* s_desc = reinterpret_cast<int4*>(smem + L::desc);
    volatile int16_t* s_last = reinterpret_cast<volatile int16_t*>(smem + L::last);
    const uint32_t bar0 = sbase + L::bars;
    // barriers: desc_full / desc_empty (steps, with lse and delta); q_full / q_empty, do_full / do_empty (stages);
    // kv_full / kv_empty; s, dp (scores, do.v complete); p, ds (written by the softmax warps); acc (dk, dv of the pair complete);
    // dv (of the pair complete: its rows leave during dk's last product); acc_free (read and set to zero)
    const uint32_t desc_full = bar0, desc_empty = bar0 + 32, bar_dv = bar0 + 64, q_full = bar0 + 96,
                   q_empty = bar0 + 112, do_full = bar0 + 128, do_empty = bar0 + 144, kv_full = bar0 + 160, kv_empty = bar0 + 168,
                   bar_s = bar0 + 176, bar_dp = bar0 + 184, bar_p = bar0 + 192, bar_ds = bar0 + 200, bar_acc = bar0 + 208,
                   bar_acc_free = bar0 + 216, bar_clc = bar0 + 224;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 232);
    auto arrive = [&](uint32_t bar) {                         // behind what the whole warp has done so far
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };

    if (tid == 0) {
        for (int i = 0; i < BKV_DESCS; ++i) {
            mbar_init(desc_full + 8 * i, 1);
            mbar_init(desc_empty + 8 * i, 10);                // eight softmax warps, TMA, MMA
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full + 8 * i, 1);
            mbar_init(q_empty + 8 * i, 1);
            mbar_init(do_full + 8 * i, 1);
            mbar_init(do_empty + 8 * i, 1);
        }
        mbar_init(kv_full, 1);
        mbar_init(kv_empty, 1);
        mbar_init(bar_s, 1);
        mbar_init(bar_dp, 1);
        mbar_init(bar_p, 8);
        mbar_init(bar_ds, 8);
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, 8);
        mbar_init(bar_clc, 1);
        mbar_init(bar_dv, 1);
        mbar_fence_init();
    }
    for (int i = tid; i < 2 * BKV_MAXG * 4; i += BKV_THREADS) s_dn[i] = 0.f;
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    int n_step = 0;                                           // steps taken over
    int4 d, loc;                                              // the step's words
    auto next_step = [&]() -> int {                           // its flags
        const int slot = n_step & (BKV_DESCS - 1);
        ok = warp_wait(desc_full + slot * 8, (n_step / BKV_DESCS) & 1);
        d = s_desc[2 * slot];
        loc = s_desc[2 * slot + 1];
        d.y = ok ? __shfl_sync(0xffffffffu, d.y, 0) : BKV_STOP;
        return d.y;
    };
    auto release_step = [&]() { arrive(desc_empty + (n_step++ & (BKV_DESCS - 1)) * 8); };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(BWD_REGS_LOW));
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer
            int ni = 0, pairs = 0;                                // steps with queries, pairs that have some
#pragma unroll 1
            while (ok) {
                next_step();
                release_step();
                if (d.y & BKV_STOP) break;
                if (d.y & BKV_EMPTY) continue;
                const int hkv = loc.z, b = loc.w;
                if (d.y & BKV_FIRST) {
                    if (pairs > 0) ok = warp_wait(kv_empty, (pairs - 1) & 1);
                    if (!ok) break;
                    if (lane == 0) {
                        const int t[2] = {loc.x, loc.y};
                        mbar_expect_tx(kv_full, ((t[0] >= 0) + (t[1] >= 0)) * 64 * (DK + DV) * 2);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (t[u] < 0) continue;
#pragma unroll
                            for (int sub = 0; sub < DK / 64; ++sub)
                                tma_load_4d(sbase + L::kv + sub * 16384 + u * 8192, &map_k, sub * 64, hkv, t[u] * 64, b, kv_full);
#pragma unroll
                            for (int sub = 0; sub < DV / 64; ++sub)
                                tma_load_4d(sbase + L::kv + 128 * DK * 2 + sub * 16384 + u * 8192, &map_v, sub * 64, hkv, t[u] * 64, b, kv_full);
                        }
                    }
                    __syncwarp();
                    ++pairs;
                }
                const int st = ni & 1, par = ((ni >> 1) - 1) & 1, hq = hkv * G + d.z;
                if (lane == 0 && ni >= 2) {                       // into L2 while the stages are still read
#pragma unroll
                    for (int sub = 0; sub < DK / 64; ++sub) tma_prefetch_4d(&map_q, sub * 64, hq, d.x, b);
#pragma unroll
                    for (int sub = 0; sub < DV / 64; ++sub) tma_prefetch_4d(&map_do, sub * 64, hq, d.x, b);
                }
                __syncwarp();
                if (ni >= 2) ok = warp_wait(q_empty + st * 8, par);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(q_full + st * 8, 128 * DK * 2);
#pragma unroll
                    for (int sub = 0; sub < DK / 64; ++sub)
                        tma_load_4d(sbase + L::q + st * (128 * DK * 2) + sub * 16384, &map_q, sub * 64, hq, d.x, b, q_full + st * 8);
                }
                __syncwarp();
                if (ni >= 2) ok = warp_wait(do_empty + st * 8, par);
                if (!ok) {
                    warp_wait(q_full + st * 8, (ni >> 1) & 1);    // nothing may still be on its way into shared memory
                    break;
                }
                if (lane == 0) {
                    mbar_expect_tx(do_full + st * 8, 128 * DV * 2);
#pragma unroll
                    for (int sub = 0; sub < DV / 64; ++sub)
                        tma_load_4d(sbase + L::dos + st * (128 * DV * 2) + sub * 16384, &map_do, sub * 64, hq, d.x, b, do_full + st * 8);
                }
                __syncwarp();
                ++ni;
            }
            if (!ok) {
                if (pairs > 0) warp_wait(kv_full, (pairs - 1) & 1);
                for (int i = max(0, ni - 2); i < ni; ++i) {
                    warp_wait(q_full + (i & 1) * 8, (i >> 1) & 1);
                    warp_wait(do_full + (i & 1) * 8, (i >> 1) & 1);
                }
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------ MMA issuer
            constexpr uint32_t id_s = umma_idesc_bf16(128, 128, false);
            constexpr uint32_t id_dv = umma_idesc_bf16(128, DV, true), id_dk = umma_idesc_bf16(128, DK, true);
            const uint32_t kl = umma_desc_lo(sbase + L::kv, 16), vl = umma_desc_lo(sbase + L::kv + 128 * DK * 2, 16);
            auto scores = [&](int st) {                           // K Q^T
                tc_fence_after();
                const uint32_t ql = umma_desc_lo(sbase + L::q + st * (128 * DK * 2), 16);
#pragma unroll
                for (int h = 0; h < DK / 64; ++h) umma_ss_x4<2, 2>(tmem + C_S, kl + h * 1024, ql + h * 1024, id_s, h > 0);
                umma_commit(bar_s);
            };
            auto products = [&](int st, bool last) {              // V dO^T
                tc_fence_after();
                const uint32_t dl = umma_desc_lo(sbase + L::dos + st * (128 * DV * 2), 16);
#pragma unroll
                for (int h = 0; h < DV / 64; ++h) umma_ss_x4<2, 2>(tmem + C_DP, vl + h * 1024, dl + h * 1024, id_s, h > 0);
                umma_commit(bar_dp);
                if (last) umma_commit(kv_empty);
            };
            int ni = 0, pairs = 0;
            int f = next_step();
            release_step();
#pragma unroll 1
            while (ok && !(f & BKV_STOP)) {
                if (f & BKV_EMPTY) {
                    f = next_step();
                    release_step();
                    continue;
                }
                if (f & BKV_FIRST) {
                    ok = warp_wait(kv_full, pairs & 1);
                    if (ok) ok = warp_wait(q_full + (ni & 1) * 8, (ni >> 1) & 1);
                    if (!ok) break;
                    scores(ni & 1);
                    ok = warp_wait(do_full + (ni & 1) * 8, (ni >> 1) & 1);
                    if (!ok) break;
                    products(ni & 1, (f & BKV_LAST) != 0);
                    ok = warp_wait(bar_acc_free, pairs & 1);
                    ++pairs;
                }
                const int st = ni & 1, nst = st ^ 1, npar = ((ni + 1) >> 1) & 1;
                const uint32_t m01 = f & BKV_ACT0 ? 0u : 0xffffffffu, m23 = f & BKV_ACT1 ? 0u : 0xffffffffu;
                const bool last = (f & BKV_LAST) != 0;
                if (ok) ok = warp_wait(bar_p, ni & 1);
                if (!ok) break;
                tc_fence_after();
                {                                                 // dv += p dO
                    const uint32_t dl = umma_desc_lo(sbase + L::dos + st * (128 * DV * 2), 16384);
#pragma unroll
                    for (int h = 0; h < 2; ++h) umma_ts_x4_lanes<128>(tmem + C_DV, tmem + C_S + h * 64, dl + h * 512, id_dv, m01, m23);
                    umma_commit(do_empty + st * 8);
                    if (last) umma_commit(bar_dv);
                }
                int fn = BKV_STOP;
                if (!last) {                                      // the next scores as soon as p has been used
                    fn = next_step();
                    release_step();
                    if (ok) ok = warp_wait(q_full + nst * 8, npar);
                    if (!ok) break;
                    scores(nst);
                }
                ok = warp_wait(bar_ds, ni & 1);
                if (!ok) break;
                tc_fence_after();
                {                                                 // dk += ds Q
                    const uint32_t ql = umma_desc_lo(sbase + L::q + st * (128 * DK * 2), 16384);
#pragma unroll
                    for (int h = 0; h < 2; ++h) umma_ts_x4_lanes<128>(tmem + C_DK, tmem + C_DP + h * 64, ql + h * 512, id_dk, m01, m23);
                    umma_commit(q_empty + st * 8);
                }
                if (last) {
                    umma_commit(bar_acc);
                    f = next_step();
                    release_step();
                } else {
                    ok = warp_wait(do_full + nst * 8, npar);
                    if (!ok) break;
                    products(nst, (fn & BKV_LAST) != 0);
                    f = fn;
                }
                ++ni;
            }
        } else if (warp == 2) {
            // ------------------------------------------------------------ planner: blocks, their steps, lse and delta of the queries
            int n = 0, asked = 0, answers = 0;                    // steps, take-over requests
            int block = blockIdx.x;
            const bool persist = !SMALL || gridDim.x > BKV_SMALL;
            auto open = [&]() {
                if (n >= BKV_DESCS) ok = warp_wait(desc_empty + (n & (BKV_DESCS - 1)) * 8, (n / BKV_DESCS - 1) & 1);
                return ok;
            };
            auto put = [&](int4 x, int4 y) {
                const int slot = n & (BKV_DESCS - 1);
                if (lane == 0) {
                    s_desc[2 * slot] = x;
                    s_desc[2 * slot + 1] = y;
                }
                arrive(desc_full + slot * 8);
                ++n;
            };
            auto request = [&]() {
                if (lane == 0) {
                    fence_async_smem();
                    mbar_expect_tx(bar_clc, 16);
                    request_block(sbase + L::clc, bar_clc);
                }
                __syncwarp();
                ++asked;
            };
#pragma unroll 1
            while (ok) {
                // Block `item` of a head: the item-th pair of the tiles whose block some head of the group selected, in their order
                // (neighbours see nearly the same queries), then what is unselected of tiles 2 item and 2 item + 1, which only
                // their own blocks' queries see; in halves, the first `halves` blocks are the pairs alone, the others the rest.
                const bool rest_only = SMALL && halves && block >= halves;
                if (rest_only) block -= halves;
                const int hbase = block / (BKV_HEADS * ctas_per_head) * BKV_HEADS, hcount = min(BKV_HEADS, heads - hbase);
                const int within = block - hbase * ctas_per_head;
                const int item = within / hcount, head = hbase + within % hcount;
                const int hkv = head % HKV, b = head / HKV;
                auto selected = [&](int kt) -> bool {
                    bool s = false;
#pragma unroll 1
                    for (int gi = 0; gi < G; ++gi) s |= types_i[(((long)b * TN + kt / cpb) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0;
                    return s;
                };
                int chosen[2] = {-1, -1}, rest[2] = {-1, -1};
                unsigned mine = 0;                                // bit i: tile 2 item + i is selected
                int cnt = 0;
#pragma unroll 1
                for (int base = 0; base < NT; base += 32) {
                    const unsigned m = __ballot_sync(0xffffffffu, base + lane < NT && selected(base + lane));
                    const int k = __popc(m);
                    if (2 * item >= base && 2 * item < base + 32) mine = m >> (2 * item - base);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int r = 2 * item + i - cnt;
                        if (r >= 0 && r < k) chosen[i] = base + __fns(m, 0, r + 1);
                    }
                    cnt += k;
                    if (cnt >= 2 * item + 2 && base + 32 > 2 * item + 1) break;
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (!((mine >> i) & 1) && 2 * item + i < NT) rest[i] = 2 * item + i;
                if (rest_only) chosen[0] = -1;
                bool requested = !persist || chosen[0] < 0;       // a step or none: ask for the next block at once
                if (persist && requested) request();
                if (chosen[0] >= 0) {
                    // last query tile of every (tile, head): the sequence's if the head selected the block, else the own block's
                    __syncwarp();
#pragma unroll 1
                    for (int i = lane; i < 2 * BKV_MAXG; i += 32) {
                        const int kt = i / BKV_MAXG ? chosen[1] : chosen[0], gi = i % BKV_MAXG;
                        int last = -1;
                        if (kt >= 0 && gi < G) {
                            const int blk = kt / cpb, blk_end = (blk + 1) * nbs;
                            const bool s = G == 1 || types_i[(((long)b * TN + blk) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0;
                            if (s && blk_end < T) last = NTq - 1;
                            else if (own) last = min((blk_end - 1) / ATT_BM, NTq - 1);
                        }
                        s_last[i] = (int16_t)last;
                    }
                    __syncwarp();
                }
#pragma unroll 1
                for (int pass = chosen[0] < 0; ok && pass < (SMALL && halves && !rest_only ? 1 : 2); ++pass) {
                    const bool sums = pass == 0;
                    const int t[2] = {sums ? chosen[0] : rest[0], sums ? chosen[1] : rest[1]};
                    if (t[0] < 0 && t[1] < 0) continue;
                    const int4 where = make_int4(t[0], t[1], hkv, b);
                    int first[2], end[2], own_last[2];            // tile u: query tiles [first, last(head)]
                    bool any[2] = {false, false};
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        end[u] = (t[u] / cpb + 1) * nbs;
                        first[u] = t[u] < 0 ? NTq : own ? t[u] * 64 / ATT_BM : end[u] / ATT_BM;
                        own_last[u] = t[u] >= 0 && own ? min((end[u] - 1) / ATT_BM, NTq - 1) : -1;
                    }
                    auto last_of = [&](int u, int gi) -> int { return sums ? (int)s_last[u * BKV_MAXG + gi] : own_last[u]; };
                    for (int gi = 0; gi < G; ++gi) {
                        any[0] |= last_of(0, gi) >= first[0];
                        any[1] |= last_of(1, gi) >= first[1];
                    }
                    const int base = (sums ? BKV_SUMS : 0) | (any[0] ? BKV_ANY0 : 0) | (any[1] ? BKV_ANY1 : 0);
                    if (!any[0] && !any[1]) {
                        if (open()) put(make_int4(0, base | BKV_EMPTY, 0, 0), where);
                        continue;
                    }
                    int held = -1, h_qt = 0, h_gi = 0, h_prev = 0;    // the step that is announced once it is known whether another follows
                    float nl[4], nd[4];
                    auto announce = [&](int more) {
                        if (!open()) return;
                        float* x = reinterpret_cast<float*>(smem + L::stat + (n & (BKV_DESCS - 1)) * 1024);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            x[lane + 32 * i] = nl[i];
                            x[128 + lane + 32 * i] = nd[i];
                        }
                        put(make_int4(h_qt * ATT_BM, held | more, h_gi, h_prev), where);
                    };
                    int prev = -1;
#pragma unroll 1
                    for (int gi = 0; ok && gi < G; ++gi) {
                        const int l0 = last_of(0, gi), l1 = last_of(1, gi), hi = max(l0, l1);
                        int sel = sums ? BKV_SEL0 | BKV_SEL1 : 0;
                        if (sums && G > 1) {
                            sel = 0;
#pragma unroll
                            for (int u = 0; u < 2; ++u)
                                if (t[u] >= 0 && types_i[(((long)b * TN + t[u] / cpb) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0)
                                    sel |= u ? BKV_SEL1 : BKV_SEL0;
                        }
#pragma unroll 1
                        for (int qt = min(l0 >= first[0] ? first[0] : NTq, l1 >= first[1] ? first[1] : NTq); ok && qt <= hi; ++qt) {
                            const int act = (qt >= first[0] && qt <= l0 ? BKV_ACT0 : 0) | (qt >= first[1] && qt <= l1 ? BKV_ACT1 : 0);
                            if (!act) continue;
                            if (held >= 0) announce(0);
                            held = base | act | sel | (prev < 0 ? BKV_FIRST : 0) | (prev >= 0 && prev != gi ? BKV_FLUSH : 0);
                            h_qt = qt;
                            h_gi = gi;
                            h_prev = prev;
                            prev = gi;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {         // a query behind the end has probability 0
                                const int q = qt * ATT_BM + lane + 32 * i;
                                const long r = ((long)b * T + q) * HQ + hkv * G + gi;
                                nl[i] = q < T ? -lse[r] : -INFINITY;
                                nd[i] = q < T ? -delta[r] : 0.f;
                            }
                        }
                    }
                    if (ok) announce(BKV_LAST);
                    // the pair's last steps are under way: early enough to work out the next block, late enough to leave it to an SM
                    // that is free earlier
                    if (persist && ok && sums) {
                        request();
                        requested = true;
                    }
                }
                if (!persist) break;
                if (ok && !requested) request();                  // (the chosen pair had no step)
                if (asked > answers) {                            // (also after a failed wait: the answer is on its way)
                    const bool came = warp_wait(bar_clc, answers & 1);
                    ++answers;
                    ok = ok && came;
                }
                if (!ok || !taken_block(sbase + L::clc, block)) break;
                __syncwarp();
            }
            if (ok && open()) put(make_int4(0, BKV_STOP, 0, 0), make_int4(0, 0, 0, 0));
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(BWD_REGS_HIGH));
        // ------------------------------------------------------------ softmax: one key per thread and half, 64 queries each
        const int quad = warp & 3, half = (warp - 4) >> 2, u = quad >> 1, part = (quad & 1) * 2 + half;
        const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t t_s = t_lane + C_S + half * 64, t_dp = t_lane + C_DP + half * 64;
        const float sl2 = scale * kLog2e;
        unsigned char* const out = smem + L::out + (warp - 4) * 4096;
        int ni = 0, pairs = 0;                                // steps with queries, pairs that have some
        float dn = 0.f;
        auto flush = [&](int gi, int f) {                     // one slot per (key tile, head, warp): a fixed order of summation
            dn = warp_sum(dn);
            if (lane == 0 && (f & BKV_SUMS)) s_dn[(u * BKV_MAXG + gi) * 4 + part] = dn;
            dn = 0.f;
        };
        auto zero = [&](uint32_t col) {
            uint32_t z[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) z[e] = 0;
            tmem_st32(t_lane + col, z);
            tmem_st32(t_lane + col + 32, z);
        };
        auto block_col = [&](int blk) -> uint32_t { return blk < DV / 64 ? C_DV + blk * 64 : C_DK + (blk - DV / 64) * 64; };
        // this warp's rows of dv and dk: 64 columns at a time through its own 4 KB, then zeros for the next pair
        auto finish = [&](bool any, bool acc) {
            const int kt = u ? loc.y : loc.x, row0 = kt * 64 + (quad & 1) * 32;
#pragma unroll 1
            for (int blk = half; blk < NB; blk += 2) {
                if (acc) {                                    // dv is complete while dk's last product is still under way
                    ok = warp_wait(blk < DV / 64 ? bar_dv : bar_acc, pairs & 1);
                    if (!ok) return;
                    tc_fence_after();
                }
                uint32_t w[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) w[e] = 0;
                if (acc) {
                    if (any) {
                        uint32_t r0[32], r1[32];
                        tmem_ld32(t_lane + block_col(blk), r0);
                        tmem_ld32(t_lane + block_col(blk) + 32, r1);
                        tmem_ld_wait();
                        const float f = blk < DV / 64 ? 1.f : scale;
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            w[e] = pack_bf16(__uint_as_float(r0[2 * e]) * f, __uint_as_float(r0[2 * e + 1]) * f);
                            w[16 + e] = pack_bf16(__uint_as_float(r1[2 * e]) * f, __uint_as_float(r1[2 * e + 1]) * f);
                        }
                    }
                    zero(block_col(blk));
                }
                if (lane == 0) tma_store_wait_read();         // the block before has left
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<uint4*>(out + lane * 128 + ((i ^ (lane & 7)) << 4)) =
                        make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
                fence_async_smem();
                __syncwarp();
                if (lane == 0 && kt >= 0 && row0 < T) {
                    if (blk < DV / 64) tma_store_4d(&map_dv, smem_u32(out), blk * 64, loc.z, row0, loc.w);
                    else tma_store_4d(&map_dk, smem_u32(out), (blk - DV / 64) * 64, loc.z, row0, loc.w);
                    tma_store_commit();
                }
            }
        };
        // (one warp)  the pair's sums of ds for every head, which are then zero again
        auto write_sums = [&](bool some) {
#pragma unroll 1
            for (int i = lane; i < 2 * G; i += 32) {
                const int v = i / G, gi = i - v * G, kt = v ? loc.y : loc.x;
                float* x = s_dn + (v * BKV_MAXG + gi) * 4;
                const float sum = some ? (x[0] + x[1]) + (x[2] + x[3]) : 0.f;
                x[0] = x[1] = x[2] = x[3] = 0.f;
                if (kt >= 0) dnats_part[((long)loc.w * NT + kt) * HQ + loc.z * G + gi] = sum;
            }
            __syncwarp();
        };
        auto release_acc = [&]() {
            tmem_st_wait();
            tc_fence_before();
            arrive(bar_acc_free);
        };
#pragma unroll 1
        for (int blk = half; blk < NB; blk += 2) zero(block_col(blk));
        release_acc();
        int end_own = 0;                                      // end of the own block
#pragma unroll 1
        while (true) {
            const int f = next_step();
            if (!ok || (f & BKV_STOP)) break;
            if (f & BKV_EMPTY) {
                release_step();
                finish(false, false);
                if (warp == 4) write_sums(false);
                continue;
            }
            const bool act = (f & (BKV_ACT0 << u)) != 0;
            const int kt = u ? loc.y : loc.x;
            if (f & BKV_FIRST) end_own = (kt / cpb + 1) * nbs;
            const int blk_end = end_own - d.x;                // relative to the first query
            const float* st = reinterpret_cast<const float*>(smem + L::stat + (n_step & (BKV_DESCS - 1)) * 1024) + half * 64;
            ok = warp_wait(bar_s, ni & 1);
            if (!ok) break;
            tc_fence_after();
            if (f & BKV_FLUSH) flush(d.w, f);                 // (every warp has left the pair before: its sums have been written)
            uint32_t r[64];
            if (act) {
                uint32_t(&r0)[32] = *reinterpret_cast<uint32_t(*)[32]>(r);
                uint32_t(&r1)[32] = *reinterpret_cast<uint32_t(*)[32]>(r + 32);
                tmem_ld32(t_s, r0);
                tmem_ld32(t_s + 32, r1);
                tmem_ld_wait();
                if (blk_end > half * 64 || !(f & (BKV_SEL0 << u))) {          // not all of them behind the own block and seeing it
                    const int lo = (own ? kt * 64 + (quad & 1) * 32 + lane - d.x : blk_end) - half * 64;
                    const int hi = (f & (BKV_SEL0 << u)) ? 64 : blk_end - half * 64;
#pragma unroll
                    for (int e = 0; e < 64; ++e)
                        if (e < lo || e >= hi) r[e] = 0xff800000u;
                }
                const uint64_t sc2 = pack2(sl2, sl2);
#pragma unroll
                for (int h = 0; h < 2; ++h) {                 // (in halves: what is held in registers has to fit)
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const int e = h * 16 + i;
                        const float4 l4 = *reinterpret_cast<const float4*>(st + 2 * e);
                        float x0, x1, x2, x3;
                        unpack2(fma2(pack2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), sc2, pack2(l4.x, l4.y)), x0, x1);
                        unpack2(fma2(pack2(__uint_as_float(r[2 * e + 2]), __uint_as_float(r[2 * e + 3])), sc2, pack2(l4.z, l4.w)), x2, x3);
                        x0 = ex2(x0), x1 = ex2(x1), x2 = ex2(x2), x3 = ex2(x3);
                        r[2 * e] = __float_as_uint(x0), r[2 * e + 1] = __float_as_uint(x1);
                        r[2 * e + 2] = __float_as_uint(x2), r[2 * e + 3] = __float_as_uint(x3);
                        pk[i] = pack_bf16(x0, x1);
                        pk[i + 1] = pack_bf16(x2, x3);
                    }
                    tmem_st16(t_s + h * 16, pk);
                }
                tmem_st_wait();
            }
            tc_fence_before();
            arrive(bar_p);
            ok = warp_wait(bar_dp, ni & 1);
            if (!ok) break;
            tc_fence_after();
            if (act) {
                uint64_t sum = 0;
                auto gradients = [&](auto behind) {
                    constexpr bool later = decltype(behind)::value;
                    uint32_t x0[32], x1[32];
                    tmem_ld32(t_dp, x0);
                    tmem_ld32(t_dp + 32, x1);
                    tmem_ld_wait();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t pk[16];
                        uint32_t(&x)[32] = h ? x1 : x0;
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {
                            const float4 d4 = *reinterpret_cast<const float4*>(st + 128 + h * 32 + 2 * e);
                            const uint32_t* p = r + h * 32 + 2 * e;
                            const uint64_t a = mul2(pack2(__uint_as_float(p[0]), __uint_as_float(p[1])),
                                                    add2(pack2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1])), pack2(d4.x, d4.y)));
                            const uint64_t c = mul2(pack2(__uint_as_float(p[2]), __uint_as_float(p[3])),
                                                    add2(pack2(__uint_as_float(x[2 * e + 2]), __uint_as_float(x[2 * e + 3])), pack2(d4.z, d4.w)));
                            pk[e] = close2(a);
                            pk[e + 1] = close2(c);
                            if (later) {
                                sum = add2(sum, add2(a, c));
                            } else {                              // queries of the own block do not count
                                float a0, a1, c0, c1;
                                unpack2(a, a0, a1);
                                unpack2(c, c0, c1);
                                const int at = half * 64 + h * 32 + 2 * e;
                                sum = add2(sum, add2(pack2(at >= blk_end ? a0 : 0.f, at + 1 >= blk_end ? a1 : 0.f),
                                                     pack2(at + 2 >= blk_end ? c0 : 0.f, at + 3 >= blk_end ? c1 : 0.f)));
                            }
                        }
                        tmem_st16(t_dp + h * 16, pk);
                    }
                };
                if (blk_end <= half * 64) gradients(std::true_type());       // all of them behind the own block
                else gradients(std::false_type());
                dn += hsum2(sum);
                tmem_st_wait();
            }
            tc_fence_before();
            arrive(bar_ds);
            release_step();
            ++ni;
            if (!(f & BKV_LAST)) continue;
            finish((f & (BKV_ANY0 << u)) != 0, true);
            if (ok) ok = warp_wait(bar_acc, pairs & 1);       // (a phase passes by every warp: some have blocks of dv only)
            if (!ok) break;
            ++pairs;
            flush(d.z, f);                                    // behind the products of the pair, which warp 4 has joined in: it has
            release_acc();                                    // written the sums of the pair before, also if this one is a single step
            if (warp == 4) {                                  // in front of its part in the next step, behind which others flush again
                if (f & BKV_SUMS) ok = warp_wait(bar_acc_free, pairs & 1);
                if (!ok) break;
                write_sums((f & BKV_SUMS) != 0);
            }
        }
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int DK, int DV>
static int launch_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                           const int* types_i, void* dq, void* dk, void* dv, float* delta, float* dnats_part, int B, int T,
                           int HQ, int HKV, int HN, int nbs, float scale, int own_chunk, int compat, cudaStream_t st) {
    const int NT = (T + 63) / 64, NTq = (T + ATT_BM - 1) / ATT_BM;
    const int TN = (T + nbs - 1) / nbs;
    if (NTq > 32767) {                                       // the dk, dv kernel keeps numbers of query tiles in 16 bits
        set_error("natsl_attn_bwd: T=%d is too long (max %d)", T, 32767 * ATT_BM);
        return NATSL_ERR_TOO_LARGE;
    }
    auto k1 = attn_bwd_dq_kernel<DK, DV>;
    const int per_head = (NT + 1) / 2, heads = HKV * B, blocks = per_head * heads;      // pairs of key tiles
    const bool few = blocks <= BKV_SMALL;
    const int halves = few && NT > 1 ? blocks : 0;
    auto k2 = few ? attn_bwd_dkdv_kernel<DK, DV, true> : attn_bwd_dkdv_kernel<DK, DV, false>;
    cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, DqSmem<DK, DV>::total);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvSmem<DK, DV>::total);
    if (e != cudaSuccess) {
        set_error("natsl_attn_bwd: cannot reserve %d B of shared memory (%s)", DkvSmem<DK, DV>::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mdo, mdq, mdk, mdv;
    int* status = nullptr;
    int rc = encode_bthd_map(&mq, q, B, T, HQ, DK, 128, "natsl_attn_bwd(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, HKV, DK, 64, "natsl_attn_bwd(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T, HKV, DV, 64, "natsl_attn_bwd(v)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mdo, d_o, B, T, HQ, DV, 128, "natsl_attn_bwd(do)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mdq, dq, B, T, HQ, DK, 32, "natsl_attn_bwd(dq)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mdk, dk, B, T, HKV, DK, 32, "natsl_attn_bwd(dk)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mdv, dv, B, T, HKV, DV, 32, "natsl_attn_bwd(dv)");
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    auto bf = [](const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); };
    const int own = own_chunk && !compat;
    k1<<<NTq * HQ * B, BDQ_THREADS, DqSmem<DK, DV>::total, st>>>(mq, mk, mv, mdo, mdq, bf(q), bf(o), bf(d_o), lse, types_i, delta, T, HQ, HKV,
                                                                 HN, TN, nbs, scale, own, HQ * B, status);
    rc = check_launch("natsl_attn_bwd (dq)");
    if (rc != NATSL_OK) return rc;
    k2<<<blocks + halves, BKV_THREADS, DkvSmem<DK, DV>::total, st>>>(mq, mk, mv, mdo, mdk, mdv, lse, delta, types_i, dnats_part, T, HQ,
                                                                     HKV, HN, TN, nbs, scale, own, heads, per_head, halves, status);
    return check_launch("natsl_attn_bwd (dk, dv)");
}

}  // namespace natsl

extern "C" int natsl_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                              const int32_t* types_i, void* dq, void* dk, void* dv, float* delta, float* dnats_part, int B,
                              int T, int HQ, int HKV, int HN, int DK, int DV, int nbs, float scale, int flags,
                              void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && v && o && d_o && lse && types_i && dq && dk && dv && delta && dnats_part, NATSL_ERR_NULL,
                  "natsl_attn_bwd: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && HQ > 0 && HKV > 0 && HN > 0 && HQ % HKV == 0 && HQ % HN == 0, NATSL_ERR_BAD_SHAPE,
                  "natsl_attn_bwd: bad shape B=%d T=%d HQ=%d HKV=%d HN=%d", B, T, HQ, HKV, HN);
    NATSL_REQUIRE(HQ / HKV <= 16, NATSL_ERR_UNSUPPORTED, "natsl_attn_bwd: at most 16 query heads per key/value head");
    NATSL_REQUIRE(nbs >= 64 && nbs % 64 == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_attn_bwd: nats_block_size must be a multiple of 64 (got %d)", nbs);
    NATSL_REQUIRE(HQ <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_attn_bwd: B and HQ must be <= 65535");
    const int own = (flags & NATSL_FLAG_ATTN_OWN_CHUNK) ? 1 : 0;
    const int compat = (flags & NATSL_FLAG_BWD_REFERENCE_COMPAT) ? 1 : 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define NATSL_AB_CASE(KK, VV) \
    if (DK == KK && DV == VV) \
        return launch_attn_bwd<KK, VV>(q, k, v, o, d_o, lse, types_i, dq, dk, dv, delta, dnats_part, B, T, HQ, HKV, HN, nbs, \
                                       scale, own, compat, st);
    NATSL_AB_CASE(64, 64)
    NATSL_AB_CASE(64, 128)
    NATSL_AB_CASE(128, 64)
    NATSL_AB_CASE(128, 128)
#undef NATSL_AB_CASE
    set_error("natsl_attn_bwd: unsupported head dims DK=%d DV=%d (64 or 128 each)", DK, DV);
    return NATSL_ERR_UNSUPPORTED;
}
