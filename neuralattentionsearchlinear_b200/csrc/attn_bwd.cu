// Backward of the chunk-masked softmax branch (src/nats/ops/attns/attns.py:1562-1759; preprocess :357-372,
// dq :383-708, dk/dv :719-982).  Key s is visible to query t when its block is softmax-selected and lies
// entirely before t, or when both are in the same block and s <= t (the forward's mask).  With
//     p = exp2(scale*log2(e) * q.k - lse),   delta = rowsum(o * do),   ds = p * (do.v - delta)
// the gradients are dq = scale * ds k, dk = scale * ds^T q, dv = p^T do.
//
// Two kernels on the 5th-generation tensor cores, both deterministic (no atomics; every reduction has a fixed order).
// Warp roles as in the forward (320 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 softmax with 16 query
// rows each, four threads per row.  All score tiles are 128 queries x 64 keys with the queries in the TMEM lanes.
//   attn_bwd_dq_kernel    one CTA per (128 queries, query head), two per SM: walks the visible 64-key tiles, dq stays in
//                         TMEM; also writes delta (the preprocess kernel of the reference folded in).  ds goes back to
//                         TMEM (over do.v) as the A operand of ds k.
//   attn_bwd_dkdv_kernel  one CTA per two selected 64-key tiles of a key/value head (walks the 128-query tiles that see
//                         either) or per eight unselected ones (own blocks only); accumulates dk^T and dv^T (head dim in
//                         the lanes, keys in the columns) of two key tiles in TMEM; p and ds go to shared memory as the B
//                         operands of do^T p and q^T ds.  It also sums ds over the later blocks' queries: the reference's
//                         `dnats` column for the softmax branch (attns.py:922, 975-978), per (64-key tile, query head).
// `compat` reproduces the reference's default backward, which drops every own-block entry of ds and p
// (attns.py:590-591, 631-633, 842, 884 with the flag passed at mixed_attn_gdn.py:237) while lse and delta still
// come from the full forward.
// Every mbarrier wait has an iteration limit; on expiry the CTA records a status, stops issuing work, still frees its
// TMEM and returns.
#include "attn_tc.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr float kLog2e = 1.4426950408889634f;

// ------------------------------------------------------------------------------------------------- dq
template <int DK, int DV>
struct DqSmem {
    // 128 / 128: one V stage (its tile is free as soon as do.v is done) keeps the CTA at half an SM's shared memory
    static constexpr int VST = DK + DV == 256 ? 1 : 2;
    static constexpr int q = 0;                               // DK/64 sub-tiles [128][64]; at the end the dq staging
    static constexpr int dos = q + 128 * DK * 2;              // DV/64 sub-tiles [128][64]
    static constexpr int k = dos + 128 * DV * 2;              // 2 stages x DK/64 sub-tiles [64][64]
    static constexpr int v = k + 2 * 64 * DK * 2;             // VST stages x DV/64 sub-tiles [64][64]
    static constexpr int bars = v + VST * 64 * DV * 2;
    static constexpr int list = bars + 160;                   // visible key tiles (16 bits each), NT entries
    static int total(int NT) { return list + ((NT * 2 + 15) & ~15); }
};

template <int DK, int DV>
__global__ void __launch_bounds__(TC_THREADS, 2)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                   const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse,
                   const int* __restrict__ types_i, __nv_bfloat16* __restrict__ dq, float* __restrict__ delta_out, int T, int HQ,
                   int HKV, int HN, int TN, int nbs, float scale, int own, int* status) {
    using L = DqSmem<DK, DV>;
    constexpr int VST = L::VST;
    constexpr uint32_t C_S = 0, C_DP = 64, C_DQ = 128;        // TMEM columns: scores; do.v, then ds; dq
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int it = (int)gridDim.x - 1 - (int)blockIdx.x;      // heavy (late) query tiles first
    const int hq = blockIdx.y, b = blockIdx.z;
    const int hkv = hq / (HQ / HKV), hn = hq / (HQ / HN);
    const int q0 = it * ATT_BM;
    const int* selp = types_i + ((long)b * TN * HN + hn) * 2;  // column 0
    const long tstride = (long)HN * 2;
    const uint32_t s_q = sbase + L::q, s_do = sbase + L::dos, s_k = sbase + L::k, s_v = sbase + L::v;
    const uint32_t bar0 = sbase + L::bars;
    const uint32_t bar_q = bar0, bar_k_full = bar0 + 8, bar_k_empty = bar0 + 24, bar_v_full = bar0 + 40, bar_v_empty = bar0 + 56,
                   bar_s = bar0 + 72, bar_dp = bar0 + 80, bar_s_free = bar0 + 88, bar_ds = bar0 + 96, bar_done = bar0 + 104;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 112);
    int* s_count = reinterpret_cast<int*>(smem + L::bars + 116);
    uint16_t* s_list = reinterpret_cast<uint16_t*>(smem + L::list);
    const int span0 = (q0 / nbs) * nbs / 64;                  // first key tile of the own span
    const int cpb = nbs / 64;

    if (tid == 0) {
        mbar_init(bar_q, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_k_full + 8 * i, 1);
            mbar_init(bar_k_empty + 8 * i, 1);
            mbar_init(bar_v_full + 8 * i, 1);
            mbar_init(bar_v_empty + 8 * i, 1);
        }
        mbar_init(bar_s, 1);
        mbar_init(bar_dp, 1);
        mbar_init(bar_s_free, 8);                             // one arrival per softmax warp
        mbar_init(bar_ds, 8);
        mbar_init(bar_done, 1);
        mbar_fence_init();
        mbar_expect_tx(bar_q, 128 * (DK + DV) * 2);
#pragma unroll
        for (int sub = 0; sub < DK / 64; ++sub) tma_load_4d(s_q + sub * 16384, &map_q, sub * 64, hq, q0, b, bar_q);
#pragma unroll
        for (int sub = 0; sub < DV / 64; ++sub) tma_load_4d(s_do + sub * 16384, &map_do, sub * 64, hq, q0, b, bar_q);
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), TC_TMEM_COLS);
    if (warp == 2) {
        // visible key tiles in ascending order: sub-tiles of selected blocks before the own span, then the own span
        // (whose entries are masked per element)
        const int n_cand = min((q0 + ATT_BM + 63) / 64, (T + 63) / 64);
        int count = 0;
#pragma unroll 1
        for (int base = 0; base < n_cand; base += 32) {
            const int kt = base + lane;
            const bool vis = kt < n_cand && (kt >= span0 || selp[(long)(kt / cpb) * tstride] != 0);
            const unsigned m = __ballot_sync(0xffffffffu, vis);
            if (vis) s_list[count + __popc(m & ((1u << lane) - 1))] = (uint16_t)kt;
            count += __popc(m);
        }
        if (lane == 0) *s_count = count;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int n_tiles = *s_count;                             // >= 1: the own span is never empty
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
#pragma unroll 1
        for (int j = 0; ok && j < n_tiles; ++j) {
            const int ks = j & 1, vs = j % VST, t0 = s_list[j] * 64;
            if (j >= 2) ok = warp_wait(bar_k_empty + ks * 8, ((j >> 1) - 1) & 1);
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar_k_full + ks * 8, 64 * DK * 2);
#pragma unroll
                for (int sub = 0; sub < DK / 64; ++sub)
                    tma_load_4d(s_k + ks * (64 * DK * 2) + sub * 8192, &map_k, sub * 64, hkv, t0, b, bar_k_full + ks * 8);
#pragma unroll
                for (int sub = 0; sub < DV / 64; ++sub) tma_prefetch_4d(&map_v, sub * 64, hkv, t0, b);
            }
            __syncwarp();
            if (j >= VST) ok = warp_wait(bar_v_empty + vs * 8, ((j / VST) - 1) & 1);
            if (!ok) break;
            if (lane == 0) {
                mbar_expect_tx(bar_v_full + vs * 8, 64 * DV * 2);
#pragma unroll
                for (int sub = 0; sub < DV / 64; ++sub)
                    tma_load_4d(s_v + vs * (64 * DV * 2) + sub * 8192, &map_v, sub * 64, hkv, t0, b, bar_v_full + vs * 8);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t id_s = umma_idesc_bf16(128, 64, false);
        constexpr uint32_t id_dq = umma_idesc_bf16(128, DK, true);
        auto issue_s = [&](int j) {                           // S = Q K_j^T
            const uint32_t kt = s_k + (j & 1) * (64 * DK * 2);
            const uint32_t ql = umma_desc_lo(s_q, 16), kl = umma_desc_lo(kt, 16);
#pragma unroll
            for (int h = 0; h < DK / 64; ++h) umma_ss_x4<2, 2>(tmem + C_S, ql + h * 1024, kl + h * 512, id_s, h > 0);
            umma_commit(bar_s);
        };
        auto issue_dp = [&](int j) {                          // dO V_j^T
            const uint32_t vt = s_v + (j % VST) * (64 * DV * 2);
            const uint32_t dl = umma_desc_lo(s_do, 16), vl = umma_desc_lo(vt, 16);
#pragma unroll
            for (int h = 0; h < DV / 64; ++h) umma_ss_x4<2, 2>(tmem + C_DP, dl + h * 1024, vl + h * 512, id_s, h > 0);
            umma_commit(bar_dp);
            umma_commit(bar_v_empty + (j % VST) * 8);
        };
        ok = warp_wait(bar_q, 0);
        if (ok) ok = warp_wait(bar_k_full, 0);
        if (ok) {
            tc_fence_after();
            issue_s(0);
        }
        if (ok) ok = warp_wait(bar_v_full, 0);
        if (ok) {
            tc_fence_after();
            issue_dp(0);
        }
#pragma unroll 1
        for (int j = 0; ok && j < n_tiles; ++j) {
            const int jn = j + 1;
            if (jn < n_tiles) {                               // the next scores as soon as these have been read
                ok = warp_wait(bar_k_full + (jn & 1) * 8, (jn >> 1) & 1);
                if (ok) ok = warp_wait(bar_s_free, j & 1);
                if (!ok) break;
                tc_fence_after();
                issue_s(jn);
            }
            ok = warp_wait(bar_ds, j & 1);
            if (!ok) break;
            tc_fence_after();
            const uint32_t kt = s_k + (j & 1) * (64 * DK * 2);
            umma_ts_x4<128>(tmem + C_DQ, tmem + C_DP, umma_desc_lo(kt, 8192), id_dq, j > 0);
            umma_commit(jn < n_tiles ? bar_k_empty + (j & 1) * 8 : bar_done);
            if (jn < n_tiles) {
                ok = warp_wait(bar_v_full + (jn % VST) * 8, (jn / VST) & 1);
                if (!ok) break;
                tc_fence_after();
                issue_dp(jn);                                 // behind ds k in the tensor pipe: ds may be overwritten
            }
        }
    } else {
        // ------------------------------------------------------------ softmax (8 warps)
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int row_a = quad * 32 + half * 16 + (lane >> 2), row_b = row_a + 8;
        const int cq = (lane & 3) * 2;
        const int t_a = q0 + row_a, t_b = q0 + row_b;
        const uint32_t t_rows = tmem + ((uint32_t)(quad * 32 + half * 16) << 16);
        const float sl2 = scale * kLog2e;
        // delta = rowsum(o * do): four threads per row
        auto row_delta = [&](int t) -> float {
            float s = 0.f;
            if (t < T) {
                const long off = (((long)b * T + t) * HQ + hq) * DV + (lane & 3) * 8;
#pragma unroll
                for (int c = 0; c < DV / 32; ++c) {
                    const uint4 x = *reinterpret_cast<const uint4*>(o + off + c * 32);
                    const uint4 y = *reinterpret_cast<const uint4*>(d_o + off + c * 32);
                    const uint32_t* xw = reinterpret_cast<const uint32_t*>(&x);
                    const uint32_t* yw = reinterpret_cast<const uint32_t*>(&y);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 u = unpack_bf16(xw[e]), w = unpack_bf16(yw[e]);
                        s += u.x * w.x + u.y * w.y;
                    }
                }
            }
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            return s;
        };
        const float del_a = row_delta(t_a), del_b = row_delta(t_b);
        float lse_a = 0.f, lse_b = 0.f;
        if (t_a < T) lse_a = lse[((long)b * T + t_a) * HQ + hq];
        if (t_b < T) lse_b = lse[((long)b * T + t_b) * HQ + hq];
        if ((lane & 3) == 0) {
            if (t_a < T) delta_out[((long)b * T + t_a) * HQ + hq] = del_a;
            if (t_b < T) delta_out[((long)b * T + t_b) * HQ + hq] = del_b;
        }
#pragma unroll 1
        for (int j = 0; j < n_tiles; ++j) {
            ok = warp_wait(bar_s, j & 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t sr[32], pr[16];
            tmem_ld_16x256b_x8(t_rows + C_S, sr);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_s_free);
            const int kt = s_list[j];
            if (kt >= span0) {
                // own-span tile: per row the visible keys are columns [0, limit] (attn_walk.cuh: visible()); an invisible
                // score becomes -inf, its p zero
                const int s0 = kt * 64, blk = s0 / nbs, blk_end = (blk + 1) * nbs;
                const bool selb = selp[(long)blk * tstride] != 0;
                int lim_a = T - 1 - s0, lim_b = lim_a;
                if (t_a < blk_end) lim_a = own ? min(lim_a, t_a - s0) : -1;
                else if (!selb) lim_a = -1;
                if (t_b < blk_end) lim_b = own ? min(lim_b, t_b - s0) : -1;
                else if (!selb) lim_b = -1;
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int c = 8 * k + cq + e;
                        if (c > lim_a) sr[4 * k + e] = 0xff800000u;
                        if (c > lim_b) sr[4 * k + 2 + e] = 0xff800000u;
                    }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    sr[4 * k + e] = __float_as_uint(ex2(fmaf(__uint_as_float(sr[4 * k + e]), sl2, (e >> 1) ? -lse_b : -lse_a)));
            ok = warp_wait(bar_dp, j & 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t dr[32];
            tmem_ld_16x256b_x8(t_rows + C_DP, dr);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                pr[2 * k] = pack_bf16(__uint_as_float(sr[4 * k]) * (__uint_as_float(dr[4 * k]) - del_a),
                                      __uint_as_float(sr[4 * k + 1]) * (__uint_as_float(dr[4 * k + 1]) - del_a));
                pr[2 * k + 1] = pack_bf16(__uint_as_float(sr[4 * k + 2]) * (__uint_as_float(dr[4 * k + 2]) - del_b),
                                          __uint_as_float(sr[4 * k + 3]) * (__uint_as_float(dr[4 * k + 3]) - del_b));
            }
            tmem_st_16x128b_x8(t_rows + C_DP, pr);            // ds over the first 32 columns of do.v
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_ds);
        }
        if (ok) ok = warp_wait(bar_done, 0);
        unsigned char* stage = smem + L::q;
        if (ok) {
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < DK; c0 += 64) {
                uint32_t r[32];
                tmem_ld_16x256b_x8(t_rows + C_DQ + c0, r);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int chunk = (c0 >> 3) + k;
                    *reinterpret_cast<uint32_t*>(stage + swz<DK * 2>(row_a, chunk) + (lane & 3) * 4) =
                        pack_bf16(__uint_as_float(r[4 * k]) * scale, __uint_as_float(r[4 * k + 1]) * scale);
                    *reinterpret_cast<uint32_t*>(stage + swz<DK * 2>(row_b, chunk) + (lane & 3) * 4) =
                        pack_bf16(__uint_as_float(r[4 * k + 2]) * scale, __uint_as_float(r[4 * k + 3]) * scale);
                }
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");       // every softmax warp reaches it, also after a failed wait
        if (ok)
            store_tile<128, DK, 256>(stage, dq + (((long)b * T + q0) * HQ + hq) * DK, (long)HQ * DK, min(128, T - q0), tid - 64);
    }
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, TC_TMEM_COLS);
}

// ------------------------------------------------------------------------------------------------- dk, dv
constexpr int BKV_MAXG = 16;
template <int DK, int DV>
struct DkvSmem {
    // A stage is [do | q], both as [128][64] sub-tiles.  With a head dim of 64 the M = 128 products read the 64 columns
    // behind the tile as well (the next sub-tile, always inside the buffers) and those result rows are never used.
    static constexpr int stage_bytes = 128 * (DK + DV) * 2;
    static constexpr int stage = 0;                           // 2 stages
    static constexpr int kv = stage + 2 * stage_bytes;        // per key tile: DK/64 + DV/64 sub-tiles [64][64]
    static constexpr int kv_bytes = 64 * (DK + DV) * 2;
    static constexpr int p = kv + 2 * kv_bytes;               // p [128 queries][64 keys]
    static constexpr int ds = p + 16384;                      // ds, same layout
    static constexpr int dn = ds + 16384;                     // dnats parts [2 tiles][16 heads][8 warps]
    static constexpr int last = dn + 2 * BKV_MAXG * 8 * 4;    // last query tile [2 tiles][16 heads]
    static constexpr int tiles = last + 2 * BKV_MAXG * 4;     // key tiles of this CTA [8]
    static constexpr int bars = tiles + 32;
    static constexpr int total = bars + 96;
    static_assert(total <= 227 * 1024, "one CTA per SM");
};

// What a CTA walks: for every query head of the group the query tiles that see either key tile, and inside a query
// tile the key tiles that it sees.  All roles step through the same sequence.
struct DkvWalk {
    const int* last;                                          // shared memory [2][16]; -1: no query tile
    int first[2];
    int G;
    int gi, qt, u;
    __device__ __forceinline__ bool active(int uu) const { return qt >= first[uu] && qt <= last[uu * BKV_MAXG + gi]; }
    __device__ __forceinline__ void enter() {                 // first query tile of head gi
        const int l0 = last[gi], l1 = last[BKV_MAXG + gi];
        qt = min(l0 >= first[0] ? first[0] : 0x7fffffff, l1 >= first[1] ? first[1] : 0x7fffffff);
        u = 0;
    }
    // moves to the first (gi, qt, u) at or after the current one; false at the end
    __device__ __forceinline__ bool settle() {
#pragma unroll 1
        while (gi < G) {
            const int hi = max(last[gi], last[BKV_MAXG + gi]);
#pragma unroll 1
            for (; qt <= hi; ++qt, u = 0) {
                if (u == 0 && active(0)) return true;
                if (u <= 1 && active(1)) {
                    u = 1;
                    return true;
                }
            }
            if (++gi < G) enter();
        }
        return false;
    }
    __device__ __forceinline__ bool begin() {
        gi = 0;
        enter();
        return settle();
    }
    __device__ __forceinline__ bool next() {
        ++u;
        return settle();
    }
    __device__ __forceinline__ bool next_query() {
        u = 2;
        return settle();
    }
    __device__ __forceinline__ bool first_of_query() const { return u == 0 || !active(0); }
    __device__ __forceinline__ bool last_of_query() const { return u == 1 || !active(1); }
};

// The key tiles of unselected blocks, one after the other: only queries of their own block see them.
constexpr int BKV_OWN = 8;                                    // tiles per CTA
struct OwnWalk {
    const volatile int* tiles;
    int n, G, nbs, NTq;
    int u, gi, qt, last;
    __device__ __forceinline__ void enter() {
        const int k0 = tiles[u] * 64;
        qt = k0 / ATT_BM;
        last = min(((k0 / nbs + 1) * nbs - 1) / ATT_BM, NTq - 1);
    }
    __device__ __forceinline__ bool begin() {
        u = gi = 0;
        if (n > 0) enter();
        return n > 0;
    }
    __device__ __forceinline__ bool next() {
        if (++qt > last) {
            if (++gi == G) {
                gi = 0;
                if (++u == n) return false;
            }
            enter();
        }
        return true;
    }
    __device__ __forceinline__ bool first_of_tile() const { return gi == 0 && qt == tiles[u] * 64 / ATT_BM; }
};

// Heads whose CTAs are interleaved, heaviest first: the last CTAs to start are then light ones, and q and do of that many
// heads (2 MB each at 4096 x 128) stay in L2 for the CTAs of a head that run at the same time.
constexpr int BKV_HEADS = 32;

template <int DK, int DV>
__global__ void __launch_bounds__(TC_THREADS, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                     const float* __restrict__ lse, const float* __restrict__ delta, const int* __restrict__ types_i,
                     __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, float* __restrict__ dnats_part, int T, int HQ,
                     int HKV, int HN, int TN, int nbs, float scale, int own, int heads, int ctas_per_head, int* status) {
    using L = DkvSmem<DK, DV>;
    // TMEM: scores 2 x 64 columns, do.v 2 x 64, then two accumulator pairs dv^T (64), dk^T (64)
    constexpr uint32_t C_S = 0, C_DP = 128, C_ACC = 256;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int hbase = (int)blockIdx.x / (BKV_HEADS * ctas_per_head) * BKV_HEADS, hcount = min(BKV_HEADS, heads - hbase);
    const int within = (int)blockIdx.x - hbase * ctas_per_head;
    const int item = within / hcount, head = hbase + within % hcount;
    const int hkv = head % HKV, b = head / HKV;
    const int G = HQ / HKV, cpb = nbs / 64;
    const int NT = (T + 63) / 64, NTq = (T + ATT_BM - 1) / ATT_BM;
    float* s_dn = reinterpret_cast<float*>(smem + L::dn);
    int* s_last = reinterpret_cast<int*>(smem + L::last);
    volatile int* s_tile = reinterpret_cast<volatile int*>(smem + L::tiles);
    const uint32_t bar0 = sbase + L::bars;
    const uint32_t bar_full = bar0, bar_empty = bar0 + 16, bar_kv = bar0 + 32, bar_s = bar0 + 48, bar_p = bar0 + 64, bar_acc = bar0 + 72;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::bars + 80);
    volatile int* s_nsel = reinterpret_cast<volatile int*>(smem + L::bars + 84);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 1);
            mbar_init(bar_kv + 8 * i, 1);
            mbar_init(bar_s + 8 * i, 1);
        }
        mbar_init(bar_p, 8);                                  // one arrival per softmax warp
        mbar_init(bar_acc, 1);
        mbar_fence_init();
    }
    for (int i = tid; i < 2 * BKV_MAXG * 8; i += TC_THREADS) s_dn[i] = 0.f;
    if (warp == 2) {
        // Key tiles in the order: those of selected blocks (of any head of the group), then the others.  The first
        // ceil(n / 2) CTAs of a head take two selected tiles each: neighbours see nearly the same queries, so the pair
        // shares the loads of q and do (64 KB per 128 x 64 scores of one tile).  The next ones take eight unselected
        // tiles, the rest of the CTAs have nothing to do.
        auto selected = [&](int kt) -> bool {
            bool s = false;
#pragma unroll 1
            for (int gi = 0; gi < G; ++gi) s |= types_i[(((long)b * TN + kt / cpb) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0;
            return s;
        };
        constexpr int KEEP = 4;                               // ballots kept from the counting pass (8192 tokens)
        unsigned kept[KEEP];
        int n_sel = 0;
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            kept[i] = __ballot_sync(0xffffffffu, i * 32 + lane < NT && selected(i * 32 + lane));
            n_sel += __popc(kept[i]);
        }
#pragma unroll 1
        for (int base = KEEP * 32; base < NT; base += 32)
            n_sel += __popc(__ballot_sync(0xffffffffu, base + lane < NT && selected(base + lane)));
        const int n_pairs = (n_sel + 1) / 2;
        const bool mine_sel = item < n_pairs;
        const int r0 = mine_sel ? 2 * item : (item - n_pairs) * BKV_OWN;
        const int want = mine_sel ? 2 : BKV_OWN;              // ranks [r0, r0 + want) among the tiles of that kind
        if (lane < BKV_OWN) s_tile[lane] = -1;
        __syncwarp();
        int cnt = 0;
        auto place = [&](int base, unsigned ms) {
            const unsigned in = base + 32 <= NT ? 0xffffffffu : (1u << (NT - base)) - 1;
            const unsigned m = mine_sel ? ms : in & ~ms;
            const int r = cnt + __popc(m & ((1u << lane) - 1)) - r0;
            if (((m >> lane) & 1) && r >= 0 && r < want) s_tile[r] = base + lane;
            cnt += __popc(m);
        };
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (i * 32 < NT) place(i * 32, kept[i]);
#pragma unroll 1
        for (int base = KEEP * 32; base < NT && cnt < r0 + want; base += 32)
            place(base, __ballot_sync(0xffffffffu, base + lane < NT && selected(base + lane)));
        __syncwarp();
        if (lane == 0) *s_nsel = n_sel;
        // query tiles [first, last] of every (selected tile, head): the own block's from the keys on, the later ones if the
        // head selected the block
#pragma unroll 1
        for (int i = lane; mine_sel && i < 2 * BKV_MAXG; i += 32) {
            const int kt = s_tile[i / BKV_MAXG], gi = i % BKV_MAXG;
            int last = -1;
            if (kt >= 0 && gi < G) {
                const int blk = kt / cpb, blk_end = (blk + 1) * nbs;
                const bool s = G == 1 || types_i[(((long)b * TN + blk) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0;
                if (s && blk_end < T) last = NTq - 1;
                else if (own) last = min((blk_end - 1) / ATT_BM, NTq - 1);
            }
            s_last[i] = last;
        }
    }
    __syncthreads();
    const int n_pairs = (*s_nsel + 1) / 2;
    const bool paired = item < n_pairs;
    if (s_tile[0] < 0) return;                                // no tile of either kind is left for this CTA
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int tile[2] = {s_tile[0], s_tile[1]};
    int n_own = 0;
    while (n_own < BKV_OWN && s_tile[n_own] >= 0) ++n_own;
    DkvWalk w;
    w.last = s_last;
    w.G = G;
#pragma unroll
    for (int u = 0; u < 2; ++u) w.first[u] = tile[u] < 0 ? NTq : own ? tile[u] * 64 / ATT_BM : ((tile[u] / cpb + 1) * nbs) / ATT_BM;
    auto has_items = [&](int u) -> bool {
#pragma unroll 1
        for (int gi = 0; gi < G; ++gi)
            if (s_last[u * BKV_MAXG + gi] >= w.first[u]) return true;
        return false;
    };
    OwnWalk ow;
    ow.tiles = s_tile;
    ow.n = own ? n_own : 0;
    ow.G = G;
    ow.nbs = nbs;
    ow.NTq = NTq;
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        auto load_kv = [&](int slot, int kt, uint32_t bar) {
            const uint32_t dst = sbase + L::kv + slot * L::kv_bytes;
#pragma unroll
            for (int sub = 0; sub < DK / 64; ++sub) tma_load_4d(dst + sub * 8192, &map_k, sub * 64, hkv, kt * 64, b, bar);
#pragma unroll
            for (int sub = 0; sub < DV / 64; ++sub)
                tma_load_4d(dst + 64 * DK * 2 + sub * 8192, &map_v, sub * 64, hkv, kt * 64, b, bar);
        };
        auto load_q = [&](int stg, int gi, int qt) {
            const uint32_t base = sbase + L::stage + stg * L::stage_bytes;
#pragma unroll
            for (int sub = 0; sub < DK / 64; ++sub)
                tma_load_4d(base + 128 * DV * 2 + sub * 16384, &map_q, sub * 64, hkv * G + gi, qt * ATT_BM, b, bar_full + stg * 8);
#pragma unroll
            for (int sub = 0; sub < DV / 64; ++sub)
                tma_load_4d(base + sub * 16384, &map_do, sub * 64, hkv * G + gi, qt * ATT_BM, b, bar_full + stg * 8);
        };
        int n = 0;
        if (paired) {
            if (lane == 0)
                for (int u = 0; u < 2; ++u)
                    if (has_items(u)) {
                        mbar_expect_tx(bar_kv + u * 8, L::kv_bytes);
                        load_kv(u, tile[u], bar_kv + u * 8);
                    }
            __syncwarp();
#pragma unroll 1
            for (bool more = w.begin(); more; more = w.next_query(), ++n) {
                const int stg = n & 1;
                if (n >= 2) ok = warp_wait(bar_empty + stg * 8, ((n >> 1) - 1) & 1);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(bar_full + stg * 8, L::stage_bytes);
                    load_q(stg, w.gi, w.qt);
                    if (w.qt + 2 < NTq) {                     // warm L2 for the tile this stage most likely receives next
#pragma unroll
                        for (int sub = 0; sub < DK / 64; ++sub)
                            tma_prefetch_4d(&map_q, sub * 64, hkv * G + w.gi, (w.qt + 2) * ATT_BM, b);
#pragma unroll
                        for (int sub = 0; sub < DV / 64; ++sub)
                            tma_prefetch_4d(&map_do, sub * 64, hkv * G + w.gi, (w.qt + 2) * ATT_BM, b);
                    }
                }
                __syncwarp();
            }
        } else {
#pragma unroll 1
            for (bool more = ow.begin(); more; more = ow.next(), ++n) {
                const int stg = n & 1;
                if (n >= 2) ok = warp_wait(bar_empty + stg * 8, ((n >> 1) - 1) & 1);
                if (!ok) break;
                if (lane == 0) {                              // every item brings its own copy of k and v
                    mbar_expect_tx(bar_full + stg * 8, L::stage_bytes + L::kv_bytes);
                    load_kv(stg, s_tile[ow.u], bar_full + stg * 8);
                    load_q(stg, ow.gi, ow.qt);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        constexpr uint32_t id_s = umma_idesc_bf16(128, 64, false);
        constexpr uint32_t id_acc = umma_idesc_bf16(128, 64, true) | (1u << 15);         // A MN-major too
        auto scores = [&](int n, int stg, int kv) {           // S and dO V^T of item n into buffer n & 1
            stg = __shfl_sync(0xffffffffu, stg, 0);
            kv = __shfl_sync(0xffffffffu, kv, 0);
            n = __shfl_sync(0xffffffffu, n, 0) & 1;
            tc_fence_after();
            const uint32_t dl = umma_desc_lo(sbase + L::stage + stg * L::stage_bytes, 16), ql = dl + (128 * DV * 2 >> 4);
            const uint32_t kl = umma_desc_lo(sbase + L::kv + kv * L::kv_bytes, 16), vl = kl + (64 * DK * 2 >> 4);
#pragma unroll
            for (int h = 0; h < DK / 64; ++h) umma_ss_x4<2, 2>(tmem + C_S + n * 64, ql + h * 1024, kl + h * 512, id_s, h > 0);
#pragma unroll
            for (int h = 0; h < DV / 64; ++h) umma_ss_x4<2, 2>(tmem + C_DP + n * 64, dl + h * 1024, vl + h * 512, id_s, h > 0);
            umma_commit(bar_s + n * 8);
        };
        auto accumulate = [&](int stg, int slot, bool cont, bool release) {
            stg = __shfl_sync(0xffffffffu, stg, 0);
            slot = __shfl_sync(0xffffffffu, slot, 0);
            tc_fence_after();
            const uint32_t dl = umma_desc_lo(sbase + L::stage + stg * L::stage_bytes, 16384), ql = dl + (128 * DV * 2 >> 4);
            const uint32_t pl = umma_desc_lo(sbase + L::p, 8192), dsl = umma_desc_lo(sbase + L::ds, 8192);
            const uint32_t acc = tmem + C_ACC + slot * 128;
#pragma unroll
            for (int h = 0; h < 2; ++h)                       // dv^T += do^T p
                umma_ss_x4<128, 128>(acc, dl + h * 512, pl + h * 512, id_acc, cont || h > 0);
#pragma unroll
            for (int h = 0; h < 2; ++h)                       // dk^T += q^T ds
                umma_ss_x4<128, 128>(acc + 64, ql + h * 512, dsl + h * 512, id_acc, cont || h > 0);
            umma_commit(bar_acc);
            if (release) umma_commit(bar_empty + stg * 8);
        };
        if (paired) {
            DkvWalk a = w;                                    // one item ahead: scores
            bool more = w.begin(), ahead = a.begin();
            int na = 0, nq_a = -1, nq = -1;                   // items issued; query tiles entered by a / w
            bool kv_seen[2] = {false, false}, started[2] = {false, false};
            auto step_ahead = [&]() {
                if (a.first_of_query()) {
                    ++nq_a;
                    ok = warp_wait(bar_full + (nq_a & 1) * 8, (nq_a >> 1) & 1);
                }
                if (ok && !kv_seen[a.u]) ok = warp_wait(bar_kv + a.u * 8, 0);
                kv_seen[a.u] = true;
                if (ok) scores(na, nq_a & 1, a.u);
                ++na;
                ahead = a.next();
            };
            // The scores of the next item go ahead of this item's products (their buffer was read before bar_p of item
            // i - 1) unless their tiles are still on the way: the stage that the producer fills after them is the one
            // that these products release.  (One place that issues scores and one that issues products: inlined at every
            // turn of the sequence, with descriptors formed for each product, this warp had 150 KB of code.)
            auto ready = [&]() {
                return __all_sync(0xffffffffu, !a.first_of_query() || mbar_test_wait(bar_full + ((nq_a + 1) & 1) * 8, ((nq_a + 1) >> 1) & 1));
            };
#pragma unroll 1
            for (int i = 0; ok && more;) {
                if (ahead && na <= i + 1 && (na == i || ready())) {
                    step_ahead();
                    if (na == i + 1) continue;
                }
                if (ok) ok = warp_wait(bar_p, i & 1);
                if (!ok) break;
                if (w.first_of_query()) ++nq;
                accumulate(nq & 1, w.u, started[w.u], w.last_of_query());
                started[w.u] = true;
                more = w.next();
                ++i;
            }
        } else {
            OwnWalk a = ow;
            bool more = ow.begin(), ahead = a.begin();
            int na = 0;
            auto step_ahead = [&]() {
                ok = warp_wait(bar_full + (na & 1) * 8, (na >> 1) & 1);
                if (ok) scores(na, na & 1, na & 1);
                ++na;
                ahead = a.next();
            };
#pragma unroll 1
            for (int i = 0; ok && more;) {
                if (ahead && na <= i + 1 &&
                    (na == i || __all_sync(0xffffffffu, mbar_test_wait(bar_full + (na & 1) * 8, (na >> 1) & 1)))) {
                    step_ahead();
                    if (na == i + 1) continue;
                }
                // the accumulators of tile u - 2 were read before the softmax warps arrived here for the item before
                if (ok) ok = warp_wait(bar_p, i & 1);
                if (!ok) break;
                accumulate(i & 1, ow.u & 1, !ow.first_of_tile(), true);
                more = ow.next();
                ++i;
            }
        }
    } else {
        // ------------------------------------------------------------ softmax (8 warps)
        const int quad = warp & 3, half = (warp - 2) >> 2, sw = warp - 2;
        const int row_a = quad * 32 + half * 16 + (lane >> 2), row_b = row_a + 8;
        const int cq = (lane & 3) * 2;
        const uint32_t t_rows = tmem + ((uint32_t)(quad * 32 + half * 16) << 16);
        const float sl2 = scale * kLog2e;
        unsigned char* p_t = smem + L::p;
        unsigned char* ds_t = smem + L::ds;
        float lse_a = 0.f, lse_b = 0.f, del_a = 0.f, del_b = 0.f;
        auto load_rows = [&](int gi, int qt) {
            const int t_a = qt * ATT_BM + row_a, t_b = t_a + 8;
            const long r = ((long)b * T + t_a) * HQ + hkv * G + gi;
            lse_a = t_a < T ? lse[r] : 0.f;
            del_a = t_a < T ? delta[r] : 0.f;
            lse_b = t_b < T ? lse[r + 8L * HQ] : 0.f;
            del_b = t_b < T ? delta[r + 8L * HQ] : 0.f;
        };
        // p and ds of item i (key tile kt, query tile qt; `sel`: later blocks see the keys) into registers, bf16 pairs; adds
        // the ds of later blocks' queries to dn.  Returns once the products of the previous item have read p and ds.
        uint32_t sr[32];
        auto item_p = [&](int i, int kt, int qt, bool sel, float& dn) -> bool {
            bool ok = warp_wait(bar_s + (i & 1) * 8, (i >> 1) & 1);
            if (!ok) return false;
            tc_fence_after();
            uint32_t dr[32];
            tmem_ld_16x256b_x8(t_rows + C_S + (i & 1) * 64, sr);
            tmem_ld_16x256b_x8(t_rows + C_DP + (i & 1) * 64, dr);
            tmem_ld_wait();
            const int t_a = qt * ATT_BM + row_a, t_b = t_a + 8;
            const int s0 = kt * 64, blk_end = (kt / cpb + 1) * nbs;
            if (qt * ATT_BM < blk_end) {
                // rows of the own block see columns [0, t - s0], rows behind it all or none
                const int lim_a = t_a >= blk_end ? (sel ? 63 : -1) : (own ? t_a - s0 : -1);
                const int lim_b = t_b >= blk_end ? (sel ? 63 : -1) : (own ? t_b - s0 : -1);
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int c = 8 * k + cq + e;
                        if (c > lim_a) sr[4 * k + e] = 0xff800000u;
                        if (c > lim_b) sr[4 * k + 2 + e] = 0xff800000u;
                    }
            }
            float sum_a = 0.f, sum_b = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float p0 = ex2(fmaf(__uint_as_float(sr[4 * k]), sl2, -lse_a));
                const float p1 = ex2(fmaf(__uint_as_float(sr[4 * k + 1]), sl2, -lse_a));
                const float p2 = ex2(fmaf(__uint_as_float(sr[4 * k + 2]), sl2, -lse_b));
                const float p3 = ex2(fmaf(__uint_as_float(sr[4 * k + 3]), sl2, -lse_b));
                const float d0 = p0 * (__uint_as_float(dr[4 * k]) - del_a), d1 = p1 * (__uint_as_float(dr[4 * k + 1]) - del_a);
                const float d2 = p2 * (__uint_as_float(dr[4 * k + 2]) - del_b), d3 = p3 * (__uint_as_float(dr[4 * k + 3]) - del_b);
                sum_a += d0 + d1;
                sum_b += d2 + d3;
                sr[4 * k] = pack_bf16(p0, p1);
                sr[4 * k + 1] = pack_bf16(p2, p3);
                sr[4 * k + 2] = pack_bf16(d0, d1);
                sr[4 * k + 3] = pack_bf16(d2, d3);
            }
            dn += (t_a >= blk_end ? sum_a : 0.f) + (t_b >= blk_end ? sum_b : 0.f);
            if (i > 0) ok = warp_wait(bar_acc, (i - 1) & 1);
            return ok;
        };
        auto item_write = [&]() {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t oa = swz<128>(row_a, k) + (lane & 3) * 4, ob = swz<128>(row_b, k) + (lane & 3) * 4;
                *reinterpret_cast<uint32_t*>(p_t + oa) = sr[4 * k];
                *reinterpret_cast<uint32_t*>(p_t + ob) = sr[4 * k + 1];
                *reinterpret_cast<uint32_t*>(ds_t + oa) = sr[4 * k + 2];
                *reinterpret_cast<uint32_t*>(ds_t + ob) = sr[4 * k + 3];
            }
            fence_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p);
        };
        // dk, dv of key tile kt from accumulator pair `slot` (zeros without `any`): lane = head-dim index, columns = keys.
        // Transposed through the p and ds tiles, which no product reads at that time, so that the rows leave in 16-byte
        // pieces (two-byte stores straight from the registers took 8000 clocks a tile, most of an unselected tile's time).
        // Every softmax warp calls it, also after a failed wait (`good` false: nothing is read or stored).
        auto finish = [&](int kt, int slot, bool any, bool good) {
            const int d = quad * 32 + lane;
            const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + C_ACC + slot * 128 + half * 32;
            tc_fence_after();
            uint32_t r[32];
            if (good && quad * 32 < DV) {
                tmem_ld32(acc, r);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    *reinterpret_cast<__nv_bfloat16*>(p_t + swz<DV * 2>(half * 32 + c, d >> 3) + (d & 7) * 2) =
                        __float2bfloat16(any ? __uint_as_float(r[c]) : 0.f);
            }
            if (good && quad * 32 < DK) {
                tmem_ld32(acc + 64, r);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    *reinterpret_cast<__nv_bfloat16*>(ds_t + swz<DK * 2>(half * 32 + c, d >> 3) + (d & 7) * 2) =
                        __float2bfloat16(any ? __uint_as_float(r[c]) * scale : 0.f);
            }
            tc_fence_before();
            asm volatile("bar.sync 2, 256;" ::: "memory");
            const long tok = (long)b * T + kt * 64;
            const int n_valid = good ? min(64, T - kt * 64) : 0;
            store_tile<64, DV, 256>(p_t, dv + (tok * HKV + hkv) * DV, (long)HKV * DV, n_valid, tid - 64);
            store_tile<64, DK, 256>(ds_t, dk + (tok * HKV + hkv) * DK, (long)HKV * DK, n_valid, tid - 64);
            asm volatile("bar.sync 2, 256;" ::: "memory");
        };
        int i = 0;
        if (paired) {
            float dn[2] = {0.f, 0.f};
            auto flush = [&](int gi) {                        // one slot per (key tile, head, warp): a fixed order of summation
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    dn[u] = warp_sum(dn[u]);
                    if (lane == 0) s_dn[(u * BKV_MAXG + gi) * 8 + sw] = dn[u];
                    dn[u] = 0.f;
                }
            };
            int gi = 0;
#pragma unroll 1
            for (bool more = w.begin(); more; more = w.next(), ++i) {
                if (w.gi != gi) {
                    flush(gi);
                    gi = w.gi;
                }
                if (w.first_of_query()) load_rows(gi, w.qt);
                const int kt = w.u ? tile[1] : tile[0];
                // rows behind the own block are in the walk only where the head selected the block; in a tile that holds
                // both, the flag decides
                bool sel = true;
                if (G > 1 && w.qt * ATT_BM < (kt / cpb + 1) * nbs)
                    sel = types_i[(((long)b * TN + kt / cpb) * HN + (hkv * G + gi) / (HQ / HN)) * 2] != 0;
                float add = 0.f;
                ok = item_p(i, kt, w.qt, sel, add);
                if (!ok) break;
                item_write();
                if (w.u) dn[1] += add; else dn[0] += add;
            }
            flush(gi);
            if (ok && i > 0) ok = warp_wait(bar_acc, (i - 1) & 1);
#pragma unroll 1
            for (int u = 0; u < (tile[1] >= 0 ? 2 : 1); ++u) finish(s_tile[u], u, has_items(u), ok);
        } else if (!own) {
#pragma unroll 1
            for (int u = 0; u < n_own; ++u) finish(s_tile[u], 0, false, true);
        } else {
            int done = 0;                                     // tiles written
            float unused = 0.f;
            bool more = ow.begin();
#pragma unroll 1
            while (true) {
                if (more) {
                    load_rows(ow.gi, ow.qt);
                    if (ok) ok = item_p(i, s_tile[ow.u], ow.qt, false, unused);
                } else if (ok) {
                    ok = warp_wait(bar_acc, (i - 1) & 1);
                }
                if (!more || ow.u > done) {                   // the previous item was its tile's last
                    finish(s_tile[done], done & 1, true, ok);
                    ++done;
                }
                if (!more) break;
                if (ok) item_write();
                more = ow.next();
                ++i;
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");       // every softmax warp reaches it, also after a failed wait
        const int n_tiles = paired ? 2 : n_own;
#pragma unroll 1
        for (int e = tid - 64; e < n_tiles * G; e += 256) {
            const int u = e / G, gi = e % G;
            if (s_tile[u] < 0) continue;
            const float* p = s_dn + (u * BKV_MAXG + gi) * 8;
            dnats_part[((long)b * NT + s_tile[u]) * HQ + hkv * G + gi] =
                paired ? ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7])) : 0.f;
        }
    }
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
    const int smem = DqSmem<DK, DV>::total(NT);
    if (smem > 227 * 1024) {
        set_error("natsl_attn_bwd: T=%d needs %d B of shared memory (max %d)", T, smem, 227 * 1024);
        return NATSL_ERR_TOO_LARGE;
    }
    auto k1 = attn_bwd_dq_kernel<DK, DV>;
    auto k2 = attn_bwd_dkdv_kernel<DK, DV>;
    cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvSmem<DK, DV>::total);
    if (e != cudaSuccess) {
        set_error("natsl_attn_bwd: cannot reserve %d B of shared memory (%s)", smem, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mdo;
    int* status = nullptr;
    int rc = encode_bthd_map(&mq, q, B, T, HQ, DK, 128, "natsl_attn_bwd(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, HKV, DK, 64, "natsl_attn_bwd(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T, HKV, DV, 64, "natsl_attn_bwd(v)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mdo, d_o, B, T, HQ, DV, 128, "natsl_attn_bwd(do)");
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    auto bf = [](const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); };
    const int own = own_chunk && !compat;
    k1<<<dim3(NTq, HQ, B), TC_THREADS, smem, st>>>(mq, mk, mv, mdo, bf(o), bf(d_o), lse, types_i, reinterpret_cast<__nv_bfloat16*>(dq),
                                                  delta, T, HQ, HKV, HN, TN, nbs, scale, own, status);
    rc = check_launch("natsl_attn_bwd (dq)");
    if (rc != NATSL_OK) return rc;
    // ceil(n / 2) + ceil((NT - n) / 8) CTAs per head for n selected tiles, known on the device only
    const int per_head = NT / 2 + 1, heads = HKV * B;
    k2<<<per_head * heads, TC_THREADS, DkvSmem<DK, DV>::total, st>>>(
        mq, mk, mv, mdo, lse, delta, types_i, reinterpret_cast<__nv_bfloat16*>(dk), reinterpret_cast<__nv_bfloat16*>(dv), dnats_part, T,
        HQ, HKV, HN, TN, nbs, scale, own, heads, per_head, status);
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
