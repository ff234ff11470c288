// Gated-delta-rule recurrence AND chunk output in one walk for any of the built head dims (K in {64, 128}, value
// columns in slices of 32 or 64) and any nats_block_size: the counterpart of gdn_walk_tc.cu for shapes the tcgen05 kernel
// has no tiles for, and for few (batch, head) pairs, where slices of the value dim are what fills the SMs.
// One CTA per (batch, head, BV value columns) walks the 64-token chunks in order; per chunk c (S = state it reads):
//     v' = u - e^{carry} w S                                                                        (w warps)
//     o  = scale (rstd_q e^{g+carry} q S + P v')                                                    (q warps)
//     S <- e^{g_last+carry} S + k^T (v' rstd_k e^{g_last-g})      if the chunk updates the state     (w warps)
// which is src/nats/ops/common/chunk_delta_h.py:189-324 fused with src/nats/ops/common/chunk_o.py:124-215; with
// nats_block_size > 64 the chunks of an unselected block update a temporary state that is rolled back at its end
// (src/nats/ops/gated_delta_rule/fused_recurrent.py:221-228, 276-281).
// What bounds it: the serial chain of a chunk (w S -> v' -> k^T v'' -> bf16 copy of S), so its products run as small
// mma.sync steps of four warps (a tcgen05 round trip through TMEM costs more than these whole products), the output side
// runs on four other warps, and TMA keeps the next chunk's tiles in flight.  Against the recurrence and
// the output as two kernels the per-chunk states (K x V bf16 written and read) never leave the SM.
#include "tc_common.cuh"
#include "warp_gemm.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

// w warps 0-3, q warps 4-7.  With 32 columns (few CTAs, the chain is everything) a ninth warp issues the TMA loads; with 64
// columns warp 4, which has the least P v' work, does: nine warps would leave 96 registers a thread at two CTAs per SM
// and spill (262 against 168 us at B = 16, T = 4096, H = 16, K = V = 64; the ninth warp is worth 10 % at 32 columns).
template <int BV>
constexpr bool gw_tma_warp = BV == 32;
template <int BV>
constexpr int gw_threads = gw_tma_warp<BV> ? 288 : 256;

template <int K, int BV>
struct GwSmem {
    static constexpr int NST = 2;
    static constexpr int w = 0, q = w + 64 * K * 2, k = q + 64 * K * 2, p = k + 64 * K * 2, u = p + 8192;
    static constexpr int stage = u + 64 * BV * 2;
    static constexpr int sb = NST * stage;                    // bf16 copy of the state [K][BV]
    static constexpr int vs = sb + K * BV * 2;                // v'' [64][BV]   (v' replaces u in its stage)
    static constexpr int bars = vs + 64 * BV * 2;
    static constexpr int meta = bars + 64;                    // per chunk g_last, selected (float2), then the backup
    static int total(int NT, bool with_save) { return meta + NT * 8 + (with_save ? K * BV * 4 : 0); }
};

// Fragment loads from tiles of 64-column sub-tiles ([64 rows][64 columns] each, 128-byte swizzle: what TMA writes).
__device__ __forceinline__ void load_a_sub(uint32_t tile, int row0, int k0, int lane, uint32_t (&a)[4]) {
    load_a<128>(tile + (k0 >> 6) * 8192, row0, k0 & 63, lane, a);
}
__device__ __forceinline__ void load_a_t_sub(uint32_t tile, int m0, int k0, int lane, uint32_t (&a)[4]) {
    load_a_t<128>(tile + (m0 >> 6) * 8192, m0 & 63, k0, lane, a);
}

template <int K, int BV>
__global__ void __launch_bounds__(gw_threads<BV>, K == 64 && BV == 64 ? 2 : 1)
gdn_walk_mma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_q,
                    const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_u,
                    const __grid_constant__ CUtensorMap map_p, const float* __restrict__ gcs,
                    const float* __restrict__ krstd, const float* __restrict__ qrstd, const int* __restrict__ types_i,
                    const int* __restrict__ indices, const int* __restrict__ n_blocks, const float* __restrict__ h0,
                    __nv_bfloat16* __restrict__ o, float* __restrict__ ht, float* hstart, const void* __restrict__ last_types,
                    int last_f32, int last_stride, int T, int H, int HN, int V, int TN, int nbs, float scale, int decay, int trailing_quirk,
                    int* status) {
    using L = GwSmem<K, BV>;
    constexpr int MT = K / 64, NTL = BV / 8, NSUB = K / 64;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, qd = lane & 3;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int v0 = blockIdx.x * BV, h = blockIdx.y, b = blockIdx.z;
    const int hn = h / (H / HN);
    const int NT = (T + 63) / 64, cpb = nbs / 64;
    float2* s_meta = reinterpret_cast<float2*>(smem + L::meta);              // per chunk: g_last, selected
    float* save_p = reinterpret_cast<float*>(smem + L::meta + NT * 8);
    const uint32_t bar_full = sbase + L::bars, bar_empty = bar_full + 8 * L::NST;
    if (tid == 0) {
        for (int i = 0; i < L::NST; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 8);
        }
        mbar_fence_init();
    }
    for (int c = tid; c < NT; c += gw_threads<BV>) {
        s_meta[c] = make_float2(gcs[((long)b * T + min(c * 64 + 63, T - 1)) * H + h],
                                types_i[(((long)b * TN + c / cpb) * HN + hn) * 2 + 1] != 0 ? 1.f : 0.f);
    }
    __syncthreads();

    auto issue = [&](int c) {                               // one thread: all tiles of chunk c into stage c % NST
        const int t0 = c * 64;
        const bool act = cpb > 1 || s_meta[c].y != 0.f;
        const uint32_t full = bar_full + (c % L::NST) * 8, base = sbase + (c % L::NST) * L::stage;
        mbar_expect_tx(full, (act ? 3 : 2) * 64 * K * 2 + 8192 + 64 * BV * 2);
#pragma unroll
        for (int sub = 0; sub < NSUB; ++sub) {
            tma_load_4d(base + L::w + sub * 8192, &map_w, sub * 64, h, t0, b, full);
            tma_load_4d(base + L::q + sub * 8192, &map_q, sub * 64, h, t0, b, full);
            if (act) tma_load_4d(base + L::k + sub * 8192, &map_k, sub * 64, h, t0, b, full);
        }
        tma_load_4d(base + L::p, &map_p, 0, h, t0, b, full);
        tma_load_4d(base + L::u, &map_u, v0, h, t0, b, full);
    };
    constexpr bool kTmaWarp = gw_tma_warp<BV>;
    const bool loader = warp == (kTmaWarp ? 8 : 4) && lane == 0;
    if (loader) {
        prefetch_tensormap(&map_w); prefetch_tensormap(&map_q); prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_u); prefetch_tensormap(&map_p);
        for (int c = 0; c < L::NST && c < NT; ++c) issue(c);
    }
    if (kTmaWarp && warp == 8) {
        if (loader)
            for (int c = L::NST; c < NT; ++c) {
                if (!mbar_wait(bar_empty + (c % L::NST) * 8, (c / L::NST - 1) & 1, status)) break;
                issue(c);
            }
        return;
    }

    const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
    const int last_sel = nsel > 0 ? indices[(((long)b * TN + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
    const bool is_q = warp >= 4;
    const int r0 = (warp & 3) * 16, ra = r0 + gq, rb = ra + 8;              // token rows of this lane
    const int krow0 = warp * (K / 4);                                       // state rows of a w warp
    const uint32_t sb = sbase + L::sb;
    auto bar_all = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };

    float S[MT][NTL][4];
    if (!is_q) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                float2 lo = make_float2(0.f, 0.f), hi = lo;
                if (h0) {
                    const float* p = h0 + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + nt * 8 + qd * 2;
                    lo = *reinterpret_cast<const float2*>(p);
                    hi = *reinterpret_cast<const float2*>(p + 8L * V);
                }
                S[mt][nt][0] = lo.x; S[mt][nt][1] = lo.y; S[mt][nt][2] = hi.x; S[mt][nt][3] = hi.y;
            }
    }
    auto publish = [&] {                                                    // bf16 copy of the state
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                const int r = krow0 + mt * 16 + gq;
                *reinterpret_cast<uint32_t*>(smem + L::sb + swz<BV * 2>(r, nt) + qd * 4) = pack_bf16(S[mt][nt][0], S[mt][nt][1]);
                *reinterpret_cast<uint32_t*>(smem + L::sb + swz<BV * 2>(r + 8, nt) + qd * 4) = pack_bf16(S[mt][nt][2], S[mt][nt][3]);
            }
    };
    // fp32 copy of the state times `mul` to global memory
    auto store_state = [&](float* dst, float mul) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                float* p = dst + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + nt * 8 + qd * 2;
                *reinterpret_cast<float2*>(p) = make_float2(S[mt][nt][0] * mul, S[mt][nt][1] * mul);
                *reinterpret_cast<float2*>(p + 8L * V) = make_float2(S[mt][nt][2] * mul, S[mt][nt][3] * mul);
            }
    };
    if (!is_q) publish();
    bar_all();

    // A chunk is a chain of short steps of a few warps, so what is not a product counts too: offsets are 32-bit and advance
    // with the chunk, nothing is divided, and a failed (bounded) wait only stops further waiting -- the chunk is computed
    // on whatever the tiles hold, the status word says that the results are invalid.
    const float* g_p = gcs + ((long)b * T) * H + h;
    const float* rs_p = (is_q ? qrstd : krstd) + ((long)b * T) * H + h;
    __nv_bfloat16* o_p = o + ((long)b * T * H + h) * V + v0;
    float ga, gb, fa, fb, ga_n, gb_n, fa_n, fb_n;
    // cumsum of the log decay and the l2 norm factor (k rows on w warps, q rows on q warps) of this lane's two rows
    auto load_rows = [&](int t0, float& g0, float& g1, float& f0, float& f1) {
        const int ta = min(t0 + ra, T - 1) * H, tb = min(t0 + rb, T - 1) * H;
        g0 = g_p[ta];
        g1 = g_p[tb];
        f0 = t0 + ra < T ? rs_p[ta] : 0.f;
        f1 = t0 + rb < T ? rs_p[tb] : 0.f;
    };
    load_rows(0, ga, gb, fa, fb);
    constexpr bool kKeep = BV == 32;                                        // registers for 64 columns would spill
    uint32_t off_a[NTL], off_b[NTL];                                        // this lane's places in a [64][BV] tile
#pragma unroll
    for (int nt = 0; nt < NTL; ++nt) {
        off_a[nt] = swz<BV * 2>(ra, nt) + qd * 4;
        off_b[nt] = swz<BV * 2>(rb, nt) + qd * 4;
    }
    float carry = 0.f, carry_save = 0.f, blk_g = 0.f;
    const int c_last = (TN - 1) * cpb;                                      // first chunk of the last block
    bool ok = true;
    int sub = 0, stg = 0, par = 0;                                          // chunk within its block, tile stage, its parity
    bool may_carry = decay && (!trailing_quirk || 0 < last_sel);
    int blk = 0;

    for (int c = 0; c < NT; ++c) {
        const float2 meta = *reinterpret_cast<const float2*>(smem + L::meta + c * 8);
        const float gl = meta.x;
        const bool sel = meta.y != 0.f, active = cpb > 1 || sel;
        const bool block_end = sub == cpb - 1 || c == NT - 1;
        const bool restore = cpb > 1 && block_end && !sel;
        const uint32_t base = sbase + stg * L::stage;
        unsigned char* base_p = smem + stg * L::stage;
        load_rows(min(c + 1, NT - 1) * 64, ga_n, gb_n, fa_n, fb_n);         // consumed by the next chunk
        if (sub == 0) {
            carry_save = carry;
            blk_g = 0.f;
            if (!is_q && cpb > 1 && !sel) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < NTL; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) save_p[((mt * NTL + nt) * 4 + e) * 128 + tid] = S[mt][nt][e];
            }
        }
        if (c == c_last && hstart && !is_q) store_state(hstart, __expf(carry));
        blk_g += gl;
        const float ec = __expf(carry), dec = __expf(gl + carry);
        // rows past the end of a ragged last chunk have zero k and u; their cumsum only has to stay finite
        const float f0 = is_q ? fa * __expf(ga + carry) : fa * __expf(fminf(gl - ga, 80.f));
        const float f1 = is_q ? fb * __expf(gb + carry) : fb * __expf(fminf(gl - gb, 80.f));
        // the stage the previous chunk has left takes the tiles after next
        if (!kTmaWarp && loader && c >= 1 && c + L::NST - 1 < NT && ok) {
            ok = mbar_wait(bar_empty + ((c - 1) % L::NST) * 8, ((c - 1) / L::NST) & 1, status);
            if (ok) issue(c + L::NST - 1);
        }
        if (!kTmaWarp) __syncwarp();
        if (ok) ok = mbar_wait(bar_full + stg * 8, par, status);
        float acc[NTL][4];
        zero_acc(acc);
        const uint32_t at = base + (is_q ? L::q : L::w);
#pragma unroll
        for (int kk = 0; kk < K / 16; ++kk) {
            uint32_t a[4];
            load_a_sub(at, r0, kk * 16, lane, a);
#pragma unroll
            for (int p = 0; p < NTL / 2; ++p) {
                uint32_t bb[4];
                load_b_kn<BV * 2>(sb, kk * 16, p * 16, lane, bb);
                mma_bf16(acc[2 * p], a, bb[0], bb[1]);
                mma_bf16(acc[2 * p + 1], a, bb[2], bb[3]);
            }
        }
        unsigned char* vp_p = base_p + L::u;
        if (!is_q) {
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                if (!kKeep) {
                    off_a[nt] = swz<BV * 2>(ra, nt) + qd * 4;
                    off_b[nt] = off_a[nt] + 8 * BV * 2;                     // same swizzle eight rows on (128-byte rows)
                }
                const float2 xa = unpack_bf16(*reinterpret_cast<const uint32_t*>(vp_p + off_a[nt]));
                const float2 xb = unpack_bf16(*reinterpret_cast<const uint32_t*>(vp_p + off_b[nt]));
                const float a0 = xa.x - ec * acc[nt][0], a1 = xa.y - ec * acc[nt][1];
                const float b0 = xb.x - ec * acc[nt][2], b1 = xb.y - ec * acc[nt][3];
                *reinterpret_cast<uint32_t*>(vp_p + off_a[nt]) = pack_bf16(a0, a1);
                *reinterpret_cast<uint32_t*>(vp_p + off_b[nt]) = pack_bf16(b0, b1);
                if (active) {
                    *reinterpret_cast<uint32_t*>(smem + L::vs + off_a[nt]) = pack_bf16(a0 * f0, a1 * f0);
                    *reinterpret_cast<uint32_t*>(smem + L::vs + off_b[nt]) = pack_bf16(b0 * f1, b1 * f1);
                }
            }
        }
        bar_all();                                         // v', v'' written; every warp is done with this copy of S
        if (is_q) {
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                acc[nt][0] *= f0; acc[nt][1] *= f0;
                acc[nt][2] *= f1; acc[nt][3] *= f1;
            }
            const uint32_t vp = smem_u32(vp_p);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                if (kk <= (warp & 3)) {
                    uint32_t a[4];
                    load_a<128>(base + L::p, r0, kk * 16, lane, a);
#pragma unroll
                    for (int p = 0; p < NTL / 2; ++p) {
                        uint32_t bb[4];
                        load_b_kn<BV * 2>(vp, kk * 16, p * 16, lane, bb);
                        mma_bf16(acc[2 * p], a, bb[0], bb[1]);
                        mma_bf16(acc[2 * p + 1], a, bb[2], bb[3]);
                    }
                }
            }
            // output rows through the q rows only this warp reads, so that a row leaves in 16-byte pieces
#pragma unroll
            for (int nt = 0; nt < NTL; ++nt) {
                *reinterpret_cast<uint32_t*>(base_p + L::q + swz<128>(ra, nt) + qd * 4) = pack_bf16(acc[nt][0] * scale, acc[nt][1] * scale);
                *reinterpret_cast<uint32_t*>(base_p + L::q + swz<128>(rb, nt) + qd * 4) = pack_bf16(acc[nt][2] * scale, acc[nt][3] * scale);
            }
            __syncwarp();
            __nv_bfloat16* o_c = o_p + (long)c * 64 * H * V;
#pragma unroll
            for (int j = 0; j < NTL / 2; ++j) {
                const int r = r0 + (lane + 32 * j) / NTL, ch = (lane + 32 * j) % NTL;
                if (c * 64 + r < T)
                    *reinterpret_cast<uint4*>(o_c + r * H * V + ch * 8) =
                        *reinterpret_cast<const uint4*>(base_p + L::q + swz<128>(r, ch));
            }
            // orders v' and these rows (written with ordinary stores) before the next tiles that TMA writes there
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + stg * 8);
        } else {
            if (active && !restore) {                      // the last update of a rolled-back block is never read
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < NTL; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) S[mt][nt][e] *= dec;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t bb[NTL / 2][4];
#pragma unroll
                    for (int p = 0; p < NTL / 2; ++p) load_b_kn<BV * 2>(sbase + L::vs, kk * 16, p * 16, lane, bb[p]);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        uint32_t a[4];
                        load_a_t_sub(base + L::k, krow0 + mt * 16, kk * 16, lane, a);
#pragma unroll
                        for (int p = 0; p < NTL / 2; ++p) {
                            mma_bf16(S[mt][2 * p], a, bb[p][0], bb[p][1]);
                            mma_bf16(S[mt][2 * p + 1], a, bb[p][2], bb[p][3]);
                        }
                    }
                }
            }
            if (restore) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < NTL; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) S[mt][nt][e] = save_p[((mt * NTL + nt) * 4 + e) * 128 + tid];
            }
            if (active) publish();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + stg * 8);
        }
        if (active) {
            carry = 0.f;
            bar_all();                                     // the new copy of S is complete
        } else if (may_carry) {
            carry += gl;
        }
        if (restore) carry = carry_save + (may_carry ? blk_g : 0.f);
        ga = ga_n; gb = gb_n; fa = fa_n; fb = fb_n;
        if (++stg == L::NST) { stg = 0; par ^= 1; }
        if (block_end) {
            sub = 0;
            ++blk;
            may_carry = decay && (!trailing_quirk || blk < last_sel);
        } else {
            ++sub;
        }
    }
    if (is_q || !ok) return;
    if (ht) store_state(ht, 1.f);
    if (hstart && T % nbs == 0) {
        // the last block is complete: the decoder starts from the state behind it if its own type is linear, else from
        // the state in front of it, decayed over it
        const long li = (long)b * last_stride + hn * 2 + 1;
        const float lt = last_f32 ? reinterpret_cast<const float*>(last_types)[li]
                                  : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(last_types)[li]);
        if (lt > 0.f) {
            store_state(hstart, 1.f);
        } else if (decay) {
            const float f = __expf(blk_g);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < NTL; ++nt) {
                    float* p = hstart + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + nt * 8 + qd * 2;
                    float2 x = *reinterpret_cast<float2*>(p), y = *reinterpret_cast<float2*>(p + 8L * V);
                    x.x *= f; x.y *= f; y.x *= f; y.y *= f;
                    *reinterpret_cast<float2*>(p) = x;
                    *reinterpret_cast<float2*>(p + 8L * V) = y;
                }
        }
    }
}

template <int K, int BV>
static int launch_walk_mma(const void* q, const void* k, const void* w, const void* u, const void* pmat, const float* gcs,
                           const float* krstd, const float* qrstd, const int* types_i, const int* indices, const int* n_blocks,
                           const float* h0, void* o, float* ht, float* hstart, const void* last_types, int last_f32, int last_stride, int B, int T,
                           int H, int HN, int V, int nbs, float scale, int flags, cudaStream_t st) {
    using L = GwSmem<K, BV>;
    const char* who = "natsl_gdn_walk";
    const int NT = (T + 63) / 64;
    const int smem = L::total(NT, nbs > 64);
    NATSL_REQUIRE((long)T * H < (1l << 31) && 64l * H * V < (1l << 31), NATSL_ERR_TOO_LARGE,
                  "natsl_gdn_walk: T * H and 64 * H * V must be below 2^31");
    NATSL_REQUIRE(smem <= 227 * 1024, NATSL_ERR_TOO_LARGE, "natsl_gdn_walk: T=%d needs %d B of shared memory (max %d)", T, smem, 227 * 1024);
    auto kern = gdn_walk_mma_kernel<K, BV>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
        set_error("natsl_gdn_walk: cannot reserve %d B of shared memory (%s)", smem, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mw, mq, mk, mu, mp;
    int rc = encode_bthd_map(&mw, w, B, T, H, K, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mq, q, B, T, H, K, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, H, K, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mu, u, B, T, H, V, 64, who, BV);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mp, pmat, B, T, H, 64, 64, who);
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    kern<<<dim3(V / BV, H, B), gw_threads<BV>, smem, st>>>(
        mw, mq, mk, mu, mp, gcs, krstd, qrstd, types_i, indices, n_blocks, h0, reinterpret_cast<__nv_bfloat16*>(o), ht, hstart,
        last_types, last_f32, last_stride, T, H, HN, V, (T + nbs - 1) / nbs, nbs, scale, (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0,
        (flags & NATSL_FLAG_NO_TRAILING_QUIRK) ? 0 : 1, status);
    return check_launch(who);
}

}  // namespace natsl

extern "C" int natsl_gdn_walk(const void* q, const void* k, const void* w, const void* u, const void* pmat, const float* gcs,
                              const float* k_rstd, const float* q_rstd, const int32_t* types_i, const int32_t* indices,
                              const int32_t* n_blocks, const float* h0, void* o, float* ht, float* hstart,
                              const void* last_types, int last_dtype, int last_stride, int B, int T, int H, int HN, int K, int V, int nbs,
                              float scale, int flags, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && w && u && pmat && gcs && k_rstd && q_rstd && types_i && indices && n_blocks && o, NATSL_ERR_NULL,
                  "natsl_gdn_walk: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0, NATSL_ERR_BAD_SHAPE, "natsl_gdn_walk: bad shape");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_gdn_walk: B, H <= 65535");
    NATSL_REQUIRE(nbs >= 64 && nbs % 64 == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_gdn_walk: nats_block_size must be a multiple of 64 (got %d)", nbs);
    NATSL_REQUIRE(!hstart || T % nbs != 0 || (last_types && (last_dtype == NATSL_DT_F32 || last_dtype == NATSL_DT_BF16)),
                  NATSL_ERR_NULL, "natsl_gdn_walk: the block-start state of a complete last block needs that block's types");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int f32 = last_dtype == NATSL_DT_F32;
#define NATSL_GW(KK, BB) \
    return launch_walk_mma<KK, BB>(q, k, w, u, pmat, gcs, k_rstd, q_rstd, types_i, indices, n_blocks, h0, o, ht, hstart, \
                                   last_types, f32, last_stride, B, T, H, HN, V, nbs, scale, flags, st)
    // 32 value columns per CTA while that still leaves no second wave, 64 otherwise (the w, q, k and P tiles are then read
    // half as often).
    const bool narrow = V % 64 != 0 || (long)B * H * (V / 32) <= 148;
    if (V % 32 == 0 && V >= 64) {
        if (K == 64) { if (narrow) NATSL_GW(64, 32); else NATSL_GW(64, 64); }
        if (K == 128) { if (narrow) NATSL_GW(128, 32); else NATSL_GW(128, 64); }
    }
#undef NATSL_GW
    set_error("natsl_gdn_walk: unsupported head dims K=%d V=%d (K in {64, 128}, V a multiple of 32 from 64 on)", K, V);
    return NATSL_ERR_UNSUPPORTED;
}
