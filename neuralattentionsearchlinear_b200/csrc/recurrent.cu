// fp32 reference-precision path: token-by-token linear recurrence with re-roll, and a plain fp32
// chunk-masked softmax attention.  These follow the reference's decode kernel
//   src/nats/ops/gated_delta_rule/fused_recurrent.py:128-358  (Mamba2 twin: src/nats/ops/mamba/fused_recurrent.py:121-322)
// per token:  S <- e^{g_t} S;  v' = beta_t (v_t - S^T k_t)  [delta rule] or v_t [Mamba2];  S <- S + k_t v'^T;
//             o_t = scale * S^T q_t;   at the end of a block that is not selected the state is rolled back to the
//             block-start state (decayed by the block's total log decay when decay over skipped blocks is on).
// They serve fp32 inputs (parity to 1e-4 against the naive recurrent form) and short sequences; the bf16
// chunked tensor-core kernels are the throughput path.  CUDA-core fp32 math only.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

template <typename T>
__device__ __forceinline__ float ldf(const T* p, long i);
template <>
__device__ __forceinline__ float ldf<float>(const float* p, long i) { return p[i]; }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long i) { return __bfloat162float(p[i]); }
template <typename T>
__device__ __forceinline__ void stf(T* p, long i, float v);
template <>
__device__ __forceinline__ void stf<float>(float* p, long i, float v) { p[i] = v; }
template <>
__device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, long i, float v) { p[i] = __float2bfloat16(v); }

// ------------------------------------------------------------------------------------------------ token recurrence
// Serial over the tokens, so what bounds it is the chain of one token: S^T k -> v' -> S.  Eight lanes share one state column
// (K / 8 rows each, in registers), so both dots of a token (S^T k and S^T q: o = scale (e^g S^T q + (q.k) v')) take K / 8
// multiply-adds and one round of three shuffles; everything that does not depend on the state (norms, q.k, e^g) is prepared
// for a group of tokens at a time in shared memory by four other warps, one group ahead, from rows that cp.async brings one
// group further ahead.  At B = 2, T = 512, H = 4, K = V = 64, fp32: 472 -> 74 us (it was a warp per eight columns, five
// shuffles for each of 16 sums per token, loads per token).
constexpr int REC_THREADS = 128, REC_COLS = REC_THREADS / 8;         // each of the two roles: compute, preparation
template <int K>
constexpr int rec_ch = K <= 128 ? 32 : 16;          // tokens per prepared group

template <typename T, int K>
struct RecSmem {
    static constexpr int CH = rec_ch<K>;
    // raw rows of one group: q, k [CH][K], v [CH][REC_COLS]
    static constexpr int rq = 0, rk = rq + CH * K * (int)sizeof(T), rv = rk + CH * K * (int)sizeof(T);
    static constexpr int raw = rv + CH * REC_COLS * (int)sizeof(T);
    // prepared group, fp32: q, k, v and [CH] float4 (e^g, g, beta, q.k)
    static constexpr int q = 0, k = q + CH * K * 4, v = k + CH * K * 4, sc = v + CH * REC_COLS * 4, group = sc + CH * 16;
    static constexpr int groups = 2 * raw, total = groups + 2 * group;
};

template <typename T, int K>
__global__ void __launch_bounds__(2 * REC_THREADS)
linear_recurrent_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                        const float* __restrict__ g, const T* __restrict__ beta, const int* __restrict__ types_i,
                        const float* h0, T* __restrict__ o, float* ht,
                        float* hstart, int Tlen, int H, int HN, int V, int TN, int nbs, float scale,
                        int gdn, int decay, int use_l2norm, const float* hstart_in,
                        const float* __restrict__ gsum_in, int t_off, int step_mode) {
    // step_mode (decoding): the Tlen tokens continue a block that already holds t_off tokens; h0 is the current state,
    // hstart_in the state at the start of that block, gsum_in [B,H] its log decay so far.  A block only ends where
    // (t_off + t + 1) is a multiple of nbs, and ht receives the current state instead of the state after the last
    // selected block (fused_recurrent.py:128-358 with initial_state / initial_state_current / g_cumsum).
    using L = RecSmem<T, K>;
    constexpr int CH = L::CH, R4 = K / 32;             // float4 rows per lane
    extern __shared__ __align__(16) unsigned char smem[];
    const bool prep = threadIdx.x >= REC_THREADS;      // warps 4-7 prepare, warps 0-3 compute
    const int tid = threadIdx.x & (REC_THREADS - 1), lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, b = blockIdx.z;
    const int c0 = blockIdx.x * REC_COLS, n_cols = min(REC_COLS, V - c0);
    const long tok0 = (long)b * Tlen;
    const int n_grp = (Tlen + CH - 1) / CH;
    // named barriers: prepared group `i & 1` is full (1, 2) / has been consumed (3, 4)
    auto sync = [](int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(2 * REC_THREADS) : "memory"); };
    auto arrive = [](int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(2 * REC_THREADS) : "memory"); };

    if (prep) {
        const bool vec = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 7) == 0;
        auto fetch = [&](int grp) {                    // raw rows of a group of tokens, 8 bytes a copy
            const int t0 = grp * CH, n = min(CH, Tlen - t0);
            unsigned char* raw = smem + (grp & 1) * L::raw;
            if (!vec) {                                // tensors that do not start on 8 bytes: element by element
                T* e = reinterpret_cast<T*>(raw);
                for (int i = tid; i < n * K; i += REC_THREADS) {
                    const long src = ((tok0 + t0 + i / K) * H + h) * K + i % K;
                    e[L::rq / sizeof(T) + i] = q[src];
                    e[L::rk / sizeof(T) + i] = k[src];
                }
                for (int i = tid; i < n * REC_COLS; i += REC_THREADS)
                    if (i % REC_COLS < n_cols) e[L::rv / sizeof(T) + i] = v[((tok0 + t0 + i / REC_COLS) * H + h) * V + c0 + i % REC_COLS];
                cp_async_commit();
                return;
            }
            constexpr int EPC = 8 / (int)sizeof(T), QC = K / EPC;
            for (int i = tid; i < n * QC; i += REC_THREADS) {
                const int t = i / QC, c = (i % QC) * EPC;
                const long src = ((tok0 + t0 + t) * H + h) * K + c;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(raw + L::rq + (t * K + c) * sizeof(T))), "l"(q + src));
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(raw + L::rk + (t * K + c) * sizeof(T))), "l"(k + src));
            }
            const int VC = n_cols / EPC;               // V is a multiple of 8
            for (int i = tid; i < n * VC; i += REC_THREADS) {
                const int t = i / VC, c = (i % VC) * EPC;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(raw + L::rv + (t * REC_COLS + c) * sizeof(T))),
                             "l"(v + ((tok0 + t0 + t) * H + h) * V + c0 + c));
            }
            cp_async_commit();
        };
        fetch(0);
        for (int grp = 0; grp < n_grp; ++grp) {
            const int t0 = grp * CH, n = min(CH, Tlen - t0);
            if (grp + 1 < n_grp) { fetch(grp + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
            asm volatile("bar.sync 5, %0;" ::"n"(REC_THREADS) : "memory");       // every warp's raw rows have landed
            if (grp >= 2) sync(3 + (grp & 1));
            unsigned char* out = smem + L::groups + (grp & 1) * L::group;
            float *s_q = reinterpret_cast<float*>(out + L::q), *s_k = reinterpret_cast<float*>(out + L::k);
            float* s_v = reinterpret_cast<float*>(out + L::v);
            float4* s_sc = reinterpret_cast<float4*>(out + L::sc);
            const T* rq = reinterpret_cast<const T*>(smem + (grp & 1) * L::raw + L::rq);
            const T* rk = reinterpret_cast<const T*>(smem + (grp & 1) * L::raw + L::rk);
            const T* rv = reinterpret_cast<const T*>(smem + (grp & 1) * L::raw + L::rv);
#pragma unroll 2
            for (int t = warp; t < n; t += REC_THREADS / 32) {      // one warp per token
                float qv[K / 32], kv[K / 32], sq = 0.f, sk = 0.f, qk = 0.f;
                const long i = (tok0 + t0 + t) * H + h;
                const float gt = g[i], bt = gdn ? ldf(beta, i) : 0.f;
#pragma unroll
                for (int j = 0; j < K / 32; ++j) {
                    qv[j] = ldf(rq, t * K + lane + 32 * j);
                    kv[j] = ldf(rk, t * K + lane + 32 * j);
                    sq += qv[j] * qv[j];
                    sk += kv[j] * kv[j];
                }
                if (use_l2norm) {
                    const float a = rsqrtf(warp_sum(sq) + 1e-6f), c = rsqrtf(warp_sum(sk) + 1e-6f);
#pragma unroll
                    for (int j = 0; j < K / 32; ++j) { qv[j] *= a; kv[j] *= c; }
                }
#pragma unroll
                for (int j = 0; j < K / 32; ++j) {
                    s_q[t * K + lane + 32 * j] = qv[j];
                    s_k[t * K + lane + 32 * j] = kv[j];
                    qk += qv[j] * kv[j];
                }
                qk = warp_sum(qk);
                if (lane == 0) s_sc[t] = make_float4(__expf(gt), gt, bt, qk);
            }
            for (int i = tid; i < n * REC_COLS; i += REC_THREADS) s_v[i] = (i % REC_COLS) < n_cols ? ldf(rv, i) : 0.f;
            __threadfence_block();
            arrive(1 + (grp & 1));
            asm volatile("bar.sync 5, %0;" ::"n"(REC_THREADS) : "memory");       // the raw rows may be overwritten
        }
        return;
    }

    const int col = warp * 4 + (lane >> 3), part = lane & 7, vc = c0 + col;
    const bool col_ok = vc < V;
    const int hn = h / (H / HN);
    // row part * 4 + 32 i + e of the state column in S[i].e
    float4 S[R4], S0[R4], Sfin[R4];
    auto at = [&](int i, int e) { return (((long)b * H + h) * K + part * 4 + 32 * i + e) * V + vc; };
    auto rd = [&](const float* p, int i) {
        return col_ok ? make_float4(p[at(i, 0)], p[at(i, 1)], p[at(i, 2)], p[at(i, 3)]) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
#pragma unroll
    for (int i = 0; i < R4; ++i) {
        S[i] = Sfin[i] = h0 ? rd(h0, i) : make_float4(0.f, 0.f, 0.f, 0.f);
        S0[i] = hstart_in ? rd(hstart_in, i) : S[i];
    }
    float gsum = gsum_in ? gsum_in[(long)b * H + h] : 0.f;
    T* op = o + (tok0 * H + h) * V + (col_ok ? vc : 0);
    int left = nbs - t_off % nbs;                      // tokens to the end of the current block
    for (int grp = 0; grp < n_grp; ++grp) {
        const int t0 = grp * CH, n = min(CH, Tlen - t0);
        const unsigned char* in = smem + L::groups + (grp & 1) * L::group;
        const float *s_q = reinterpret_cast<const float*>(in + L::q), *s_k = reinterpret_cast<const float*>(in + L::k);
        const float* s_v = reinterpret_cast<const float*>(in + L::v);
        const float4* s_sc = reinterpret_cast<const float4*>(in + L::sc);
        sync(1 + (grp & 1));
        // one token's operands, read one token ahead of their use
        struct Tok {
            float4 sc, kk[R4], qq[R4];
            float vin;
        };
        auto rd_tok = [&](int t, Tok& x) {
            x.sc = s_sc[t];
            x.vin = s_v[t * REC_COLS + col];
#pragma unroll
            for (int i = 0; i < R4; ++i) {
                x.kk[i] = *reinterpret_cast<const float4*>(s_k + t * K + part * 4 + 32 * i);
                x.qq[i] = *reinterpret_cast<const float4*>(s_q + t * K + part * 4 + 32 * i);
            }
        };
        auto run_tok = [&](const Tok& x) {
            float dk0 = 0.f, dk1 = 0.f, dq0 = 0.f, dq1 = 0.f;
#pragma unroll
            for (int i = 0; i < R4; ++i) {
                dk0 += S[i].x * x.kk[i].x; dk1 += S[i].y * x.kk[i].y; dk0 += S[i].z * x.kk[i].z; dk1 += S[i].w * x.kk[i].w;
                dq0 += S[i].x * x.qq[i].x; dq1 += S[i].y * x.qq[i].y; dq0 += S[i].z * x.qq[i].z; dq1 += S[i].w * x.qq[i].w;
            }
            float dk = dk0 + dk1, dq = dq0 + dq1;
            const float eg = x.sc.x;
#pragma unroll
            for (int i = 0; i < R4; ++i) { S[i].x *= eg; S[i].y *= eg; S[i].z *= eg; S[i].w *= eg; }
#pragma unroll
            for (int off = 4; off > 0; off >>= 1) {
                dk += __shfl_xor_sync(0xffffffffu, dk, off);
                dq += __shfl_xor_sync(0xffffffffu, dq, off);
            }
            const float vn = gdn ? x.sc.z * (x.vin - eg * dk) : x.vin;
#pragma unroll
            for (int i = 0; i < R4; ++i) {
                S[i].x += x.kk[i].x * vn; S[i].y += x.kk[i].y * vn;
                S[i].z += x.kk[i].z * vn; S[i].w += x.kk[i].w * vn;
            }
            if (part == 0 && col_ok) stf(op, 0, (eg * dq + x.sc.w * vn) * scale);
            op += (long)H * V;
            gsum += x.sc.y;
        };
        for (int t = 0; t < n;) {
            // tokens up to the end of the block (or of the group): no tests inside
            const int stop = min(n, t + left);
            left -= stop - t;
            Tok x, y;
            rd_tok(t, x);
            for (; t + 1 < stop; t += 2) {
                rd_tok(t + 1, y);
                run_tok(x);
                rd_tok(min(t + 2, n - 1), x);
                run_tok(y);
            }
            if (t < stop) {
                run_tok(x);
                ++t;
            }
            if (left == 0 || (!step_mode && t0 + t == Tlen)) {
                const int sel = types_i[(((long)b * TN + (t_off + t0 + t - 1) / nbs) * HN + hn) * 2 + 1];
                const float roll = decay ? __expf(gsum) : 1.f;
#pragma unroll
                for (int i = 0; i < R4; ++i) {
                    if (sel) Sfin[i] = S[i];
                    else S[i] = make_float4(S0[i].x * roll, S0[i].y * roll, S0[i].z * roll, S0[i].w * roll);
                    S0[i] = S[i];
                }
                gsum = 0.f;
                left = nbs;
            }
        }
        if (grp + 2 < n_grp) arrive(3 + (grp & 1));
    }
    if (!col_ok) return;
    auto wr = [&](float* p, int i, const float4 x) { p[at(i, 0)] = x.x; p[at(i, 1)] = x.y; p[at(i, 2)] = x.z; p[at(i, 3)] = x.w; };
#pragma unroll
    for (int i = 0; i < R4; ++i) {
        if (ht) wr(ht, i, step_mode ? S[i] : Sfin[i]);
        if (hstart) wr(hstart, i, S0[i]);
    }
}

// ------------------------------------------------------------------------------------------------ fp32 attention
// One CTA per 16 queries of a head: key tiles of 64 in shared memory (skipped whole where no key of the tile is visible),
// scores as 2 x 4 register blocks, online softmax over the tile by the eight lanes that share a query, then the value product
// as DV / 16 columns per thread.  CUDA cores only; at these sizes latency and shared-memory reads bound it, so the next tile's
// rows are in flight while one is computed.  B = 2, T = 512, H = 4, 64 / 64: 443 -> 53 us (one warp per query, every lane
// walking whole key rows on its own).
constexpr int AF_Q = 16, AF_K = 64;

template <int DK, int DV>
struct AfSmem {
    static constexpr int LDK = DK + 4, LDV = DV + 4, LDP = AF_K + 4;          // pitches in floats: 16-byte rows, spread banks
    static constexpr int q = 0, k = q + AF_Q * LDK, v = k + AF_K * LDK, p = v + AF_K * LDV, total = (p + AF_Q * LDP) * 4;
};

template <typename T, int DK, int DV>
__global__ void __launch_bounds__(128)
attn_fp32_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                 const int* __restrict__ types_i, T* __restrict__ o, float* __restrict__ lse, int Tlen, int HQ, int HKV,
                 int HN, int TN, int nbs, float scale, int own_chunk) {
    using L = AfSmem<DK, DV>;
    extern __shared__ __align__(16) float sm[];
    float *s_q = sm + L::q, *s_k = sm + L::k, *s_v = sm + L::v, *s_p = sm + L::p;
    const int tid = threadIdx.x;
    const int n_qt = (Tlen + AF_Q - 1) / AF_Q;
    const int q0 = (n_qt - 1 - (int)blockIdx.x) * AF_Q, hq = blockIdx.y, b = blockIdx.z;      // longest walks first
    const int hkv = hq / (HQ / HKV), hn = hq / (HQ / HN);
    const int nq = min(AF_Q, Tlen - q0);
    for (int i = tid; i < AF_Q * DK; i += 128) {
        const int r = i / DK, d = i % DK;
        s_q[r * L::LDK + d] = r < nq ? ldf(q, (((long)b * Tlen + q0 + r) * HQ + hq) * DK + d) * scale : 0.f;
    }
    // scores: queries qi, qi + 8 and keys kj + 16 m; softmax and values: query tid / 8, eight lanes each
    const int qi = tid >> 4, kj = tid & 15, qr = tid >> 3, ql = tid & 7;
    float m = -INFINITY, l = 0.f, acc[DV / 8];
#pragma unroll
    for (int d = 0; d < DV / 8; ++d) acc[d] = 0.f;
    const int kend = q0 + nq;                            // keys below the last query
    const int tblk_lo = q0 / nbs, tblk_hi = (q0 + nq - 1) / nbs;
    auto sel = [&](int blk) { return types_i[(((long)b * TN + blk) * HN + hn) * 2] != 0; };
    for (int k0 = 0; k0 < kend; k0 += AF_K) {
        // with blocks of a multiple of 64 a key tile lies in one block, and whole tiles are skipped
        const int blk = k0 / nbs;
        const bool one = nbs % AF_K == 0;
        const bool own = own_chunk && blk >= tblk_lo && blk <= tblk_hi, past = blk < tblk_hi && sel(blk);
        if (one && !own && !past) continue;              // uniform over the CTA
        const int nk = min(AF_K, Tlen - k0);
        __syncthreads();                                 // the previous tile is consumed
        for (int i = tid; i < AF_K * (DK / 4); i += 128) {
            const int r = i / (DK / 4), d = (i % (DK / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < nk) {
                const T* p = k + (((long)b * Tlen + k0 + r) * HKV + hkv) * DK + d;
                x = make_float4(ldf(p, 0), ldf(p, 1), ldf(p, 2), ldf(p, 3));
            }
            *reinterpret_cast<float4*>(s_k + r * L::LDK + d) = x;
        }
        bool wild = false;                               // an infinity or NaN among the values of the tile
        for (int i = tid; i < AF_K * (DV / 4); i += 128) {
            const int r = i / (DV / 4), d = (i % (DV / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < nk) {
                const T* p = v + (((long)b * Tlen + k0 + r) * HKV + hkv) * DV + d;
                x = make_float4(ldf(p, 0), ldf(p, 1), ldf(p, 2), ldf(p, 3));
            }
            *reinterpret_cast<float4*>(s_v + r * L::LDV + d) = x;
            wild |= !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w));
        }
        wild = __syncthreads_or(wild);
        float sc[2][4] = {};
#pragma unroll 4
        for (int d = 0; d < DK; d += 4) {
            float4 a[2], c[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = *reinterpret_cast<const float4*>(s_q + (qi + 8 * i) * L::LDK + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const float4*>(s_k + (kj + 16 * j) * L::LDK + d);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sc[i][j] += a[i].x * c[j].x;
                    sc[i][j] += a[i].y * c[j].y;
                    sc[i][j] += a[i].z * c[j].z;
                    sc[i][j] += a[i].w * c[j].w;
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = q0 + qi + 8 * i, s = k0 + kj + 16 * j, tb = t / nbs, sb = one ? blk : s / nbs;
                const bool vis = s < Tlen && ((sb < tb && (one ? past : sel(sb))) || (own_chunk && sb == tb && s <= t));
                s_p[(qi + 8 * i) * L::LDP + kj + 16 * j] = vis ? sc[i][j] : -INFINITY;
            }
        __syncthreads();
        float mt = -INFINITY, x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = s_p[qr * L::LDP + ql + 8 * j];
            mt = fmaxf(mt, x[j]);
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, off));
        const float mn = fmaxf(m, mt), al = mn == -INFINITY ? 1.f : __expf(m - mn);
        float ps = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = x[j] == -INFINITY ? -0.f : __expf(x[j] - mn);      // -0: the key is not visible
            ps += x[j];
            s_p[qr * L::LDP + ql + 8 * j] = x[j];
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, off);
        l = l * al + ps;
        m = mn;
        __syncwarp();                                    // the eight lanes of a query sit in one warp
#pragma unroll
        for (int d = 0; d < DV / 8; ++d) acc[d] *= al;
        if (wild) {                                      // 0 times such a value is not 0: only the visible keys count
            for (int j = 0; j < AF_K; ++j) {
                const float pj = s_p[qr * L::LDP + j];
                if (__float_as_uint(pj) == 0x80000000u) continue;
#pragma unroll
                for (int d = 0; d < DV / 8; ++d) acc[d] += pj * s_v[j * L::LDV + ql * 4 + 32 * (d / 4) + d % 4];
            }
            continue;
        }
        for (int j = 0; j < AF_K; j += 4) {
            const float4 pj = *reinterpret_cast<const float4*>(s_p + qr * L::LDP + j);
#pragma unroll
            for (int d = 0; d < DV / 32; ++d) {          // columns ql * 4 + 32 d .. + 3
                const float* vp = s_v + j * L::LDV + ql * 4 + 32 * d;
                const float4 v0 = *reinterpret_cast<const float4*>(vp), v1 = *reinterpret_cast<const float4*>(vp + L::LDV),
                             v2 = *reinterpret_cast<const float4*>(vp + 2 * L::LDV), v3 = *reinterpret_cast<const float4*>(vp + 3 * L::LDV);
                acc[4 * d] += pj.x * v0.x; acc[4 * d] += pj.y * v1.x; acc[4 * d] += pj.z * v2.x; acc[4 * d] += pj.w * v3.x;
                acc[4 * d + 1] += pj.x * v0.y; acc[4 * d + 1] += pj.y * v1.y; acc[4 * d + 1] += pj.z * v2.y; acc[4 * d + 1] += pj.w * v3.y;
                acc[4 * d + 2] += pj.x * v0.z; acc[4 * d + 2] += pj.y * v1.z; acc[4 * d + 2] += pj.z * v2.z; acc[4 * d + 2] += pj.w * v3.z;
                acc[4 * d + 3] += pj.x * v0.w; acc[4 * d + 3] += pj.y * v1.w; acc[4 * d + 3] += pj.z * v2.w; acc[4 * d + 3] += pj.w * v3.w;
            }
        }
    }
    if (qr >= nq) return;
    const bool has = l > 0.f;
    const long ob = ((long)b * Tlen + q0 + qr) * HQ + hq;
#pragma unroll
    for (int d = 0; d < DV / 32; ++d)
#pragma unroll
        for (int e = 0; e < 4; ++e) stf(o, ob * DV + ql * 4 + 32 * d + e, has ? acc[4 * d + e] / l : 0.f);
    if (ql == 0) lse[ob] = has ? (m + logf(l)) * 1.44269504f : 0.f;
}

template <typename T>
static int launch_recurrent(const void* q, const void* k, const void* v, const float* g, const void* beta,
                            const int* types_i, const float* h0, void* o, float* ht, float* hstart, int B, int T_, int H,
                            int HN, int K, int V, int nbs, float scale, int gdn, int decay, int l2, cudaStream_t st,
                            const float* hstart_in = nullptr, const float* gsum_in = nullptr, int t_off = 0,
                            int step_mode = 0) {
    const int TN = (t_off + T_ + nbs - 1) / nbs;
    dim3 grid((V + REC_COLS - 1) / REC_COLS, H, B);
    cudaError_t e = cudaSuccess;
#define NATSL_REC(KK) \
    e = cudaFuncSetAttribute(linear_recurrent_kernel<T, KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, RecSmem<T, KK>::total); \
    if (e == cudaSuccess) linear_recurrent_kernel<T, KK><<<grid, 2 * REC_THREADS, RecSmem<T, KK>::total, st>>>( \
        reinterpret_cast<const T*>(q), reinterpret_cast<const T*>(k), reinterpret_cast<const T*>(v), g, \
        reinterpret_cast<const T*>(beta), types_i, h0, reinterpret_cast<T*>(o), ht, hstart, T_, H, HN, V, TN, nbs, scale, gdn, decay, l2, \
        hstart_in, gsum_in, t_off, step_mode)
    if (K == 32) { NATSL_REC(32); }
    else if (K == 64) { NATSL_REC(64); }
    else if (K == 96) { NATSL_REC(96); }
    else if (K == 128) { NATSL_REC(128); }
    else if (K == 192) { NATSL_REC(192); }
    else if (K == 256) { NATSL_REC(256); }
    else {
        set_error("natsl_linear_recurrent_fwd: unsupported key dim K=%d (32, 64, 96, 128, 192 or 256)", K);
        return NATSL_ERR_UNSUPPORTED;
    }
#undef NATSL_REC
    if (e != cudaSuccess) {
        set_error("natsl_linear_recurrent_fwd: cannot reserve shared memory (%s)", cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return check_launch("natsl_linear_recurrent_fwd");
}

template <typename T>
static int launch_attn_fp32(const void* q, const void* k, const void* v, const int* types_i, void* o, float* lse, int B,
                            int T_, int HQ, int HKV, int HN, int DK, int DV, int nbs, float scale, int own,
                            cudaStream_t st) {
    const int TN = (T_ + nbs - 1) / nbs;
    dim3 grid((T_ + AF_Q - 1) / AF_Q, HQ, B);
    cudaError_t e = cudaSuccess;
#define NATSL_AF(DKK, DVV) \
    e = cudaFuncSetAttribute(attn_fp32_kernel<T, DKK, DVV>, cudaFuncAttributeMaxDynamicSharedMemorySize, AfSmem<DKK, DVV>::total); \
    if (e == cudaSuccess) attn_fp32_kernel<T, DKK, DVV><<<grid, 128, AfSmem<DKK, DVV>::total, st>>>( \
        reinterpret_cast<const T*>(q), reinterpret_cast<const T*>(k), reinterpret_cast<const T*>(v), types_i, \
        reinterpret_cast<T*>(o), lse, T_, HQ, HKV, HN, TN, nbs, scale, own)
    if (DK == 64 && DV == 64) { NATSL_AF(64, 64); }
    else if (DK == 32 && DV == 32) { NATSL_AF(32, 32); }
    else if (DK == 128 && DV == 64) { NATSL_AF(128, 64); }
    else if (DK == 64 && DV == 128) { NATSL_AF(64, 128); }
    else if (DK == 128 && DV == 128) { NATSL_AF(128, 128); }
    else {
        set_error("natsl_attn_fwd_fp32: unsupported head dims DK=%d DV=%d", DK, DV);
        return NATSL_ERR_UNSUPPORTED;
    }
#undef NATSL_AF
    if (e != cudaSuccess) {
        set_error("natsl_attn_fwd_fp32: cannot reserve shared memory (%s)", cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return check_launch("natsl_attn_fwd_fp32");
}

}  // namespace natsl

extern "C" int natsl_linear_recurrent_fwd(int rule, int dtype, const void* q, const void* k, const void* v,
                                          const float* g, const void* beta, const int32_t* types_i, const float* h0,
                                          void* o, float* ht, float* hstart, int B, int T, int H, int HN, int K, int V,
                                          int nbs, float scale, int flags, int use_l2norm, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && v && g && types_i && o, NATSL_ERR_NULL, "natsl_linear_recurrent_fwd: null pointer");
    NATSL_REQUIRE(rule == NATSL_RULE_GDN || rule == NATSL_RULE_MAMBA, NATSL_ERR_UNSUPPORTED, "natsl_linear_recurrent_fwd: bad rule");
    NATSL_REQUIRE(rule != NATSL_RULE_GDN || beta, NATSL_ERR_NULL, "natsl_linear_recurrent_fwd: beta is required for the delta rule");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0 && V % 8 == 0 && nbs > 0, NATSL_ERR_BAD_SHAPE,
                  "natsl_linear_recurrent_fwd: bad shape (V must be a multiple of 8)");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_linear_recurrent_fwd: B, H <= 65535");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int gdn = rule == NATSL_RULE_GDN, decay = (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0;
    if (dtype == NATSL_DT_F32)
        return launch_recurrent<float>(q, k, v, g, beta, types_i, h0, o, ht, hstart, B, T, H, HN, K, V, nbs, scale, gdn, decay, use_l2norm, st);
    if (dtype == NATSL_DT_BF16)
        return launch_recurrent<__nv_bfloat16>(q, k, v, g, beta, types_i, h0, o, ht, hstart, B, T, H, HN, K, V, nbs, scale, gdn, decay, use_l2norm, st);
    set_error("natsl_linear_recurrent_fwd: dtype must be f32 or bf16");
    return NATSL_ERR_UNSUPPORTED;
}

extern "C" int natsl_linear_recurrent_step(int rule, int dtype, const void* q, const void* k, const void* v, const float* g,
                                           const void* beta, const int32_t* types_i, const float* h_cur,
                                           const float* h_start, const float* gsum, int t_off, void* o, float* h_cur_out,
                                           float* h_start_out, int B, int T, int H, int HN, int K, int V, int nbs,
                                           float scale, int flags, int use_l2norm, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && v && g && types_i && h_cur && h_start && gsum && o && h_cur_out && h_start_out, NATSL_ERR_NULL,
                  "natsl_linear_recurrent_step: null pointer");
    NATSL_REQUIRE(rule == NATSL_RULE_GDN || rule == NATSL_RULE_MAMBA, NATSL_ERR_UNSUPPORTED, "natsl_linear_recurrent_step: bad rule");
    NATSL_REQUIRE(rule != NATSL_RULE_GDN || beta, NATSL_ERR_NULL, "natsl_linear_recurrent_step: beta is required for the delta rule");
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0 && V % 8 == 0 && nbs > 0 && t_off >= 0 && t_off < nbs,
                  NATSL_ERR_BAD_SHAPE, "natsl_linear_recurrent_step: bad shape (V a multiple of 8, 0 <= t_off < nbs)");
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_linear_recurrent_step: B, H <= 65535");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int gdn = rule == NATSL_RULE_GDN, decay = (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0;
    if (dtype == NATSL_DT_F32)
        return launch_recurrent<float>(q, k, v, g, beta, types_i, h_cur, o, h_cur_out, h_start_out, B, T, H, HN, K, V, nbs, scale,
                                       gdn, decay, use_l2norm, st, h_start, gsum, t_off, 1);
    if (dtype == NATSL_DT_BF16)
        return launch_recurrent<__nv_bfloat16>(q, k, v, g, beta, types_i, h_cur, o, h_cur_out, h_start_out, B, T, H, HN, K, V, nbs,
                                               scale, gdn, decay, use_l2norm, st, h_start, gsum, t_off, 1);
    set_error("natsl_linear_recurrent_step: dtype must be f32 or bf16");
    return NATSL_ERR_UNSUPPORTED;
}

extern "C" int natsl_attn_fwd_fp32(int dtype, const void* q, const void* k, const void* v, const int32_t* types_i, void* o,
                                   float* lse, int B, int T, int HQ, int HKV, int HN, int DK, int DV, int nbs, float scale,
                                   int flags, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && v && types_i && o && lse, NATSL_ERR_NULL, "natsl_attn_fwd_fp32: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && HQ > 0 && HKV > 0 && HN > 0 && HQ % HKV == 0 && HQ % HN == 0 && nbs > 0,
                  NATSL_ERR_BAD_SHAPE, "natsl_attn_fwd_fp32: bad shape");
    NATSL_REQUIRE(HQ <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_attn_fwd_fp32: B, HQ <= 65535");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int own = (flags & NATSL_FLAG_ATTN_OWN_CHUNK) ? 1 : 0;
    if (dtype == NATSL_DT_F32) return launch_attn_fp32<float>(q, k, v, types_i, o, lse, B, T, HQ, HKV, HN, DK, DV, nbs, scale, own, st);
    if (dtype == NATSL_DT_BF16)
        return launch_attn_fp32<__nv_bfloat16>(q, k, v, types_i, o, lse, B, T, HQ, HKV, HN, DK, DV, nbs, scale, own, st);
    set_error("natsl_attn_fwd_fp32: dtype must be f32 or bf16");
    return NATSL_ERR_UNSUPPORTED;
}
