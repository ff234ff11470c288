// Gated-delta-rule linear branch for head dims that hold the state and every operand to fp32 precision between bf16 tensors
// (K = 192, any V in slices of 32, any nats_block_size): chunk preparation, then recurrence and output in one walk.
// Per 64-token chunk (S = state it reads, T' = (I + A)^-1 diag(beta), A = strictLower(beta kn kn^T e^{g_i - g_j})):
//     v' = T' (v - rstd_k e^{g+carry} k S)                                                          (w warps)
//     o  = scale (rstd_q e^{g+carry} q S + P v')                                                    (q warps)
//     S <- e^{g_last+carry} S + k^T (v' rstd_k e^{g_last-g})      if the chunk updates the state     (w warps)
// (src/nats/ops/common/chunk_delta_h.py:189-324 and src/nats/ops/common/chunk_o.py:124-215, with the inverse applied inside the
// walk instead of to w and u before it).  q, k and v are exact in bf16.  Everything computed (S, T', P, v - .., v', v'') enters
// its products as the sum of bf16 parts: three where the result stays in the state (24 bits), two where it only reaches the
// output, which is rounded to 8; the sums themselves and the state are fp32.
// What bounds it: the serial chain of a chunk (k S -> T' r -> v' -> k^T v'' -> parts of S), so eight warps share each of its
// products (16 rows x 16 columns each) and eight others form the output; one of those issues the next tiles' loads at the
// barriers behind which their buffers are free (a warp of its own would leave 96 registers a thread, which spill).
// B = 2, T = 2048, H = 6, V = 384: preparation 32 us, walk 172 us (5.4 us a chunk), op 221 us.  Against float64 the outputs are
// off by their rounding (1.66e-3, as those of the token recurrence, which takes 1.1 ms), the final state by 0.9 - 1.0e-7 for
// decays of 0.7 a token and 0.8e-7 for slower ones (token recurrence 0.7 - 0.8e-7 and up to 1.2e-6).  With w, u, v' and S
// rounded to bf16, as for the other head dims, the op took 132 us and was off by 3.7e-3, its final state by 2.5e-3.
#include "tc_common.cuh"
#include "warp_gemm.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

constexpr int SP_LD = 66, SP_TP = 320;                        // row pitch of fp32 tiles; bf16 of a token row: T' x 3, P x 2

// x0 + e0, x1 + e1 as the sum of N bf16 pairs, largest first (e: what rounding to fp32 has left over)
template <int N>
__device__ __forceinline__ void split_bf16(float x0, float x1, uint32_t (&p)[N], float e0 = 0.f, float e1 = 0.f) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i == N - 1) {
            x0 += e0;
            x1 += e1;
        }
        p[i] = pack_bf16(x0, x1);
        const float2 f = unpack_bf16(p[i]);
        x0 -= f.x;
        x1 -= f.y;
    }
}

// acc + low += d with nothing lost: what acc cannot hold goes to low
__device__ __forceinline__ void add_exact(float& acc, float& low, float d) {
    const float s = acc + d, t = s - acc;
    low += (acc - (s - t)) + (d - t);
    acc = s;
}

// ------------------------------------------------------------------------------------------------ preparation
template <int K>
struct SpPrep {
    // the q tile becomes P [64][66] fp32 and W (fp64), the k tile T [64][66] fp64: three CTAs per SM
    static constexpr int q = 0, W = q + 64 * SP_LD * 4, k = q + 64 * K * 2, T = k;
    static constexpr int A = T + 64 * SP_LD * 8, gd = A + 64 * SP_LD * 4;
    static constexpr int vec = gd + 65 * 8, total = vec + 3 * 64 * 4;
    static_assert(W + 3 * 16 * 17 * 8 <= k && 64 * K * 2 <= 64 * SP_LD * 8, "P and W fit over q, k under T");
    static_assert(W % 8 == 0 && T % 8 == 0 && gd % 8 == 0 && 3 * (total + 1024) <= 228 * 1024, "doubles; three CTAs");
};

template <int K>
__global__ void __launch_bounds__(256, 3)
gdn_split_prep_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const float* __restrict__ g,
                      const void* __restrict__ beta, int beta_f32, __nv_bfloat16* __restrict__ tp, float* __restrict__ kf_out,
                      float* __restrict__ qf_out, float* __restrict__ vf_out, float* __restrict__ egl_out, int T, int H, int use_l2norm) {
    using L = SpPrep<K>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, qd = lane & 3;
    const int h = blockIdx.y, b = blockIdx.z, t0 = blockIdx.x * 64, valid = min(64, T - t0);
    const long tok0 = (long)b * T + t0;
    unsigned char* qs_p = smem + L::q;
    const uint32_t qs = smem_u32(qs_p), ks = smem_u32(smem + L::k);
    float *As = reinterpret_cast<float*>(smem + L::A), *Ps = reinterpret_cast<float*>(qs_p);
    double *Ts = reinterpret_cast<double*>(smem + L::T), *Ws = reinterpret_cast<double*>(smem + L::W);
    double* s_g = reinterpret_cast<double*>(smem + L::gd);
    auto kn = [&](int r) -> double& { return *reinterpret_cast<double*>(&As[r * SP_LD + 64]); };     // in A's padding: 1 / norm of k
    float *s_b = reinterpret_cast<float*>(smem + L::vec), *s_kr = s_b + 64, *s_qr = s_kr + 64;

    load_tile_async<64, K, 256>(qs, q + (tok0 * H + h) * K, (long)H * K, valid, tid);
    load_tile_async<64, K, 256>(ks, k + (tok0 * H + h) * K, (long)H * K, valid, tid);
    cp_async_commit();
    // Chunk-local cumsum of g, two warps, in fp64: its differences are what counts, and over 64 tokens an fp32 sum is off by 4e-6
    // where the product of the tokens' own decays is not.
    double x = 0.;
    if (tid < 64) {
        float bv = 0.f;
        if (tid < valid) {
            const long i = (tok0 + tid) * H + h;
            x = g[i];
            bv = beta_f32 ? reinterpret_cast<const float*>(beta)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(beta)[i]);
        }
        s_b[tid] = bv;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += u;
        }
        if (tid == 31) s_g[64] = x;
    }
    cp_async_wait<0>();
    __syncthreads();
    if (tid < 64) s_g[tid] = tid < 32 ? x : x + s_g[64];
    for (int r = warp * 8; r < warp * 8 + 8; ++r) {           // row norms of q and k
        float sq = 0.f, sk = 0.f;
        if (lane < K / 8) {
            const uint4 a = *reinterpret_cast<const uint4*>(qs_p + swz<K * 2>(r, lane));
            const uint4 c = *reinterpret_cast<const uint4*>(smem + L::k + swz<K * 2>(r, lane));
            const uint32_t *aw = reinterpret_cast<const uint32_t*>(&a), *cw = reinterpret_cast<const uint32_t*>(&c);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 u = unpack_bf16(aw[j]), w = unpack_bf16(cw[j]);
                sq += u.x * u.x + u.y * u.y;
                sk += w.x * w.x + w.y * w.y;
            }
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        if (lane == 0) {
            s_qr[r] = use_l2norm ? rsqrtf(sq + 1e-6f) : 1.f;
            kn(r) = use_l2norm ? 1. / sqrt((double)sk + 1e-6) : 1.;
            s_kr[r] = (float)kn(r);
        }
    }
    // warps 0-3: k k^T, warps 4-7: q k^T; a warp holds 16 rows, columns up to the diagonal.  Each 16-wide step of the contraction
    // is added in fp32 arithmetic of its own: the tensor core's running sum truncates.
    const bool kk_warp = warp < 4;
    const int rblk = kk_warp ? warp : 7 - warp, r0 = rblk * 16;
    float acc[8][4];
    zero_acc(acc);
#pragma unroll 2
    for (int kk = 0; kk < K / 16; ++kk) {
        uint32_t a[4];
        load_a<K * 2>(kk_warp ? ks : qs, r0, kk * 16, lane, a);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            if (p > rblk) break;
            uint32_t bb[4];
            load_b_nk<K * 2>(ks, p * 16, kk * 16, lane, bb);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16(d, a, bb[2 * e], bb[2 * e + 1]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[2 * p + e][j] += d[j];
            }
        }
    }
    __syncthreads();                                          // norms and cumsum known, products done: q may be overwritten
    if (tid < valid) {                                        // factors of the rows of k S, q S and v'', decay over the chunk
        const long i = (tok0 + tid) * H + h;
        // rounded once, vf held in two parts: an error of theirs is one of the whole row
        const double eg = exp(s_g[tid]), kr = kn(tid);
        kf_out[i] = (float)(kr * eg);
        qf_out[i] = (float)(s_qr[tid] * eg);
        const double vf = kr * exp(s_g[63] - s_g[tid]);
        vf_out[i] = (float)vf;
        vf_out[i + (long)gridDim.z * T * H] = (float)(vf - (float)vf);
        if (tid == 0) egl_out[((long)b * gridDim.x + blockIdx.x) * H + h] = (float)exp(s_g[63]);
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = r0 + gq + 8 * (e >> 1), j = nt * 8 + 2 * qd + (e & 1);
            const float gam = j <= i ? expf((float)(s_g[i] - s_g[j])) * s_kr[j] : 0.f;
            if (kk_warp) As[i * SP_LD + j] = j < i ? acc[nt][e] * s_b[i] * s_kr[i] * gam : 0.f;
            else Ps[i * SP_LD + j] = acc[nt][e] * s_qr[i] * gam;
        }
    for (int i = tid; i < 64 * SP_LD; i += 256) Ts[i] = 0.;
    __syncthreads();
    // T = (I + A)^-1 in fp64 (its three parts hold 24 bits): the diagonal blocks by forward substitution (a lane per column), then block diagonal by block diagonal
    // T_ij = -T_ii sum_m A_im T_mj
    if (warp < 4 && lane < 16) {
        const int d0 = warp * 16;
        double xc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            double s = i == lane ? 1. : 0.;
#pragma unroll
            for (int j = 0; j < i; ++j) s -= As[(d0 + i) * SP_LD + d0 + j] * xc[j];
            xc[i] = s;
            Ts[(d0 + i) * SP_LD + d0 + lane] = s;
        }
    }
    __syncthreads();
    for (int d = 1; d < 4; ++d) {
        const int n = (4 - d) * 256;
        for (int e = tid; e < n; e += 256) {
            const int j = e >> 8, r = (e >> 4) & 15, c = e & 15, i = j + d;
            double s = 0.;
            for (int m = j * 16; m < i * 16; ++m) s += As[(i * 16 + r) * SP_LD + m] * Ts[m * SP_LD + j * 16 + c];
            Ws[(j * 16 + r) * 17 + c] = s;
        }
        __syncthreads();
        for (int e = tid; e < n; e += 256) {
            const int j = e >> 8, r = (e >> 4) & 15, c = e & 15, i = j + d;
            double s = 0.;
#pragma unroll
            for (int m = 0; m < 16; ++m) s -= Ts[(i * 16 + r) * SP_LD + i * 16 + m] * Ws[(j * 16 + m) * 17 + c];
            Ts[(i * 16 + r) * SP_LD + j * 16 + c] = s;
        }
        __syncthreads();
    }
    for (int e = tid; e < 64 * 8; e += 256) {
        const int r = e >> 3, c8 = (e & 7) * 8;
        if (r >= valid) continue;
        uint32_t out[5][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t t3[3], p2[2];
            const double x0 = Ts[r * SP_LD + c8 + 2 * j] * s_b[c8 + 2 * j], x1 = Ts[r * SP_LD + c8 + 2 * j + 1] * s_b[c8 + 2 * j + 1];
            split_bf16((float)x0, (float)x1, t3, (float)(x0 - (float)x0), (float)(x1 - (float)x1));
            split_bf16(Ps[r * SP_LD + c8 + 2 * j], Ps[r * SP_LD + c8 + 2 * j + 1], p2);
            out[0][j] = t3[0]; out[1][j] = t3[1]; out[2][j] = t3[2]; out[3][j] = p2[0]; out[4][j] = p2[1];
        }
        __nv_bfloat16* dst = tp + ((tok0 + r) * H + h) * SP_TP + c8;
#pragma unroll
        for (int p = 0; p < 5; ++p) *reinterpret_cast<uint4*>(dst + p * 64) = make_uint4(out[p][0], out[p][1], out[p][2], out[p][3]);
    }
}

// ------------------------------------------------------------------------------------------------ walk
constexpr int SW_W = 8, SW_THREADS = 32 * 2 * SW_W, SW_BV = 32;

template <int K>
struct SwSmem {
    static constexpr int kq = 0, kq_bytes = 2 * 64 * K * 2;   // 2 stages of [k | q], sub-tiles [64][64]
    static constexpr int t = kq + 2 * kq_bytes, p = t + 3 * 8192, v = p + 2 * 8192;         // v: 2 stages [64][32]
    static constexpr int s = v + 2 * 4096, s_bytes = K * 64;  // parts of S [K][32]
    static constexpr int r = s + 3 * s_bytes, vp = r + 3 * 4096, vs = vp + 2 * 4096;        // parts of r, v', v'' [64][32]
    static constexpr int bars = vs + 3 * 4096, meta = bars + 64;
    static int total(int NT) { return meta + NT * 8; }
};

// ROLL: blocks of more than one chunk, whose state is kept for a roll-back (its 24 registers would spill elsewhere).
template <int K, bool ROLL>
__global__ void __launch_bounds__(SW_THREADS, 1)
gdn_split_walk_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_tp,
                      const float* __restrict__ kf, const float* __restrict__ qf, const float* __restrict__ vf,
                      const float* __restrict__ egl, const int* __restrict__ types_i, const int* __restrict__ indices,
                      const int* __restrict__ n_blocks, const float* __restrict__ h0, __nv_bfloat16* __restrict__ o,
                      float* __restrict__ ht, float* hstart,
                      const void* __restrict__ last_types, int last_f32, int last_stride, int T, int H, int HN, int V, int TN, int nbs,
                      float scale, int decay, int trailing_quirk, int* status) {
    using L = SwSmem<K>;
    constexpr int MT = K / 64, NSUB = K / 64, BV = SW_BV;     // 16-row tiles of the state per w warp: K / 4 rows
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, qd = lane & 3;
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const int v0 = blockIdx.x * BV, h = blockIdx.y, b = blockIdx.z, hn = h / (H / HN);
    const int NT = (T + 63) / 64, cpb = ROLL ? nbs / 64 : 1;
    float2* s_meta = reinterpret_cast<float2*>(smem + L::meta);              // per chunk: decay, selected
    const uint32_t full_kq = sbase + L::bars, full_t = full_kq + 16, full_p = full_kq + 24;
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) mbar_init(full_kq + 8 * i, 1);
        mbar_fence_init();
    }
    for (int c = tid; c < NT; c += SW_THREADS)
        s_meta[c] = make_float2(egl[((long)b * NT + c) * H + h],
                                types_i[(((long)b * TN + c / cpb) * HN + hn) * 2 + 1] != 0 ? 1.f : 0.f);
    __syncthreads();

    const bool loader = warp == SW_W && lane == 0;            // of the q warp with the fewest products
    auto load_kq = [&](int c) {
        const uint32_t dst = sbase + L::kq + (c & 1) * L::kq_bytes, bar = full_kq + (c & 1) * 8;
        mbar_expect_tx(bar, L::kq_bytes + 4096);
#pragma unroll
        for (int sub = 0; sub < NSUB; ++sub) {
            tma_load_4d(dst + sub * 8192, &map_k, sub * 64, h, c * 64, b, bar);
            tma_load_4d(dst + 64 * K * 2 + sub * 8192, &map_q, sub * 64, h, c * 64, b, bar);
        }
        tma_load_4d(sbase + L::v + (c & 1) * 4096, &map_v, v0, h, c * 64, b, bar);
    };
    auto load_t = [&](int c) {
        mbar_expect_tx(full_t, 3 * 8192);
#pragma unroll
        for (int p = 0; p < 3; ++p) tma_load_4d(sbase + L::t + p * 8192, &map_tp, p * 64, h, c * 64, b, full_t);
    };
    auto load_p = [&](int c) {
        mbar_expect_tx(full_p, 2 * 8192);
#pragma unroll
        for (int p = 0; p < 2; ++p) tma_load_4d(sbase + L::p + p * 8192, &map_tp, (3 + p) * 64, h, c * 64, b, full_p);
    };
    if (loader) {
        prefetch_tensormap(&map_q); prefetch_tensormap(&map_k); prefetch_tensormap(&map_v); prefetch_tensormap(&map_tp);
        load_kq(0);
        load_t(0);
        load_p(0);
        if (NT > 1) load_kq(1);
    }
    __syncwarp();

    const int nsel = n_blocks[((long)b * HN + hn) * 2 + 1];
    const int last_sel = nsel > 0 ? indices[(((long)b * TN + (nsel - 1)) * HN + hn) * 2 + 1] : -1;
    const bool is_q = warp >= SW_W;
    const int rg = warp & 3, n0 = ((warp >> 2) & 1) * 16;     // row group, first of 16 columns
    const int r0 = rg * 16, ra = r0 + gq, rb = ra + 8, krow0 = rg * (K / 4);
    auto bar_w = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    auto bar_all = [] { asm volatile("bar.sync 2, 512;" ::: "memory"); };
    // byte offset of this lane's pair of columns n0 + 8 nt + 2 qd in row `row` of a [..][32] tile
    auto at = [&](int row, int nt) { return swz<64>(row, (n0 >> 3) + nt) + qd * 4; };

    float S[MT][2][4], save[ROLL ? MT : 1][2][4];
    if (!is_q) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float2 lo = make_float2(0.f, 0.f), hi = lo;
                if (h0) {
                    const float* p = h0 + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + n0 + nt * 8 + qd * 2;
                    lo = *reinterpret_cast<const float2*>(p);
                    hi = *reinterpret_cast<const float2*>(p + 8L * V);
                }
                S[mt][nt][0] = lo.x; S[mt][nt][1] = lo.y; S[mt][nt][2] = hi.x; S[mt][nt][3] = hi.y;
            }
    }
    auto publish = [&] {                                      // the parts of S that the products read
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    uint32_t p[3];
                    split_bf16(S[mt][nt][2 * hh], S[mt][nt][2 * hh + 1], p);
                    const uint32_t off = at(krow0 + mt * 16 + gq + 8 * hh, nt);
#pragma unroll
                    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(smem + L::s + i * L::s_bytes + off) = p[i];
                }
    };
    auto store_state = [&](float* dst, float mul) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float* p = dst + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + n0 + nt * 8 + qd * 2;
                *reinterpret_cast<float2*>(p) = make_float2(S[mt][nt][0] * mul, S[mt][nt][1] * mul);
                *reinterpret_cast<float2*>(p + 8L * V) = make_float2(S[mt][nt][2] * mul, S[mt][nt][3] * mul);
            }
    };
    if (!is_q) publish();
    bar_all();

    const float *f_p = (is_q ? qf : kf) + (long)b * T * H + h, *u_p = vf + (long)b * T * H + h;
    const long u_low = (long)gridDim.z * T * H;               // second part of vf
    // this lane's two rows: factors of k S or q S, and of v'' (zero past the end)
    auto load_rows = [&](int t0, float& f0, float& f1, float2& u0, float2& u1) {
        const long ta = (long)min(t0 + ra, T - 1) * H, tb = (long)min(t0 + rb, T - 1) * H;
        f0 = f_p[ta];
        f1 = f_p[tb];
        u0 = u1 = make_float2(0.f, 0.f);
        if (is_q) return;
        if (t0 + ra < T) u0 = make_float2(u_p[ta], u_p[ta + u_low]);
        if (t0 + rb < T) u1 = make_float2(u_p[tb], u_p[tb + u_low]);
    };
    float fa, fb, fa_n, fb_n;
    float2 ua, ub, ua_n, ub_n;
    load_rows(0, fa, fb, ua, ub);
    float carry = 1.f, carry_save = 1.f, blk_dec = 1.f;       // decays as factors: carried over skipped chunks, over the block
    const int c_last = (TN - 1) * cpb;                        // first chunk of the last block
    bool ok = true;
    int sub = 0, blk = 0;
    bool may_carry = decay && (!trailing_quirk || 0 < last_sel);

    for (int c = 0; c < NT; ++c) {
        const float2 meta = s_meta[c];
        const float dec_c = meta.x;                           // decay over the chunk
        const bool sel = meta.y != 0.f, active = cpb > 1 || sel;
        const bool block_end = sub == cpb - 1 || c == NT - 1;
        const bool restore = cpb > 1 && block_end && !sel;
        const uint32_t kt = sbase + L::kq + (c & 1) * L::kq_bytes;
        load_rows(min(c + 1, NT - 1) * 64, fa_n, fb_n, ua_n, ub_n);
        if (sub == 0) {
            carry_save = carry;
            blk_dec = 1.f;
            if (ROLL && !is_q && !sel) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) save[mt][nt][e] = S[mt][nt][e];
            }
        }
        if (c == c_last && hstart && !is_q) store_state(hstart, carry);
        blk_dec *= dec_c;
        const float dec = dec_c * carry, ea = fa * carry, eb = fb * carry;
        if (ok) ok = mbar_wait(full_kq + (c & 1) * 8, (c >> 1) & 1, status);
        // ---- k S (three parts of S) or q S (two).  The largest part is added step by step in fp32 arithmetic.
        float acc[2][4], low[2][4];
        zero_acc(acc);
        zero_acc(low);
        {
            const uint32_t tile = kt + (is_q ? 64 * K * 2 : 0);
#pragma unroll 4
            for (int kk = 0; kk < K / 16; ++kk) {
                uint32_t a[4], bb[4];
                load_a<128>(tile + (kk >> 2) * 8192, r0, (kk & 3) * 16, lane, a);
                if (!is_q) {
                    load_b_kn<64>(sbase + L::s + 2 * L::s_bytes, kk * 16, n0, lane, bb);
                    mma_bf16(low[0], a, bb[0], bb[1]);
                    mma_bf16(low[1], a, bb[2], bb[3]);
                }
                load_b_kn<64>(sbase + L::s + L::s_bytes, kk * 16, n0, lane, bb);
                mma_bf16(low[0], a, bb[0], bb[1]);
                mma_bf16(low[1], a, bb[2], bb[3]);
                load_b_kn<64>(sbase + L::s, kk * 16, n0, lane, bb);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    float d[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_bf16(d, a, bb[2 * nt], bb[2 * nt + 1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[nt][e] += d[e];
                }
            }
        }
        if (!is_q) {
            // ---- r = v - rstd_k e^{g+carry} k S
            const unsigned char* vt = smem + L::v + (c & 1) * 4096;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const uint32_t off = at(hh ? rb : ra, nt);
                    const float2 x = unpack_bf16(*reinterpret_cast<const uint32_t*>(vt + off));
                    uint32_t p[3];
                    const float f = hh ? -eb : -ea;
                    split_bf16(fmaf(f, acc[nt][2 * hh], fmaf(f, low[nt][2 * hh], x.x)),
                               fmaf(f, acc[nt][2 * hh + 1], fmaf(f, low[nt][2 * hh + 1], x.y)), p);
#pragma unroll
                    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(smem + L::r + i * 4096 + off) = p[i];
                }
            bar_w();                                          // r complete
            if (ok) ok = mbar_wait(full_t, c & 1, status);
            // ---- v' = T' r: T' is lower triangular
            zero_acc(acc);
            zero_acc(low);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                if (kk > rg) break;
                uint32_t th[4], tm[4], tl[4], bh[4], bm[4], bl[4];
                load_a<128>(sbase + L::t, r0, kk * 16, lane, th);
                load_a<128>(sbase + L::t + 8192, r0, kk * 16, lane, tm);
                load_a<128>(sbase + L::t + 16384, r0, kk * 16, lane, tl);
                load_b_kn<64>(sbase + L::r, kk * 16, n0, lane, bh);
                load_b_kn<64>(sbase + L::r + 4096, kk * 16, n0, lane, bm);
                load_b_kn<64>(sbase + L::r + 8192, kk * 16, n0, lane, bl);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma_bf16(low[nt], tl, bh[2 * nt], bh[2 * nt + 1]);
                    mma_bf16(low[nt], th, bl[2 * nt], bl[2 * nt + 1]);
                    mma_bf16(low[nt], tm, bm[2 * nt], bm[2 * nt + 1]);
                    mma_bf16(low[nt], tm, bh[2 * nt], bh[2 * nt + 1]);
                    mma_bf16(low[nt], th, bm[2 * nt], bm[2 * nt + 1]);
                    float d[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_bf16(d, th, bh[2 * nt], bh[2 * nt + 1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) add_exact(acc[nt][e], low[nt][e], d[e]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const uint32_t off = at(hh ? rb : ra, nt);
                    const float x0 = acc[nt][2 * hh] + low[nt][2 * hh], x1 = acc[nt][2 * hh + 1] + low[nt][2 * hh + 1];
                    uint32_t p2[2], p3[3];
                    split_bf16(x0, x1, p2);
#pragma unroll
                    for (int i = 0; i < 2; ++i) *reinterpret_cast<uint32_t*>(smem + L::vp + i * 4096 + off) = p2[i];
                    if (active) {
                        // (acc + low) f, what rounding leaves over going into the last part
                        const float2 f = hh ? ub : ua;
                        float y[2], e[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const float m = acc[nt][2 * hh + j], t = m * f.x;
                            const float z = fmaf(low[nt][2 * hh + j], f.x, fmaf(m, f.y, fmaf(m, f.x, -t)));
                            y[j] = t + z;
                            e[j] = z - (y[j] - t);
                        }
                        split_bf16(y[0], y[1], p3, e[0], e[1]);
#pragma unroll
                        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(smem + L::vs + i * 4096 + off) = p3[i];
                    }
                }
        }
        bar_all();                                            // v', v'' written; every warp is done with these parts of S, and with T'
        if (loader && ok && c + 1 < NT) load_t(c + 1);
        __syncwarp();
        if (is_q) {
            // ---- o = scale (q S + P v'): P is lower triangular
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[nt][e] = (e < 2 ? ea : eb) * (acc[nt][e] + low[nt][e]);
            if (ok) ok = mbar_wait(full_p, c & 1, status);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                if (kk > rg) break;
                uint32_t ph[4], pm[4], bh[4], bm[4];
                load_a<128>(sbase + L::p, r0, kk * 16, lane, ph);
                load_a<128>(sbase + L::p + 8192, r0, kk * 16, lane, pm);
                load_b_kn<64>(sbase + L::vp, kk * 16, n0, lane, bh);
                load_b_kn<64>(sbase + L::vp + 4096, kk * 16, n0, lane, bm);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma_bf16(acc[nt], pm, bh[2 * nt], bh[2 * nt + 1]);
                    mma_bf16(acc[nt], ph, bm[2 * nt], bm[2 * nt + 1]);
                    mma_bf16(acc[nt], ph, bh[2 * nt], bh[2 * nt + 1]);
                }
            }
            __nv_bfloat16* oc = o + (((long)b * T + c * 64) * H + h) * V + v0 + n0 + qd * 2;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                if (c * 64 + ra < T)
                    *reinterpret_cast<uint32_t*>(oc + (long)ra * H * V + nt * 8) = pack_bf16(acc[nt][0] * scale, acc[nt][1] * scale);
                if (c * 64 + rb < T)
                    *reinterpret_cast<uint32_t*>(oc + (long)rb * H * V + nt * 8) = pack_bf16(acc[nt][2] * scale, acc[nt][3] * scale);
            }
        } else {
            if (active && !restore) {                         // the last update of a rolled-back block is never read
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    zero_acc(acc);
                    zero_acc(low);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        uint32_t a[4], bb[4];
                        const int m0 = krow0 + mt * 16;
                        load_a_t<128>(kt + (m0 >> 6) * 8192, m0 & 63, kk * 16, lane, a);
#pragma unroll
                        for (int p = 2; p > 0; --p) {
                            load_b_kn<64>(sbase + L::vs + p * 4096, kk * 16, n0, lane, bb);
                            mma_bf16(low[0], a, bb[0], bb[1]);
                            mma_bf16(low[1], a, bb[2], bb[3]);
                        }
                        load_b_kn<64>(sbase + L::vs, kk * 16, n0, lane, bb);
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) {
                            float d[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_bf16(d, a, bb[2 * nt], bb[2 * nt + 1]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[nt][e] += d[e];
                        }
                    }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) S[mt][nt][e] = fmaf(dec, S[mt][nt][e], low[nt][e]) + acc[nt][e];
                }
            }
            if (ROLL && restore) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) S[mt][nt][e] = save[mt][nt][e];
            }
            if (active) publish();
        }
        bar_all();                                            // the new parts of S are complete; the chunk's tiles are done with
        if (loader && ok && c + 1 < NT) {
            load_p(c + 1);
            if (c + 2 < NT) load_kq(c + 2);
        }
        __syncwarp();
        if (active) carry = 1.f;
        else if (may_carry) carry *= dec_c;
        if (restore) carry = carry_save * (may_carry ? blk_dec : 1.f);
        fa = fa_n; fb = fb_n; ua = ua_n; ub = ub_n;
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
        // the last block is complete: the decoder starts from the state behind it if its own type is linear, else from the state
        // in front of it, decayed over it
        const long li = (long)b * last_stride + hn * 2 + 1;
        const float lt = last_f32 ? reinterpret_cast<const float*>(last_types)[li]
                                  : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(last_types)[li]);
        if (lt > 0.f) {
            store_state(hstart, 1.f);
        } else if (decay) {
            const float f = blk_dec;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    float* p = hstart + (((long)b * H + h) * K + krow0 + mt * 16 + gq) * V + v0 + n0 + nt * 8 + qd * 2;
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        float2* x = reinterpret_cast<float2*>(p + hh * 8L * V);
                        *x = make_float2(x->x * f, x->y * f);
                    }
                }
        }
    }
}

}  // namespace
}  // namespace natsl

extern "C" int natsl_gdn_split_prep(const void* q, const void* k, const float* g, const void* beta, int beta_dtype, void* tp, float* kf,
                                    float* qf, float* vf, float* egl, int B, int T, int H, int K, int use_l2norm, void* stream) {
    using namespace natsl;
    const char* who = "natsl_gdn_split_prep";
    NATSL_REQUIRE(q && k && g && beta && tp && kf && qf && vf && egl, NATSL_ERR_NULL, "%s: null pointer", who);
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0, NATSL_ERR_BAD_SHAPE, "%s: bad shape", who);
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "%s: B, H <= 65535", who);
    NATSL_REQUIRE(K == 192, NATSL_ERR_UNSUPPORTED, "%s: unsupported key dim K=%d (192)", who, K);
    NATSL_REQUIRE(beta_dtype == NATSL_DT_F32 || beta_dtype == NATSL_DT_BF16, NATSL_ERR_UNSUPPORTED, "%s: beta must be bf16 or f32", who);
    NATSL_REQUIRE(aligned_to(16, q, k, tp), NATSL_ERR_UNSUPPORTED, "%s: q, k and the result must start on 16 bytes", who);
    auto kern = gdn_split_prep_kernel<192>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SpPrep<192>::total);
    if (e != cudaSuccess) {
        set_error("%s: cannot reserve %d B of shared memory (%s)", who, SpPrep<192>::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    kern<<<dim3((T + 63) / 64, H, B), 256, SpPrep<192>::total, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __nv_bfloat16*>(q), reinterpret_cast<const __nv_bfloat16*>(k), g, beta, beta_dtype == NATSL_DT_F32,
        reinterpret_cast<__nv_bfloat16*>(tp), kf, qf, vf, egl, T, H, use_l2norm);
    return check_launch(who);
}

extern "C" int natsl_gdn_split_walk(const void* q, const void* k, const void* v, const void* tp, const float* kf, const float* qf,
                                    const float* vf, const float* egl, const int32_t* types_i, const int32_t* indices, const int32_t* n_blocks,
                                    const float* h0, void* o, float* ht, float* hstart, const void* last_types, int last_dtype,
                                    int last_stride, int B, int T, int H, int HN, int K, int V, int nbs, float scale, int flags,
                                    void* stream) {
    using namespace natsl;
    const char* who = "natsl_gdn_split_walk";
    NATSL_REQUIRE(q && k && v && tp && kf && qf && vf && egl && types_i && indices && n_blocks && o, NATSL_ERR_NULL, "%s: null pointer", who);
    NATSL_REQUIRE(B > 0 && T > 0 && H > 0 && HN > 0 && H % HN == 0, NATSL_ERR_BAD_SHAPE, "%s: bad shape", who);
    NATSL_REQUIRE(H <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "%s: B, H <= 65535", who);
    NATSL_REQUIRE(K == 192 && V > 0 && V % 32 == 0, NATSL_ERR_UNSUPPORTED, "%s: unsupported head dims K=%d V=%d (K = 192, V a multiple of 32)",
                  who, K, V);
    NATSL_REQUIRE(nbs >= 64 && nbs % 64 == 0, NATSL_ERR_UNSUPPORTED, "%s: nats_block_size must be a multiple of 64 (got %d)", who, nbs);
    NATSL_REQUIRE(!hstart || T % nbs != 0 || (last_types && (last_dtype == NATSL_DT_F32 || last_dtype == NATSL_DT_BF16)), NATSL_ERR_NULL,
                  "%s: the block-start state of a complete last block needs that block's types", who);
    NATSL_REQUIRE(aligned_to(16, h0, o, ht, hstart), NATSL_ERR_UNSUPPORTED, "%s: states and output must start on 16 bytes", who);
    const int smem = SwSmem<192>::total((T + 63) / 64);
    NATSL_REQUIRE(smem <= 227 * 1024, NATSL_ERR_TOO_LARGE, "%s: T=%d needs %d B of shared memory (max %d)", who, T, smem, 227 * 1024);
    auto kern = nbs > 64 ? gdn_split_walk_kernel<192, true> : gdn_split_walk_kernel<192, false>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
        set_error("%s: cannot reserve %d B of shared memory (%s)", who, smem, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mt;
    int rc = encode_bthd_map(&mq, q, B, T, H, K, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T, H, K, 64, who);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T, H, V, 64, who, SW_BV);
    if (rc == NATSL_OK) rc = encode_bthd_map(&mt, tp, B, T, H, SP_TP, 64, who);
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    kern<<<dim3(V / SW_BV, H, B), SW_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        mq, mk, mv, mt, kf, qf, vf, egl, types_i, indices, n_blocks, h0, reinterpret_cast<__nv_bfloat16*>(o), ht, hstart, last_types,
        last_dtype == NATSL_DT_F32, last_stride, T, H, HN, V, (T + nbs - 1) / nbs, nbs, scale, (flags & NATSL_FLAG_DECAY_SKIPPED) ? 1 : 0,
        (flags & NATSL_FLAG_NO_TRAILING_QUIRK) ? 0 : 1, status);
    return check_launch(who);
}
