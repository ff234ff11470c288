// One decoding token of a whole NAtSL layer (GDN or Mamba2) in four launches: projections -> {linear-branch step, softmax
// attention over the cached keys, mixing weights} -> branch merge -> output projection.
//   src/nats/layers/natsl_attn_gdn.py:389-666 with one new token (Mamba2: src/nats/layers/natsl_attn_mamba2.py:330-599);
//   linear branch  src/nats/ops/gated_delta_rule/fused_recurrent.py:128-358, src/nats/ops/mamba/fused_recurrent.py:121-322;
//   softmax branch src/nats/ops/mixed_ops/mixed_attn_gdn.py:475-504 (SDPA over the cache under its visibility mask).
// What bounds it: at batch 1 the layer reads its weights once (33 MB at hidden 1024..2048) and does almost no arithmetic,
// so the floor is the weight read plus the dependent launches; issued step by step from Python (about 80 launches,
// several host reads) the same token took 1.4 ms of host time.  A request of 777 + 48 tokens at hidden 2048, batch 1:
// 70 -> 1.6 ms; 2048 + 32 tokens at hidden 1024, batch 32: 50 -> 4.2 ms (prefill included in both).
//   * proj / out: "skinny" products y[b, n] = x[b, :] . W[n, :].  The weight rows are the M side of mma.m16n8k16, the
//     batch the N side, so a weight element is loaded once, straight from global memory into the A fragment: with the k
//     index permuted inside every 32-wide group a lane's fragment is one 16-byte load per row (the same permutation on
//     both operands leaves the sum unchanged).  Weight loads do not depend on the previous kernel and are issued before
//     the programmatic-launch wait.
//   * core: three kinds of CTA in one grid.  Every CTA recomputes the short convolution of the channels it needs (four
//     taps), which costs less than a launch in between, and loads everything but the projections (states, tails, weights,
//     the first keys and values) before it waits for them.  The recurrence reads the state once: S^T k and S^T q are formed
//     together (o = e^g S^T q + (q.k) v').  Attention splits the 64-key units of the finished blocks over CTAs; a warp
//     takes 16 keys of a unit, several units on their way through shared memory.
//     On the device, tokens back to back (us; before: one step of 8 or 16 keys ahead in registers, ranges of units per split, all
//     mixing rows in one CTA): 32 rows, 2000 tokens, 16 heads of 64 51.3 -> 41.0; 4 rows, 1000 tokens, 32 heads of 128 / 64 36.7 -> 26.6; 16
//     rows, 2000 tokens, 16 heads of 128 61.4 -> 50.4; 64 rows, 40 tokens 157 -> 155; 1 row, 300 tokens, 6 heads of 128 / 256 14.8 -> 15.2,
//     1000 tokens 16.8 -> 15.9.
//   * merge: combines the splits, both RMS norms, mixing weights and gate; extra CTAs shift the convolution tails.
// All state (recurrent state, tails, decay sums, pooled input, key/value rows) is updated in place.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

using bf16 = __nv_bfloat16;
constexpr int DS_THREADS = 128;               // core CTAs
constexpr int DS_MAXK = 256;
constexpr int DS_MIX = 512, DS_MIX_ROWS = 16; // channels and rows per CTA of the mixing logits
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ float rb(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ float bf(const bf16* p, long i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ float ldw(const void* p, int f32, long i) {
    return f32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}

// natsl_decode_args with typed pointers (same layout).
struct Args {
    int B, hidden, H, K, V, HQ, HN, nbs, pos, cap, n_done, rule;
    int attn_conv, silu, own_chunk, decay, neg_eigval, mix_sigmoid;
    int qn_f32, kn_f32, alog_f32, dt_f32, w12_f32, types_f32;
    float norm_eps, l2_eps, mix_eps, scale_attn, scale_lin, reserved;
    const bf16 *x, *w_q, *w_k, *w_v, *w_a, *w_b, *w_g, *w_o, *w_mix;
    const bf16 *cw_q, *cw_k, *cw_v, *cb_q, *cb_k, *cb_v;
    const void *qn_w, *kn_w, *A_log, *dt_bias, *w1, *w2, *types, *types_new;
    bf16 *conv_q, *conv_k, *conv_v;
    float *state, *start, *g_block, *pool_sum;
    bf16 *k_cache, *v_cache, *out;
    unsigned char* workspace;
    int64_t workspace_bytes;
};
static_assert(sizeof(Args) == sizeof(natsl_decode_args), "argument layout");

// ------------------------------------------------------------------------------------------------ skinny products
struct SkinnySeg {
    const bf16* w;                            // [rows, Kdim]
    int rows, out_off, tile0;
};
struct SkinnyArgs {
    SkinnySeg seg[6];
    int nseg, B, Kdim, y_stride;
    const bf16* x;                            // [B, Kdim]
    bf16* y;                                  // [B, y_stride]
    float* pool;                              // [B, Kdim] += x, or NULL
};

// NB groups of 8 batch rows; WM warps side by side over weight rows (16 each), WK warps over the contraction.
template <int NB, int WM, int WK>
__global__ void __launch_bounds__(256) skinny_kernel(const SkinnyArgs a) {
    constexpr int R = 16 * WM, UN = NB > 4 ? 2 : 4;
    __shared__ float red[WK][R][NB * 8 + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wk = warp / WM, g = lane >> 2, t = lane & 3;
    int s = 0;
#pragma unroll
    for (int i = 1; i < 6; ++i)
        if (i < a.nseg && (int)blockIdx.x >= a.seg[i].tile0) s = i;
    const bf16* w = a.seg[s].w;
    const int rows = a.seg[s].rows, row0 = ((int)blockIdx.x - a.seg[s].tile0) * R + wm * 16;
    const int ra = min(row0 + g, rows - 1), rbw = min(row0 + g + 8, rows - 1);
    const int nc = a.Kdim / 32, c0 = nc * wk / WK, c1 = nc * (wk + 1) / WK;
    const uint4* pa = reinterpret_cast<const uint4*>(w + (long)ra * a.Kdim) + t;
    const uint4* pb = reinterpret_cast<const uint4*>(w + (long)rbw * a.Kdim) + t;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 wa[UN], wb[UN];
    auto load_w = [&](int c) {
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const bool ok = c + u < c1;
            wa[u] = ok ? __ldg(pa + (c + u) * 4) : zero;
            wb[u] = ok ? __ldg(pb + (c + u) * 4) : zero;
        }
    };
    load_w(c0);
    pdl_wait();
    pdl_trigger();
    float acc[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    for (int c = c0; c < c1; c += UN) {
        uint4 ca[UN], cb[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) { ca[u] = wa[u]; cb[u] = wb[u]; }
        if (c + UN < c1) load_w(c + UN);
        uint4 xv[UN][NB];                                 // all activation fragments of these steps in flight at once
#pragma unroll
        for (int u = 0; u < UN; ++u)
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                const int row = n * 8 + g;
                xv[u][n] = row < a.B && c + u < c1 ? *(reinterpret_cast<const uint4*>(a.x + (long)row * a.Kdim) + (c + u) * 4 + t) : zero;
            }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const uint32_t f0[4] = {ca[u].x, cb[u].x, ca[u].y, cb[u].y}, f1[4] = {ca[u].z, cb[u].z, ca[u].w, cb[u].w};
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                mma_bf16(acc[n], f0, xv[u][n].x, xv[u][n].y);
                mma_bf16(acc[n], f1, xv[u][n].z, xv[u][n].w);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) red[wk][wm * 16 + g + 8 * (e >> 1)][n * 8 + 2 * t + (e & 1)] = acc[n][e];
    __syncthreads();
    const int tile_row0 = ((int)blockIdx.x - a.seg[s].tile0) * R;
    for (int i = tid; i < R * a.B; i += 256) {
        const int r = i % R, b = i / R;
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < WK; ++k) v += red[k][r][b];
        if (tile_row0 + r < rows) a.y[(long)b * a.y_stride + a.seg[s].out_off + tile_row0 + r] = __float2bfloat16(v);
    }
    if (a.pool)
        for (int i = blockIdx.x * 256 + tid; i < a.B * a.Kdim; i += gridDim.x * 256) a.pool[i] += __bfloat162float(a.x[i]);
}

// ------------------------------------------------------------------------------------------------ core
struct CoreArgs {
    Args a;
    const bf16* raw;                          // [B, NR]: q | k | v | gate | a | b
    bf16* o_lin;                              // [B, H*V]
    float* wlog;                              // [B, n_slices, 2*HQ] partial mixing logits
    float* part;                              // [B, HQ, S, DV + 2]
    float* gnew;                              // [B, H]
    int NR, S, n_mix, n_attn, n_rec, vs, n_slices;
};

// What a convolution needs besides the new input: the tail (the last four inputs), weights, bias.  None of it is written by
// the kernels in front of this one in the step, so it is loaded before the programmatic-launch wait.
struct Conv {
    uint2 tail, w;
    float bias;
    __device__ __forceinline__ void load(const bf16* tails, const bf16* weights, const bf16* biases, long row, int d) {
        tail = *reinterpret_cast<const uint2*>(tails + row * 4);
        w = *reinterpret_cast<const uint2*>(weights + (long)d * 4);
        bias = biases ? bf(biases, d) : 0.f;
    }
    // rounded to bf16 like the layer's own convolution output
    __device__ __forceinline__ float operator()(float x_new, int silu) const {
        const float2 t0 = unpack_bf16(tail.x), t1 = unpack_bf16(tail.y), w0 = unpack_bf16(w.x), w1 = unpack_bf16(w.y);
        float acc = bias;
        acc += w0.x * t0.y;
        acc += w0.y * t1.x;
        acc += w1.x * t1.y;
        acc += w1.y * x_new;
        return rb(silu ? acc * (1.f / (1.f + __expf(-acc))) : acc);
    }
};

template <int NTHR>
__device__ __forceinline__ float block_sum(float v, float* s_red, int tid) {
    v = warp_sum(v);
    __syncthreads();
    if ((tid & 31) == 0) s_red[tid >> 5] = v;
    __syncthreads();
    float r = 0.f;
#pragma unroll
    for (int i = 0; i < NTHR / 32; ++i) r += s_red[i];
    return r;
}

// Two sums over the block with one pair of barriers; s_red: 2 x NTHR / 32 floats.
template <int NTHR>
__device__ __forceinline__ void block_sum2(float& u, float& v, float* s_red, int tid) {
    u = warp_sum(u);
    v = warp_sum(v);
    __syncthreads();
    if ((tid & 31) == 0) {
        s_red[tid >> 5] = u;
        s_red[NTHR / 32 + (tid >> 5)] = v;
    }
    __syncthreads();
    u = v = 0.f;
#pragma unroll
    for (int i = 0; i < NTHR / 32; ++i) {
        u += s_red[i];
        v += s_red[NTHR / 32 + i];
    }
}

// VS value columns (32 or 64) per CTA: rows of the state rg + RP i, four columns per thread.
template <int VS>
__device__ void core_recurrence(const CoreArgs& c, int idx, float* sm) {
    constexpr int TPR = VS / 4, RP = DS_THREADS / TPR;    // threads per state row, rows per pass
    const Args& a = c.a;
    const int tid = threadIdx.x, K = a.K, V = a.V, H = a.H, HK = H * K, HV = H * V;
    const int nvs = V / VS, vs = idx % nvs, h = (idx / nvs) % H, b = idx / (nvs * H);
    const bool gdn = a.rule == NATSL_RULE_GDN;
    float* s_q = sm;                           // [256]
    float* s_k = sm + DS_MAXK;                 // [256]
    float* s_v = s_k + DS_MAXK;                // [VS]
    float* s_red = s_v + VS;                // [8]
    float* s_dot = s_red + 8;                  // [2][RP][VS]
    const bf16* raw = c.raw + (long)b * c.NR;
    const int rg = tid / TPR, c4 = (tid % TPR) * 4, col = vs * VS + c4;
    float* Sp = a.state + (((long)b * H + h) * K) * V + col;
    constexpr int NREG = 8;
    float4 S[NREG];
#pragma unroll
    for (int i = 0; i < NREG; ++i)
        if (rg + RP * i < K) S[i] = *reinterpret_cast<const float4*>(Sp + (long)(rg + RP * i) * V);
    Conv cq[2], ck[2], cv;
#pragma unroll
    for (int j = 0; j < 2; ++j)
        if (tid + j * DS_THREADS < K) {
            const int d = h * K + tid + j * DS_THREADS;
            cq[j].load(a.conv_q, a.cw_q, a.cb_q, (long)b * HK + d, d);
            ck[j].load(a.conv_k, a.cw_k, a.cb_k, (long)b * HK + d, d);
        }
    const int dv = h * V + vs * VS + (tid & (VS - 1));
    cv.load(a.conv_v, a.cw_v, a.cb_v, (long)b * HV + dv, dv);
    const float dtb = ldw(a.dt_bias, a.dt_f32, h), alog = expf(ldw(a.A_log, a.alog_f32, h));
    const float gsum = a.types_new ? a.g_block[(long)b * H + h] : 0.f;
    pdl_wait();
    float rq2[2], rk2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
        if (tid + j * DS_THREADS < K) {
            rq2[j] = bf(raw, h * K + tid + j * DS_THREADS);
            rk2[j] = bf(raw, HK + h * K + tid + j * DS_THREADS);
        }
    const float rv = bf(raw, 2 * HK + dv), z = bf(raw, 2 * HK + 2 * HV + h) + dtb;
    const float braw = gdn ? bf(raw, 2 * HK + 2 * HV + H + h) : 0.f;
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = tid + j * DS_THREADS;
        if (i < K) {
            const float qv = cq[j](rq2[j], a.silu), kv = ck[j](rk2[j], a.silu);
            s_q[i] = qv;
            s_k[i] = kv;
            sq += qv * qv;
            sk += kv * kv;
        }
    }
    const float sp = z > 20.f ? z : log1pf(expf(z));
    const float gt = -alog * sp;
    if (tid < VS) {
        float vv = cv(rv, a.silu);
        if (!gdn) vv = rb(vv * sp);
        s_v[tid] = vv;
    }
    block_sum2<DS_THREADS>(sq, sk, s_red, tid);
    const float eps = gdn ? 1e-6f : a.l2_eps;
    const float rq = rsqrtf(sq + eps), rk = rsqrtf(sk + eps);
    float qk = 0.f;
    for (int i = tid; i < K; i += DS_THREADS) {
        // the delta rule normalises in fp32 inside the recurrence, the Mamba2 layer in front of it (rounded to bf16)
        const float qn = gdn ? s_q[i] * rq : rb(s_q[i] * rq), kn = gdn ? s_k[i] * rk : rb(s_k[i] * rk);
        s_q[i] = qn;
        s_k[i] = kn;
        qk += qn * kn;
    }
    qk = block_sum<DS_THREADS>(qk, s_red, tid);         // its barriers also publish s_q, s_k
    float4 dk = make_float4(0, 0, 0, 0), dq = dk;
    auto add = [&](const float4 s, int r) {
        const float kk = s_k[r], qq = s_q[r];
        dk.x += s.x * kk; dk.y += s.y * kk; dk.z += s.z * kk; dk.w += s.w * kk;
        dq.x += s.x * qq; dq.y += s.y * qq; dq.z += s.z * qq; dq.w += s.w * qq;
    };
#pragma unroll
    for (int i = 0; i < NREG; ++i)
        if (rg + RP * i < K) add(S[i], rg + RP * i);
    for (int r = rg + RP * NREG; r < K; r += RP) add(*reinterpret_cast<const float4*>(Sp + (long)r * V), r);
    float* d0 = s_dot + rg * VS + c4;
    *reinterpret_cast<float4*>(d0) = dk;
    *reinterpret_cast<float4*>(d0 + RP * VS) = dq;
    __syncthreads();
    if (tid < VS) {
        float tk = 0.f, tq = 0.f;
#pragma unroll
        for (int i = 0; i < RP; ++i) { tk += s_dot[i * VS + tid]; tq += s_dot[(RP + i) * VS + tid]; }
        const float eg = __expf(gt);
        float vv = s_v[tid];
        if (gdn) {
            float beta = rb(1.f / (1.f + expf(-braw)));
            if (a.neg_eigval) beta *= 2.f;
            vv = beta * (vv - eg * tk);
        }
        s_v[tid] = vv;
        c.o_lin[(long)b * HV + h * V + vs * VS + tid] = __float2bfloat16((eg * tq + qk * vv) * a.scale_lin);
    }
    __syncthreads();
    const float eg = __expf(gt);
    const float4 vn = *reinterpret_cast<const float4*>(s_v + c4);
    const bool ends = a.types_new != nullptr;
    float* Bp = a.start + (((long)b * H + h) * K) * V + col;
    float roll = 1.f;
    bool sel = false;
    if (ends) {
        const int hn = h / (H / a.HN);
        sel = rintf(ldw(a.types_new, a.types_f32, ((long)b * a.HN + hn) * 2 + 1)) == 1.f;
        roll = a.decay ? __expf(gsum + gt) : 1.f;
    }
    auto upd = [&](float4 s, int r) {
        const float kk = s_k[r];
        s.x = eg * s.x + kk * vn.x; s.y = eg * s.y + kk * vn.y; s.z = eg * s.z + kk * vn.z; s.w = eg * s.w + kk * vn.w;
        if (ends) {                                       // the block is complete: keep its updates or roll them back
            float4* bp = reinterpret_cast<float4*>(Bp + (long)r * V);
            if (!sel) {
                s = *bp;
                s.x *= roll; s.y *= roll; s.z *= roll; s.w *= roll;
            }
            *bp = s;
        }
        *reinterpret_cast<float4*>(Sp + (long)r * V) = s;
    };
#pragma unroll
    for (int i = 0; i < NREG; ++i)
        if (rg + RP * i < K) upd(S[i], rg + RP * i);
    for (int r = rg + RP * NREG; r < K; r += RP) upd(*reinterpret_cast<const float4*>(Sp + (long)r * V), r);
    if (vs == 0 && tid == 0) c.gnew[(long)b * H + h] = gt;
}

__device__ __forceinline__ float warp_max_redux(float x) {
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}

// Keys and values leave L2 first: a token reads each of them once, and what stays is weights and states (a token of 32 rows, 2048
// tokens, 16 heads of 64: 47.1 -> 42.6 us; 16 rows, 16 heads of 128: 58.4 -> 51.7 us).
__device__ __forceinline__ uint64_t evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void copy_first(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}

// Ring of a warp of the attention: steps of 16 keys; three of them where four CTAs then still share an SM, else two (at 128/128
// three CTAs), or one (launch_core).
template <int DK, int DV, bool DEEP> struct Ring {
    static constexpr int step = 16 * (DK + DV) * 2, D = !DEEP ? 1 : DK + DV == 128 ? 3 : 2, bytes = 4 * D * step;
};

template <int DK, int DV, bool DEEP>
__device__ void core_attention(const CoreArgs& c, int idx, float* sm) {
    const Args& a = c.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = idx % c.S, hq = (idx / c.S) % a.HQ, b = idx / (c.S * a.HQ);
    const int HK = a.H * a.K, HV = a.H * a.V;
    constexpr int LK = DK / 8, LV = DV / 8, KG = 32 / LK, VG = 32 / LV;      // lanes per row, rows per load
    float* s_q = sm;                                   // [DK] query, scaled
    float* s_kn = s_q + DK;                            // [DK] new key
    float* s_vn = s_kn + DK;                           // [DV] new value
    float* s_ml = s_vn + DV;                           // [4][2]
    float* s_red = s_ml + 8;                           // [8]
    float* s_acc = s_red + 8;                          // [4][DV]
    const bool last = s == c.S - 1;
    float m = -INFINITY, l = 0.f;
    uint64_t acc2[4] = {0, 0, 0, 0};
    const bf16* kb = a.k_cache + ((long)b * a.cap * a.HQ + hq) * DK + (lane % LK) * 8;
    const bf16* vb = a.v_cache + ((long)b * a.cap * a.HQ + hq) * DV + (lane % LV) * 8;
    // A step of a warp = 16 keys, its quarter of a selected 64-key unit of this split (32 units' selection bits per load, by ballot),
    // then of the current block.  Keys and values come through the warp's own ring in shared memory, D steps deep: the first D are
    // on their way before the wait for the projections, and a split of few units is no chain of loads (one step ahead in
    // registers, 8 keys at head dims 128, it was: 4 rows of 32 heads, 1030 tokens: attention 14.5 us behind the wait).
    using R = Ring<DK, DV, DEEP>;
    constexpr int D = R::D, KS = 16, NK = KS / KG, NV = KS / VG;
    static_assert(LK >= NK && NV >= 1, "lanes per row");
    extern __shared__ __align__(16) unsigned char ring_all[];
    unsigned char* const ring = ring_all + warp * (D * R::step);
    const uint32_t ring_s = smem_u32(ring);
    const uint64_t hint = evict_first();
    const int hn = hq / (a.HQ / a.HN), upb = a.nbs / 64;
    const int n_units = a.n_done * upb;
    const int own0 = a.own_chunk ? a.pos / a.nbs * a.nbs : a.pos;               // keys of the current block before the new token
    const long tstride = (long)a.HN * 2;
    const long tbase = ((long)b * a.n_done * a.HN + hn) * 2;
    auto chosen = [&](int u, int end) -> bool { return u < end && ldw(a.types, a.types_f32, tbase + (long)(u / upb) * tstride) > 0.5f; };
    // Which units are this split's.  Up to 32 (2048 tokens), and up to 64 where a range would be less than four, every split reads all
    // selection bits and takes every S-th selected unit, then every S-th unit of the current block: equal shares, where a range of
    // its own holds none of them or all (4 rows of 32 heads, 16 units over 5 splits: the last CTA had twice the mean).  Otherwise, a
    // range of its own, 32 units at a time, whose shares even out (whole tokens, ranges / shares, us: 16 heads of 64, 1 row,
    // 2000 tokens 16.1 / 15.2, 3300 tokens 16.8 / 16.3, 8 rows, 2600 tokens 23.8 / 25.2, 4 rows, 5500 tokens 23.6 / 25.4, 8000
    // tokens 28.5 / 31.1).
    const bool few = n_units <= 32 || (n_units <= 64 && n_units < 4 * c.S);
    unsigned mask = 0, more = 0;                        // units base .. base + 31 that are left; of few, the ones behind
    int base = 0, end = 0, own_unit = last ? 0 : 1 << 20, own_step = 1;
    if (few) {
        const unsigned all = __ballot_sync(0xffffffffu, chosen(lane, n_units)), behind = __ballot_sync(0xffffffffu, chosen(32 + lane, n_units));
        const unsigned below = (1u << lane) - 1;
        mask = __ballot_sync(0xffffffffu, (all >> lane & 1) && __popc(all & below) % c.S == s);
        more = __ballot_sync(0xffffffffu, (behind >> lane & 1) && (__popc(all) + __popc(behind & below)) % c.S == s);
        const int rank = (__popc(all) + __popc(behind)) % c.S;             // of the units of the current block
        own_unit = s - rank + (s < rank ? c.S : 0);
        own_step = c.S;
    } else {
        end = (int)((long)n_units * (s + 1) / c.S);
        base = (int)((long)n_units * s / c.S) - 32;
    }
    auto next = [&](int& key0) -> int {                 // keys of the warp's next step, 0 at the end
        if (mask == 0 && more) {
            mask = more;
            more = 0;
            base = 32;
        }
        while (mask == 0 && base + 32 < end) {
            base += 32;
            mask = __ballot_sync(0xffffffffu, chosen(base + lane, end));
        }
        if (mask) {
            key0 = (base + __ffs(mask) - 1) * 64 + warp * 16;
            mask &= mask - 1;
            return KS;
        }
        key0 = own0 + own_unit * 64 + warp * 16;
        if (own_unit >= 1 << 20 || key0 >= a.pos) return 0;
        own_unit += own_step;
        return min(KS, a.pos - key0);
    };
    auto fetch = [&](int slot) -> int {                 // the next step into `slot`; always one group of copies
        int key0 = 0;
        const int n = next(key0);
        if (n > 0) {
            const uint32_t dst = ring_s + slot * R::step + lane * 16;
#pragma unroll
            for (int i = 0; i < NK; ++i) copy_first(dst + i * 512, kb + (long)(key0 + min(i * KG + lane / LK, n - 1)) * a.HQ * DK, hint);
#pragma unroll
            for (int i = 0; i < NV; ++i)
                copy_first(dst + KS * DK * 2 + i * 512, vb + (long)(key0 + min(i * VG + lane / LV, n - 1)) * a.HQ * DV, hint);
        }
        cp_async_commit();
        return n;
    };
    int count[D];                                       // keys of the steps on their way
#pragma unroll
    for (int i = 0; i < D; ++i) count[i] = fetch(i);

    // ---- query of this head, and (last split) the new token's key and value: they wait for the projections
    {
        const int dk = hq * DK + (tid & (DK - 1)), dv = hq * DV + (tid & (DV - 1));
        Conv cq, ck, cv;
        float wq = 1.f, wk = 1.f;
        if (a.attn_conv) {
            cq.load(a.conv_q, a.cw_q, a.cb_q, (long)b * HK + dk, dk);
            ck.load(a.conv_k, a.cw_k, a.cb_k, (long)b * HK + dk, dk);
            cv.load(a.conv_v, a.cw_v, a.cb_v, (long)b * HV + dv, dv);
        }
        if (a.qn_w) {
            wq = ldw(a.qn_w, a.qn_f32, tid & (DK - 1));
            wk = ldw(a.kn_w, a.kn_f32, tid & (DK - 1));
        }
        pdl_wait();
        const bf16* raw = c.raw + (long)b * c.NR;
        float qv = bf(raw, dk), kv = bf(raw, HK + dk), vv = bf(raw, 2 * HK + dv);
        if (a.attn_conv) {
            qv = cq(qv, a.silu);
            kv = ck(kv, a.silu);
            vv = cv(vv, a.silu);
        }
        if (a.qn_w) {
            float sq = tid < DK ? qv * qv : 0.f, sk = tid < DK ? kv * kv : 0.f;
            block_sum2<DS_THREADS>(sq, sk, s_red, tid);
            qv = rb(qv * rsqrtf(sq / DK + a.norm_eps) * wq);
            kv = rb(kv * rsqrtf(sk / DK + a.norm_eps) * wk);
        }
        if (tid < DK) {
            s_q[tid] = qv * (a.scale_attn * kLog2e);
            s_kn[tid] = kv;
            if (last) a.k_cache[(((long)b * a.cap + a.pos) * a.HQ + hq) * DK + tid] = __float2bfloat16(kv);
        }
        if (last && tid < DV) {
            s_vn[tid] = vv;
            a.v_cache[(((long)b * a.cap + a.pos) * a.HQ + hq) * DV + tid] = __float2bfloat16(vv);
        }
    }
    __syncthreads();
    uint64_t q2[4];
    {
        const int d0 = (lane % LK) * 8;
#pragma unroll
        for (int e = 0; e < 4; ++e) q2[e] = pack2(s_q[d0 + 2 * e], s_q[d0 + 2 * e + 1]);
    }
    // Scores: a row's LK lanes each hold a part of its dot product.  The lanes hand half of their rows' parts to each other until one
    // row is left per lane (eight shuffles for eight rows of sixteen lanes, where summing row by row takes 32), so that a lane
    // has the score of one key, my_key, shared with LK / NK - 1 others, and the probabilities need no shared memory.
    int my_key = lane / LK, src[NV];                    // src: lane that has the probability of this lane's i-th value row
#pragma unroll
    for (int n = NK, o = LK / 2; n > 1; n >>= 1, o >>= 1) my_key += (lane & o) ? n / 2 * KG : 0;
    const bool counts = (lane & (LK / NK - 1)) == 0;    // one of the lanes that share a key
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int key = i * VG + lane / LV;
        src[i] = key % KG * LK;
#pragma unroll
        for (int n = NK, o = LK / 2; n > 1; n >>= 1, o >>= 1) src[i] += (key / KG) & (n / 2) ? o : 0;
    }
    auto step = [&](const unsigned char* at, int n_keys) {
        float d[NK];
#pragma unroll
        for (int i = 0; i < NK; ++i) {
            const uint4 kr = *reinterpret_cast<const uint4*>(at + i * 512 + lane * 16);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&kr);
            uint64_t x = mul2(open2(w[0]), q2[0]);
#pragma unroll
            for (int e = 1; e < 4; ++e) x = fma2(open2(w[e]), q2[e], x);
            d[i] = hsum2(x);
        }
        int o = LK / 2;
#pragma unroll
        for (int n = NK; n > 1; n >>= 1, o >>= 1) {
            const bool hi = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < n / 2; ++i) {
                const float keep = hi ? d[i + n / 2] : d[i], give = hi ? d[i] : d[i + n / 2];
                d[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
#pragma unroll
        for (int r = LK / NK / 2; r > 0; r >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], r);
        const float sc = my_key < n_keys ? d[0] : -INFINITY;
        // scores of -inf (infinite keys) weigh nothing, also while there is nothing else
        const float mn = fmaxf(m, warp_max_redux(sc));
        if (mn != m) {                                  // (the same in all lanes)
            const float al = mn == -INFINITY ? 1.f : exp2f(m - mn);
            l *= al;
#pragma unroll
            for (int e = 0; e < 4; ++e) acc2[e] = mul2(acc2[e], pack2(al, al));
            m = mn;
        }
        const float p = sc == -INFINITY ? 0.f : exp2f(sc - m);
        l += counts ? p : 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float pj = __shfl_sync(0xffffffffu, p, src[i]);
            const uint4 vr = *reinterpret_cast<const uint4*>(at + KS * DK * 2 + i * 512 + lane * 16);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&vr);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc2[e] = fma2(pack2(pj, pj), open2(w[e]), acc2[e]);
        }
    };
    int slot = 0;
    while (count[0] > 0) {
        cp_async_wait<D - 1>();
        __syncwarp();
        step(ring + slot * R::step, count[0]);
        __syncwarp();                                   // every lane has read the slot
#pragma unroll
        for (int i = 0; i + 1 < D; ++i) count[i] = count[i + 1];
        count[D - 1] = fetch(slot);
        slot = slot + 1 == D ? 0 : slot + 1;
    }
    cp_async_wait<0>();
    // sum the key groups of a warp, then the warps
    l = warp_sum(l);
    float acc[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) unpack2(acc2[e], acc[2 * e], acc[2 * e + 1]);
#pragma unroll
    for (int o = LV; o < 32; o <<= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if (lane < LV)
#pragma unroll
        for (int e = 0; e < 8; ++e) s_acc[warp * DV + lane * 8 + e] = acc[e];
    if (lane == 0) { s_ml[warp * 2] = m; s_ml[warp * 2 + 1] = l; }
    float s_new = -INFINITY;                            // score of the new token
    if (last && a.own_chunk) s_new = block_sum<DS_THREADS>(tid < DK ? s_q[tid] * s_kn[tid] : 0.f, s_red, tid);
    __syncthreads();
    float M = s_new;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, s_ml[w * 2]);
    float* part = c.part + (((long)b * a.HQ + hq) * c.S + s) * (DV + 2);
    if (tid < DV) {
        // a part without a finite score holds zeros, or the NaN of a score or value, which goes on as it is
        float L = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float f = s_ml[w * 2] == -INFINITY ? 1.f : exp2f(s_ml[w * 2] - M);
            L += f * s_ml[w * 2 + 1];
            o += f * s_acc[w * DV + tid];
        }
        if (s_new != -INFINITY) {
            const float p = exp2f(s_new - M);
            L += p;
            o += p * s_vn[tid];
        }
        part[2 + tid] = o;
        if (tid == 0) { part[0] = M; part[1] = L; }
    }
}

// Partial logits of the mixing weights: DS_MIX_ROWS rows of w_mix [2 HQ, H K] times one slice of DS_MIX channels of the convolved
// query of one batch row (the merge adds the slices up).  A CTA's weights, four rows a warp, are on their way before the wait for the
// projections; all rows in one CTA took 11 us from there, four rounds of loads one after the other.
__device__ void core_mix_logits(const CoreArgs& c, int idx, float* sm) {
    const Args& a = c.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int HK = a.H * a.K, rows = 2 * a.HQ, groups = (rows + DS_MIX_ROWS - 1) / DS_MIX_ROWS;
    const int r0 = idx % groups * DS_MIX_ROWS + warp * (DS_MIX_ROWS / 4), slice = idx / groups % c.n_slices, b = idx / (groups * c.n_slices);
    const int d0 = slice * DS_MIX;
    constexpr int PER = DS_MIX / DS_THREADS, RW = DS_MIX_ROWS / 4;
    Conv cq[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int d = min(d0 + tid + j * DS_THREADS, HK - 1);
        cq[j].load(a.conv_q, a.cw_q, a.cb_q, (long)b * HK + d, d);
    }
    uint4 wr[RW][DS_MIX / 256];                             // channels (lane + 32 i) * 8 .. + 7
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int i = 0; i < DS_MIX / 256; ++i) {
            const int d = d0 + (lane + 32 * i) * 8;
            wr[r][i] = d < HK && r0 + r < rows ? *reinterpret_cast<const uint4*>(a.w_mix + (long)(r0 + r) * HK + d) : make_uint4(0, 0, 0, 0);
        }
    pdl_wait();
    float x[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) x[j] = bf(c.raw + (long)b * c.NR, min(d0 + tid + j * DS_THREADS, HK - 1));
#pragma unroll
    for (int j = 0; j < PER; ++j) sm[tid + j * DS_THREADS] = d0 + tid + j * DS_THREADS < HK ? cq[j](x[j], a.silu) : 0.f;
    __syncthreads();
    float acc[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) acc[r] = 0.f;
#pragma unroll
    for (int i = 0; i < DS_MIX / 256; ++i) {
        if (d0 + (lane + 32 * i) * 8 >= HK) continue;
        float q[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) q[e] = sm[(lane + 32 * i) * 8 + e];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&wr[r][i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16(w[e]);
                acc[r] += f.x * q[2 * e];
                acc[r] += f.y * q[2 * e + 1];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float v = warp_sum(acc[r]);
        if (lane == 0 && r0 + r < rows) c.wlog[((long)b * c.n_slices + slice) * rows + r0 + r] = v;
    }
}

template <int DK, int DV, bool DEEP>
__global__ void __launch_bounds__(DS_THREADS, 4) decode_core_kernel(const CoreArgs c) {
    __shared__ __align__(16) float sm[2 * DS_MAXK + 64 + 8 + 2 * DS_THREADS * 4];
    static_assert(2 * DK + DV + 16 + 4 * DV <= 2 * DS_MAXK + 64 + 8 + 2 * DS_THREADS * 4, "attention scratch");
    pdl_trigger();
    // The mixing logits, then attention, then the recurrence, whose CTAs are the shorter ones.  (In turn, so that both end together:
    // tokens of 32 rows, 2048 tokens, 47.1 -> 49.8 us, 16 rows of 128 / 128 61 -> 65 us; the recurrence first: 50.8 and 65 us.)
    const int idx = blockIdx.x;
    if (idx < c.n_mix) core_mix_logits(c, idx, sm);
    else if (idx < c.n_mix + c.n_attn) core_attention<DK, DV, DEEP>(c, idx - c.n_mix, sm);
    else if (c.vs == 64) core_recurrence<64>(c, idx - c.n_mix - c.n_attn, sm);
    else core_recurrence<32>(c, idx - c.n_mix - c.n_attn, sm);
}

// ------------------------------------------------------------------------------------------------ merge
struct MergeArgs {
    Args a;
    const bf16 *raw, *o_lin;
    const float *wlog, *part, *gnew;
    bf16* y;                                  // [B, H*V]
    int NR, S, n_slices, n_heads;             // n_heads = B * HQ, four to a CTA, then the CTAs of the tails
};

// One warp per (batch, head), DV / 32 channels per lane: nothing but warp shuffles between the loads, which are issued up front.
template <int DV>
__global__ void __launch_bounds__(128) decode_merge_kernel(const MergeArgs c) {
    constexpr int E = DV / 32;
    const Args& a = c.a;
    const int tid = threadIdx.x, lane = tid & 31, HK = a.H * a.K, HV = a.H * a.V;
    const int n_cta = (c.n_heads + 3) / 4;
    float w1[E], w2[E];
    const bool tails = (int)blockIdx.x >= n_cta;
    if (!tails)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            w1[e] = a.w1 ? ldw(a.w1, a.w12_f32, lane * E + e) : 1.f;
            w2[e] = a.w2 ? ldw(a.w2, a.w12_f32, lane * E + e) : 1.f;
        }
    pdl_wait();
    pdl_trigger();
    if (tails) {
        // convolution tails: drop the oldest input, append the new one; decay sums of the current block
        const long i = (long)(blockIdx.x - n_cta) * 128 + tid;
        const int per = 2 * HK + HV;
        if (i < (long)a.B * per) {
            const int b = (int)(i / per);
            int d = (int)(i % per);
            const bf16 x = c.raw[(long)b * c.NR + d];
            bf16* tail;
            if (d < HK) tail = a.conv_q + ((long)b * HK + d) * 4;
            else if (d < 2 * HK) tail = a.conv_k + ((long)b * HK + d - HK) * 4;
            else tail = a.conv_v + ((long)b * HV + d - 2 * HK) * 4;
            uint2 tw = *reinterpret_cast<const uint2*>(tail);
            tw.x = (tw.x >> 16) | (tw.y << 16);
            tw.y = (tw.y >> 16) | ((uint32_t)*reinterpret_cast<const unsigned short*>(&x) << 16);
            *reinterpret_cast<uint2*>(tail) = tw;
        }
        if (i < a.B * a.H) a.g_block[i] = a.types_new ? 0.f : a.g_block[i] + c.gnew[i];
        return;
    }
    const int unit = blockIdx.x * 4 + (tid >> 5);
    if (unit >= c.n_heads) return;
    const int hq = unit % a.HQ, b = unit / a.HQ;
    const float* part = c.part + (long)unit * c.S * (DV + 2);
    const int d0 = hq * DV + lane * E;
    float x1[E], gg[E], o[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        x1[e] = bf(c.o_lin, (long)b * HV + d0 + e);
        gg[e] = bf(c.raw, (long)b * c.NR + 2 * HK + HV + d0 + e);
        o[e] = 0.f;
    }
    // splits s = lane, lane + 32 (at most 64); the values of the first four are on their way before their weights are known
    constexpr int AHEAD = 4;
    float m0 = -INFINITY, m1 = -INFINITY, s0 = 0.f, s1 = 0.f, pv[AHEAD][E];
    if (lane < c.S) { m0 = part[(long)lane * (DV + 2)]; s0 = part[(long)lane * (DV + 2) + 1]; }
    if (lane + 32 < c.S) { m1 = part[(long)(lane + 32) * (DV + 2)]; s1 = part[(long)(lane + 32) * (DV + 2) + 1]; }
#pragma unroll
    for (int s = 0; s < AHEAD; ++s)
#pragma unroll
        for (int e = 0; e < E; ++e) pv[s][e] = s < c.S ? part[(long)s * (DV + 2) + 2 + lane * E + e] : 0.f;
    float l1 = 0.f, l2 = 0.f;
    if (a.w_mix) {                                       // slices by lane, summed in their order
        float2 wl = make_float2(0.f, 0.f);
        if (lane < c.n_slices) wl = *reinterpret_cast<const float2*>(c.wlog + (((long)b * c.n_slices + lane) * a.HQ + hq) * 2);
        for (int k = 0; k < c.n_slices; ++k) {
            float2 w;
            if (k < 32) {
                w.x = __shfl_sync(0xffffffffu, wl.x, k);
                w.y = __shfl_sync(0xffffffffu, wl.y, k);
            } else {
                w = *reinterpret_cast<const float2*>(c.wlog + (((long)b * c.n_slices + k) * a.HQ + hq) * 2);
            }
            l1 += w.x;
            l2 += w.y;
        }
        l1 = rb(l1);
        l2 = rb(l2);
    }
    float M = fmaxf(m0, m1);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, k));
    const float f0 = m0 == -INFINITY ? 1.f : exp2f(m0 - M), f1 = m1 == -INFINITY ? 1.f : exp2f(m1 - M);
    const float L = warp_sum(f0 * s0 + f1 * s1);
#pragma unroll
    for (int s = 0; s < AHEAD; ++s) {
        if (s >= c.S) break;
        const float f = __shfl_sync(0xffffffffu, f0, s);
#pragma unroll
        for (int e = 0; e < E; ++e) o[e] += f * pv[s][e];
    }
#pragma unroll 4
    for (int s = AHEAD; s < c.S; ++s) {
        const float f = __shfl_sync(0xffffffffu, s < 32 ? f0 : f1, s & 31);
        const float* p = part + (long)s * (DV + 2) + 2 + lane * E;
#pragma unroll
        for (int e = 0; e < E; ++e) o[e] += f * p[e];
    }
    float q1 = 0.f, q2 = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        o[e] = rb(L == 0.f ? 0.f : o[e] / L);
        q1 += x1[e] * x1[e];
        q2 += o[e] * o[e];
    }
    const float r1 = rsqrtf(warp_sum(q1) / DV + a.mix_eps), r2 = rsqrtf(warp_sum(q2) / DV + a.mix_eps);
    float m_1 = 1.f, m_2 = 1.f;
    if (a.w_mix) {
        const float mx = fmaxf(l1, l2), e1 = expf(l1 - mx), e2 = expf(l2 - mx);
        m_1 = rb(e1 / (e1 + e2));
        m_2 = rb(e2 / (e1 + e2));
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const float v = x1[e] * r1 * w1[e] * m_1 + o[e] * r2 * w2[e] * m_2;
        const float sg = 1.f / (1.f + __expf(-gg[e]));
        c.y[(long)b * HV + d0 + e] = __float2bfloat16(a.mix_sigmoid ? v * sg : v * gg[e] * sg);
    }
}

// ------------------------------------------------------------------------------------------------ host
template <typename Arg>
cudaError_t launch_pdl(void (*kern)(const Arg), unsigned grid, unsigned block, cudaStream_t st, const Arg& arg, bool overlap = true,
                       unsigned smem = 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, arg);
}

template <int DK, int DV>
cudaError_t launch_core(const CoreArgs& c, cudaStream_t st) {
    // One slot per warp where the CTAs do not fit the SMs at once and a split has few steps, which other CTAs' loads hide: the
    // recurrence and the mixing logits, which need no ring, then share an SM four at a time at 128/128 too, and the first-level cache
    // keeps something.  At 128/128 (three CTAs per SM with two slots) also where the recurrence's CTAs are most of the grid.  Whole
    // tokens, deep / one slot, us: 16 heads of 128, 64 rows, 40 tokens 170 / 157, 1000 tokens 202 / 192, 32 rows, 600 tokens 65.6 /
    // 60.1, 16 rows, 300 tokens 35.7 / 32.8, but 16 rows, 3000 tokens 61.4 / 64.1; 16 heads of 64, 32 rows, 40 tokens 22.7 / 22.0, but
    // 2000 tokens 42 / 47.
    constexpr int FIT = DK + DV == 256 ? 3 : 4;
    const int units = c.a.n_done * (c.a.nbs / 64) + (c.a.own_chunk ? c.a.pos % c.a.nbs + 63 : 0) / 64;
    const int per = (units + c.S - 1) / c.S;
    const bool one_slot = c.n_mix + c.n_rec + c.n_attn > 148 * FIT &&
                          (per <= 4 || (FIT == 3 && (long)per * c.n_attn <= 11l * c.n_rec));
    auto kern = one_slot ? decode_core_kernel<DK, DV, false> : decode_core_kernel<DK, DV, true>;
    const int bytes = one_slot ? Ring<DK, DV, false>::bytes : Ring<DK, DV, true>::bytes;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    return launch_pdl(kern, c.n_mix + c.n_rec + c.n_attn, DS_THREADS, st, c, true, bytes);
}

// Row tiles of every segment, then the launch.  Up to 32 batch rows all eight warps share the contraction of 16 weight rows
// (most CTAs, most loads in flight; 64-row tiles left 16 CTAs for the output product at hidden 1024: 15 us a product); above
// that, warps side by side over 64 weight rows read the activations a quarter as often.
cudaError_t launch_skinny(SkinnyArgs& a, cudaStream_t st, bool overlap) {
    const int nb = (a.B + 7) / 8;
    const int R = nb <= 4 ? 16 : 64;
    int tiles = 0;
    for (int i = 0; i < a.nseg; ++i) {
        a.seg[i].tile0 = tiles;
        tiles += (a.seg[i].rows + R - 1) / R;
    }
    if (nb == 1) return launch_pdl(skinny_kernel<1, 1, 8>, tiles, 256, st, a, overlap);
    if (nb == 2) return launch_pdl(skinny_kernel<2, 1, 8>, tiles, 256, st, a, overlap);
    if (nb <= 4) return launch_pdl(skinny_kernel<4, 1, 8>, tiles, 256, st, a, overlap);
    return launch_pdl(skinny_kernel<8, 4, 2>, tiles, 256, st, a, overlap);
}

// Splits of the finished keys of one (batch, head) over CTAs: enough CTAs for four per SM, at least two 64-key units each.  At
// 128/128, where three fit with the deep ring, three per SM are better up to a few rows and worse beyond (16 heads, four / three, us a
// token: 2 rows, 2700 tokens 26.0 / 23.8, 8 rows, 2000 33.5 / 31.4, 5500 53.3 / 56.7, 16 rows, 5500 85.6 / 96.1).
int attn_splits(int B, int HQ, int units) {
    const int want = (148 * 4 + B * HQ - 1) / (B * HQ), most = units / 2;
    const int s = want < most ? want : most;
    return s < 1 ? 1 : (s > 64 ? 64 : s);
}

struct Layout {
    long raw, olin, wlog, y, part, gnew, total;
    int NR, S, slices;
};
Layout layout(const Args& a) {
    Layout l;
    const long HK = (long)a.H * a.K, HV = (long)a.H * a.V;
    l.NR = (int)(2 * HK + 2 * HV + 2 * a.H);
    l.NR = (l.NR + 7) / 8 * 8;
    l.S = attn_splits(a.B, a.HQ, a.n_done * (a.nbs / 64));
    auto up = [](long x) { return (x + 255) / 256 * 256; };
    l.raw = 0;
    l.olin = up(l.raw + 2l * a.B * l.NR);
    l.wlog = up(l.olin + 2l * a.B * HV);
    l.slices = (int)((HK + DS_MIX - 1) / DS_MIX);
    l.y = up(l.wlog + 4l * a.B * l.slices * 2 * a.HQ);
    l.gnew = up(l.y + 2l * a.B * HV);
    l.part = up(l.gnew + 4l * a.B * a.H);
    // sized for the most splits this batch can get, so that one workspace serves a request from its first token on
    const int smax = attn_splits(a.B, a.HQ, 1 << 20);
    l.total = l.part + 4l * a.B * a.HQ * smax * (HV / a.HQ + 2);
    return l;
}

int check(const Args* a) {
    NATSL_REQUIRE(a, NATSL_ERR_NULL, "natsl_decode_step: null argument block");
    NATSL_REQUIRE(a->B > 0 && a->B <= 64 && a->hidden > 0 && a->hidden % 32 == 0 && a->H > 0 && a->HQ > 0 && a->HN > 0 &&
                      a->H % a->HN == 0 && a->HQ % a->HN == 0 && a->nbs >= 64 && a->nbs % 64 == 0,
                  NATSL_ERR_BAD_SHAPE, "natsl_decode_step: bad shape (1 <= B <= 64, hidden a multiple of 32)");
    NATSL_REQUIRE(a->K % 32 == 0 && a->K <= DS_MAXK && a->V % 32 == 0 && (a->H * a->K) % a->HQ == 0 && (a->H * a->V) % a->HQ == 0,
                  NATSL_ERR_UNSUPPORTED, "natsl_decode_step: head dims K=%d V=%d (multiples of 32, K <= 256)", a->K, a->V);
    const int DK = a->H * a->K / a->HQ, DV = a->H * a->V / a->HQ;
    NATSL_REQUIRE((DK == 64 || DK == 128) && (DV == 64 || DV == 128), NATSL_ERR_UNSUPPORTED,
                  "natsl_decode_step: softmax head dims %d / %d (64 or 128 each)", DK, DV);
    return NATSL_OK;
}

}  // namespace
}  // namespace natsl

extern "C" int64_t natsl_decode_workspace_bytes(const natsl_decode_args* args) {
    using namespace natsl;
    const Args* a = reinterpret_cast<const Args*>(args);
    const int rc = check(a);
    return rc == NATSL_OK ? layout(*a).total : rc;
}

extern "C" int natsl_decode_step(const natsl_decode_args* args, void* stream) {
    using namespace natsl;
    int rc = check(reinterpret_cast<const Args*>(args));
    if (rc != NATSL_OK) return rc;
    const Args& a = *reinterpret_cast<const Args*>(args);
    NATSL_REQUIRE(a.x && a.out && a.w_q && a.w_k && a.w_v && a.w_a && a.w_g && a.w_o && a.cw_q && a.cw_k && a.cw_v && a.A_log &&
                      a.dt_bias && a.conv_q && a.conv_k && a.conv_v && a.state && a.start && a.g_block && a.k_cache &&
                      a.v_cache && a.workspace && (a.n_done == 0 || a.types) && (a.rule != NATSL_RULE_GDN || a.w_b),
                  NATSL_ERR_NULL, "natsl_decode_step: null pointer");
    NATSL_REQUIRE(aligned_to(16, a.x, a.w_q, a.w_k, a.w_v, a.w_a, a.w_b, a.w_g, a.w_o, a.w_mix, a.state, a.start, a.k_cache, a.v_cache,
                             a.workspace) &&
                      aligned_to(8, a.cw_q, a.cw_k, a.cw_v, a.conv_q, a.conv_k, a.conv_v),
                  NATSL_ERR_UNSUPPORTED, "natsl_decode_step: a tensor does not start on 16 bytes (convolution weights and tails: 8)");
    NATSL_REQUIRE(a.pos >= 0 && a.pos < a.cap && a.n_done >= 0 && a.n_done == a.pos / a.nbs, NATSL_ERR_BAD_SHAPE,
                  "natsl_decode_step: pos=%d cap=%d finished blocks=%d", a.pos, a.cap, a.n_done);
    NATSL_REQUIRE((a.types_new != nullptr) == ((a.pos + 1) % a.nbs == 0), NATSL_ERR_BAD_SHAPE,
                  "natsl_decode_step: types_new belongs to the token that completes a block");
    const Layout l = layout(a);
    NATSL_REQUIRE(a.workspace_bytes >= l.total, NATSL_ERR_TOO_LARGE, "natsl_decode_step: workspace of %ld bytes, %ld needed",
                  (long)a.workspace_bytes, l.total);
    rc = check_device(a.x, "natsl_decode_step");
    if (rc != NATSL_OK) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    unsigned char* ws = a.workspace;
    const int HK = a.H * a.K, HV = a.H * a.V, DK = HK / a.HQ, DV = HV / a.HQ;
    bf16* raw = reinterpret_cast<bf16*>(ws + l.raw);

    SkinnyArgs p = {};
    p.seg[0] = {a.w_q, HK, 0, 0};
    p.seg[1] = {a.w_k, HK, HK, 0};
    p.seg[2] = {a.w_v, HV, 2 * HK, 0};
    p.seg[3] = {a.w_g, HV, 2 * HK + HV, 0};
    p.seg[4] = {a.w_a, a.H, 2 * HK + 2 * HV, 0};
    p.seg[5] = {a.w_b, a.H, 2 * HK + 2 * HV + a.H, 0};
    p.nseg = a.rule == NATSL_RULE_GDN ? 6 : 5;
    p.B = a.B;
    p.Kdim = a.hidden;
    p.y_stride = l.NR;
    p.x = a.x;
    p.y = raw;
    p.pool = a.pool_sum;
    // the first launch waits for everything in front of it (its early weight loads must not overtake a kernel that writes
    // them), the other three overlap their prologues with the one before
    cudaError_t e = launch_skinny(p, st, false);

    CoreArgs c = {};
    c.a = a;
    c.raw = raw;
    c.o_lin = reinterpret_cast<bf16*>(ws + l.olin);
    c.wlog = reinterpret_cast<float*>(ws + l.wlog);
    c.part = reinterpret_cast<float*>(ws + l.part);
    c.gnew = reinterpret_cast<float*>(ws + l.gnew);
    c.NR = l.NR;
    c.S = l.S;
    c.n_attn = a.B * a.HQ * l.S;
    // 64 columns per recurrence CTA (half the convolution work) once 32 would take more than one wave
    c.vs = a.K <= 64 && a.V % 64 == 0 && (long)a.B * a.H * (a.V / 32) > 148 * 4 ? 64 : 32;
    c.n_rec = a.B * a.H * (a.V / c.vs);
    c.n_slices = l.slices;
    c.n_mix = a.w_mix ? a.B * l.slices * ((2 * a.HQ + DS_MIX_ROWS - 1) / DS_MIX_ROWS) : 0;
    if (e == cudaSuccess)
        e = DK == 64 ? (DV == 64 ? launch_core<64, 64>(c, st) : launch_core<64, 128>(c, st))
                     : (DV == 64 ? launch_core<128, 64>(c, st) : launch_core<128, 128>(c, st));

    MergeArgs g = {};
    g.a = a;
    g.raw = raw;
    g.o_lin = c.o_lin;
    g.wlog = c.wlog;
    g.part = c.part;
    g.gnew = c.gnew;
    g.y = reinterpret_cast<bf16*>(ws + l.y);
    g.NR = l.NR;
    g.S = l.S;
    g.n_slices = l.slices;
    g.n_heads = a.B * a.HQ;
    const unsigned tails = (unsigned)(((long)a.B * (2 * HK + HV) + 127) / 128);
    if (e == cudaSuccess)
        e = launch_pdl(DV == 64 ? decode_merge_kernel<64> : decode_merge_kernel<128>, (g.n_heads + 3) / 4 + tails, 128, st, g);

    SkinnyArgs o = {};
    o.seg[0] = {a.w_o, a.hidden, 0, 0};
    o.nseg = 1;
    o.B = a.B;
    o.Kdim = HV;
    o.y_stride = a.hidden;
    o.x = g.y;
    o.y = a.out;
    if (e == cudaSuccess) e = launch_skinny(o, st, true);
    if (e != cudaSuccess) {
        set_error("natsl_decode_step: CUDA error %d (%s)", (int)e, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return check_launch("natsl_decode_step");
}
