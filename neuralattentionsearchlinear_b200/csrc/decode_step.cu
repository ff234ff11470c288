// One decoding token of a whole NAtSL layer (GDN or Mamba2) in four launches: projections -> {linear-branch step, softmax
// attention over the cached keys, mixing weights} -> branch merge -> output projection.
//   src/nats/layers/natsl_attn_gdn.py:389-666 with one new token (Mamba2: src/nats/layers/natsl_attn_mamba2.py:330-599);
//   linear branch  src/nats/ops/gated_delta_rule/fused_recurrent.py:128-358, src/nats/ops/mamba/fused_recurrent.py:121-322;
//   softmax branch src/nats/ops/mixed_ops/mixed_attn_gdn.py:475-504 (SDPA over the cache under its visibility mask).
// What bounds it: at batch 1 the layer reads its weights once (33 MB at hidden 1024..2048) and does almost no arithmetic,
// so the floor is the weight read plus the dependent launches; issued step by step from Python (about 80 launches,
// several host reads) the same token took 1.4 ms of host time.  A request of 777 + 48 tokens at hidden 2048, batch 1:
// 69.0 -> 2.9 ms; 2048 + 32 tokens at hidden 1024, batch 32: 49.1 -> 5.5 ms (prefill included in both).
//   * proj / out: "skinny" products y[b, n] = x[b, :] . W[n, :].  The weight rows are the M side of mma.m16n8k16, the
//     batch the N side, so a weight element is loaded once, straight from global memory into the A fragment: with the k
//     index permuted inside every 32-wide group a lane's fragment is one 16-byte load per row (the same permutation on
//     both operands leaves the sum unchanged).  Weight loads do not depend on the previous kernel and are issued before
//     the programmatic-launch wait.
//   * core: three kinds of CTA in one grid.  Every CTA recomputes the short convolution of the channels it needs (four
//     taps), which costs less than a launch in between.  The recurrence reads the state once: S^T k and S^T q are formed
//     together (o = e^g S^T q + (q.k) v').  Attention splits the 64-key units of the finished blocks over CTAs; a warp
//     takes 16 keys of a unit, K and V loads of all of them in flight.
//   * merge: combines the splits, both RMS norms, mixing weights and gate; extra CTAs shift the convolution tails.
// All state (recurrent state, tails, decay sums, pooled input, key/value rows) is updated in place.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

using bf16 = __nv_bfloat16;
constexpr int DS_THREADS = 128;               // core CTAs
constexpr int DS_VS = 32;                     // value columns per recurrence CTA
constexpr int DS_MAXK = 256;
constexpr int DS_WROWS = 8;                   // mixing-weight rows per CTA
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
    constexpr int R = 16 * WM, UN = NB >= 4 ? 2 : 4;
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
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            if (c + u >= c1) break;
            const uint32_t f0[4] = {ca[u].x, cb[u].x, ca[u].y, cb[u].y}, f1[4] = {ca[u].z, cb[u].z, ca[u].w, cb[u].w};
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                const int row = n * 8 + g;
                const uint4 xb = row < a.B ? *(reinterpret_cast<const uint4*>(a.x + (long)row * a.Kdim) + (c + u) * 4 + t) : zero;
                mma_bf16(acc[n], f0, xb.x, xb.y);
                mma_bf16(acc[n], f1, xb.z, xb.w);
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
    bf16* wlog;                               // [B, 2*HQ]
    float* part;                              // [B, HQ, S, DV + 2]
    float* gnew;                              // [B, H]
    int NR, S, n_attn, n_rec;
};

// Convolved channel (rounded to bf16 like the layer's own convolution output): tail = the last four inputs.
__device__ __forceinline__ float conv1(const bf16* tail, const bf16* w, const bf16* bias, float x_new, int d, int silu) {
    const uint2 tw = *reinterpret_cast<const uint2*>(tail), ww = *reinterpret_cast<const uint2*>(w + (long)d * 4);
    const float2 t0 = unpack_bf16(tw.x), t1 = unpack_bf16(tw.y), w0 = unpack_bf16(ww.x), w1 = unpack_bf16(ww.y);
    float acc = bias ? bf(bias, d) : 0.f;
    acc += w0.x * t0.y;
    acc += w0.y * t1.x;
    acc += w1.x * t1.y;
    acc += w1.y * x_new;
    return rb(silu ? acc * (1.f / (1.f + __expf(-acc))) : acc);
}

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

__device__ void core_recurrence(const CoreArgs& c, int idx, float* sm) {
    const Args& a = c.a;
    const int tid = threadIdx.x, K = a.K, V = a.V, H = a.H, HK = H * K, HV = H * V;
    const int nvs = V / DS_VS, vs = idx % nvs, h = (idx / nvs) % H, b = idx / (nvs * H);
    const bool gdn = a.rule == NATSL_RULE_GDN;
    float* s_q = sm;                           // [256]
    float* s_k = sm + DS_MAXK;                 // [256]
    float* s_v = s_k + DS_MAXK;                // [32]
    float* s_red = s_v + DS_VS;                // [8]
    float* s_dot = s_red + 8;                  // [2][16][32]
    const bf16* raw = c.raw + (long)b * c.NR;
    // state rows of this thread: rg + 16 i, four columns
    const int rg = tid >> 3, col = vs * DS_VS + (tid & 7) * 4;
    float* Sp = a.state + (((long)b * H + h) * K) * V + col;
    constexpr int NREG = 8;
    float4 S[NREG];
    pdl_wait();
#pragma unroll
    for (int i = 0; i < NREG; ++i)
        if (rg + 16 * i < K) S[i] = *reinterpret_cast<const float4*>(Sp + (long)(rg + 16 * i) * V);
    float sq = 0.f, sk = 0.f;
    for (int i = tid; i < K; i += DS_THREADS) {
        const int d = h * K + i;
        const float qv = conv1(a.conv_q + ((long)b * HK + d) * 4, a.cw_q, a.cb_q, bf(raw, d), d, a.silu);
        const float kv = conv1(a.conv_k + ((long)b * HK + d) * 4, a.cw_k, a.cb_k, bf(raw, HK + d), d, a.silu);
        s_q[i] = qv;
        s_k[i] = kv;
        sq += qv * qv;
        sk += kv * kv;
    }
    const float araw = bf(raw, 2 * HK + 2 * HV + h);
    const float z = araw + ldw(a.dt_bias, a.dt_f32, h);
    const float sp = z > 20.f ? z : log1pf(expf(z));
    const float gt = -expf(ldw(a.A_log, a.alog_f32, h)) * sp;
    if (tid < DS_VS) {
        const int d = h * V + vs * DS_VS + tid;
        float vv = conv1(a.conv_v + ((long)b * HV + d) * 4, a.cw_v, a.cb_v, bf(raw, 2 * HK + d), d, a.silu);
        if (!gdn) vv = rb(vv * sp);
        s_v[tid] = vv;
    }
    sq = block_sum<DS_THREADS>(sq, s_red, tid);
    sk = block_sum<DS_THREADS>(sk, s_red + 4, tid);
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
        if (rg + 16 * i < K) add(S[i], rg + 16 * i);
    for (int r = rg + 16 * NREG; r < K; r += 16) add(*reinterpret_cast<const float4*>(Sp + (long)r * V), r);
    float* d0 = s_dot + rg * DS_VS + (tid & 7) * 4;
    *reinterpret_cast<float4*>(d0) = dk;
    *reinterpret_cast<float4*>(d0 + 16 * DS_VS) = dq;
    __syncthreads();
    if (tid < DS_VS) {
        float tk = 0.f, tq = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) { tk += s_dot[i * DS_VS + tid]; tq += s_dot[(16 + i) * DS_VS + tid]; }
        const float eg = __expf(gt);
        float vv = s_v[tid];
        if (gdn) {
            float beta = rb(1.f / (1.f + expf(-bf(raw, 2 * HK + 2 * HV + H + h))));
            if (a.neg_eigval) beta *= 2.f;
            vv = beta * (vv - eg * tk);
        }
        s_v[tid] = vv;
        c.o_lin[(long)b * HV + h * V + vs * DS_VS + tid] = __float2bfloat16((eg * tq + qk * vv) * a.scale_lin);
    }
    __syncthreads();
    const float eg = __expf(gt);
    const float4 vn = *reinterpret_cast<const float4*>(s_v + (tid & 7) * 4);
    const bool ends = a.types_new != nullptr;
    float* Bp = a.start + (((long)b * H + h) * K) * V + col;
    float roll = 1.f;
    bool sel = false;
    if (ends) {
        const int hn = h / (H / a.HN);
        sel = rintf(ldw(a.types_new, a.types_f32, ((long)b * a.HN + hn) * 2 + 1)) == 1.f;
        roll = a.decay ? __expf(a.g_block[(long)b * H + h] + gt) : 1.f;
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
        if (rg + 16 * i < K) upd(S[i], rg + 16 * i);
    for (int r = rg + 16 * NREG; r < K; r += 16) upd(*reinterpret_cast<const float4*>(Sp + (long)r * V), r);
    if (vs == 0 && tid == 0) c.gnew[(long)b * H + h] = gt;
}

template <int DK, int DV>
__device__ void core_attention(const CoreArgs& c, int idx, float* sm) {
    const Args& a = c.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = idx % c.S, hq = (idx / c.S) % a.HQ, b = idx / (c.S * a.HQ);
    const int HK = a.H * a.K, HV = a.H * a.V;
    constexpr int LK = DK / 8, LV = DV / 8, KG = 32 / LK, VG = 32 / LV;      // lanes per row, rows per load
    float* s_q = sm;                                   // [DK] query, scaled
    float* s_kn = s_q + DK;                            // [DK] new key
    float* s_vn = s_kn + DK;                           // [DV] new value
    float* s_p = s_vn + DV;                            // [4][16]
    float* s_ml = s_p + 64;                            // [4][2]
    float* s_red = s_ml + 8;                           // [8]
    float* s_acc = s_red + 8;                          // [4][DV]
    pdl_wait();
    const bf16* raw = c.raw + (long)b * c.NR;
    const bool last = s == c.S - 1;
    {
        float qv = 0.f, kv = 0.f;
        if (tid < DK) {
            const int d = hq * DK + tid;
            qv = bf(raw, d);
            kv = bf(raw, HK + d);
            if (a.attn_conv) {
                qv = conv1(a.conv_q + ((long)b * HK + d) * 4, a.cw_q, a.cb_q, qv, d, a.silu);
                kv = conv1(a.conv_k + ((long)b * HK + d) * 4, a.cw_k, a.cb_k, kv, d, a.silu);
            }
        }
        if (a.qn_w) {
            const float sq = block_sum<DS_THREADS>(qv * qv, s_red, tid), sk = block_sum<DS_THREADS>(kv * kv, s_red + 4, tid);
            if (tid < DK) {
                qv = rb(qv * rsqrtf(sq / DK + a.norm_eps) * ldw(a.qn_w, a.qn_f32, tid));
                kv = rb(kv * rsqrtf(sk / DK + a.norm_eps) * ldw(a.kn_w, a.kn_f32, tid));
            }
        }
        if (tid < DK) {
            s_q[tid] = qv * (a.scale_attn * kLog2e);
            s_kn[tid] = kv;
            if (last) a.k_cache[(((long)b * a.cap + a.pos) * a.HQ + hq) * DK + tid] = __float2bfloat16(kv);
        }
        if (last && tid < DV) {
            const int d = hq * DV + tid;
            float vv = bf(raw, 2 * HK + d);
            if (a.attn_conv) vv = conv1(a.conv_v + ((long)b * HV + d) * 4, a.cw_v, a.cb_v, vv, d, a.silu);
            s_vn[tid] = vv;
            a.v_cache[(((long)b * a.cap + a.pos) * a.HQ + hq) * DV + tid] = __float2bfloat16(vv);
        }
    }
    __syncthreads();
    float q8[8];
    {
        const int d0 = (lane % LK) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) q8[e] = s_q[d0 + e];
    }
    float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    const bf16* kb = a.k_cache + ((long)b * a.cap * a.HQ + hq) * DK + (lane % LK) * 8;
    const bf16* vb = a.v_cache + ((long)b * a.cap * a.HQ + hq) * DV + (lane % LV) * 8;
    float* my_p = s_p + warp * 16;
    auto unit = [&](int key0, int n_keys) {            // this warp's 16 keys from key0, the first n_keys of them valid
        constexpr int NK = 16 / KG, NV = 16 / VG;
        uint4 kr[NK], vr[NV];
#pragma unroll
        for (int i = 0; i < NK; ++i) {
            const int j = min(i * KG + lane / LK, n_keys - 1);
            kr[i] = *reinterpret_cast<const uint4*>(kb + (long)(key0 + j) * a.HQ * DK);
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int j = min(i * VG + lane / LV, n_keys - 1);
            vr[i] = *reinterpret_cast<const uint4*>(vb + (long)(key0 + j) * a.HQ * DV);
        }
#pragma unroll
        for (int i = 0; i < NK; ++i) {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&kr[i]);
            float d = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16(w[e]);
                d += f.x * q8[2 * e];
                d += f.y * q8[2 * e + 1];
            }
#pragma unroll
            for (int o = LK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (lane % LK == 0) my_p[i * KG + lane / LK] = d;
        }
        __syncwarp();
        const float sc = (lane & 15) < n_keys ? my_p[lane & 15] : -INFINITY;
        float mx = sc;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m, mx), al = exp2f(m - mn);
        const float p = exp2f(sc - mn);
        float ps = p;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        l = l * al + ps;
        m = mn;
        __syncwarp();
        if (lane < 16) my_p[lane] = p;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] *= al;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float pj = my_p[i * VG + lane / LV];
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&vr[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16(w[e]);
                acc[2 * e] += pj * f.x;
                acc[2 * e + 1] += pj * f.y;
            }
        }
        __syncwarp();
    };
    const int hn = hq / (a.HQ / a.HN), upb = a.nbs / 64;
    const int n_units = a.n_done * upb;
    const int u0 = (int)((long)n_units * s / c.S), u1 = (int)((long)n_units * (s + 1) / c.S);
    for (int u = u0; u < u1; ++u) {
        const int blk = u / upb;
        if (ldw(a.types, a.types_f32, (((long)b * a.n_done + blk) * a.HN + hn) * 2) > 0.5f) unit(u * 64 + warp * 16, 16);
    }
    if (last && a.own_chunk) {
        const int own0 = a.pos / a.nbs * a.nbs;         // keys of the current block before the new token
        for (int k0 = own0 + warp * 16; k0 < a.pos; k0 += 64) unit(k0, min(16, a.pos - k0));
    }
    // sum the key groups of a warp, then the warps
#pragma unroll
    for (int o = LV; o < 32; o <<= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if (lane < LV)
#pragma unroll
        for (int e = 0; e < 8; ++e) s_acc[warp * DV + lane * 8 + e] = acc[e];
    if (lane == 0) { s_ml[warp * 2] = m; s_ml[warp * 2 + 1] = l; }
    float own = -INFINITY;                              // score of the new token
    if (last && a.own_chunk) own = block_sum<DS_THREADS>(tid < DK ? s_q[tid] * s_kn[tid] : 0.f, s_red, tid);
    __syncthreads();
    float M = own;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, s_ml[w * 2]);
    float* part = c.part + (((long)b * a.HQ + hq) * c.S + s) * (DV + 2);
    if (tid < DV) {
        float L = 0.f, o = 0.f;
        if (M != -INFINITY) {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float f = exp2f(s_ml[w * 2] - M);
                L += f * s_ml[w * 2 + 1];
                o += f * s_acc[w * DV + tid];
            }
            if (own != -INFINITY) {
                const float p = exp2f(own - M);
                L += p;
                o += p * s_vn[tid];
            }
        }
        part[2 + tid] = o;
        if (tid == 0) { part[0] = M; part[1] = L; }
    }
}

// logits of the mixing weights: rows of w_mix [2 HQ, H K] times the convolved query of one batch row
__device__ void core_mix_logits(const CoreArgs& c, int idx) {
    const Args& a = c.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = 2 * a.HQ, groups = (rows + DS_WROWS - 1) / DS_WROWS;
    const int b = idx / groups, row0 = (idx % groups) * DS_WROWS, HK = a.H * a.K;
    extern __shared__ float s_dyn[];                   // [HK] convolved query
    pdl_wait();
    const bf16* raw = c.raw + (long)b * c.NR;
    for (int d = tid; d < HK; d += DS_THREADS)
        s_dyn[d] = conv1(a.conv_q + ((long)b * HK + d) * 4, a.cw_q, a.cb_q, bf(raw, d), d, a.silu);
    __syncthreads();
    for (int r = row0 + warp; r < min(row0 + DS_WROWS, rows); r += 4) {
        float acc = 0.f;
        for (int d = lane * 8; d < HK; d += 256) {
            const uint4 v = *reinterpret_cast<const uint4*>(a.w_mix + (long)r * HK + d);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16(w[e]);
                acc += f.x * s_dyn[d + 2 * e];
                acc += f.y * s_dyn[d + 2 * e + 1];
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) c.wlog[(long)b * rows + r] = __float2bfloat16(acc);
    }
}

template <int DK, int DV>
__global__ void __launch_bounds__(DS_THREADS) decode_core_kernel(const CoreArgs c) {
    __shared__ __align__(16) float sm[2 * DS_MAXK + DS_VS + 8 + 2 * 16 * DS_VS];
    static_assert(2 * DK + DV + 64 + 16 + 4 * DV <= 2 * DS_MAXK + DS_VS + 8 + 2 * 16 * DS_VS, "attention scratch");
    pdl_trigger();
    int idx = blockIdx.x;
    if (idx < c.n_attn) {
        core_attention<DK, DV>(c, idx, sm);
    } else if (idx < c.n_attn + c.n_rec) {
        core_recurrence(c, idx - c.n_attn, sm);
    } else {
        core_mix_logits(c, idx - c.n_attn - c.n_rec);
    }
}

// ------------------------------------------------------------------------------------------------ merge
struct MergeArgs {
    Args a;
    const bf16 *raw, *o_lin, *wlog;
    const float *part, *gnew;
    bf16* y;                                  // [B, H*V]
    int NR, S, n_heads;                       // n_heads = B * HQ CTAs of the merge itself, then the tail CTAs
};

template <int DV>
__global__ void __launch_bounds__(DV) decode_merge_kernel(const MergeArgs c) {
    const Args& a = c.a;
    const int tid = threadIdx.x, HK = a.H * a.K, HV = a.H * a.V;
    __shared__ float s_red[8];
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.x >= c.n_heads) {
        // convolution tails: drop the oldest input, append the new one; decay sums of the current block
        const long i = (long)(blockIdx.x - c.n_heads) * DV + tid;
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
    const int hq = blockIdx.x % a.HQ, b = blockIdx.x / a.HQ;
    const float* part = c.part + ((long)b * a.HQ + hq) * c.S * (DV + 2);
    float M = -INFINITY;
    for (int s = 0; s < c.S; ++s) M = fmaxf(M, part[(long)s * (DV + 2)]);
    float L = 0.f, o = 0.f;
    if (M != -INFINITY)
        for (int s = 0; s < c.S; ++s) {
            const float* p = part + (long)s * (DV + 2);
            const float f = exp2f(p[0] - M);
            L += f * p[1];
            o += f * p[2 + tid];
        }
    const float x2 = rb(L > 0.f ? o / L : 0.f);
    const int d = hq * DV + tid;
    const float x1 = bf(c.o_lin, (long)b * HV + d);
    const float s1 = block_sum<DV>(x1 * x1, s_red, tid), s2 = block_sum<DV>(x2 * x2, s_red + 4, tid);
    const float r1 = rsqrtf(s1 / DV + a.mix_eps), r2 = rsqrtf(s2 / DV + a.mix_eps);
    float m1 = 1.f, m2 = 1.f;
    if (a.w_mix) {
        const float l1 = bf(c.wlog, ((long)b * a.HQ + hq) * 2), l2 = bf(c.wlog, ((long)b * a.HQ + hq) * 2 + 1);
        const float mx = fmaxf(l1, l2), e1 = expf(l1 - mx), e2 = expf(l2 - mx);
        m1 = rb(e1 / (e1 + e2));
        m2 = rb(e2 / (e1 + e2));
    }
    const float gg = bf(c.raw, (long)b * c.NR + 2 * HK + HV + d);
    const float v = x1 * r1 * (a.w1 ? ldw(a.w1, a.w12_f32, tid) : 1.f) * m1 + x2 * r2 * (a.w2 ? ldw(a.w2, a.w12_f32, tid) : 1.f) * m2;
    const float sg = 1.f / (1.f + __expf(-gg));
    c.y[(long)b * HV + d] = __float2bfloat16(a.mix_sigmoid ? v * sg : v * gg * sg);
}

// ------------------------------------------------------------------------------------------------ host
template <typename Arg>
cudaError_t launch_pdl(void (*kern)(const Arg), unsigned grid, unsigned block, size_t smem, cudaStream_t st, const Arg& arg) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, arg);
}

// Row tiles of every segment, then the launch.  The split between weight rows and contraction per CTA follows the batch:
// few batch rows -> all warps on the contraction of 16 weight rows (most CTAs, most loads in flight); more rows -> warps
// side by side over weight rows, so that a CTA reads the activations once for 64 of them.
cudaError_t launch_skinny(SkinnyArgs& a, cudaStream_t st) {
    const int nb = (a.B + 7) / 8;
    const int R = nb == 1 ? 16 : nb == 2 ? 32 : 64;
    int tiles = 0;
    for (int i = 0; i < a.nseg; ++i) {
        a.seg[i].tile0 = tiles;
        tiles += (a.seg[i].rows + R - 1) / R;
    }
    if (nb == 1) return launch_pdl(skinny_kernel<1, 1, 8>, tiles, 256, 0, st, a);
    if (nb == 2) return launch_pdl(skinny_kernel<2, 2, 4>, tiles, 256, 0, st, a);
    if (nb <= 4) return launch_pdl(skinny_kernel<4, 4, 2>, tiles, 256, 0, st, a);
    return launch_pdl(skinny_kernel<8, 4, 2>, tiles, 256, 0, st, a);
}

// Splits of the finished keys of one (batch, head) over CTAs: enough CTAs for four per SM, at least two 64-key units each.
int attn_splits(int B, int HQ, int units) {
    const int want = (148 * 4 + B * HQ - 1) / (B * HQ), most = units / 2;
    const int s = want < most ? want : most;
    return s < 1 ? 1 : (s > 64 ? 64 : s);
}

struct Layout {
    long raw, olin, wlog, y, part, gnew, total;
    int NR, S;
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
    l.y = up(l.wlog + 2l * a.B * 2 * a.HQ);
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
    NATSL_REQUIRE(a->K % 32 == 0 && a->K <= DS_MAXK && a->V % DS_VS == 0 && (a->H * a->K) % a->HQ == 0 && (a->H * a->V) % a->HQ == 0,
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
    const int rc = check(reinterpret_cast<const Args*>(args));
    if (rc != NATSL_OK) return rc;
    const Args& a = *reinterpret_cast<const Args*>(args);
    NATSL_REQUIRE(a.x && a.out && a.w_q && a.w_k && a.w_v && a.w_a && a.w_g && a.w_o && a.cw_q && a.cw_k && a.cw_v && a.A_log &&
                      a.dt_bias && a.conv_q && a.conv_k && a.conv_v && a.state && a.start && a.g_block && a.k_cache &&
                      a.v_cache && a.workspace && (a.n_done == 0 || a.types) && (a.rule != NATSL_RULE_GDN || a.w_b),
                  NATSL_ERR_NULL, "natsl_decode_step: null pointer");
    NATSL_REQUIRE(a.pos >= 0 && a.pos < a.cap && a.n_done >= 0 && a.n_done == a.pos / a.nbs, NATSL_ERR_BAD_SHAPE,
                  "natsl_decode_step: pos=%d cap=%d finished blocks=%d", a.pos, a.cap, a.n_done);
    NATSL_REQUIRE((a.types_new != nullptr) == ((a.pos + 1) % a.nbs == 0), NATSL_ERR_BAD_SHAPE,
                  "natsl_decode_step: types_new belongs to the token that completes a block");
    const Layout l = layout(a);
    NATSL_REQUIRE(a.workspace_bytes >= l.total, NATSL_ERR_TOO_LARGE, "natsl_decode_step: workspace of %ld bytes, %ld needed",
                  (long)a.workspace_bytes, l.total);
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
    cudaError_t e = launch_skinny(p, st);

    CoreArgs c = {};
    c.a = a;
    c.raw = raw;
    c.o_lin = reinterpret_cast<bf16*>(ws + l.olin);
    c.wlog = reinterpret_cast<bf16*>(ws + l.wlog);
    c.part = reinterpret_cast<float*>(ws + l.part);
    c.gnew = reinterpret_cast<float*>(ws + l.gnew);
    c.NR = l.NR;
    c.S = l.S;
    c.n_attn = a.B * a.HQ * l.S;
    c.n_rec = a.B * a.H * (a.V / DS_VS);
    const int n_mix = a.w_mix ? a.B * ((2 * a.HQ + DS_WROWS - 1) / DS_WROWS) : 0;
    const size_t dyn = a.w_mix ? (size_t)HK * 4 : 0;
    NATSL_REQUIRE(dyn <= 40 * 1024, NATSL_ERR_TOO_LARGE, "natsl_decode_step: H*K = %d is too large", HK);
    auto core = DK == 64 ? (DV == 64 ? decode_core_kernel<64, 64> : decode_core_kernel<64, 128>)
                         : (DV == 64 ? decode_core_kernel<128, 64> : decode_core_kernel<128, 128>);
    if (e == cudaSuccess) e = launch_pdl(core, c.n_attn + c.n_rec + n_mix, DS_THREADS, dyn, st, c);

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
    g.n_heads = a.B * a.HQ;
    const unsigned tails = (unsigned)(((long)a.B * (2 * HK + HV) + DV - 1) / DV);
    if (e == cudaSuccess) e = launch_pdl(DV == 64 ? decode_merge_kernel<64> : decode_merge_kernel<128>, g.n_heads + tails, DV, 0, st, g);

    SkinnyArgs o = {};
    o.seg[0] = {a.w_o, a.hidden, 0, 0};
    o.nseg = 1;
    o.B = a.B;
    o.Kdim = HV;
    o.y_stride = a.hidden;
    o.x = g.y;
    o.y = a.out;
    if (e == cudaSuccess) e = launch_skinny(o, st);
    if (e != cudaSuccess) {
        set_error("natsl_decode_step: CUDA error %d (%s)", (int)e, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return check_launch("natsl_decode_step");
}
