// Bandwidth kernels for the steps of the NAtSL layer directly before the hybrid attention op, forward and backward:
//   short causal depthwise convolution + SiLU   (fla ShortConvolution at src/nats/layers/natsl_attn_gdn.py:329-348, 430-447)
//   RMSNorm, optionally fused with the residual add in front of it
//                                               (fla RMSNorm: per-head q/k norms natsl_attn_gdn.py:233-235, 504-505; block
//                                                norms src/nats/models/natsl_attn_gdn/modeling_natsl_attn_gdn.py:62, 110, 138-139)
//   SwiGLU  silu(a) * b                          (fla GatedMLP, modeling_natsl_attn_gdn.py:111-117)
//   mean over each block of tokens               (fla mean_pooling, natsl_attn_gdn.py:412-416; src/nats/ops/utils/pooling.py:26-57)
// All tensors bf16, math in fp32, 16-byte accesses where the row width allows.  Reductions over rows (weight gradients)
// are written as per-CTA partial sums and added up by the caller: no atomics, reproducible results.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = unpack_bf16(u[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&f)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

// ------------------------------------------------------------------------------------------------ short conv + SiLU
constexpr int CONV_W = 4;

// y[b,t,d] = act(bias[d] + sum_j w[d,j] x[b, t-(W-1)+j, d]).
// Backward: dpre = dy * act'(pre) with pre recomputed; dx[t] = sum_j w[j] dpre[t+(W-1)-j];
// dw[d,j] = sum_{b,t} dpre[t] x[t-(W-1)+j], dbias[d] = sum dpre: per-(batch, token range) partial sums
// dw_part [B * gridDim.y, D, W + 1] (column W = bias).  One thread = 8 channels x `span` tokens.
__global__ void __launch_bounds__(128)
short_conv_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                      const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ dy,
                      __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, int T, int D, int silu, int span) {
    const int cg = blockIdx.x * blockDim.x + threadIdx.x;
    if (cg * 8 >= D) return;
    const int d0 = cg * 8;
    const int t0 = blockIdx.y * span, b = blockIdx.z;
    constexpr int W = CONV_W;
    float wt[8][W], bs[8], dwa[8][W + 1];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        bs[c] = bias ? __bfloat162float(bias[d0 + c]) : 0.f;
#pragma unroll
        for (int j = 0; j < W; ++j) wt[c][j] = __bfloat162float(w[(d0 + c) * W + j]);
#pragma unroll
        for (int j = 0; j <= W; ++j) dwa[c][j] = 0.f;
    }
    auto loadx = [&](int t, float (&f)[8]) {
        if (t >= 0 && t < T) ld8(x + ((long)b * T + t) * D + d0, f);
        else {
#pragma unroll
            for (int c = 0; c < 8; ++c) f[c] = 0.f;
        }
    };
    // dpre at token t (zero outside [0, T)); xw = x[t-(W-1) .. t]
    auto dpre_at = [&](int t, const float (&xw)[W][8], float (&dp)[8]) {
        if (t < 0 || t >= T) {
#pragma unroll
            for (int c = 0; c < 8; ++c) dp[c] = 0.f;
            return;
        }
        float g[8];
        ld8(dy + ((long)b * T + t) * D + d0, g);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float a = bs[c];
#pragma unroll
            for (int j = 0; j < W; ++j) a += wt[c][j] * xw[j][c];
            if (silu) {
                const float s = sigmoidf_(a);
                dp[c] = g[c] * s * (1.f + a * (1.f - s));
            } else {
                dp[c] = g[c];
            }
        }
    };
    // xs holds x[tt-(W-1) .. tt+(W-1)] (2W-1 rows) for the current tt; dps holds dpre[tt .. tt+(W-1)]
    float xs[2 * W - 1][8], dps[W][8];
#pragma unroll
    for (int i = 0; i < 2 * W - 1; ++i) loadx(t0 - (W - 1) + i, xs[i]);
#pragma unroll
    for (int i = 0; i < W; ++i) {
        float xw[W][8];
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int c = 0; c < 8; ++c) xw[j][c] = xs[i + j][c];
        dpre_at(t0 + i, xw, dps[i]);
    }
    const int t_end = min(T, t0 + span);
    for (int tt = t0; tt < t_end; ++tt) {
        // weight gradient of token tt (tokens of this thread's own range only: each token counted once)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
#pragma unroll
            for (int j = 0; j < W; ++j) dwa[c][j] += dps[0][c] * xs[j][c];
            dwa[c][W] += dps[0][c];
        }
        // dx[tt] = sum_j w[j] dpre[tt + (W-1) - j]
        float o[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float a = 0.f;
#pragma unroll
            for (int j = 0; j < W; ++j) a += wt[c][j] * dps[W - 1 - j][c];
            o[c] = a;
        }
        st8(dx + ((long)b * T + tt) * D + d0, o);
        // slide by one token
#pragma unroll
        for (int i = 0; i < 2 * W - 2; ++i)
#pragma unroll
            for (int c = 0; c < 8; ++c) xs[i][c] = xs[i + 1][c];
        loadx(tt + W, xs[2 * W - 2]);
#pragma unroll
        for (int i = 0; i < W - 1; ++i)
#pragma unroll
            for (int c = 0; c < 8; ++c) dps[i][c] = dps[i + 1][c];
        {
            float xw[W][8];
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int c = 0; c < 8; ++c) xw[j][c] = xs[W - 1 + j][c];
            dpre_at(tt + W, xw, dps[W - 1]);
        }
    }
    float* out = dw_part + (((long)b * gridDim.y + blockIdx.y) * D + d0) * (W + 1);
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int j = 0; j <= W; ++j) out[c * (W + 1) + j] = dwa[c][j];
}

// ------------------------------------------------------------------------------------------------ RMSNorm
// One warp per row of D elements; lane owns NV vectors of VEC elements: element (j*32 + lane)*VEC + e.
template <int D>
struct RowShape {
    static constexpr int VEC = (D >= 256) ? 8 : D / 32;
    static constexpr int NV = D / (32 * VEC);
};

// Loads vector j of a row (VEC elements of this lane) as floats.
template <int D>
__device__ __forceinline__ void vec_load(const __nv_bfloat16* row, int lane, int j, float (&f)[RowShape<D>::VEC]) {
    constexpr int VEC = RowShape<D>::VEC;
    const __nv_bfloat16* q = row + (j * 32 + lane) * VEC;
    if constexpr (VEC == 8) {
        ld8(q, f);
    } else {
#pragma unroll
        for (int e = 0; e < VEC; e += 2) {
            const float2 t = unpack_bf16(*reinterpret_cast<const uint32_t*>(q + e));
            f[e] = t.x;
            f[e + 1] = t.y;
        }
    }
}
template <int D>
__device__ __forceinline__ void vec_store(__nv_bfloat16* row, int lane, int j, const float (&f)[RowShape<D>::VEC]) {
    constexpr int VEC = RowShape<D>::VEC;
    __nv_bfloat16* q = row + (j * 32 + lane) * VEC;
    if constexpr (VEC == 8) {
        st8(q, f);
    } else {
#pragma unroll
        for (int e = 0; e < VEC; e += 2) *reinterpret_cast<uint32_t*>(q + e) = pack_bf16(f[e], f[e + 1]);
    }
}
template <int D>
__device__ __forceinline__ void vec_weight(const void* w, int w_f32, int lane, int j, float (&f)[RowShape<D>::VEC]) {
    constexpr int VEC = RowShape<D>::VEC;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        const int col = (j * 32 + lane) * VEC + e;
        f[e] = w ? (w_f32 ? reinterpret_cast<const float*>(w)[col] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[col])) : 1.f;
    }
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16(x)); }

// s = x (+ res, rounded to bf16: the stored sum is what is normalised);  y = s * rsqrt(mean(s^2) + eps) * w.
// sum_out (may be NULL) receives s.  Two passes over the row (the second one hits the L1 / L2 cache).
template <int D>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res, const void* __restrict__ w,
                   int w_f32, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ sum_out, long rows, float eps) {
    constexpr int VEC = RowShape<D>::VEC, NV = RowShape<D>::NV;
    const int lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const __nv_bfloat16* xr = x + row * D;
    const __nv_bfloat16* rr = res ? res + row * D : nullptr;
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        float a[VEC];
        vec_load<D>(xr, lane, j, a);
        if (rr) {
            float r[VEC];
            vec_load<D>(rr, lane, j, r);
#pragma unroll
            for (int e = 0; e < VEC; ++e) a[e] = round_bf16(a[e] + r[e]);
            if (sum_out) vec_store<D>(sum_out + row * D, lane, j, a);
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) ss += a[e] * a[e];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / D + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        float a[VEC], ww[VEC];
        vec_load<D>(xr, lane, j, a);
        if (rr) {
            float r[VEC];
            vec_load<D>(rr, lane, j, r);
#pragma unroll
            for (int e = 0; e < VEC; ++e) a[e] = round_bf16(a[e] + r[e]);
        }
        vec_weight<D>(w, w_f32, lane, j, ww);
#pragma unroll
        for (int e = 0; e < VEC; ++e) a[e] = a[e] * rstd * ww[e];
        vec_store<D>(y + row * D, lane, j, a);
    }
}

// Narrow rows (D = 64, 128, 256: the per-head norms): D / 8 lanes per row with 16 bytes each, 32 / (D / 8) rows per warp,
// one pass with the row in registers -- a warp per 128-byte row moves too few bytes per instruction.
template <int D>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_narrow_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                          const void* __restrict__ w, int w_f32, __nv_bfloat16* __restrict__ y,
                          __nv_bfloat16* __restrict__ sum_out, long rows, float inv_n, float eps) {
    constexpr int LPR = D / 8, RPW = 32 / LPR;
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    const long row_raw = ((long)blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW + lane / LPR;
    const bool ok = row_raw < rows;
    const long row = ok ? row_raw : rows - 1;                 // keep every lane in the shuffles
    float a[8], ww[8];
    ld8(x + row * D + sub * 8, a);
    if (res) {
        float r[8];
        ld8(res + row * D + sub * 8, r);
#pragma unroll
        for (int e = 0; e < 8; ++e) a[e] = round_bf16(a[e] + r[e]);
        if (sum_out && ok) st8(sum_out + row * D + sub * 8, a);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int col = sub * 8 + e;
        ww[e] = w ? (w_f32 ? reinterpret_cast<const float*>(w)[col] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[col])) : 1.f;
    }
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += a[e] * a[e];
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rstd = rsqrtf(ss * inv_n + eps);              // 1 / D, or 1 for the l2 norm
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = a[e] * rstd * ww[e];
    if (ok) st8(y + row * D + sub * 8, a);
}

// dx = rstd (dy w - xhat mean(dy w xhat)) (+ dadd);  dw_part [gridDim.x, D] = per-CTA sums of dy xhat.
// A thread owns eight neighbouring features of its rows: the row, its gradient and what is added are read once, with the next
// turn's loads in flight, and the weights and their gradients stay in registers.  Narrow rows (D <= 256): D / 8 lanes, the rows
// of a warp side by side, no barrier.  Wide rows: D / 8 threads, 256 / (D / 8) rows of a CTA side by side, the
// partial sums of the warps through shared memory (double-buffered: one barrier a turn), 64 registers for four CTAs per SM with 86 to
// 112 bytes spilled; two rows deep takes 127 registers and half the CTAs (127 against 121 us).  Bound by memory.  L2 flushed, against a warp per row that read it twice, one row in flight:
// 32768 x 2048 with an added gradient 217 -> 121 us (traffic 82), 524288 x 128 137 -> 107 us (62).  Few rows are bound by the turns of
// a CTA (min(rows / 8, RMS_BWD_CTAS) CTAs, so eight turns of one row at 2048 features), in a graph, warm: 300 x 2048 15.5 -> 11.0 us,
// 1000 x 2048 14.9 -> 10.9, 4000 x 2048 52 -> 19, 1000 x 64 2.3 -> 2.4, 16000 x 64 4.9 -> 4.1.
constexpr int RMS_BWD_CTAS = 592;                              // four per SM, one partial sum of the weight gradient each
struct RmsBwd {
    const __nv_bfloat16 *s, *dy, *dadd;
    const void* w;
    __nv_bfloat16* dx;
    float* dw_part;                                            // NULL: no weight
    long rows;
    float inv_n, eps;                                          // 1 / D, or 1 for the l2 norm
    int w_f32, wide;                                           // wide: every tensor starts on 16 bytes
};
__device__ __forceinline__ void rms_sums(const uint64_t (&a)[4], const uint64_t (&g)[4], const uint64_t (&ww)[4], float& ss, float& c) {
    uint64_t s2 = 0, c2 = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        s2 = fma2(a[i], a[i], s2);
        c2 = fma2(mul2(g[i], ww[i]), a[i], c2);
    }
    ss = hsum2(s2);
    c = hsum2(c2);
}
// g becomes the gradient of the row in front of the added one; ss, c are the sums over the row.
__device__ __forceinline__ void rms_grad(const uint64_t (&a)[4], uint64_t (&g)[4], const uint64_t (&ww)[4], uint64_t (&dwa)[4], float ss, float c,
                                         float inv_n, float eps, bool ok) {
    const float rstd = rsqrtf(ss * inv_n + eps), m = -(c * rstd * inv_n);     // m = -mean(dy w xhat)
    const uint64_t r2 = pack2(rstd, rstd), m2 = pack2(m, m);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint64_t xh = mul2(a[i], r2);
        if (ok) dwa[i] = fma2(g[i], xh, dwa[i]);
        g[i] = mul2(r2, fma2(xh, m2, mul2(g[i], ww[i])));
    }
}
__device__ __forceinline__ void rms_store(const RmsBwd& p, long at, uint64_t (&g)[4], const uint4& add) {
    if (p.dadd) {
        uint64_t r[4];
        open8(add, r);
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = add2(g[i], r[i]);
    }
    st16(p.dx + at, close8(g), p.wide);
}

template <int D>
__global__ void __launch_bounds__(256) rmsnorm_bwd_narrow_kernel(const RmsBwd p) {
    constexpr int LPR = D / 8, RPW = 32 / LPR;
    __shared__ float s_dw[8][D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPR;
    uint64_t ww[4], dwa[4];
    weights8(p.w, p.w_f32, sub * 8, ww);
#pragma unroll
    for (int i = 0; i < 4; ++i) dwa[i] = 0;
    const long step = (long)gridDim.x * 8 * RPW;
    long row0 = ((long)blockIdx.x * 8 + warp) * RPW;           // the warp's first row of this turn
    uint4 na, ng, nr = make_uint4(0, 0, 0, 0);
    auto load = [&](long r0) {
        const long r = r0 + lane / LPR < p.rows ? r0 + lane / LPR : p.rows - 1;      // keep every lane in the shuffles
        const long at = r * D + sub * 8;
        na = ld16(p.s + at, p.wide);
        ng = ld16(p.dy + at, p.wide);
        if (p.dadd) nr = ld16(p.dadd + at, p.wide);
    };
    if (row0 < p.rows) load(row0);
    for (; row0 < p.rows; row0 += step) {
        uint64_t a[4], g[4];
        open8(na, a);
        open8(ng, g);
        const uint4 add = nr;
        if (row0 + step < p.rows) load(row0 + step);
        float ss, c;
        rms_sums(a, g, ww, ss, c);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        const bool ok = row0 + lane / LPR < p.rows;
        rms_grad(a, g, ww, dwa, ss, c, p.inv_n, p.eps, ok);
        if (ok) rms_store(p, (row0 + lane / LPR) * D + sub * 8, g, add);
    }
    if (!p.dw_part) return;
    float o8[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) unpack2(dwa[i], o8[2 * i], o8[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) o8[i] += __shfl_xor_sync(0xffffffffu, o8[i], o);
        if (lane < LPR) s_dw[warp][sub * 8 + i] = o8[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += 256) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) s += s_dw[k][i];
        p.dw_part[(long)blockIdx.x * D + i] = s;
    }
}

template <int D>
__global__ void __launch_bounds__(256, 4) rmsnorm_bwd_wide_kernel(const RmsBwd p) {
    constexpr int TPR = D / 8, RB = 256 / TPR, W = TPR / 32;   // threads of a row; rows side by side; warps of a row
    __shared__ float2 s_sum[2][8];
    __shared__ float s_dw[RB > 1 ? RB * D : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rb = tid / TPR, f0 = (tid % TPR) * 8;
    uint64_t ww[4], dwa[4];
    weights8(p.w, p.w_f32, f0, ww);
#pragma unroll
    for (int i = 0; i < 4; ++i) dwa[i] = 0;
    const long step = (long)gridDim.x * RB;
    uint4 na, ng, nr = make_uint4(0, 0, 0, 0);
    auto load = [&](long row0) {
        const long at = (row0 + rb < p.rows ? row0 + rb : p.rows - 1) * D + f0;
        na = ld16(p.s + at, p.wide);
        ng = ld16(p.dy + at, p.wide);
        if (p.dadd) nr = ld16(p.dadd + at, p.wide);
    };
    long row0 = (long)blockIdx.x * RB;
    if (row0 < p.rows) load(row0);
    for (int buf = 0; row0 < p.rows; row0 += step, buf ^= 1) {
        uint64_t a[4], g[4];
        open8(na, a);
        open8(ng, g);
        const uint4 add = nr;
        float ss, c;
        rms_sums(a, g, ww, ss, c);
        ss = warp_sum(ss);
        c = warp_sum(c);
        if (lane == 0) s_sum[buf][warp] = make_float2(ss, c);
        if (row0 + step < p.rows) load(row0 + step);
        __syncthreads();
        ss = c = 0.f;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const float2 v = s_sum[buf][rb * W + k];
            ss += v.x;
            c += v.y;
        }
        const bool ok = row0 + rb < p.rows;
        rms_grad(a, g, ww, dwa, ss, c, p.inv_n, p.eps, ok);
        if (ok) rms_store(p, (row0 + rb) * D + f0, g, add);
    }
    if (!p.dw_part) return;
    float o8[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) unpack2(dwa[i], o8[2 * i], o8[2 * i + 1]);
    if constexpr (RB == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) p.dw_part[(long)blockIdx.x * D + f0 + i] = o8[i];
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) s_dw[rb * D + f0 + i] = o8[i];
        __syncthreads();
        for (int i = tid; i < D; i += 256) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < RB; ++k) s += s_dw[k * D + i];
            p.dw_part[(long)blockIdx.x * D + i] = s;
        }
    }
}

// ------------------------------------------------------------------------------------------------ SwiGLU
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y, long n8) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
        float fa[8], fb[8], o[8];
        ld8(a + i * 8, fa);
        ld8(b + i * 8, fb);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fa[e] * sigmoidf_(fa[e]) * fb[e];
        st8(y + i * 8, o);
    }
}
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, const __nv_bfloat16* __restrict__ dy,
                  __nv_bfloat16* __restrict__ da, __nv_bfloat16* __restrict__ db, long n8) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
        float fa[8], fb[8], g[8], oa[8], ob[8];
        ld8(a + i * 8, fa);
        ld8(b + i * 8, fb);
        ld8(dy + i * 8, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float s = sigmoidf_(fa[e]);
            oa[e] = g[e] * fb[e] * s * (1.f + fa[e] * (1.f - s));
            ob[e] = g[e] * fa[e] * s;
        }
        st8(da + i * 8, oa);
        st8(db + i * 8, ob);
    }
}

// ------------------------------------------------------------------------------------------------ block mean
// y[b, c, d] = mean over the tokens of block c (the last block may be shorter), tokens added up in their order: the selection's
// decisions hang on the last bit.  One thread = a pair of channels of one block with MEAN_U rows in flight, so that few long blocks
// (4 x 1030 tokens in blocks of 256: five thousand threads of eight channels) keep the memory busy too.
constexpr int MEAN_U = 16;
__global__ void __launch_bounds__(128)
block_mean_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int T, int D, int nbs, int NB) {
    const int cp = blockIdx.x * blockDim.x + threadIdx.x;
    if (cp * 2 >= D) return;
    const int c = blockIdx.y, b = blockIdx.z;
    const int t0 = c * nbs, n = min(T, t0 + nbs) - t0;
    const uint32_t* p = reinterpret_cast<const uint32_t*>(x + ((long)b * T + t0) * D) + cp;
    const long pitch = D / 2;
    uint64_t acc = 0;
    int t = 0;
    for (; t + MEAN_U <= n; t += MEAN_U) {
        uint32_t v[MEAN_U];
#pragma unroll
        for (int i = 0; i < MEAN_U; ++i) v[i] = p[(t + i) * pitch];
#pragma unroll
        for (int i = 0; i < MEAN_U; ++i) acc = add2(acc, open2(v[i]));
    }
#pragma unroll 4
    for (; t < n; ++t) acc = add2(acc, open2(p[t * pitch]));
    const float inv = 1.f / (float)n;
    reinterpret_cast<uint32_t*>(y + ((long)b * NB + c) * D)[cp] = close2(mul2(acc, pack2(inv, inv)));
}

static inline const __nv_bfloat16* bfc(const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); }
static inline __nv_bfloat16* bfm(void* p) { return reinterpret_cast<__nv_bfloat16*>(p); }

}  // namespace natsl

using namespace natsl;

// The four taps of two neighbouring channels, one pair per tap (a tap at a time they were sixteen loads of two bytes per lane,
// which took the load unit longer than the tile).
__device__ __forceinline__ void conv_taps(const uint4& v, uint64_t& t0, uint64_t& t1, uint64_t& t2, uint64_t& t3) {
    const float2 a01 = unpack_bf16(v.x), a23 = unpack_bf16(v.y), b01 = unpack_bf16(v.z), b23 = unpack_bf16(v.w);
    t0 = pack2(a01.x, b01.x);
    t1 = pack2(a01.y, b01.y);
    t2 = pack2(a23.x, b23.x);
    t3 = pack2(a23.y, b23.y);
}

// Forward with the input tile staged in shared memory: one CTA = 128 channels x 64 tokens (+ 3 halo rows), every load
// issued at once with cp.async; warp s computes the tokens 8 s .. 8 s + 7, a lane four channels (two pairs).  8 x 4096 x 2048, L2
// flushed: 104 us a channel at a time, 88 us in pairs, 78 us with the taps in two loads (traffic 41).
constexpr int CF_TT = 64, CF_L = 32, CF_CH = 4;
__global__ void __launch_bounds__(256)
short_conv_fwd_tile_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                           const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ y, int T, int D, int silu, int wide) {
    constexpr int W = CONV_W, XR = CF_TT + W - 1, ROWB = CF_L * CF_CH * 2, CPR = ROWB / 16;
    __shared__ __align__(16) unsigned char xs[XR * ROWB];
    const int tid = threadIdx.x, lane = tid & 31, sr = tid >> 5;
    const int d_cta = blockIdx.x * CF_L * CF_CH, d0 = d_cta + lane * CF_CH;
    const int t0 = blockIdx.y * CF_TT, b = blockIdx.z;
    const bool ch_ok = d0 < D;
    const uint32_t xs_a = smem_u32(xs);
    for (int i = tid; i < XR * CPR; i += 256) {
        const int r = i / CPR, c = i % CPR;
        const int t = t0 - (W - 1) + r, dd = d_cta + c * 8;
        const bool ok = t >= 0 && t < T && dd < D;
        cp_async16(xs_a + r * ROWB + c * 16, ok ? (const void*)(x + ((long)b * T + t) * D + dd) : (const void*)x, ok ? 16 : 0);
    }
    cp_async_commit();
    static_assert(CF_CH == 4, "a thread reads 8 bytes per row: two pairs of channels");
    uint64_t wt[W][2], bs[2];                                 // [tap][pair of channels]
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int dd = (ch_ok ? d0 : 0) + 2 * c;
        bs[c] = bias ? pack2(__bfloat162float(bias[dd]), __bfloat162float(bias[dd + 1])) : 0;
        conv_taps(ld16(w + dd * W, wide), wt[0][c], wt[1][c], wt[2][c], wt[3][c]);
    }
    cp_async_wait<0>();
    __syncthreads();
    uint64_t win[W][2];
    auto row = [&](int r, uint64_t (&f)[2]) {
        const uint2 v = *reinterpret_cast<const uint2*>(xs + r * ROWB + lane * 8);
        f[0] = open2(v.x);
        f[1] = open2(v.y);
    };
    const int ts = sr * 8;
    __nv_bfloat16* yp = y + ((long)b * T + t0 + ts) * D + d0;
#pragma unroll
    for (int j = 0; j < W - 1; ++j) row(ts + j, win[j + 1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int j = 0; j < W - 1; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) win[j][c] = win[j + 1][c];
        row(ts + i + W - 1, win[W - 1]);
        uint64_t o[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            o[c] = bs[c];
#pragma unroll
            for (int j = 0; j < W; ++j) o[c] = fma2(wt[j][c], win[j][c], o[c]);
            if (silu) o[c] = silu2(o[c]);
        }
        if (ch_ok && t0 + ts + i < T) *reinterpret_cast<uint2*>(yp + (long)i * D) = make_uint2(close2(o[0]), close2(o[1]));
    }
}

extern "C" int natsl_short_conv_fwd(const void* x, const void* w, const void* bias, void* y, int B, int T, int D, int W,
                                    int silu, void* stream) {
    NATSL_REQUIRE(x && w && y, NATSL_ERR_NULL, "natsl_short_conv_fwd: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && D > 0 && D % 8 == 0 && B <= 65535, NATSL_ERR_BAD_SHAPE,
                  "natsl_short_conv_fwd: bad shape (D a multiple of 8)");
    NATSL_REQUIRE(W == CONV_W, NATSL_ERR_UNSUPPORTED, "natsl_short_conv_fwd: kernel size %d is not built (4)", W);
    NATSL_REQUIRE(natsl::aligned_to(16, x) && natsl::aligned_to(8, y), NATSL_ERR_UNSUPPORTED,
                  "natsl_short_conv_fwd: a tensor does not start on 16 bytes (y: 8)");
    dim3 grid((D + CF_L * CF_CH - 1) / (CF_L * CF_CH), (T + CF_TT - 1) / CF_TT, B);
    short_conv_fwd_tile_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(bfc(x), bfc(w), bfc(bias), bfm(y), T, D, silu,
                                                                                         aligned_to(16, w));
    return check_launch("natsl_short_conv_fwd");
}

// The same backward for span = 64 with the tiles staged in shared memory: one CTA = 128 channels x 64 tokens, all loads
// of the x tile (64 + 6 halo rows) and the dy tile (64 + 3) are issued at once with cp.async (the sliding-window form
// above has two loads in flight per thread and is bound by their latency).  What bounds it then is instruction issue, so
// a warp (64 channels, two per lane: four would need 90 registers and leave two CTAs on an SM) slides over 16 tokens with
// the window of x and of the pre-activation gradients in registers: each row is read and unpacked once and three of
// nineteen gradients are computed twice.  The weight-gradient partials of the four warps of a channel group are summed in
// shared memory in a fixed order: one partial per CTA.  A lane's two channels are a pair of floats.  8 x 4096 x 2048, L2 flushed:
// 160 us a channel at a time, 141 us in pairs with the sigmoid's division taken out (traffic 61); instruction issue (72 %) bounds it.
constexpr int CB_TT = 64, CB_CG = 32, CB_CH = 2;      // tokens per CTA, threads across channels, channels per thread
constexpr int CB_GR = 2, CB_WT = 16;                  // channel groups per CTA, tokens per warp
__global__ void __launch_bounds__(256, 4)
short_conv_bwd_tile_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                           const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ dy,
                           __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, int T, int D, int silu, int wide) {
    constexpr int W = CONV_W;
    constexpr int XR = CB_TT + 2 * (W - 1), YR = CB_TT + (W - 1);            // rows of the two tiles
    constexpr int ROWB = CB_GR * CB_CG * CB_CH * 2;                          // bytes per tile row
    constexpr int CPR = ROWB / 16;                                          // 16-byte chunks per tile row
    static_assert(CB_TT / CB_WT * CB_GR == 8 && W == 4 && CB_CH == 2, "eight warps; a lane reads 4 bytes per row");
    extern __shared__ __align__(16) unsigned char smem_cb[];
    unsigned char* xs = smem_cb;
    unsigned char* ys = smem_cb + XR * ROWB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = warp & (CB_GR - 1), sr = warp / CB_GR;
    const int d_cta = blockIdx.x * CB_GR * CB_CG * CB_CH;
    const int t0 = blockIdx.y * CB_TT, b = blockIdx.z;
    const int d0 = d_cta + (grp * CB_CG + lane) * CB_CH;
    const bool ch_ok = d0 < D;
    {
        const uint32_t xs_a = smem_u32(xs), ys_a = smem_u32(ys);
        for (int i = tid; i < XR * CPR; i += 256) {
            const int r = i / CPR, c = i % CPR;
            const int t = t0 - (W - 1) + r, dd = d_cta + c * 8;
            const bool ok = t >= 0 && t < T && dd < D;
            cp_async16(xs_a + r * ROWB + c * 16, ok ? (const void*)(x + ((long)b * T + t) * D + dd) : (const void*)x, ok ? 16 : 0);
        }
        for (int i = tid; i < YR * CPR; i += 256) {
            const int r = i / CPR, c = i % CPR;
            const int t = t0 + r, dd = d_cta + c * 8;
            const bool ok = t < T && dd < D;
            cp_async16(ys_a + r * ROWB + c * 16, ok ? (const void*)(dy + ((long)b * T + t) * D + dd) : (const void*)dy, ok ? 16 : 0);
        }
        cp_async_commit();
    }
    const int dc = ch_ok ? d0 : 0;                             // a lane's two channels are one pair of floats
    uint64_t wt[W], bs, dwa[W + 1];
    bs = bias ? pack2(__bfloat162float(bias[dc]), __bfloat162float(bias[dc + 1])) : 0;
    conv_taps(ld16(w + dc * W, wide), wt[0], wt[1], wt[2], wt[3]);
#pragma unroll
    for (int j = 0; j <= W; ++j) dwa[j] = 0;
    cp_async_wait<0>();
    __syncthreads();
    auto row = [&](const unsigned char* tile, int r) {
        return open2(*reinterpret_cast<const uint32_t*>(tile + r * ROWB + (grp * CB_CG + lane) * 4));
    };
    // Step i of this warp: the pre-activation gradient of token ts + i (rows ts + i .. ts + i + 3 of the x tile are its
    // window; dy is zero outside the sequence) and, from the third step on, dx of token ts + i - 3, which needs the
    // gradients of tokens ts + i - 3 .. ts + i.  The weight gradients take the warp's own tokens only.
    const int ts = sr * CB_WT;
    uint64_t xw[W], dps[W];
    const uint64_t one = pack2(1.f, 1.f), neg = pack2(-1.f, -1.f);
#pragma unroll
    for (int j = 0; j < W - 1; ++j) xw[j] = row(xs, ts + j);
    auto step = [&](int i, bool own) {
        xw[W - 1] = row(xs, ts + i + W - 1);
        uint64_t g = row(ys, ts + i), a = bs;
#pragma unroll
        for (int j = 0; j < W; ++j) a = fma2(wt[j], xw[j], a);
        if (silu) {
            const uint64_t sg = sigmoid2(a);
            g = mul2(mul2(g, sg), fma2(a, fma2(sg, neg, one), one));
        }
        if (own) {
#pragma unroll
            for (int j = 0; j < W; ++j) dwa[j] = fma2(g, xw[j], dwa[j]);
            dwa[W] = add2(dwa[W], g);
        }
#pragma unroll
        for (int k = 0; k < W - 1; ++k) {
            dps[k] = dps[k + 1];
            xw[k] = xw[k + 1];
        }
        dps[W - 1] = g;
    };
#pragma unroll
    for (int k = 0; k < W; ++k) dps[k] = 0;
#pragma unroll
    for (int i = 0; i < W - 1; ++i) step(i, true);
    __nv_bfloat16* dxp = dx + ((long)b * T + t0 + ts) * D + d0;
#pragma unroll
    for (int i = W - 1; i < CB_WT + W - 1; ++i) {
        step(i, i < CB_WT);
        if (t0 + ts + i - (W - 1) < T && ch_ok) {
            uint64_t o = mul2(wt[0], dps[W - 1]);
#pragma unroll
            for (int j = 1; j < W; ++j) o = fma2(wt[j], dps[W - 1 - j], o);
            *reinterpret_cast<uint32_t*>(dxp + (long)(i - (W - 1)) * D) = close2(o);
        }
    }
    // ---- the warps' partials -> one per CTA (fixed order)
    __syncthreads();
    constexpr int NW = CB_TT / CB_WT, PER = CB_CH * (W + 1) * CB_CG;
    float* red = reinterpret_cast<float*>(smem_cb);          // [group][token warps][CB_CH * (W + 1)][32 lanes]
#pragma unroll
    for (int j = 0; j <= W; ++j) {
        float lo, hi;
        unpack2(dwa[j], lo, hi);
        red[(grp * NW + sr) * PER + j * CB_CG + lane] = lo;
        red[(grp * NW + sr) * PER + (W + 1 + j) * CB_CG + lane] = hi;
    }
    __syncthreads();
    float* part = dw_part + (((long)b * gridDim.y + blockIdx.y) * D + d_cta) * (W + 1);
    for (int e = tid; e < CB_GR * PER; e += 256) {           // in the order of the result
        const int ch = e / (W + 1), j = e % (W + 1), gr = ch / (CB_CG * CB_CH), l = ch / CB_CH % CB_CG, c = ch % CB_CH;
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < NW; ++k) a += red[(gr * NW + k) * PER + (c * (W + 1) + j) * CB_CG + l];
        if (d_cta + ch < D) part[e] = a;
    }
}

extern "C" int natsl_short_conv_bwd(const void* x, const void* w, const void* bias, const void* dy, void* dx, float* dw_part,
                                    int B, int T, int D, int W, int silu, int span, void* stream) {
    NATSL_REQUIRE(x && w && dy && dx && dw_part, NATSL_ERR_NULL, "natsl_short_conv_bwd: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && D > 0 && D % 8 == 0 && B <= 65535 && span > 0, NATSL_ERR_BAD_SHAPE,
                  "natsl_short_conv_bwd: bad shape (D a multiple of 8)");
    NATSL_REQUIRE(W == CONV_W, NATSL_ERR_UNSUPPORTED, "natsl_short_conv_bwd: kernel size %d is not built (4)", W);
    NATSL_REQUIRE(natsl::aligned_to(16, x, dy) && natsl::aligned_to(span == CB_TT ? 4 : 16, dx), NATSL_ERR_UNSUPPORTED,
                  "natsl_short_conv_bwd: a tensor does not start on 16 bytes (dx: 4 with spans of 64 tokens)");
    const int groups = D / 8;
    if (span == CB_TT) {
        constexpr int smem = ((CB_TT + 2 * (CONV_W - 1)) + (CB_TT + CONV_W - 1)) * CB_GR * CB_CG * CB_CH * 2;
        static_assert(smem >= 8 * CB_CH * (CONV_W + 1) * CB_CG * 4, "the partial sums are reduced over the tiles");
        cudaError_t e = cudaFuncSetAttribute(short_conv_bwd_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            set_error("natsl_short_conv_bwd: cannot reserve %d B of shared memory (%s)", smem, cudaGetErrorString(e));
            return NATSL_ERR_CUDA;
        }
        dim3 grid((D + CB_GR * CB_CG * CB_CH - 1) / (CB_GR * CB_CG * CB_CH), (T + CB_TT - 1) / CB_TT, B);
        short_conv_bwd_tile_kernel<<<grid, 256, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
            bfc(x), bfc(w), bfc(bias), bfc(dy), bfm(dx), dw_part, T, D, silu, aligned_to(16, w));
        return check_launch("natsl_short_conv_bwd");
    }
    dim3 grid((groups + 127) / 128, (T + span - 1) / span, B);
    short_conv_bwd_kernel<<<grid, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(bfc(x), bfc(w), bfc(bias), bfc(dy), bfm(dx),
                                                                                   dw_part, T, D, silu, span);
    return check_launch("natsl_short_conv_bwd");
}

#define NATSL_ROW_DISPATCH(CALL)                                                               \
    switch (D) {                                                                               \
        case 512: CALL(512); break;                                                            \
        case 1024: CALL(1024); break;                                                          \
        case 2048: CALL(2048); break;                                                          \
        default:                                                                               \
            set_error("unsupported row width D=%d (64, 128, 256, 512, 1024 or 2048)", D);      \
            return NATSL_ERR_UNSUPPORTED;                                                      \
    }

extern "C" int natsl_rmsnorm_fwd(const void* x, const void* res, const void* w, int w_dtype, void* y, void* sum_out, long rows,
                                 int D, float eps, void* stream) {
    NATSL_REQUIRE(x && y, NATSL_ERR_NULL, "natsl_rmsnorm_fwd: null pointer");
    NATSL_REQUIRE(rows > 0, NATSL_ERR_BAD_SHAPE, "natsl_rmsnorm_fwd: empty input");
    NATSL_REQUIRE(w_dtype == NATSL_DT_BF16 || w_dtype == NATSL_DT_F32, NATSL_ERR_UNSUPPORTED, "natsl_rmsnorm_fwd: weight must be bf16 or f32");
    NATSL_REQUIRE(natsl::aligned_to(16, x, res, y, sum_out), NATSL_ERR_UNSUPPORTED, "natsl_rmsnorm_fwd: a tensor does not start on 16 bytes");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (D == 64 || D == 128 || D == 256) {
        const int rpc = 8 * (32 / (D / 8));                  // rows per CTA
        const unsigned gridn = (unsigned)((rows + rpc - 1) / rpc);
#define NATSL_NARROW(DD) rmsnorm_fwd_narrow_kernel<DD><<<gridn, 256, 0, st>>>(bfc(x), bfc(res), w, w_dtype == NATSL_DT_F32, bfm(y), bfm(sum_out), rows, 1.f / DD, eps)
        if (D == 64) NATSL_NARROW(64);
        else if (D == 128) NATSL_NARROW(128);
        else NATSL_NARROW(256);
#undef NATSL_NARROW
        return check_launch("natsl_rmsnorm_fwd");
    }
    const unsigned grid = (unsigned)((rows + 7) / 8);
#define NATSL_CALL(DD) rmsnorm_fwd_kernel<DD><<<grid, 256, 0, st>>>(bfc(x), bfc(res), w, w_dtype == NATSL_DT_F32, bfm(y), bfm(sum_out), rows, eps)
    NATSL_ROW_DISPATCH(NATSL_CALL)
#undef NATSL_CALL
    return check_launch("natsl_rmsnorm_fwd");
}

extern "C" int natsl_rmsnorm_bwd(const void* s, const void* w, int w_dtype, const void* dy, const void* dadd, void* dx,
                                 float* dw_part, int n_part, long rows, int D, float eps, void* stream) {
    NATSL_REQUIRE(s && dy && dx && dw_part, NATSL_ERR_NULL, "natsl_rmsnorm_bwd: null pointer");
    NATSL_REQUIRE(rows > 0 && n_part > 0, NATSL_ERR_BAD_SHAPE, "natsl_rmsnorm_bwd: empty input");
    NATSL_REQUIRE(w_dtype == NATSL_DT_BF16 || w_dtype == NATSL_DT_F32, NATSL_ERR_UNSUPPORTED, "natsl_rmsnorm_bwd: weight must be bf16 or f32");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const RmsBwd p = {bfc(s), bfc(dy), bfc(dadd), w, bfm(dx), dw_part, rows, D > 0 ? 1.f / D : 0.f, eps, w_dtype == NATSL_DT_F32,
                      aligned_to(16, s, dy, dadd, dx)};
    switch (D) {
        case 64: rmsnorm_bwd_narrow_kernel<64><<<n_part, 256, 0, st>>>(p); break;
        case 128: rmsnorm_bwd_narrow_kernel<128><<<n_part, 256, 0, st>>>(p); break;
        case 256: rmsnorm_bwd_narrow_kernel<256><<<n_part, 256, 0, st>>>(p); break;
        case 512: rmsnorm_bwd_wide_kernel<512><<<n_part, 256, 0, st>>>(p); break;
        case 1024: rmsnorm_bwd_wide_kernel<1024><<<n_part, 256, 0, st>>>(p); break;
        case 2048: rmsnorm_bwd_wide_kernel<2048><<<n_part, 256, 0, st>>>(p); break;
        default:
            set_error("unsupported row width D=%d (64, 128, 256, 512, 1024 or 2048)", D);
            return NATSL_ERR_UNSUPPORTED;
    }
    return check_launch("natsl_rmsnorm_bwd");
}

// y = x * rsqrt(sum(x^2) + eps) and its backward: the narrow rows' kernels with the sum of squares in the place of its mean.
extern "C" int natsl_l2norm_fwd(const void* x, void* y, int64_t rows, int D, float eps, void* stream) {
    NATSL_REQUIRE(x && y, NATSL_ERR_NULL, "natsl_l2norm_fwd: null pointer");
    NATSL_REQUIRE(rows > 0, NATSL_ERR_BAD_SHAPE, "natsl_l2norm_fwd: empty input");
    NATSL_REQUIRE(D == 64 || D == 128 || D == 256, NATSL_ERR_UNSUPPORTED, "natsl_l2norm_fwd: row width D=%d (64, 128 or 256)", D);
    NATSL_REQUIRE(aligned_to(16, x, y), NATSL_ERR_UNSUPPORTED, "natsl_l2norm_fwd: x and y must start on 16 bytes");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const unsigned grid = (unsigned)((rows + 8 * (256 / D) - 1) / (8 * (256 / D)));
    if (D == 64) rmsnorm_fwd_narrow_kernel<64><<<grid, 256, 0, st>>>(bfc(x), nullptr, nullptr, 0, bfm(y), nullptr, rows, 1.f, eps);
    else if (D == 128) rmsnorm_fwd_narrow_kernel<128><<<grid, 256, 0, st>>>(bfc(x), nullptr, nullptr, 0, bfm(y), nullptr, rows, 1.f, eps);
    else rmsnorm_fwd_narrow_kernel<256><<<grid, 256, 0, st>>>(bfc(x), nullptr, nullptr, 0, bfm(y), nullptr, rows, 1.f, eps);
    return check_launch("natsl_l2norm_fwd");
}

extern "C" int natsl_l2norm_bwd(const void* x, const void* dy, void* dx, int64_t rows, int D, float eps, void* stream) {
    NATSL_REQUIRE(x && dy && dx, NATSL_ERR_NULL, "natsl_l2norm_bwd: null pointer");
    NATSL_REQUIRE(rows > 0, NATSL_ERR_BAD_SHAPE, "natsl_l2norm_bwd: empty input");
    NATSL_REQUIRE(D == 64 || D == 128 || D == 256, NATSL_ERR_UNSUPPORTED, "natsl_l2norm_bwd: row width D=%d (64, 128 or 256)", D);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const RmsBwd p = {bfc(x), bfc(dy), nullptr, nullptr, bfm(dx), nullptr, rows, 1.f, eps, 0, aligned_to(16, x, dy, dx)};
    const long turns = (rows + 8 * (256 / D) - 1) / (8 * (256 / D));
    const unsigned grid = (unsigned)(turns < RMS_BWD_CTAS ? turns : RMS_BWD_CTAS);
    if (D == 64) rmsnorm_bwd_narrow_kernel<64><<<grid, 256, 0, st>>>(p);
    else if (D == 128) rmsnorm_bwd_narrow_kernel<128><<<grid, 256, 0, st>>>(p);
    else rmsnorm_bwd_narrow_kernel<256><<<grid, 256, 0, st>>>(p);
    return check_launch("natsl_l2norm_bwd");
}

extern "C" int natsl_swiglu_fwd(const void* a, const void* b, void* y, long n, void* stream) {
    NATSL_REQUIRE(a && b && y, NATSL_ERR_NULL, "natsl_swiglu_fwd: null pointer");
    NATSL_REQUIRE(n > 0 && n % 8 == 0, NATSL_ERR_BAD_SHAPE, "natsl_swiglu_fwd: element count must be a positive multiple of 8");
    NATSL_REQUIRE(natsl::aligned_to(16, a, b, y), NATSL_ERR_UNSUPPORTED, "natsl_swiglu_fwd: a tensor does not start on 16 bytes");
    const long n8 = n / 8;
    const unsigned grid = (unsigned)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
    swiglu_fwd_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(bfc(a), bfc(b), bfm(y), n8);
    return check_launch("natsl_swiglu_fwd");
}

extern "C" int natsl_swiglu_bwd(const void* a, const void* b, const void* dy, void* da, void* db, long n, void* stream) {
    NATSL_REQUIRE(a && b && dy && da && db, NATSL_ERR_NULL, "natsl_swiglu_bwd: null pointer");
    NATSL_REQUIRE(n > 0 && n % 8 == 0, NATSL_ERR_BAD_SHAPE, "natsl_swiglu_bwd: element count must be a positive multiple of 8");
    NATSL_REQUIRE(natsl::aligned_to(16, a, b, dy, da, db), NATSL_ERR_UNSUPPORTED, "natsl_swiglu_bwd: a tensor does not start on 16 bytes");
    const long n8 = n / 8;
    const unsigned grid = (unsigned)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
    swiglu_bwd_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(bfc(a), bfc(b), bfc(dy), bfm(da), bfm(db), n8);
    return check_launch("natsl_swiglu_bwd");
}

extern "C" int natsl_block_mean(const void* x, void* y, int B, int T, int D, int nbs, void* stream) {
    NATSL_REQUIRE(x && y, NATSL_ERR_NULL, "natsl_block_mean: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && D > 0 && D % 8 == 0 && nbs > 0 && B <= 65535, NATSL_ERR_BAD_SHAPE,
                  "natsl_block_mean: bad shape (D a multiple of 8)");
    const int NB = (T + nbs - 1) / nbs;
    NATSL_REQUIRE(NB <= 65535, NATSL_ERR_TOO_LARGE, "natsl_block_mean: too many blocks");
    NATSL_REQUIRE(natsl::aligned_to(4, x, y), NATSL_ERR_UNSUPPORTED, "natsl_block_mean: a tensor does not start on 4 bytes");
    dim3 grid((D / 2 + 127) / 128, NB, B);
    block_mean_kernel<<<grid, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(bfc(x), bfm(y), T, D, nbs, NB);
    return check_launch("natsl_block_mean");
}

// ------------------------------------------------------------------------------------------------ cache growth
// One contiguous run per batch entry moved to another pitch (a cache's key or value rows into a longer buffer).  Bandwidth: four
// 16-byte loads in flight per thread; the framework's strided element copy took 151 us for 134 MB, this one 41 us.
__global__ void __launch_bounds__(256) copy_batches_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, long n, long dst_pitch,
                                                           long src_pitch) {
    const uint4* s = src + blockIdx.y * src_pitch;
    uint4* d = dst + blockIdx.y * dst_pitch;
    const long i0 = (long)blockIdx.x * 1024 + threadIdx.x;
    uint4 x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (i0 + e * 256 < n) x[e] = s[i0 + e * 256];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (i0 + e * 256 < n) d[i0 + e * 256] = x[e];
}
extern "C" int natsl_copy_batches(void* dst, const void* src, int B, int64_t bytes, int64_t dst_pitch, int64_t src_pitch, void* stream) {
    NATSL_REQUIRE(dst && src, NATSL_ERR_NULL, "natsl_copy_batches: null pointer");
    NATSL_REQUIRE(B > 0 && B <= 65535 && bytes > 0 && bytes <= dst_pitch && bytes <= src_pitch, NATSL_ERR_BAD_SHAPE,
                  "natsl_copy_batches: bad shape");
    NATSL_REQUIRE(((bytes | dst_pitch | src_pitch) & 15) == 0 && natsl::aligned_to(16, dst, src), NATSL_ERR_UNSUPPORTED,
                  "natsl_copy_batches: addresses, sizes and pitches must be multiples of 16 bytes");
    const long n = bytes / 16;
    NATSL_REQUIRE((n + 1023) / 1024 <= 0x7fffffffL, NATSL_ERR_TOO_LARGE, "natsl_copy_batches: too large");
    copy_batches_kernel<<<dim3((unsigned)((n + 1023) / 1024), B), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<uint4*>(dst), reinterpret_cast<const uint4*>(src), n, dst_pitch / 16, src_pitch / 16);
    return check_launch("natsl_copy_batches");
}

// ------------------------------------------------------------------------------------------------ cross entropy rows
// One CTA per row of bf16 logits [rows, vocab]: loss_rows[r] = (logsumexp(l) - l[y]) if y != ignore else 0, and the
// logits are overwritten with their gradient (softmax(l) - onehot(y)) * inv_denom (zero for ignored rows), bf16.
// Two passes over the row: maximum and sum of exponentials (online, fp32), then the gradient.
__global__ void __launch_bounds__(256)
xent_rows_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, float* __restrict__ loss_rows,
                 int vocab, long long ignore_index, float inv_denom) {
    __shared__ float s_m[8], s_s[8];
    const long row = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __nv_bfloat16* lr = logits + row * (long)vocab;
    const long long y = labels[row];
    const bool ok = y != ignore_index;
    const int n8 = vocab / 8;
    float m = -INFINITY, s = 0.f;
    for (int i = tid; i < n8; i += 256) {
        float f[8];
        natsl::ld8(lr + i * 8, f);
        float mx = f[0];
#pragma unroll
        for (int e = 1; e < 8; ++e) mx = fmaxf(mx, f[e]);
        const float mn = fmaxf(m, mx);
        float acc = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc += __expf(f[e] - mn);
        s = s * __expf(m - mn) + acc;
        m = mn;
    }
    for (int i = n8 * 8 + tid; i < vocab; i += 256) {          // tail (vocab not a multiple of 8)
        const float f = __bfloat162float(lr[i]);
        const float mn = fmaxf(m, f);
        s = s * __expf(m - mn) + __expf(f - mn);
        m = mn;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
        const float mn = fmaxf(m, m2);
        s = (mn == -INFINITY) ? 0.f : s * __expf(m - mn) + s2 * __expf(m2 - mn);
        m = mn;
    }
    if (lane == 0) {
        s_m[warp] = m;
        s_s[warp] = s;
    }
    __syncthreads();
    float M = s_m[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) M = fmaxf(M, s_m[w]);
    float S = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) S += (s_m[w] == -INFINITY) ? 0.f : s_s[w] * __expf(s_m[w] - M);
    const float lse = M + __logf(S);
    if (tid == 0) loss_rows[row] = ok ? lse - __bfloat162float(lr[ok ? y : 0]) : 0.f;
    __syncthreads();                                           // the target logit is read before the row is overwritten
    const float sc = ok ? inv_denom : 0.f;
    for (int i = tid; i < n8; i += 256) {
        float f[8];
        natsl::ld8(lr + i * 8, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float p = __expf(f[e] - lse) - ((long long)(i * 8 + e) == y ? 1.f : 0.f);
            f[e] = p * sc;
        }
        natsl::st8(lr + i * 8, f);
    }
    for (int i = n8 * 8 + tid; i < vocab; i += 256) {
        const float p = __expf(__bfloat162float(lr[i]) - lse) - ((long long)i == y ? 1.f : 0.f);
        lr[i] = __float2bfloat16(p * sc);
    }
}

extern "C" int natsl_xent_rows(void* logits, const void* labels, float* loss_rows, long rows, int vocab, long ignore_index,
                               float inv_denom, void* stream) {
    NATSL_REQUIRE(logits && labels && loss_rows, NATSL_ERR_NULL, "natsl_xent_rows: null pointer");
    NATSL_REQUIRE(rows > 0 && rows <= 0x7fffffffL && vocab > 0, NATSL_ERR_BAD_SHAPE, "natsl_xent_rows: bad shape");
    NATSL_REQUIRE((reinterpret_cast<uintptr_t>(logits) & 15) == 0 && vocab % 8 == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_xent_rows: rows must be 16-byte aligned (vocab a multiple of 8)");
    xent_rows_kernel<<<(unsigned)rows, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<__nv_bfloat16*>(logits), reinterpret_cast<const long long*>(labels), loss_rows, vocab,
        (long long)ignore_index, inv_denom);
    return check_launch("natsl_xent_rows");
}
