// Output mixing of the hybrid layer: two-input RMSNorm with per-row mixing weights and a swish gate,
//   y = (x1 * rstd1 * w1 * a + x2 * rstd2 * w2 * b) * g * sigmoid(g),   rstd = 1 / sqrt(mean(x^2) + eps)
// (x1 = linear-branch output, x2 = softmax-branch output, (a, b) = learned per-(token, head) weights).
// Replaces the forward of FusedMultiInputRMSNormGated, src/nats/modules/fused_norm_gate.py:38-182
// (module :1354-1429).  Pure bandwidth: one warp per row of D elements, 16-byte loads and stores, fp32 math.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

constexpr long NORM_GATE_GRID = 148 * 8;

__device__ __forceinline__ float load_scalar(const void* p, int dtype, long i) {
    return dtype == NATSL_DT_F32 ? reinterpret_cast<const float*>(p)[i]
                                 : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

// Rows a warp has in flight: D / 8 lanes per row with 16 bytes each, 32 / (D / 8) rows side by side.
template <int D>
struct MixShape {
    static constexpr int LPR = D / 8, RPW = 32 / LPR;
};
template <int LPR>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One pass with the rows in registers.  Bandwidth once the arithmetic is out of the way: pairs of features (two floats per
// instruction), weights kept in registers over all rows of a warp, no division.  524288 x 128, L2 flushed: 129 -> 113 us (traffic 82).
template <int D>
__global__ void __launch_bounds__(256)
norm_gate_mix_kernel(const __nv_bfloat16* __restrict__ x1, const __nv_bfloat16* __restrict__ x2,
                     const __nv_bfloat16* __restrict__ g, const void* __restrict__ xw, int xw_dtype,
                     const void* __restrict__ w1, const void* __restrict__ w2, int w_dtype,
                     __nv_bfloat16* __restrict__ y, long rows, float eps, int activation) {
    constexpr int LPR = MixShape<D>::LPR, RPW = MixShape<D>::RPW;
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    uint64_t p1[4], p2[4];
    weights8(w1, w_dtype == NATSL_DT_F32, sub * 8, p1);
    weights8(w2, w_dtype == NATSL_DT_F32, sub * 8, p2);
    for (long row0 = ((long)blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW; row0 < rows; row0 += (long)gridDim.x * 8 * RPW) {
        const bool ok = row0 + lane / LPR < rows;
        const long row = ok ? row0 + lane / LPR : rows - 1;   // keep every lane in the shuffles
        const long base = row * D + sub * 8;
        const uint4 ua = *reinterpret_cast<const uint4*>(x1 + base), ub = *reinterpret_cast<const uint4*>(x2 + base),
                    ug = *reinterpret_cast<const uint4*>(g + base);
        float m1 = 1.f, m2 = 1.f;
        if (xw) { m1 = load_scalar(xw, xw_dtype, row * 2); m2 = load_scalar(xw, xw_dtype, row * 2 + 1); }
        uint64_t a[4], b[4], gg[4], q1 = 0, q2 = 0;
        open8(ua, a);
        open8(ub, b);
        open8(ug, gg);
#pragma unroll
        for (int i = 0; i < 4; ++i) { q1 = fma2(a[i], a[i], q1); q2 = fma2(b[i], b[i], q2); }
        const float s1 = row_sum<LPR>(hsum2(q1)), s2 = row_sum<LPR>(hsum2(q2));
        const float r1 = rsqrtf(s1 / D + eps) * m1, r2 = rsqrtf(s2 / D + eps) * m2;
        const uint64_t f1 = pack2(r1, r1), f2 = pack2(r2, r2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t v = fma2(mul2(a[i], p1[i]), f1, mul2(mul2(b[i], p2[i]), f2)), sg = sigmoid2(gg[i]);
            a[i] = mul2(v, activation == 1 ? sg : mul2(gg[i], sg));
        }
        if (ok) *reinterpret_cast<uint4*>(y + base) = close8(a);
    }
}


// Backward of the output mixing (src/nats/modules/fused_norm_gate.py:353, :657).  With n = x * rstd and
// v = n1 w1 a + n2 w2 b,  y = v * s(g):   dv = dy s(g),  dg = dy v s'(g),  da = <dv, n1 w1>,  db = <dv, n2 w2>,
// dx = rstd (dn - n mean(dn n)) with dn1 = dv w1 a (dn2 likewise; the sum of dn1 n1 is a da), and the weight gradients
// dw1 = sum_rows dv n1 a, dw2 = sum_rows dv n2 b.  The same rows per warp, strided over a fixed grid, the next rows' loads in
// flight; every CTA writes one partial sum of the weight gradients (dw_part [grid, 2, D] fp32; the caller adds the CTAs up), so
// nothing is accumulated atomically.
template <int D>
__global__ void __launch_bounds__(256, 2)
norm_gate_mix_bwd_kernel(const __nv_bfloat16* __restrict__ x1, const __nv_bfloat16* __restrict__ x2,
                         const __nv_bfloat16* __restrict__ g, const void* __restrict__ xw, int xw_dtype,
                         const void* __restrict__ w1, const void* __restrict__ w2, int w_dtype,
                         const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx1,
                         __nv_bfloat16* __restrict__ dx2, __nv_bfloat16* __restrict__ dg, float* __restrict__ dxw,
                         float* __restrict__ dw_part, long rows, float eps, int activation, int wide) {
    constexpr int LPR = MixShape<D>::LPR, RPW = MixShape<D>::RPW;
    __shared__ float s_dw[8][2][D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPR;
    uint64_t p1[4], p2[4], dw1[4], dw2[4];
    weights8(w1, w_dtype == NATSL_DT_F32, sub * 8, p1);
    weights8(w2, w_dtype == NATSL_DT_F32, sub * 8, p2);
#pragma unroll
    for (int i = 0; i < 4; ++i) dw1[i] = dw2[i] = 0;
    const long step = (long)gridDim.x * 8 * RPW;
    long row = ((long)blockIdx.x * 8 + warp) * RPW + lane / LPR;
    uint4 na, nb, ng, nd;
    float n1m = 1.f, n2m = 1.f;
    auto load = [&](long r) {
        r = r < rows ? r : rows - 1;                           // keep every lane in the shuffles
        const long base = r * D + sub * 8;
        na = ld16(x1 + base, wide);
        nb = ld16(x2 + base, wide);
        ng = ld16(g + base, wide);
        nd = ld16(dy + base, wide);
        if (xw) { n1m = load_scalar(xw, xw_dtype, r * 2); n2m = load_scalar(xw, xw_dtype, r * 2 + 1); }
    };
    if (row - lane / LPR < rows) load(row);
    const uint64_t one = pack2(1.f, 1.f), neg = pack2(-1.f, -1.f);
    for (; row - lane / LPR < rows; row += step) {
        const bool ok = row < rows;
        uint64_t a[4], b[4], gg[4], d[4], q1 = 0, q2 = 0;
        open8(na, a);
        open8(nb, b);
        open8(ng, gg);
        open8(nd, d);
        const float m1 = n1m, m2 = n2m;
        if (row - lane / LPR + step < rows) load(row + step);
#pragma unroll
        for (int i = 0; i < 4; ++i) { q1 = fma2(a[i], a[i], q1); q2 = fma2(b[i], b[i], q2); }
        const float r1 = rsqrtf(row_sum<LPR>(hsum2(q1)) / D + eps), r2 = rsqrtf(row_sum<LPR>(hsum2(q2)) / D + eps);
        const uint64_t e1 = pack2(r1, r1), e2 = pack2(r2, r2), k1 = pack2(m1, m1), k2 = pack2(m2, m2);
        uint64_t da2 = 0, db2 = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t n1 = mul2(a[i], e1), n2 = mul2(b[i], e2), u1 = mul2(n1, p1[i]), u2 = mul2(n2, p2[i]);
            const uint64_t v = fma2(u1, k1, mul2(u2, k2)), sg = sigmoid2(gg[i]), om = fma2(sg, neg, one);       // 1 - sg
            const uint64_t s = activation == 1 ? sg : mul2(gg[i], sg);
            const uint64_t sp = mul2(sg, activation == 1 ? om : fma2(gg[i], om, one));
            const uint64_t dv = mul2(d[i], s);
            d[i] = mul2(mul2(d[i], v), sp);                    // dg
            da2 = fma2(dv, u1, da2);
            db2 = fma2(dv, u2, db2);
            if (ok) {
                dw1[i] = fma2(mul2(dv, n1), k1, dw1[i]);
                dw2[i] = fma2(mul2(dv, n2), k2, dw2[i]);
            }
            gg[i] = dv;
            a[i] = n1;
            b[i] = n2;
        }
        const float da = row_sum<LPR>(hsum2(da2)), db = row_sum<LPR>(hsum2(db2));
        const float c1 = -m1 * da / D, c2 = -m2 * db / D;
        const uint64_t h1 = pack2(c1, c1), h2 = pack2(c2, c2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = mul2(e1, fma2(a[i], h1, mul2(mul2(gg[i], p1[i]), k1)));
            b[i] = mul2(e2, fma2(b[i], h2, mul2(mul2(gg[i], p2[i]), k2)));
        }
        if (ok) {
            const long base = row * D + sub * 8;
            st16(dx1 + base, close8(a), wide);
            st16(dx2 + base, close8(b), wide);
            st16(dg + base, close8(d), wide);
            if (dxw && sub == 0) { dxw[row * 2] = da; dxw[row * 2 + 1] = db; }
        }
    }
    float o1[8], o2[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        unpack2(dw1[i], o1[2 * i], o1[2 * i + 1]);
        unpack2(dw2[i], o2[2 * i], o2[2 * i + 1]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) {                   // the rows side by side in the warp
            o1[i] += __shfl_xor_sync(0xffffffffu, o1[i], o);
            o2[i] += __shfl_xor_sync(0xffffffffu, o2[i], o);
        }
        if (lane < LPR) {
            s_dw[warp][0][sub * 8 + i] = o1[i];
            s_dw[warp][1][sub * 8 + i] = o2[i];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * D; i += 256) {
        float s = 0.f;
#pragma unroll
        for (int wv = 0; wv < 8; ++wv) s += s_dw[wv][i / D][i % D];
        dw_part[(long)blockIdx.x * 2 * D + i] = s;
    }
}

}  // namespace natsl

extern "C" int natsl_norm_gate_mix(const void* x1, const void* x2, const void* g, const void* xw, int xw_dtype,
                                   const void* w1, const void* w2, int w_dtype, void* y, long rows, int D, float eps,
                                   int activation, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(x1 && x2 && g && y, NATSL_ERR_NULL, "natsl_norm_gate_mix: null pointer");
    NATSL_REQUIRE(rows > 0, NATSL_ERR_BAD_SHAPE, "natsl_norm_gate_mix: empty input");
    NATSL_REQUIRE(activation == 0 || activation == 1, NATSL_ERR_UNSUPPORTED, "natsl_norm_gate_mix: activation 0 (swish) or 1 (sigmoid)");
    NATSL_REQUIRE((xw_dtype == NATSL_DT_BF16 || xw_dtype == NATSL_DT_F32) && (w_dtype == NATSL_DT_BF16 || w_dtype == NATSL_DT_F32),
                  NATSL_ERR_UNSUPPORTED, "natsl_norm_gate_mix: weights must be bf16 or f32");
    NATSL_REQUIRE(natsl::aligned_to(16, x1, x2, g, y), NATSL_ERR_UNSUPPORTED, "natsl_norm_gate_mix: a tensor does not start on 16 bytes");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int wpb = 8;
    const long rpc = (long)wpb * (32 / (D > 0 ? (D / 8 > 0 ? D / 8 : 1) : 1));      // rows per CTA and turn
    const long turns = (rows + rpc - 1) / rpc;
    const unsigned grid = (unsigned)(turns < NORM_GATE_GRID ? turns : NORM_GATE_GRID);
#define NATSL_NG(DD) norm_gate_mix_kernel<DD><<<grid, wpb * 32, 0, st>>>( \
        reinterpret_cast<const __nv_bfloat16*>(x1), reinterpret_cast<const __nv_bfloat16*>(x2), \
        reinterpret_cast<const __nv_bfloat16*>(g), xw, xw_dtype, w1, w2, w_dtype, reinterpret_cast<__nv_bfloat16*>(y), rows, eps, activation)
    if (D == 64) NATSL_NG(64);
    else if (D == 128) NATSL_NG(128);
    else if (D == 256) NATSL_NG(256);
    else {
        set_error("natsl_norm_gate_mix: unsupported row width D=%d (64, 128 or 256)", D);
        return NATSL_ERR_UNSUPPORTED;
    }
#undef NATSL_NG
    return check_launch("natsl_norm_gate_mix");
}

extern "C" int natsl_norm_gate_mix_bwd(const void* x1, const void* x2, const void* g, const void* xw, int xw_dtype,
                                       const void* w1, const void* w2, int w_dtype, const void* dy, void* dx1, void* dx2,
                                       void* dg, float* dxw, float* dw_part, int n_part, long rows, int D, float eps,
                                       int activation, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(x1 && x2 && g && dy && dx1 && dx2 && dg && dw_part, NATSL_ERR_NULL, "natsl_norm_gate_mix_bwd: null pointer");
    NATSL_REQUIRE((xw == nullptr) == (dxw == nullptr), NATSL_ERR_NULL,
                  "natsl_norm_gate_mix_bwd: the mixing weights and their gradient go together");
    NATSL_REQUIRE(rows > 0 && n_part > 0 && n_part <= 65535, NATSL_ERR_BAD_SHAPE, "natsl_norm_gate_mix_bwd: bad sizes");
    NATSL_REQUIRE(activation == 0 || activation == 1, NATSL_ERR_UNSUPPORTED, "natsl_norm_gate_mix_bwd: activation 0 (swish) or 1 (sigmoid)");
    NATSL_REQUIRE((xw_dtype == NATSL_DT_BF16 || xw_dtype == NATSL_DT_F32) && (w_dtype == NATSL_DT_BF16 || w_dtype == NATSL_DT_F32),
                  NATSL_ERR_UNSUPPORTED, "natsl_norm_gate_mix_bwd: weights must be bf16 or f32");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    auto bf = [](const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); };
    auto bm = [](void* p) { return reinterpret_cast<__nv_bfloat16*>(p); };
    const int wide = aligned_to(16, x1, x2, g, dy, dx1, dx2, dg);
#define NATSL_NGB(DD) norm_gate_mix_bwd_kernel<DD><<<n_part, 256, 0, st>>>(bf(x1), bf(x2), bf(g), xw, xw_dtype, w1, w2, w_dtype, \
        bf(dy), bm(dx1), bm(dx2), bm(dg), dxw, dw_part, rows, eps, activation, wide)
    if (D == 64) NATSL_NGB(64);
    else if (D == 128) NATSL_NGB(128);
    else if (D == 256) NATSL_NGB(256);
    else {
        set_error("natsl_norm_gate_mix_bwd: unsupported row width D=%d (64, 128 or 256)", D);
        return NATSL_ERR_UNSUPPORTED;
    }
#undef NATSL_NGB
    return check_launch("natsl_norm_gate_mix_bwd");
}
