// Small steps of a layer's training path as one kernel each, forward and backward: the decays, betas and step sizes
// (src/nats/layers/natsl_attn_gdn.py:461-480, src/nats/layers/natsl_attn_mamba2.py:402-440), the gradient of the block mean, the sums
// of per-CTA partial weight gradients, and the gradient of the block types.  As torch operations they were about ninety of the 165
// launches of a Mamba2 layer's training step, ten microseconds of host time and a pass over memory each.
#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

using bf16 = __nv_bfloat16;
__device__ __forceinline__ float ldx(const void* p, int f32, long i) {
    return f32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}
__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ------------------------------------------------------------------------------------------------ gates
// dt = softplus(a + dt_bias), g = -e^{A_log} dt, beta = sigmoid(b) (times two), v_out = v dt.  A CTA works on GATE_T / H rows at a
// time, a thread per (row, head); the values of those rows are scaled 16 bytes at a time.  Bound by reading v once and writing it once.
constexpr int GATE_T = 256;
struct GateArgs {
    const bf16 *a, *b, *v;                    // [rows,H], [rows,H] or NULL, [rows,H,V] or NULL
    const void *A_log, *dt_bias;
    int alog_f32, dtb_f32, neg, H, V, wide, dbeta_f32;
    long rows;
    float* g;                                 // forward
    bf16 *beta, *v_out;
    const float* dg;                          // backward
    const void* dbeta;
    const bf16* dv_out;
    bf16 *da, *db, *dv;
    float* part;                              // [gridDim.x, 2, H]: gradients of A_log, dt_bias
};

__global__ void __launch_bounds__(GATE_T) gates_fwd_kernel(const GateArgs p) {
    __shared__ float s_dt[GATE_T];
    const int tid = threadIdx.x, R = GATE_T / p.H, n = R * p.H;
    const long row0 = (long)blockIdx.x * R;
    const int m = (int)min((long)n, (p.rows - row0) * p.H);            // (row, head) pairs of this CTA
    if (tid < m) {
        const long i = row0 * p.H + tid;
        const int h = tid % p.H;
        const float dt = softplus(__bfloat162float(p.a[i]) + ldx(p.dt_bias, p.dtb_f32, h));
        p.g[i] = -expf(ldx(p.A_log, p.alog_f32, h)) * dt;
        s_dt[tid] = dt;
        if (p.b) {
            const float y = rbf(1.f / (1.f + expf(-__bfloat162float(p.b[i]))));
            p.beta[i] = __float2bfloat16(p.neg ? 2.f * y : y);
        }
    }
    if (!p.v) return;
    __syncthreads();
    const int cpr = p.V / 8;
    for (int i = tid; i < m * cpr; i += GATE_T) {
        const long at = row0 * p.H * p.V + (long)i * 8;
        const float dt = s_dt[i / cpr];
        const uint64_t d2 = pack2(dt, dt);
        uint64_t x[4];
        open8(ld16(p.v + at, p.wide), x);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = mul2(x[e], d2);
        st16(p.v_out + at, close8(x), p.wide);
    }
}

// A fixed grid walks the rows; every thread keeps the sums of its head, every CTA writes one partial sum.
__global__ void __launch_bounds__(GATE_T) gates_bwd_kernel(const GateArgs p) {
    __shared__ float s_dt[GATE_T], s_ddt[GATE_T], s_sum[2][GATE_T];
    const int tid = threadIdx.x, R = GATE_T / p.H, n = R * p.H, h = tid % p.H, cpr = p.V / 8;
    const float A = expf(ldx(p.A_log, p.alog_f32, h)), bias = ldx(p.dt_bias, p.dtb_f32, h);
    float sum_a = 0.f, sum_b = 0.f;
    for (long row0 = (long)blockIdx.x * R; row0 < p.rows; row0 += (long)gridDim.x * R) {
        const int m = (int)min((long)n, (p.rows - row0) * p.H);
        const long i0 = row0 * p.H;
        float z = 0.f, dt = 0.f;
        if (tid < m) {
            z = __bfloat162float(p.a[i0 + tid]) + bias;
            dt = softplus(z);
        }
        if (p.dv_out) {
            s_dt[tid] = dt;
            __syncthreads();
            // V / 8 (a power of two, at most 32) lanes per (row, head)
            for (int i = tid; i < (m * cpr + GATE_T - 1) / GATE_T * GATE_T; i += GATE_T) {
                const bool ok = i < m * cpr;
                const long at = i0 * p.V + (long)(ok ? i : 0) * 8;
                const float d = s_dt[ok ? i / cpr : 0];
                const uint64_t d2 = pack2(d, d);
                uint64_t x[4], y[4], s2 = 0;
                open8(ld16(p.dv_out + at, p.wide), x);
                open8(ld16(p.v + at, p.wide), y);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s2 = fma2(x[e], y[e], s2);
                    x[e] = mul2(x[e], d2);
                }
                float s = hsum2(s2);
                for (int o = cpr / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (ok) {
                    st16(p.dv + at, close8(x), p.wide);
                    if (i % cpr == 0) s_ddt[i / cpr] = s;
                }
            }
            __syncthreads();
        }
        if (tid < m) {
            const float dgv = p.dg ? p.dg[i0 + tid] : 0.f;
            const float ddt = -A * dgv + (p.dv_out ? s_ddt[tid] : 0.f);
            const float ez = expf(z), dz = z > 20.f ? ddt : ddt * (ez / (ez + 1.f));
            sum_a += dgv * (-A * dt);
            sum_b += dz;
            p.da[i0 + tid] = __float2bfloat16(dz);
            if (p.db) {
                const float y = rbf(1.f / (1.f + expf(-__bfloat162float(p.b[i0 + tid]))));
                const float db = p.dbeta ? ldx(p.dbeta, p.dbeta_f32, i0 + tid) : 0.f;
                p.db[i0 + tid] = __float2bfloat16((p.neg ? 2.f * db : db) * ((1.f - y) * y));
            }
        }
    }
    s_sum[0][tid] = tid < n ? sum_a : 0.f;
    s_sum[1][tid] = tid < n ? sum_b : 0.f;
    __syncthreads();
    for (int i = tid; i < 2 * p.H; i += GATE_T) {
        const int w = i / p.H, hh = i % p.H;
        float s = 0.f;
        for (int r = 0; r < R; ++r) s += s_sum[w][r * p.H + hh];
        p.part[(long)blockIdx.x * 2 * p.H + i] = s;
    }
}

// ------------------------------------------------------------------------------------------------ block mean, backward
__global__ void __launch_bounds__(256)
block_mean_bwd_kernel(const bf16* __restrict__ dy, bf16* __restrict__ dx, int T, int D, int nbs, int NB, int wide) {
    const int cpr = D / 8, b = blockIdx.y;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long)T * cpr) return;
    const int t = (int)(i / cpr), c = (int)(i % cpr), blk = t / nbs;
    const float n = (float)(min(T, (blk + 1) * nbs) - blk * nbs);
    const uint4 v = ld16(dy + ((long)b * NB + blk) * D + c * 8, wide);
    const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16(u[e]);
        o[e] = pack_bf16(f.x / n, f.y / n);
    }
    st16(dx + ((long)b * T + t) * D + c * 8, make_uint4(o[0], o[1], o[2], o[3]), wide);
}

// ------------------------------------------------------------------------------------------------ sums of partial gradients
// out[n] = sum_p part[p, n].  A CTA: 32 columns x 32 threads; a thread adds up every 32nd row in four sums (rows 128 apart each, what is
// left over in the first), then the four in pairs, and a warp the 32 threads of a column as a tree: the same order on every run.
struct ColArgs {
    const float* part;
    void *o0, *o1;
    int P, N, mode, f0, f1;                   // mode 0: o0[n]; 1: the second half to o1; w > 1: groups of w + 1, the last to o1
};
__global__ void __launch_bounds__(1024) column_sums_kernel(const ColArgs a) {
    __shared__ float s[32][33];
    const int c = threadIdx.x, r = threadIdx.y, n = blockIdx.x * 32 + c;
    float x0 = 0.f, x1 = 0.f, x2 = 0.f, x3 = 0.f;
    if (n < a.N) {
        const float* p = a.part + n;
        int k = r;
        for (; k + 96 < a.P; k += 128) {
            x0 += p[(long)k * a.N];
            x1 += p[(long)(k + 32) * a.N];
            x2 += p[(long)(k + 64) * a.N];
            x3 += p[(long)(k + 96) * a.N];
        }
        for (; k < a.P; k += 32) x0 += p[(long)k * a.N];
    }
    s[r][c] = (x0 + x1) + (x2 + x3);
    __syncthreads();
    const float v = warp_sum(s[c][r]);                        // warp r: column r of the CTA
    const int m = blockIdx.x * 32 + r;
    if (c == 0 && m < a.N) {
        void* o = a.o0;
        int f = a.f0;
        long at = m;
        if (a.mode == 1 && m >= a.N / 2) { o = a.o1; f = a.f1; at = m - a.N / 2; }
        if (a.mode > 1) {
            const int g = m / (a.mode + 1), j = m % (a.mode + 1);
            if (j == a.mode) { o = a.o1; f = a.f1; at = g; }
            else at = (long)g * a.mode + j;
        }
        if (!o) return;
        if (f) reinterpret_cast<float*>(o)[at] = v;
        else reinterpret_cast<bf16*>(o)[at] = __float2bfloat16(v);
    }
}

// ------------------------------------------------------------------------------------------------ gradient of the block types
// out [B,TN,HN,2]: column 0 the sum of the softmax branch's per-tile sums [B,NT,HQ] over a block and the heads of the selection group
// where the block is selected, column 1 that of the linear branch's [B,NT,H] (block size 64: one tile per block).
__global__ void __launch_bounds__(256)
types_grad_kernel(const float* __restrict__ pa, const float* __restrict__ pl, const int* __restrict__ types_i, void* __restrict__ out, int f32,
                  int n, int TN, int HN, int HQ, int H) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int hn = i % HN;
    const long bt = i / HN;                                   // b * TN + t
    float s = 0.f, l = 0.f;
    for (int e = 0; e < HQ / HN; ++e) s += pa[bt * HQ + hn * (HQ / HN) + e];
    for (int e = 0; e < H / HN; ++e) l += pl[bt * H + hn * (H / HN) + e];
    if (!types_i[2l * i]) s = s * 0.f;
    if (f32) *reinterpret_cast<float2*>(reinterpret_cast<float*>(out) + 2l * i) = make_float2(s, l);
    else *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(out) + 2l * i) = pack_bf16(s, l);
}

bool dt_ok(int d) { return d == NATSL_DT_BF16 || d == NATSL_DT_F32; }
const bf16* cb(const void* p) { return reinterpret_cast<const bf16*>(p); }
bf16* mb(void* p) { return reinterpret_cast<bf16*>(p); }

}  // namespace
}  // namespace natsl

extern "C" int natsl_gates_fwd(const void* a, const void* b, const void* v, const void* A_log, int alog_dtype, const void* dt_bias,
                               int dtb_dtype, int neg_eigval, float* g, void* beta, void* v_out, int64_t rows, int H, int V, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(a && A_log && dt_bias && g && !b == !beta && !v == !v_out, NATSL_ERR_NULL, "natsl_gates_fwd: null pointer");
    NATSL_REQUIRE(rows > 0 && H > 0 && H <= GATE_T && (!v || (V > 0 && V % 8 == 0)), NATSL_ERR_BAD_SHAPE, "natsl_gates_fwd: bad shape");
    NATSL_REQUIRE(dt_ok(alog_dtype) && dt_ok(dtb_dtype), NATSL_ERR_UNSUPPORTED, "natsl_gates_fwd: A_log and dt_bias must be bf16 or f32");
    GateArgs p = {};
    p.a = cb(a); p.b = cb(b); p.v = cb(v); p.A_log = A_log; p.dt_bias = dt_bias;
    p.alog_f32 = alog_dtype == NATSL_DT_F32; p.dtb_f32 = dtb_dtype == NATSL_DT_F32; p.neg = neg_eigval; p.H = H; p.V = V;
    p.wide = aligned_to(16, v, v_out); p.rows = rows; p.g = g; p.beta = mb(beta); p.v_out = mb(v_out);
    const long R = GATE_T / H, grid = (rows + R - 1) / R;
    NATSL_REQUIRE(grid <= 0x7fffffffL, NATSL_ERR_TOO_LARGE, "natsl_gates_fwd: too many rows");
    gates_fwd_kernel<<<(unsigned)grid, GATE_T, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
    return check_launch("natsl_gates_fwd");
}

extern "C" int natsl_gates_bwd(const void* a, const void* b, const void* v, const void* A_log, int alog_dtype, const void* dt_bias,
                               int dtb_dtype, int neg_eigval, const float* dg, const void* dbeta, int dbeta_dtype, const void* dv_out, void* da,
                               void* db, void* dv, float* part, int n_part, int64_t rows, int H, int V, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(a && A_log && dt_bias && da && part && !b == !db && !dv_out == !dv && (v || !dv_out), NATSL_ERR_NULL,
                  "natsl_gates_bwd: null pointer");
    NATSL_REQUIRE(rows > 0 && H > 0 && H <= GATE_T && n_part > 0 && (!dv_out || V == 32 || V == 64 || V == 128 || V == 256), NATSL_ERR_BAD_SHAPE,
                  "natsl_gates_bwd: bad shape");
    NATSL_REQUIRE(dt_ok(alog_dtype) && dt_ok(dtb_dtype) && dt_ok(dbeta_dtype), NATSL_ERR_UNSUPPORTED, "natsl_gates_bwd: bf16 or f32");
    GateArgs p = {};
    p.a = cb(a); p.b = cb(b); p.v = cb(v); p.A_log = A_log; p.dt_bias = dt_bias;
    p.alog_f32 = alog_dtype == NATSL_DT_F32; p.dtb_f32 = dtb_dtype == NATSL_DT_F32; p.neg = neg_eigval; p.H = H; p.V = V;
    p.wide = aligned_to(16, v, dv_out, dv); p.rows = rows; p.dg = dg; p.dbeta = dbeta; p.dbeta_f32 = dbeta_dtype == NATSL_DT_F32;
    p.dv_out = cb(dv_out); p.da = mb(da); p.db = mb(db); p.dv = mb(dv); p.part = part;
    gates_bwd_kernel<<<n_part, GATE_T, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
    return check_launch("natsl_gates_bwd");
}

extern "C" int natsl_block_mean_bwd(const void* dy, void* dx, int B, int T, int D, int nbs, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(dy && dx, NATSL_ERR_NULL, "natsl_block_mean_bwd: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && D > 0 && D % 8 == 0 && nbs > 0 && B <= 65535, NATSL_ERR_BAD_SHAPE,
                  "natsl_block_mean_bwd: bad shape (D a multiple of 8)");
    const long grid = ((long)T * (D / 8) + 255) / 256;
    NATSL_REQUIRE(grid <= 0x7fffffffL, NATSL_ERR_TOO_LARGE, "natsl_block_mean_bwd: too large");
    block_mean_bwd_kernel<<<dim3((unsigned)grid, B), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(cb(dy), mb(dx), T, D, nbs, (T + nbs - 1) / nbs,
                                                                                                      aligned_to(16, dy, dx));
    return check_launch("natsl_block_mean_bwd");
}

extern "C" int natsl_column_sums(const float* part, int P, int N, int mode, void* out0, int out0_dtype, void* out1, int out1_dtype, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(part && out0, NATSL_ERR_NULL, "natsl_column_sums: null pointer");
    NATSL_REQUIRE(P > 0 && N > 0 && mode >= 0 && (mode != 1 || (N % 2 == 0 && out1)) && (mode < 2 || N % (mode + 1) == 0), NATSL_ERR_BAD_SHAPE,
                  "natsl_column_sums: bad shape");
    NATSL_REQUIRE(dt_ok(out0_dtype) && dt_ok(out1_dtype), NATSL_ERR_UNSUPPORTED, "natsl_column_sums: bf16 or f32");
    const ColArgs a = {part, out0, out1, P, N, mode, out0_dtype == NATSL_DT_F32, out1_dtype == NATSL_DT_F32};
    column_sums_kernel<<<(N + 31) / 32, dim3(32, 32), 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
    return check_launch("natsl_column_sums");
}

extern "C" int natsl_types_grad(const float* attn_tiles, const float* linear_tiles, const int32_t* types_i, void* out, int out_dtype, int B, int TN,
                                int HN, int HQ, int H, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(attn_tiles && linear_tiles && types_i && out, NATSL_ERR_NULL, "natsl_types_grad: null pointer");
    NATSL_REQUIRE(B > 0 && TN > 0 && HN > 0 && HQ % HN == 0 && H % HN == 0 && (long)B * TN * HN <= 0x3fffffffL, NATSL_ERR_BAD_SHAPE,
                  "natsl_types_grad: bad shape");
    NATSL_REQUIRE(dt_ok(out_dtype), NATSL_ERR_UNSUPPORTED, "natsl_types_grad: bf16 or f32");
    const int n = B * TN * HN;
    types_grad_kernel<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(attn_tiles, linear_tiles, types_i, out,
                                                                                         out_dtype == NATSL_DT_F32, n, TN, HN, HQ, H);
    return check_launch("natsl_types_grad");
}
