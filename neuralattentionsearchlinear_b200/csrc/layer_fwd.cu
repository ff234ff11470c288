// The steps of a NAtSL layer between its projection GEMMs and its output GEMM, forward without gradients, as one call:
// selection (hard softmax of the block logits), decays, short convolutions with the norms of both branches, mixing weights,
// selection tables, both attention branches on two streams, and what a decoding cache keeps
// (src/nats/layers/natsl_attn_gdn.py:411-650, src/nats/layers/natsl_attn_mamba2.py:352-590).
// Why one call: a prompt of a thousand tokens is some 200 us of device work in 46 launches that took the host 900 us to
// issue from Python (about 30 of them torch elementwise kernels over small tensors); the large-batch case read and wrote
// every projection two or three times (convolution, norm, cast) on its way.  What each kernel is bound by stands beside it.
#include "layer_fwd.cuh"
#include "tc_common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float bf(const bf16* p, long i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ float ldw(const void* p, int f32, long i) {
    return f32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}

// ------------------------------------------------------------------------------------------------ convolutions + norms
// Short causal convolution + SiLU of the q, k and v projections with the row norms behind it, each projection read once:
//   lin  = conv, conv / ||conv|| (Mamba2 q, k) or conv * dt (Mamba2 v);   attn = RMS norm of conv or of the raw projection;
//   conv = the convolution itself where the mixing weights or the softmax branch need it beside a normed copy.
// A lane owns 4 channels (8-byte accesses, 128 channels per warp; with 8 the registers leave half the warps) and slides over
// TT tokens with the next four rows in flight; a norm group (a head) is 16 or 32 neighbouring lanes.  The three convolutions and
// two norms as kernels of their own took 402 us at B = 16, T = 4096, 1024 channels each.  Instruction issue is what bounds it
// (69 % of the slots at B = 8, 21 warps per SM active, DRAM 42 % busy): the taps, norms and scales work on pairs of channels (two floats per instruction), the bf16 rounding of
// the convolution is also what is stored, and tokens past the end are computed and not stored, so the four tokens of a step
// have no branch between them.  Alone, L2 flushed: 16 x 4096 tokens, 1024 channels each 268 us (559 us one channel at a time, 12
// instead of 24 warps per SM), Mamba2 4 x 4096, 32 heads 246 us (444).  The budget for 24 warps is 80 registers, and the widest of
// the modes spills 58 bytes; with five blocks per SM nothing spills, to the same time for the delta rule (266 us) and a longer one
// for Mamba2 (255 us).
constexpr int CONV_CH = 128, CONV_CTAS = 6;                // channels of a block; blocks per SM
struct ConvSeg {
    const bf16 *x, *w, *bias;
    bf16 *lin, *attn, *conv, *tail;
    const void* nw;                           // norm weights [DK] (attn)
    int nw_f32, D, lin_mode, attn_mode;       // lin 0 plain 1 l2 norm 2 times dt; attn 0 none 1 norm of conv 2 norm of raw
    int lin_lanes, attn_lanes, head, blk0;    // lanes of a norm group; channels per head (dt); first grid block
};
struct ConvArgs {
    ConvSeg seg[3];
    const float* dt;
    int T, H, silu, TT;
    float l2_eps, norm_eps;
};

// One segment's run of tokens; ATTN and LIN are the segment's modes.
template <int ATTN, int LIN>
__device__ __forceinline__ void conv_run(const ConvArgs& a, const ConvSeg& s, const float* bias, int b, int d0, int t0, int t1, int lane) {
    const int D = s.D;
    const bool ok = d0 < D, biased = s.bias != nullptr, silu = a.silu;
    const int dd = ok ? d0 : D - 4;                        // idle lanes stay in the shuffles
    uint64_t w[4][2], nw[2];                               // [tap][pair of channels]
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint2 u0 = *reinterpret_cast<const uint2*>(s.w + (long)(dd + 2 * c) * 4),
                    u1 = *reinterpret_cast<const uint2*>(s.w + (long)(dd + 2 * c + 1) * 4);
        const float2 a01 = unpack_bf16(u0.x), a23 = unpack_bf16(u0.y), b01 = unpack_bf16(u1.x), b23 = unpack_bf16(u1.y);
        w[0][c] = pack2(a01.x, b01.x);
        w[1][c] = pack2(a01.y, b01.y);
        w[2][c] = pack2(a23.x, b23.x);
        w[3][c] = pack2(a23.y, b23.y);
        if (ATTN) {
            const int i = (dd + 2 * c) & (s.attn_lanes * 4 - 1);
            nw[c] = pack2(ldw(s.nw, s.nw_f32, i), ldw(s.nw, s.nw_f32, i + 1));
        }
    }
    const int lanes = ATTN ? s.attn_lanes : s.lin_lanes, lin_lanes = s.lin_lanes;
    const float inv_n = 1.f / (lanes * 4), norm_eps = a.norm_eps, l2_eps = a.l2_eps;      // 1/n of a power of two
    const long at = ((long)b * a.T + t0) * D + dd;
    const bf16* x = s.x + at;                              // the token at hand
    bf16 *lin = s.lin + at, *attn = ATTN ? s.attn + at : nullptr, *conv = s.conv ? s.conv + at : nullptr;
    const float* dt = LIN == 2 ? a.dt + ((long)b * a.T + t0) * a.H + dd / s.head : nullptr;
    auto ld = [&](int ahead) { return *reinterpret_cast<const uint2*>(x + (long)ahead * D); };
    auto open = [](const uint2& v, uint64_t (&f)[2]) {
        f[0] = open2(v.x);
        f[1] = open2(v.y);
    };
    const uint2 zero = make_uint2(0, 0);
    uint64_t h[3][2];                                      // inputs of the three tokens before, oldest first
#pragma unroll
    for (int i = 0; i < 3; ++i) open(t0 - 3 + i >= 0 ? ld(i - 3) : zero, h[i]);
    uint2 nxt[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) nxt[i] = t0 + i < t1 ? ld(i) : zero;
    auto group_sum = [&](const uint64_t (&f)[2], int n) {  // over n = 16 or 32 lanes
        const uint64_t s2 = fma2(f[1], f[1], mul2(f[0], f[0]));
        float lo, hi;
        unpack2(s2, lo, hi);
        float ss = lo + hi;
        if (n > 16) ss += __shfl_xor_sync(0xffffffffu, ss, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        return ss;
    };
#pragma unroll 1
    for (int tb = t0; tb < t1; tb += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool store = ok && tb + i < t1;
            uint64_t r[2], y[2];
            open(nxt[i], r);
            nxt[i] = tb + i + 4 < t1 ? ld(4) : zero;
#pragma unroll
            for (int c = 0; c < 2; ++c) y[c] = 0;
            if (biased) {
#pragma unroll
                for (int c = 0; c < 2; ++c) y[c] = *reinterpret_cast<const uint64_t*>(bias + lane * 4 + 2 * c);
            }
            uint2 yb;
            uint32_t* yw = reinterpret_cast<uint32_t*>(&yb);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                y[c] = fma2(w[3][c], r[c], fma2(w[2][c], h[2][c], fma2(w[1][c], h[1][c], fma2(w[0][c], h[0][c], y[c]))));
                h[0][c] = h[1][c];
                h[1][c] = h[2][c];
                h[2][c] = r[c];
            }
            if (silu) {
#pragma unroll
                for (int c = 0; c < 2; ++c) y[c] = silu2(y[c]);
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                yw[c] = close2(y[c]);
                if (ATTN == 1 || LIN) y[c] = open2(yw[c]);
            }
            auto put_scaled = [&](bf16* p, const uint64_t (&f)[2], float scale, bool norm) {
                const uint64_t sc = pack2(scale, scale);
                uint2 v;
                uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                for (int c = 0; c < 2; ++c) vw[c] = close2(norm ? mul2(mul2(f[c], sc), nw[c]) : mul2(f[c], sc));
                if (store) *reinterpret_cast<uint2*>(p) = v;
            };
            if (conv && store) *reinterpret_cast<uint2*>(conv) = yb;
            if (ATTN == 1) put_scaled(attn, y, rsqrtf(group_sum(y, lanes) * inv_n + norm_eps), true);
            if (ATTN == 2) put_scaled(attn, r, rsqrtf(group_sum(r, lanes) * inv_n + norm_eps), true);
            if (LIN == 0 && store) *reinterpret_cast<uint2*>(lin) = yb;
            if (LIN == 1) put_scaled(lin, y, rsqrtf(group_sum(y, lin_lanes) + l2_eps), false);
            if (LIN == 2) put_scaled(lin, y, tb + i < t1 ? *dt : 0.f, false);
            x += D;
            lin += D;
            if (ATTN) attn += D;
            if (conv) conv += D;
            if (LIN == 2) dt += a.H;
        }
    }
    if (s.tail && t1 == a.T && ok) {                       // the last four inputs, oldest first
        const bf16* e = s.x + ((long)b * a.T + a.T - 4) * D + dd;
#pragma unroll
        for (int i = 0; i < 4; ++i) nxt[i] = *reinterpret_cast<const uint2*>(e + (long)i * D);
        const bf16* n0 = reinterpret_cast<const bf16*>(&nxt[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            bf16 o4[4] = {n0[c], n0[4 + c], n0[8 + c], n0[12 + c]};
            *reinterpret_cast<uint2*>(s.tail + ((long)b * D + d0 + c) * 4) = *reinterpret_cast<const uint2*>(o4);
        }
    }
}

__global__ void __launch_bounds__(128, CONV_CTAS) conv_norm_kernel(const ConvArgs a) {
    __shared__ __align__(16) float bias[CONV_CH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.z;
    const int si = (int)blockIdx.x >= a.seg[2].blk0 ? 2 : (int)blockIdx.x >= a.seg[1].blk0 ? 1 : 0;
    const ConvSeg& s = a.seg[si];
    const int base = ((int)blockIdx.x - s.blk0) * CONV_CH, t0 = ((int)blockIdx.y * 4 + warp) * a.TT, t1 = min(a.T, t0 + a.TT);
    if (s.bias) {
        bias[threadIdx.x] = base + (int)threadIdx.x < s.D ? bf(s.bias, base + threadIdx.x) : 0.f;
        __syncthreads();
    }
    if (t0 >= a.T) return;
#define NATSL_CONV(A, L) \
    if (s.attn_mode == A && s.lin_mode == L) conv_run<A, L>(a, s, bias, b, base + lane * 4, t0, t1, lane)
    NATSL_CONV(0, 0);
    NATSL_CONV(1, 0);
    NATSL_CONV(2, 0);
    NATSL_CONV(0, 1);
    NATSL_CONV(1, 1);
    NATSL_CONV(2, 1);
    NATSL_CONV(0, 2);
#undef NATSL_CONV
}

// ------------------------------------------------------------------------------------------------ decoding state
// log decay and pooled layer input of the tokens behind the last complete block: g_block [B,H], pool_sum [B,hidden]
__global__ void __launch_bounds__(256)
block_rest_kernel(const float* __restrict__ g, const bf16* __restrict__ x, float* __restrict__ g_block, float* __restrict__ pool,
                  int T, int H, int hidden, int rest) {
    const int i = blockIdx.x * 256 + threadIdx.x, b = blockIdx.y;
    if (i < hidden) {
        float s = 0.f;
        for (int t = T - rest; t < T; ++t) s += bf(x, ((long)b * T + t) * hidden + i);
        pool[(long)b * hidden + i] = s;
    }
    if (i < H) {
        float s = 0.f;
        for (int t = T - rest; t < T; ++t) s += g[((long)b * T + t) * H + i];
        g_block[(long)b * H + i] = s;
    }
}

// ------------------------------------------------------------------------------------------------ two streams
// The linear branch runs on a side stream of high priority, so that its CTAs are placed ahead of the softmax branch's
// remaining ones whenever an SM frees up: the serial walk starts earlier and the attention CTAs fill in around it (0.523 -
// 0.542 against 0.559 - 0.561 ms for the whole op at B = 8, T = 4096, H = 16).  The caller's stream forks to it and joins
// again before the call returns, so every buffer may belong to the caller's stream alone.  With NATSL_HYBRID_PLAIN_PRIORITY
// the linear branch stays on the caller's stream and the other one takes a side stream of normal priority.  Streams and events
// belong to the calling thread (one stream of a kind per device, given back with the thread): calls of two threads do not queue behind each other,
// and a thread that captures a graph takes nobody else's work into it.
struct SideStream {
    struct {
        cudaStream_t stream[2];              // of normal, of high priority
        cudaEvent_t ev[3];
    } dev[64] = {};
    ~SideStream() {
        for (auto& d : dev) {
            for (auto& e : d.ev)
                if (e) cudaEventDestroy(e);
            for (auto& s : d.stream)
                if (s) cudaStreamDestroy(s);
        }
    }
};
thread_local SideStream t_side;

int side_stream(int high, cudaStream_t* side, cudaEvent_t** ev) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= 64)) e = cudaErrorInvalidDevice;
    if (e == cudaSuccess && !t_side.dev[dev].stream[high]) {
        int lo = 0, hi = 0;
        e = cudaDeviceGetStreamPriorityRange(&lo, &hi);
        if (e == cudaSuccess)
            e = cudaStreamCreateWithPriority(&t_side.dev[dev].stream[high], cudaStreamNonBlocking, high && hi < 0 ? -1 : 0);
    }
    for (int i = 0; i < 3 && e == cudaSuccess; ++i)
        if (!t_side.dev[dev].ev[i]) e = cudaEventCreateWithFlags(&t_side.dev[dev].ev[i], cudaEventDisableTiming);
    if (e != cudaSuccess) {
        set_error("cannot create the side stream: %s", cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    *side = t_side.dev[dev].stream[high];
    *ev = t_side.dev[dev].ev;
    return NATSL_OK;
}

int stream_after(cudaStream_t waiter, cudaStream_t done, cudaEvent_t ev) {
    cudaError_t e = cudaEventRecord(ev, done);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(waiter, ev, 0);
    if (e != cudaSuccess) {
        set_error("cannot order two streams: %s", cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return NATSL_OK;
}

long up256(long x) { return (x + 255) / 256 * 256; }

struct HybridLayout {
    long w, u, p, gcs, kr, qr, egl, total;
};
// The delta rule with K = 192 runs natsl_gdn_split_prep and natsl_gdn_split_walk (gcs, kr, qr hold kf, qf, vf and p holds tp).
bool split_rule(const natsl_hybrid_args& a) { return a.rule == NATSL_RULE_GDN && a.K == 192; }
HybridLayout hybrid_layout(const natsl_hybrid_args& a) {
    HybridLayout l = {};
    const long n = (long)a.B * a.T * a.H;
    const bool gdn = a.rule == NATSL_RULE_GDN, split = split_rule(a);
    if (a.options & NATSL_HYBRID_FP32) return l;
    l.gcs = 0;
    l.kr = up256(l.gcs + 4 * n);
    l.qr = up256(l.kr + (gdn ? 4 * n : 0));
    l.w = up256(l.qr + (split ? 8 * n : gdn ? 4 * n : 0));
    l.u = up256(l.w + (gdn && !split ? 2 * n * a.K : 0));
    l.p = up256(l.u + (gdn && !split ? 2 * n * a.V : 0));
    l.egl = up256(l.p + (split ? 2 * n * 320 : gdn ? 2 * n * 64 : 0));
    l.total = up256(l.egl + (split ? 4l * a.B * ((a.T + 63) / 64) * a.H : 0));
    return l;
}

int check_hybrid(const natsl_hybrid_args& a) {
    NATSL_REQUIRE(a.q_attn && a.k_attn && a.v_attn && a.q && a.k && a.v && a.g && a.types && a.o_attn && a.lse && a.o_lin &&
                      a.types_i && a.indices && a.n_blocks && a.n_chunks_lin && a.attn_n_iters && (a.workspace || (a.options & NATSL_HYBRID_FP32)) &&
                      (a.rule != NATSL_RULE_GDN || a.beta),
                  NATSL_ERR_NULL, "natsl_hybrid_forward: null pointer");
    NATSL_REQUIRE(a.B > 0 && a.T > 0 && a.H > 0 && a.HN > 0 && a.H % a.HN == 0 && a.HQ > 0 && a.HQ % a.HN == 0 && a.HKV > 0 &&
                      a.HQ % a.HKV == 0 && a.nbs >= 64 && a.nbs % 64 == 0,
                  NATSL_ERR_BAD_SHAPE, "natsl_hybrid_forward: bad shape");
    NATSL_REQUIRE(a.rule == NATSL_RULE_GDN || (a.rule == NATSL_RULE_MAMBA && ((a.K == 128 && a.V == 64) || (a.options & NATSL_HYBRID_FP32))),
                  NATSL_ERR_UNSUPPORTED,
                  "natsl_hybrid_forward: Mamba2 is built for K = 128, V = 64 (got K=%d V=%d)", a.K, a.V);
    NATSL_REQUIRE((a.options & NATSL_HYBRID_FP32) || aligned_to(16, a.q_attn, a.k_attn, a.v_attn, a.q, a.k, a.v, a.h0, a.o_attn, a.o_lin, a.ht,
                                                                a.hstart, a.workspace),
                  NATSL_ERR_UNSUPPORTED, "natsl_hybrid_forward: q, k, v, states, outputs and workspace must start on 16 bytes");
    // the token recurrence behind this option steps over the end of an unfinished last block and knows no types of its own
    // for a finished one: its block-start state is not the one a decoder rolls back to
    NATSL_REQUIRE(!((a.options & NATSL_HYBRID_FP32) && a.hstart), NATSL_ERR_UNSUPPORTED,
                  "natsl_hybrid_forward: no block-start state of fp32 tensors");
    NATSL_REQUIRE(a.workspace_bytes >= hybrid_layout(a).total, NATSL_ERR_TOO_LARGE, "natsl_hybrid_forward: workspace of %ld bytes, %ld needed",
                  (long)a.workspace_bytes, hybrid_layout(a).total);
    return NATSL_OK;
}

// Both branches.  types_dtype TBL_LOGITS: a.types are logits, types_raw receives the sampled types.  `before_attn` is launched
// beside the linear branch.
template <typename F>
int hybrid_forward(const natsl_hybrid_args& a, void* types_raw, cudaStream_t st, F before_attn) {
    cudaStream_t side = st;
    cudaEvent_t* ev = nullptr;
    const bool high = !(a.options & NATSL_HYBRID_PLAIN_PRIORITY);
    int rc = side_stream(high, &side, &ev);
    if (rc != NATSL_OK) return rc;
    const cudaStream_t lin = high ? side : st, att = high ? st : side;
    const HybridLayout l = hybrid_layout(a);
    unsigned char* ws = reinterpret_cast<unsigned char*>(a.workspace);
    float* gcs = reinterpret_cast<float*>(ws + l.gcs);
    const int TN = (a.T + a.nbs - 1) / a.nbs;
    const bool gdn = a.rule == NATSL_RULE_GDN;
    if (a.options & NATSL_HYBRID_FP32) {
        // reference-precision kernels; the recurrence is the longer chain and starts first
        rc = launch_tables(a.types, a.types_dtype, types_raw, a.B, TN, a.HN, a.T, a.nbs, a.types_i, a.indices, a.n_blocks,
                           a.n_chunks_lin, a.starting_h_idx, a.attn_n_iters, st);
        if (rc == NATSL_OK) rc = stream_after(side, st, ev[0]);
        if (rc == NATSL_OK)
            rc = natsl_linear_recurrent_fwd(a.rule, NATSL_DT_F32, a.q, a.k, a.v, a.g, a.beta, a.types_i, a.h0, a.o_lin, a.ht, a.hstart, a.B,
                                            a.T, a.H, a.HN, a.K, a.V, a.nbs, a.scale_lin, a.decay ? NATSL_FLAG_DECAY_SKIPPED : 0,
                                            a.use_l2norm, lin);
        if (rc == NATSL_OK)
            rc = natsl_attn_fwd_fp32((a.options & NATSL_HYBRID_ATTN_BF16) ? NATSL_DT_BF16 : NATSL_DT_F32, a.q_attn, a.k_attn, a.v_attn,
                                     a.types_i, a.o_attn, a.lse, a.B, a.T, a.HQ, a.HKV, a.HN, a.DK, a.DV, a.nbs, a.scale_attn,
                                     a.own_attn ? NATSL_FLAG_ATTN_OWN_CHUNK : 0, att);
        const int join = stream_after(st, side, ev[2]);
        return rc != NATSL_OK ? rc : join;
    }
    rc = stream_after(side, st, ev[0]);
    // the preparation reads no tables: it starts while they are built
    const bool split = split_rule(a);
    if (rc == NATSL_OK && split) {
        rc = natsl_gdn_split_prep(a.q, a.k, a.g, a.beta, a.beta_dtype, ws + l.p, gcs, reinterpret_cast<float*>(ws + l.kr),
                                  reinterpret_cast<float*>(ws + l.qr), reinterpret_cast<float*>(ws + l.egl), a.B, a.T, a.H, a.K,
                                  a.use_l2norm, lin);
    } else if (rc == NATSL_OK && gdn) {
        auto prep = (a.K == 128 && a.V == 128 && !(a.options & NATSL_HYBRID_PREP_MMA)) ? natsl_gdn_chunk_prep_tc : natsl_gdn_chunk_prep_ex;
        rc = prep(a.q, a.k, a.v, a.g, a.beta, a.beta_dtype, ws + l.w, ws + l.u, gcs, reinterpret_cast<float*>(ws + l.kr),
                  reinterpret_cast<float*>(ws + l.qr), ws + l.p, a.B, a.T, a.H, a.K, a.V, a.use_l2norm, lin);
    } else if (rc == NATSL_OK && !a.gcs) {
        rc = natsl_chunk_local_cumsum(a.g, gcs, a.B, a.T, a.H, lin);
    }
    if (rc == NATSL_OK)
        rc = launch_tables(a.types, a.types_dtype, types_raw, a.B, TN, a.HN, a.T, a.nbs, a.types_i, a.indices, a.n_blocks,
                           a.n_chunks_lin, a.starting_h_idx, a.attn_n_iters, att);
    if (rc == NATSL_OK) rc = stream_after(lin, att, ev[1]);
    const int flags = (a.decay ? NATSL_FLAG_DECAY_SKIPPED : 0);
    const void* last = types_raw ? (const void*)(reinterpret_cast<bf16*>(types_raw) + (long)(TN - 1) * a.HN * 2) : a.last_types;
    const int last_dtype = types_raw ? NATSL_DT_BF16 : a.last_dtype;
    const bool tc_walk = gdn && a.K == 128 && a.V == 128 && a.nbs == 64 && a.T <= 65536 && !(a.options & NATSL_HYBRID_WALK_MMA);
    if (rc == NATSL_OK && split) {
        rc = natsl_gdn_split_walk(a.q, a.k, a.v, ws + l.p, gcs, reinterpret_cast<float*>(ws + l.kr), reinterpret_cast<float*>(ws + l.qr),
                                  reinterpret_cast<float*>(ws + l.egl), a.types_i, a.indices, a.n_blocks, a.h0, a.o_lin, a.ht, a.hstart, last, last_dtype, a.last_stride, a.B,
                                  a.T, a.H, a.HN, a.K, a.V, a.nbs, a.scale_lin, flags, lin);
    } else if (rc == NATSL_OK && tc_walk && (a.options & NATSL_HYBRID_WALK_VSPLIT) && a.T <= 8192 && !a.hstart) {
        rc = natsl_gdn_walk_fused_vsplit(a.q, a.k, ws + l.w, ws + l.u, ws + l.p, gcs, reinterpret_cast<float*>(ws + l.kr),
                                         reinterpret_cast<float*>(ws + l.qr), a.types_i, a.indices, a.n_blocks, a.h0, a.o_lin, a.ht, a.B,
                                         a.T, a.H, a.HN, a.K, a.V, a.nbs, a.scale_lin, flags, lin);
    } else if (rc == NATSL_OK && gdn) {
        auto walk = tc_walk ? natsl_gdn_walk_fused_ex : natsl_gdn_walk;
        rc = walk(a.q, a.k, ws + l.w, ws + l.u, ws + l.p, gcs, reinterpret_cast<float*>(ws + l.kr), reinterpret_cast<float*>(ws + l.qr),
                  a.types_i, a.indices, a.n_blocks, a.h0, a.o_lin, a.ht, a.hstart, last, last_dtype, a.last_stride, a.B, a.T, a.H, a.HN,
                  a.K, a.V, a.nbs, a.scale_lin, flags, lin);
    } else if (rc == NATSL_OK) {
        rc = natsl_mamba_walk_fused_ex(a.q, a.k, a.v, a.gcs ? a.gcs : gcs, a.types_i, a.indices, a.n_blocks, a.h0, a.o_lin, a.ht,
                                       a.hstart, last, last_dtype, a.last_stride, a.B, a.T, a.H, a.HN, a.K, a.V, a.nbs, a.scale_lin,
                                       flags, lin);
    }
    if (rc == NATSL_OK) rc = before_attn(att);
    if (rc == NATSL_OK)
        rc = natsl_attn_fwd_ex(a.q_attn, a.k_attn, a.v_attn, a.types_i, a.indices, a.attn_n_iters, a.o_attn, a.lse, a.B, a.T, a.T, 0,
                               a.HQ, a.HKV, a.HN, a.DK, a.DV, a.nbs, a.scale_attn, a.own_attn ? NATSL_FLAG_ATTN_OWN_CHUNK : 0, att);
    const int join = stream_after(st, side, ev[2]);          // also after an error: the side stream may hold work of this call
    return rc != NATSL_OK ? rc : join;
}

}  // namespace
}  // namespace natsl

extern "C" int64_t natsl_hybrid_workspace_bytes(const natsl_hybrid_args* args) {
    using namespace natsl;
    NATSL_REQUIRE(args, NATSL_ERR_NULL, "natsl_hybrid_workspace_bytes: null argument block");
    return hybrid_layout(*args).total;
}

extern "C" int natsl_hybrid_forward(const natsl_hybrid_args* args, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(args, NATSL_ERR_NULL, "natsl_hybrid_forward: null argument block");
    NATSL_REQUIRE(args->types_dtype >= 0 && args->types_dtype <= NATSL_DT_I32, NATSL_ERR_UNSUPPORTED, "natsl_hybrid_forward: bad types dtype");
    count_launches_from_here();
    int rc = check_hybrid(*args);
    if (rc == NATSL_OK) rc = check_device(args->q, "natsl_hybrid_forward");
    if (rc != NATSL_OK) return rc;
    return hybrid_forward(*args, nullptr, reinterpret_cast<cudaStream_t>(stream), [](cudaStream_t) { return (int)NATSL_OK; });
}

namespace natsl {
namespace {

struct LayerLayout {
    long q, k, v, qa, qc, g, beta, dt, hybrid, total;
};
// Intermediates of a layer's forward.  Tensors the caller keeps (k_attn, v_attn) are outputs and not listed here.
LayerLayout layer_layout(const natsl_layer_args& a, const natsl_hybrid_args& h) {
    LayerLayout l = {};
    const long n = (long)a.B * a.T, HK = (long)a.H * a.K, HV = (long)a.H * a.V;
    const bool mamba = a.rule == NATSL_RULE_MAMBA;
    long at = 0;
    auto take = [&](long& slot, long bytes) { slot = at; at = up256(at + bytes); };
    take(l.q, 2 * n * HK);
    take(l.k, 2 * n * HK);
    take(l.v, mamba ? 2 * n * HV : 0);
    take(l.qa, a.qn_w || (mamba && a.attn_conv) ? 2 * n * HK : 0);
    take(l.qc, mamba ? 2 * n * HK : 0);
    take(l.g, 4 * n * a.H);
    take(l.beta, mamba ? 0 : 2 * n * a.H);
    take(l.dt, mamba ? 8 * n * a.H : 0);
    take(l.hybrid, hybrid_layout(h).total);
    l.total = at;
    return l;
}
void hybrid_dims(const natsl_layer_args& a, natsl_hybrid_args& h) {
    h.B = a.B; h.T = a.T; h.H = a.H; h.HN = a.HN; h.K = a.K; h.V = a.V; h.HQ = h.HKV = a.HQ;
    h.DK = a.H * a.K / a.HQ; h.DV = a.H * a.V / a.HQ;
    h.nbs = a.nbs; h.rule = a.rule; h.options = a.options;
}

}  // namespace
}  // namespace natsl

extern "C" int64_t natsl_layer_workspace_bytes(const natsl_layer_args* args) {
    using namespace natsl;
    NATSL_REQUIRE(args, NATSL_ERR_NULL, "natsl_layer_workspace_bytes: null argument block");
    natsl_hybrid_args h = {};
    hybrid_dims(*args, h);
    return layer_layout(*args, h).total;
}

extern "C" int natsl_layer_forward(const natsl_layer_args* args, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(args, NATSL_ERR_NULL, "natsl_layer_forward: null argument block");
    const natsl_layer_args& a = *args;
    const bool mamba = a.rule == NATSL_RULE_MAMBA;
    NATSL_REQUIRE(a.x && a.logits && a.q_raw && a.k_raw && a.v_raw && a.w_a && (mamba || a.w_b) && a.cw_q && a.cw_k && a.cw_v && a.A_log &&
                      a.dt_bias && a.o_lin && a.o_attn && a.k_attn && a.v_attn && a.types_raw && a.tables && a.workspace && a.lse,
                  NATSL_ERR_NULL, "natsl_layer_forward: null pointer");
    NATSL_REQUIRE(a.B > 0 && a.T >= 4 && a.hidden % 32 == 0 && a.H > 0 && a.HQ > 0 && (a.H * a.K) % a.HQ == 0 && (a.H * a.V) % a.HQ == 0 &&
                      (a.H * a.K) % 32 == 0 && a.B <= 65535,
                  NATSL_ERR_BAD_SHAPE, "natsl_layer_forward: bad shape");
    natsl_hybrid_args h = {};
    hybrid_dims(a, h);
    NATSL_REQUIRE(!a.qn_w || h.DK == 64 || h.DK == 128, NATSL_ERR_UNSUPPORTED, "natsl_layer_forward: norm width %d (64 or 128)", h.DK);
    NATSL_REQUIRE(!mamba || a.K == 128, NATSL_ERR_UNSUPPORTED, "natsl_layer_forward: Mamba2 is built for K = 128");
    const LayerLayout l = layer_layout(a, h);
    NATSL_REQUIRE(a.workspace_bytes >= l.total, NATSL_ERR_TOO_LARGE, "natsl_layer_forward: workspace of %ld bytes, %ld needed",
                  (long)a.workspace_bytes, l.total);
    NATSL_REQUIRE(aligned_to(16, a.x, a.q_raw, a.k_raw, a.v_raw, a.w_a, a.w_b, a.w_mix, a.o_lin, a.o_attn, a.k_attn, a.v_attn, a.v_lin,
                             a.workspace) &&
                      aligned_to(8, a.cw_q, a.cw_k, a.cw_v, a.tail_q, a.tail_k, a.tail_v) && aligned_to(4, a.logits, a.mix),
                  NATSL_ERR_UNSUPPORTED, "natsl_layer_forward: a tensor does not start on 16 bytes (convolution weights and tails: 8)");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    unsigned char* ws = reinterpret_cast<unsigned char*>(a.workspace);
    auto cb = [](const void* p) { return reinterpret_cast<const bf16*>(p); };
    auto mb = [](void* p) { return reinterpret_cast<bf16*>(p); };
    const int HK = a.H * a.K, HV = a.H * a.V, TN = (a.T + a.nbs - 1) / a.nbs;

    NarrowArgs n = {};
    n.x = cb(a.x); n.w0 = cb(a.w_a); n.w1 = mamba ? nullptr : cb(a.w_b);
    n.n0 = a.H; n.n1 = mamba ? 0 : a.H; n.T = a.T; n.Kdim = a.hidden; n.mode = 0;
    n.A_log = a.A_log; n.dt_bias = a.dt_bias; n.alog_f32 = a.alog_f32; n.dt_f32 = a.dt_f32; n.neg_eigval = a.neg_eigval;
    n.g = reinterpret_cast<float*>(ws + l.g);
    n.dt = mamba ? reinterpret_cast<float*>(ws + l.dt) : nullptr;
    n.gcs = mamba ? n.dt + (long)a.B * a.T * a.H : nullptr;
    n.out = mb(ws + l.beta);
    count_launches_from_here();
    int rc = check_device(a.x, "natsl_layer_forward");
    if (rc == NATSL_OK) rc = launch_narrow(n, a.B, st);
    if (rc != NATSL_OK) return rc;

    // where each tensor of the two branches lives: the delta rule's k and v convolutions double as the softmax branch's
    // tensors where nothing lies between them
    const bool conv_attn = a.attn_conv, normed = a.qn_w != nullptr;
    ConvArgs c = {};
    c.dt = n.dt; c.T = a.T; c.H = a.H; c.silu = a.silu; c.l2_eps = a.l2_eps; c.norm_eps = a.norm_eps;
    bf16 *q = mb(ws + l.q), *k = mb(ws + l.k), *v = mamba ? mb(ws + l.v) : mb(a.v_attn);
    const bf16 *qa = nullptr, *q_mix = q;
    c.seg[0] = {cb(a.q_raw), cb(a.cw_q), cb(a.cb_q), q, nullptr, nullptr, mb(a.tail_q), a.qn_w, a.qn_f32, HK, mamba ? 1 : 0, 0, a.K / 4, h.DK / 4, a.K, 0};
    c.seg[1] = {cb(a.k_raw), cb(a.cw_k), cb(a.cb_k), k, nullptr, nullptr, mb(a.tail_k), a.kn_w, a.kn_f32, HK, mamba ? 1 : 0, 0, a.K / 4, h.DK / 4, a.K, 0};
    c.seg[2] = {cb(a.v_raw), cb(a.cw_v), cb(a.cb_v), v, nullptr, nullptr, mb(a.tail_v), nullptr, 0, HV, mamba ? 2 : 0, 0, 1, 1, a.V, 0};
    if (mamba) {
        c.seg[0].conv = mb(ws + l.qc);                       // the mixing weights read the query in front of its l2 norm
        q_mix = c.seg[0].conv;
    }
    if (normed) {
        c.seg[0].attn = mb(ws + l.qa);
        c.seg[1].attn = mb(a.k_attn);
        c.seg[0].attn_mode = c.seg[1].attn_mode = conv_attn ? 1 : 2;
        qa = c.seg[0].attn;
    } else if (conv_attn) {
        if (mamba) {
            c.seg[1].conv = mb(a.k_attn);
            qa = c.seg[0].conv;
        } else {
            k = mb(a.k_attn);
            c.seg[1].lin = k;
            qa = q;
        }
    } else {
        qa = cb(a.q_raw);                                    // k_attn, v_attn are the raw projections (the caller passes them)
    }
    if (conv_attn && mamba) c.seg[2].conv = mb(a.v_attn);
    if (!conv_attn && !mamba) {
        v = mb(a.v_lin);
        NATSL_REQUIRE(v, NATSL_ERR_NULL, "natsl_layer_forward: v_lin is needed beside a raw v_attn");
        c.seg[2].lin = v;
    }
    for (const ConvSeg& e : c.seg)                           // what conv_norm_kernel is built for
        NATSL_REQUIRE(e.lin && e.lin_mode >= 0 && e.lin_mode <= 2 && e.attn_mode >= 0 && e.attn_mode <= (e.lin_mode == 2 ? 0 : 2),
                      NATSL_ERR_UNSUPPORTED, "natsl_layer_forward: no convolution kernel for modes %d, %d", e.attn_mode, e.lin_mode);
    const int kb = (HK + CONV_CH - 1) / CONV_CH, vb = (HV + CONV_CH - 1) / CONV_CH;
    c.seg[1].blk0 = kb;
    c.seg[2].blk0 = 2 * kb;
    // Tokens per warp: long runs amortise the three halo rows, short ones fill the resident warps (CONV_CTAS x 4 per SM).  A run is
    // halved below 4/3 of a full wave: 26 warps per SM are one wave and a few more, and take longer than 52 with half the tokens
    // (layers of 4 x 1262 tokens, 2048 channels each: 363 us in whole with 64-token runs, 356 us with 32; of 4 x 1144: 334, 324 us).
    const long rows = (long)a.B * a.T * (2 * kb + vb), full = 148l * CONV_CTAS * 4 * 4 / 3;
    c.TT = rows / 64 >= full ? 64 : rows / 32 >= full ? 32 : rows / 16 >= full ? 16 : 8;
    conv_norm_kernel<<<dim3(2 * kb + vb, (a.T + 4 * c.TT - 1) / (4 * c.TT), a.B), 128, 0, st>>>(c);
    rc = check_launch("natsl_layer_forward (convolutions)");
    if (rc != NATSL_OK) return rc;
    if (a.g_block) {
        const int rest = a.T % a.nbs;
        const int width = a.hidden > a.H ? a.hidden : a.H;
        block_rest_kernel<<<dim3((width + 255) / 256, a.B), 256, 0, st>>>(n.g, cb(a.x), reinterpret_cast<float*>(a.g_block),
                                                                         reinterpret_cast<float*>(a.pool_sum), a.T, a.H, a.hidden, rest);
        rc = check_launch("natsl_layer_forward (state)");
        if (rc != NATSL_OK) return rc;
    }

    h.types_dtype = NATSL_DT_BF16;
    h.beta_dtype = NATSL_DT_BF16;
    h.own_attn = a.own_chunk; h.decay = a.decay; h.use_l2norm = mamba ? 0 : 1;
    h.scale_attn = a.scale_attn; h.scale_lin = a.scale_lin;
    h.q_attn = qa; h.k_attn = a.k_attn; h.v_attn = a.v_attn;
    h.q = q; h.k = k; h.v = v; h.g = n.g; h.gcs = n.gcs; h.beta = n.out; h.types = a.logits;
    h.o_attn = a.o_attn; h.lse = reinterpret_cast<float*>(a.lse); h.o_lin = a.o_lin;
    h.ht = reinterpret_cast<float*>(a.ht); h.hstart = reinterpret_cast<float*>(a.hstart);
    h.last_stride = TN * a.HN * 2;
    int32_t* tb = reinterpret_cast<int32_t*>(a.tables);
    const long nt = (long)a.B * TN * a.HN * 2;
    h.types_i = tb; h.indices = tb + nt; h.n_blocks = tb + 2 * nt; h.n_chunks_lin = h.n_blocks + 2l * a.B * a.HN;
    h.attn_n_iters = h.n_chunks_lin + (long)a.B * a.HN;
    h.workspace = ws + l.hybrid;
    h.workspace_bytes = a.workspace_bytes - l.hybrid;
    rc = check_hybrid(h);
    if (rc != NATSL_OK) return rc;
    h.types_dtype = TBL_LOGITS;
    return hybrid_forward(h, a.types_raw, st, [&](cudaStream_t s) {
        if (!a.w_mix) return (int)NATSL_OK;
        NarrowArgs m = {};
        m.x = q_mix; m.w0 = cb(a.w_mix); m.n0 = 2 * a.HQ; m.T = a.T; m.Kdim = HK; m.mode = 1; m.out = mb(a.mix);
        return launch_narrow(m, a.B, s);
    });
}
