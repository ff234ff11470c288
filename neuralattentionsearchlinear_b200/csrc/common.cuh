// Shared device helpers for the NAtSL sm_100a kernels: cp.async staging, swizzled
// shared-memory tiles, ldmatrix / mma.sync fragments, small numeric helpers, and
// the host-side error plumbing of the C-ABI.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define NATSL_CHUNK 64

namespace natsl {

// ------------------------------------------------------------------ host-side errors
void set_error(const char* fmt, ...);
int check_launch(const char* what);
void count_launches_from_here();                             // what natsl_call_kernels counts
int check_device(const void* p, const char* what);      // p must be memory of the current device

#define NATSL_REQUIRE(cond, code, ...)          \
    do {                                        \
        if (!(cond)) {                          \
            ::natsl::set_error(__VA_ARGS__);    \
            return (code);                      \
        }                                       \
    } while (0)

// Whether every pointer starts on a multiple of `n` bytes (NULL does): kernels with wide accesses take it on trust.
template <typename... P>
inline bool aligned_to(uintptr_t n, const P*... p) {
    return ((... | reinterpret_cast<uintptr_t>(p)) & (n - 1)) == 0;
}

enum : int {
    NATSL_OK = 0,
    NATSL_ERR_BAD_SHAPE = -1,
    NATSL_ERR_UNSUPPORTED = -2,
    NATSL_ERR_NULL = -3,
    NATSL_ERR_CUDA = -4,
    NATSL_ERR_TOO_LARGE = -5,
};

// ------------------------------------------------------------------ device helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte async copy global -> shared; bytes beyond src_bytes (0 or 16) are zero-filled.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Byte offset of 16-byte chunk `chunk` of row `row` in a swizzled tile whose rows are
// ROW_BYTES long (64 or a multiple of 128).  The XOR keeps the eight rows touched by one
// ldmatrix 8x8 load in eight different 16-byte bank groups.
template <int ROW_BYTES>
__device__ __forceinline__ uint32_t swz(int row, int chunk) {
    static_assert(ROW_BYTES == 64 || ROW_BYTES % 128 == 0, "row size");
    if (ROW_BYTES == 64) return row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
    return row * ROW_BYTES + ((chunk ^ (row & 7)) << 4);
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) {
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(v);
}

// Two floats in one 64-bit register pair: one instruction for both on sm_100.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t open2(uint32_t u) {       // a pair of bf16
    const float2 f = unpack_bf16(u);
    return pack2(f.x, f.y);
}
__device__ __forceinline__ uint32_t close2(uint64_t v) {
    float lo, hi;
    unpack2(v, lo, hi);
    return pack_bf16(lo, hi);
}

// Logistic function of a pair.  The reciprocal is an approximate one (off by e <= 2^-23) with a step of Newton's iteration, which
// leaves e^2 and two roundings, less than one unit of 2^-23, without a division's call and branches; with exp(-|x|) its argument lies
// in [1, 2].  In all 2 + 1.173 |x| units from __expf, one from the reciprocal, half a one each from 1 + t and, for x < 0, from the
// product with t.
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_newton(float y) {        // 1 / y, y in [1, 2]
    const float r = rcp_ftz(y);
    return fmaf(r, fmaf(-y, r, 1.f), r);
}
__device__ __forceinline__ uint64_t sigmoid2(uint64_t v) {
    // (constants as immediates of scalar instructions: a pair of them would take two registers, or two moves at every use)
    float a, b;
    unpack2(v, a, b);
    const float ta = __expf(-fabsf(a)), tb = __expf(-fabsf(b)), ya = 1.f + ta, yb = 1.f + tb;          // y in [1, 2]
    const float ra = rcp_ftz(ya), rb0 = rcp_ftz(yb);
    const uint64_t r0 = pack2(ra, rb0), r = fma2(r0, pack2(fmaf(-ya, ra, 1.f), fmaf(-yb, rb0, 1.f)), r0);
    return mul2(pack2(a < 0.f ? ta : 1.f, b < 0.f ? tb : 1.f), r);
}
__device__ __forceinline__ uint64_t silu2(uint64_t v) { return mul2(v, sigmoid2(v)); }
__device__ __forceinline__ float hsum2(uint64_t v) {
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}
// Eight bf16 as four pairs of floats, and back.
__device__ __forceinline__ void open8(const uint4& v, uint64_t (&f)[4]) {
    f[0] = open2(v.x);
    f[1] = open2(v.y);
    f[2] = open2(v.z);
    f[3] = open2(v.w);
}
__device__ __forceinline__ uint4 close8(const uint64_t (&f)[4]) { return make_uint4(close2(f[0]), close2(f[1]), close2(f[2]), close2(f[3])); }
__device__ __forceinline__ void open8(const __nv_bfloat16* p, uint64_t (&f)[4]) { open8(*reinterpret_cast<const uint4*>(p), f); }
// Sixteen bytes at any bf16 address; `wide` says that it is a multiple of 16 (uniform over the grid).
__device__ __forceinline__ uint4 ld16(const __nv_bfloat16* p, bool wide) {
    if (wide) return *reinterpret_cast<const uint4*>(p);
    const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = (uint32_t)h[2 * i] | (uint32_t)h[2 * i + 1] << 16;
    return make_uint4(u[0], u[1], u[2], u[3]);
}
__device__ __forceinline__ void st16(__nv_bfloat16* p, const uint4& v, bool wide) {
    if (wide) {
        *reinterpret_cast<uint4*>(p) = v;
        return;
    }
    unsigned short* h = reinterpret_cast<unsigned short*>(p);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[2 * i] = (unsigned short)u[i];
        h[2 * i + 1] = (unsigned short)(u[i] >> 16);
    }
}
// Eight neighbouring weights in fp32 or bf16 (ones where there are none).
__device__ __forceinline__ void weights8(const void* w, bool f32, int at, uint64_t (&f)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[i] = pack2(1.f, 1.f);
        if (w) {
            if (f32) f[i] = pack2(reinterpret_cast<const float*>(w)[at + 2 * i], reinterpret_cast<const float*>(w)[at + 2 * i + 1]);
            else f[i] = pack2(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[at + 2 * i]),
                              __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[at + 2 * i + 1]));
        }
    }
}

// ---- fragment loaders over swizzled bf16 tiles ------------------------------------
// A fragment (16 rows x 16 k) of a row-major [rows][k] tile.
template <int ROW_BYTES>
__device__ __forceinline__ void load_a(uint32_t tile, int row0, int k0, int lane, uint32_t (&a)[4]) {
    int r = row0 + (lane & 15);
    int c = (k0 >> 3) + (lane >> 4);
    ldsm_x4(tile + swz<ROW_BYTES>(r, c), a[0], a[1], a[2], a[3]);
}
// A fragment (16 m x 16 k) of A = M^T where M is stored row-major [k][m].
template <int ROW_BYTES>
__device__ __forceinline__ void load_a_t(uint32_t tile, int m0, int k0, int lane, uint32_t (&a)[4]) {
    int i = lane >> 3;
    int r = k0 + (lane & 7) + ((i >> 1) << 3);
    int c = (m0 >> 3) + (i & 1);
    ldsm_x4_t(tile + swz<ROW_BYTES>(r, c), a[0], a[1], a[2], a[3]);
}
// B fragments for two adjacent n-tiles (16 n x 16 k) when B^T is stored row-major [n][k]
// (e.g. keys [key][d] for Q K^T): b[0],b[1] -> n-tile n0, b[2],b[3] -> n-tile n0+8.
template <int ROW_BYTES>
__device__ __forceinline__ void load_b_nk(uint32_t tile, int n0, int k0, int lane, uint32_t (&b)[4]) {
    int r = n0 + (lane & 7) + ((lane >> 4) << 3);
    int c = (k0 >> 3) + ((lane >> 3) & 1);
    ldsm_x4(tile + swz<ROW_BYTES>(r, c), b[0], b[1], b[2], b[3]);
}
// B fragments for two adjacent n-tiles when B is stored row-major [k][n]
// (e.g. values [key][dv] for P V): b[0],b[1] -> n-tile n0, b[2],b[3] -> n-tile n0+8.
template <int ROW_BYTES>
__device__ __forceinline__ void load_b_kn(uint32_t tile, int k0, int n0, int lane, uint32_t (&b)[4]) {
    int r = k0 + (lane & 7) + (((lane >> 3) & 1) << 3);
    int c = (n0 >> 3) + (lane >> 4);
    ldsm_x4_t(tile + swz<ROW_BYTES>(r, c), b[0], b[1], b[2], b[3]);
}

// Copy a [ROWS][COLS] bf16 tile from global (row stride `gstride` elements) into a swizzled
// shared tile with cp.async; rows >= valid_rows are zero-filled.  NT = threads taking part.  A thread's 16-byte chunks lie
// NT / CPR rows apart: where that is a multiple of eight the swizzle is the same for all of them, and a chunk costs two additions.
template <int ROWS, int COLS, int NT>
__device__ __forceinline__ void load_tile_async(uint32_t tile, const __nv_bfloat16* g, long gstride, int valid_rows,
                                                int tid) {
    constexpr int CPR = COLS / 8;  // 16-byte chunks per row
    constexpr int TOTAL = ROWS * CPR, RS = NT / CPR;
    if constexpr (NT % CPR == 0 && RS % 8 == 0 && ROWS % RS == 0) {
        const int r0 = tid / CPR, c = tid % CPR;
        const uint32_t dst = tile + swz<COLS * 2>(r0, c);
        const __nv_bfloat16* src = g + (long)r0 * gstride + c * 8;
#pragma unroll
        for (int j = 0; j < ROWS / RS; ++j) {
            const bool ok = r0 + j * RS < valid_rows;
            cp_async16(dst + j * RS * COLS * 2, ok ? src : g, ok ? 16 : 0);
            src += RS * gstride;
        }
    } else {
#pragma unroll
        for (int i = tid; i < TOTAL; i += NT) {
            int r = i / CPR, c = i % CPR;
            bool ok = r < valid_rows;
            const __nv_bfloat16* src = g + (ok ? (long)r * gstride + c * 8 : 0);
            cp_async16(tile + swz<COLS * 2>(r, c), src, ok ? 16 : 0);
        }
    }
}

// Add four or eight bf16 values to those in global memory, each sum rounded to nearest.  With one writer per address the result is that
// of a load, an add and a store; the addition is done at the L2 cache and nothing waits for it.
__device__ __forceinline__ void red_bf16x4(__nv_bfloat16* p, uint2 v) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v2.bf16x2 [%0], {%1, %2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void red_bf16x8(__nv_bfloat16* p, uint4 v) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// Add a swizzled [ROWS][COLS] bf16 shared tile to global memory, 16 bytes per lane.
template <int ROWS, int COLS, int NT>
__device__ __forceinline__ void add_tile(const unsigned char* tile, __nv_bfloat16* g, long gstride, int valid_rows, int tid) {
    constexpr int CPR = COLS / 8;
#pragma unroll
    for (int i = tid; i < ROWS * CPR; i += NT) {
        const int r = i / CPR, c = i % CPR;
        if (r < valid_rows) red_bf16x8(g + (long)r * gstride + c * 8, *reinterpret_cast<const uint4*>(tile + swz<COLS * 2>(r, c)));
    }
}

// Store a swizzled [ROWS][COLS] bf16 shared tile to global with 16-byte coalesced stores.
template <int ROWS, int COLS, int NT>
__device__ __forceinline__ void store_tile(const unsigned char* tile, __nv_bfloat16* g, long gstride, int valid_rows,
                                           int tid) {
    constexpr int CPR = COLS / 8;
    constexpr int TOTAL = ROWS * CPR, RS = NT / CPR;
    if constexpr (NT % CPR == 0 && RS % 8 == 0 && ROWS % RS == 0) {
        const int r0 = tid / CPR, c = tid % CPR;
        const unsigned char* src = tile + swz<COLS * 2>(r0, c);
        __nv_bfloat16* dst = g + (long)r0 * gstride + c * 8;
#pragma unroll
        for (int j = 0; j < ROWS / RS; ++j) {
            if (r0 + j * RS < valid_rows)
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src + j * RS * COLS * 2);
            dst += RS * gstride;
        }
    } else {
#pragma unroll
        for (int i = tid; i < TOTAL; i += NT) {
            int r = i / CPR, c = i % CPR;
            if (r < valid_rows) {
                uint4 v = *reinterpret_cast<const uint4*>(tile + swz<COLS * 2>(r, c));
                *reinterpret_cast<uint4*>(g + (long)r * gstride + c * 8) = v;
            }
        }
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace natsl
