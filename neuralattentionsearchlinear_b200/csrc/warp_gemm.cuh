// Warp-level tile products on mma.sync for the backward kernels: one warp accumulates a 16-row strip
//     acc[16 x 8*NT8] += A[16 x k] * B[k x 8*NT8]
// from bf16 operand tiles in XOR-swizzled shared memory (swz<ROW_BYTES>() of common.cuh).  The four storage
// combinations cover every product of the backward pass without a transposed copy of any tile:
//     A_ROW   : A stored row-major [m][k]            A_TRANS : A = M^T with M stored row-major [k][m]
//     B_NK    : B^T stored row-major [n][k]          B_KN    : B stored row-major [k][n]
// Accumulator element acc[nt][e] of lane (gq = lane >> 2, qd = lane & 3) is
//     row = m0 + gq + 8 * (e >> 1),   column = n0 + 8 * nt + 2 * qd + (e & 1).
#pragma once
#include "common.cuh"

namespace natsl {

enum : int { A_ROW = 0, A_TRANS = 1 };
enum : int { B_NK = 0, B_KN = 1 };

template <int NT8>
__device__ __forceinline__ void zero_acc(float (&acc)[NT8][4]) {
#pragma unroll
    for (int i = 0; i < NT8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
}

// Addresses of a lane's ldmatrix rows.  Tiles start on a multiple of their row length (256 bytes at most), m0 is a multiple of 16
// and n0 of 8 * NT8, so a step along a row is an exclusive or with a constant and a step over rows an addition that goes into the
// instruction: one integer operation per fragment at most.  (Against addresses formed anew for every fragment, with the tile copies
// treated the same way; B = 8, T = 4096, 16 heads of 128 / 128: reverse walk 291 -> 260 us, state part 539 -> 507, 64 x 64 part
// 736 -> 709.)
template <int RB, int MODE>
__device__ __forceinline__ uint32_t a_addr(uint32_t tile, int m0, int lane) {
    if (MODE == A_ROW) return tile + swz<RB>(m0 + (lane & 15), lane >> 4);
    const int i = lane >> 3;
    return tile + swz<RB>((lane & 7) + ((i >> 1) << 3), (m0 >> 3) + (i & 1));
}
template <int RB, int MODE>
__device__ __forceinline__ void ld_a(uint32_t at, int k0, uint32_t (&a)[4]) {           // k0: a constant after unrolling
    if (MODE == A_ROW) ldsm_x4(at ^ (k0 * 2), a[0], a[1], a[2], a[3]);
    else ldsm_x4_t(at + k0 * RB, a[0], a[1], a[2], a[3]);
}
template <int RB, int MODE>
__device__ __forceinline__ uint32_t b_addr(uint32_t tile, int n0, int lane) {
    if (MODE == B_NK) return tile + swz<RB>(n0 + (lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1);
    return tile + swz<RB>((lane & 7) + (((lane >> 3) & 1) << 3), (n0 >> 3) + (lane >> 4));
}
template <int RB, int MODE>
__device__ __forceinline__ void ld_b(uint32_t at, int p, int k0, uint32_t (&b)[4]) {    // n-tiles 2 p and 2 p + 1
    if (MODE == B_NK) ldsm_x4((at ^ (k0 * 2)) + p * 16 * RB, b[0], b[1], b[2], b[3]);
    else ldsm_x4_t((at ^ (p * 32)) + k0 * RB, b[0], b[1], b[2], b[3]);
}

// acc += A[m0.., 0..KLEN) * B[0..KLEN), n0..)
template <int A_RB, int A_MODE, int B_RB, int B_MODE, int KLEN, int NT8>
__device__ __forceinline__ void warp_gemm(float (&acc)[NT8][4], uint32_t atile, int m0, uint32_t btile, int n0, int lane) {
    static_assert(NT8 % 2 == 0 && (NT8 & (NT8 - 1)) == 0 && KLEN % 16 == 0, "n-tiles come in pairs");
    const uint32_t at = a_addr<A_RB, A_MODE>(atile, m0, lane), bt = b_addr<B_RB, B_MODE>(btile, n0, lane);
#pragma unroll
    for (int k0 = 0; k0 < KLEN; k0 += 16) {
        uint32_t a[4];
        ld_a<A_RB, A_MODE>(at, k0, a);
#pragma unroll
        for (int p = 0; p < NT8 / 2; ++p) {
            uint32_t b[4];
            ld_b<B_RB, B_MODE>(bt, p, k0, b);
            mma_bf16(acc[2 * p], a, b[0], b[1]);
            mma_bf16(acc[2 * p + 1], a, b[2], b[3]);
        }
    }
}

// Write a strip (rows m0.., columns n0..) into a swizzled bf16 tile with ROW_BYTES-long rows.
template <int RB, int NT8>
__device__ __forceinline__ void store_acc_bf16(unsigned char* tile, const float (&acc)[NT8][4], int m0, int n0, int lane) {
    const int gq = lane >> 2, qd = lane & 3;
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt) {
        const int ch = (n0 >> 3) + nt;
        *reinterpret_cast<uint32_t*>(tile + swz<RB>(m0 + gq, ch) + qd * 4) = pack_bf16(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<uint32_t*>(tile + swz<RB>(m0 + gq + 8, ch) + qd * 4) = pack_bf16(acc[nt][2], acc[nt][3]);
    }
}

// Write a strip straight to global memory (row r at g + r * gstride, columns n0..), rows from `valid` on left out: neighbouring lanes
// swap halves of neighbouring n-tiles, so that a store covers whole 32-byte sectors and no staging tile or barrier is needed.
// onto: the strip is added to what is there.
template <int NT8>
__device__ __forceinline__ void store_acc_global(__nv_bfloat16* g, long gstride, const float (&acc)[NT8][4], int m0, int n0, int valid, int lane,
                                                 bool onto = false) {
    const int gq = lane >> 2, qd = lane & 3;
    const bool odd = qd & 1;
    __nv_bfloat16* pa = g + (long)(m0 + gq) * gstride + n0 + (odd ? 8 : 0) + (qd >> 1) * 4;
    __nv_bfloat16* pb = pa + 8 * gstride;
    const bool oka = m0 + gq < valid, okb = m0 + gq + 8 < valid;
#pragma unroll
    for (int p = 0; p < NT8 / 2; ++p) {
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const uint32_t x = pack_bf16(acc[2 * p][e], acc[2 * p][e + 1]), y = pack_bf16(acc[2 * p + 1][e], acc[2 * p + 1][e + 1]);
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
            const uint2 v = odd ? make_uint2(got, y) : make_uint2(x, got);
            __nv_bfloat16* to = (e ? pb : pa) + 16 * p;
            if (e ? okb : oka) {
                if (onto) red_bf16x4(to, v);
                else *reinterpret_cast<uint2*>(to) = v;
            }
        }
    }
}

// The two bf16 values at (row, column n0 + 8*nt + 2*qd, +1) of a swizzled tile (the positions acc[nt][0..1] or
// acc[nt][2..3] of the lane address).
template <int RB>
__device__ __forceinline__ float2 load_pair_bf16(const unsigned char* tile, int row, int col) {
    return unpack_bf16(*reinterpret_cast<const uint32_t*>(tile + swz<RB>(row, col >> 3) + (col & 7) * 2));
}

// Sum over the four lanes that share an accumulator row.
__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}
// Sum over the eight lanes (gq = 0..7) that share an accumulator column pair.
__device__ __forceinline__ float colgroup_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

}  // namespace natsl
