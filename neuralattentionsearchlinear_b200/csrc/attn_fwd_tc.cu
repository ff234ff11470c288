// Chunk-masked softmax attention forward on the 5th-generation tensor cores.
//
// One work item = 256 queries of one softmax head: two tiles A and B of 128 rows that share every key and value load.
// One CTA per SM works through items until none is left: it takes over blocks of the grid that have not started yet
// (cluster launch control), so the pipeline runs across items, an SM is never idle between two of them, and a kernel
// of higher priority still gets its SMs (the take-over is refused then and the CTA ends).  Roles (384 threads):
//   warps 0-3  softmax of tile A, one thread per query row (tcgen05.ld.32x32b: 128 scores of the row in registers, no
//              shuffles): mask, online softmax in base 2 with a lazily updated maximum (O in TMEM is only rescaled when
//              a row's maximum grows by more than 2^8), P (bf16 pairs) into TMEM; at the end of an item
//              O / l -> bf16 -> global memory, whole 32-byte sectors per thread;
//   warps 4-7  the same for tile B;
//   warp 8     TMA producer: the two query tiles of an item, then pairs of 64-key tiles into a K and a V ring
//              (cp.async.bulk.tensor, 128-byte swizzle, zero fill past the sequence end);
//   warps 9, 11  MMA issuers of tile A and tile B: S = Q K^T (128 x 128), O += P V with P read straight from TMEM;
//   warp 10    scheduler: takes the next item, reads its tables, works out its steps.
// TMEM (512 columns): S of A and of B (128 columns each), O of A and of B, and, where DV = 64 leaves room, P of A and of B.
//
// What bounds it: at head dims 128 the tensor core and the exponentials need the same 1024 cycles per 128 x 128 tile; two
// tiles in flight hide one behind the other.  Measured cycles per tile: 1.6 k (DK = 128, DV = 64, long lists).  The exponential
// unit is busy 45 / 56 / 59 % of the time at 128/128, 128/64, 64/64, the tensor core 48 / 45 / 31 % (T = 4096, 50 % selected);
// the rest is the chain score tile -> maximum -> exponentials -> P V of each tile.  128-key score tiles halve the number of dependent steps of 64-key ones, and shared loads
// halve the L2 traffic of one-tile CTAs.  What it took beyond that: no code that does not have to be there (with every wait
// and every planning loop unrolled in place the kernel was 110 KB, missed the instruction cache and was 1.5 x slower than at
// 50 KB), descriptors that differ by constants, and items handed out heaviest first (see Order).
// Alone, five launches in a graph (us; before: one 128-query tile and 64-key steps per CTA, two CTAs per SM):
//                                            128/128       128/64        64/128        64/64
//   B = 8,  T = 4096,  H = 16, 25 %:       261 -> 190    243 -> 158    236 -> 172    225 -> 142     (128/128: 580 -> 795 TFLOP/s)
//   B = 16, T = 4096,  H = 16, 50 %:       745 -> 599    682 -> 492    701 -> 533    629 -> 449     (128/128: 764 -> 950 TFLOP/s)
//   B = 32, T = 2048,  H = 16, 50 %:       521 -> 381    506 -> 311    494 -> 329    437 -> 271
//   B = 1,  T = 65536, H = 32, 10 %:      4266 -> 3759  3511 -> 2862  3743 -> 3191  2980 -> 2478     (128/64: 743 -> 912 TFLOP/s)
//   B = 4,  T = 1000,  H = 16, 40 %:      29.6 -> 23.2  27.2 -> 19.2  27.9 -> 21.5  25.8 -> 18.5
//   B = 1,  T = 2048,  H = 12, 40 %:      23.5 -> 26.2  20.4 -> 20.8  22.6 -> 22.9  19.9 -> 20.4     (see the launch for small grids)
//   B = 1,  T = 512,   H = 16, 40 %:      10.6 -> 11.3  10.3 -> 10.2  10.2 -> 10.8   9.6 ->  9.9
// Behind other work under the power limit (1.76 GHz) the first one takes 211 - 218 us (273).  Tried and not kept: sixteen softmax warps with half
// a row each (207 us in the first case: the halves' maxima have to meet), the exponential unit lent to one warp at a time
// (no change), a single issuing warp for both tiles (each waits for the other's softmax).
//
// Key walk, mask and output conventions as in the mma.sync kernel (attn_walk.cuh): own span first, then the selected past
// blocks; src/nats/ops/attns/attns.py:62-353 is the reference kernel this replaces.
// Every mbarrier wait has an iteration limit; on expiry the CTA stops issuing work, waits (again with a limit) for its own
// copies in flight, records a status, frees its TMEM and returns.
#include <algorithm>

#include "attn_tc.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

int attn_fwd_mma_sync(const void* q, const void* k, const void* v, const int32_t* types_i, const int32_t* indices,
                      const int32_t* attn_n_iters, void* o, float* lse, int B, int T, int HQ, int HKV, int HN, int DK,
                      int DV, int nbs, float scale, int own, cudaStream_t st);

namespace {

constexpr int AT_THREADS = 384;
constexpr int AT_ITEM = 2 * ATT_BM;                  // queries of a work item
constexpr int AT_SMS = 148;
constexpr float LAZY_RESCALE_LOG2 = 8.0f;
constexpr long AT_GROUP_BYTES = 64 << 20;            // keys and values of the heads whose items are mixed: half of L2
constexpr uint32_t AT_O_COL = 256;
constexpr int AT_CHUNK = 8, AT_CHUNKS = 4;           // steps are handed over in chunks (an item's last one may be shorter)

// K and V ring stages of 128 keys.  Three K and two V stages are the least that the issue order needs (the tiles of an item
// may be a pair apart); smaller head dims take what hides more of the load latency.
template <int DK, int DV> struct AtSmem {
    // How far the scores run ahead of the products P V.  With DV = 64 the probabilities have columns of their own, so a
    // tile's next scores are issued as soon as its softmax holds the last ones in registers (2: the softmax never waits);
    // with DV = 128 tensor memory is full, P lies over its scores and the next ones come behind P V (1).
    static constexpr int LEAD = DV == 64 ? 2 : 1;
    static constexpr int KST = DK == 64 ? 4 : 3;
    static constexpr int VST = DV == 64 ? 4 : DK == 64 ? 3 : 2;
    static constexpr int q = 0;                                  // tile A, tile B: DK/64 sub-tiles [128][64] each
    static constexpr int k = q + 2 * 128 * DK * 2;               // KST stages x DK/64 sub-tiles [128][64]
    static constexpr int v = k + KST * 128 * DK * 2;             // VST stages x DV/64 sub-tiles [128][64]
    static constexpr int bars = v + VST * 128 * DV * 2;
    static constexpr int items = bars + 384;                     // two slots of 8 ints
    static constexpr int steps = items + 64;                     // AT_CHUNKS x AT_CHUNK steps of 8 ints
    static constexpr int clc = steps + AT_CHUNKS * AT_CHUNK * 32;   // 16-byte answer of the take-over request
    static constexpr int tmem = clc + 16;
    static constexpr int total = tmem + 16;
    static_assert(total <= 232448, "shared memory of one SM");
};

// Where the gathered part of the key sequence lives (keys below k_split; see the kernel's comment).
struct RemoteKeys {
    int k_split;          // keys [0, k_split) are gathered keys
    const int* base;      // first pair of (segment g, this head): base[g * stride], or nullptr for the head-major layout
    int stride;
    int slots;            // virtual blocks per head and gathered segment
};

// Which work item a block is.  Heads in groups whose keys and values stay in L2; in a group the items with the most keys
// first, over all its heads, so that the last items of a group, and with them of the grid, are the lightest.  (Head by head
// the SMs of a 16384-token call ended between 124 and 232 us.)
struct Order {
    uint32_t n_blocks, n_heads, group, split;            // blocks per head, heads over all batches, heads of a group, see below
    uint32_t q_per_kv, q_per_sel, rem_segments;          // query heads of a key head, of a selection head; gathered segments
};
// q0: first query of the item.  With split a block is one tile of an item: only = 1 tile A, 2 tile B (0: both).  The tile goes
// through the same keys in the same order as beside the other one, so its results do not depend on the split.
__device__ __forceinline__ void locate(const Order& od, int block, int HQ, int q_off, int& q0, int& only, int& hq, int& b) {
    const uint32_t grp = (uint32_t)block / (od.group * od.n_blocks), rest = block - grp * od.group * od.n_blocks;
    const uint32_t width = min(od.group, od.n_heads - grp * od.group), level = rest / width;
    const uint32_t head = grp * od.group + rest - level * width, i = od.n_blocks - 1 - level;
    b = (int)(head / (uint32_t)HQ);
    hq = (int)head - b * HQ;
    only = od.split ? 1 + (int)(i & 1) : 0;
    q0 = q_off + (int)(od.split ? i >> 1 : i) * AT_ITEM;
}

// One work item and the order in which its pairs of 64-key units are used.  Units 0 .. n_span-1 are the own span
// (masked), the rest the selected past blocks; pair j = units 2j, 2j+1.  Tile A takes the pairs [0, end_a) and
// [next_a, n_pairs): the pairs between them hold only keys behind A's rows.  Tile B takes [first_b, n_pairs): pair 0 is
// left out if no row of B sees it.  Step i of an item = the i-th pair of A and the i-th pair of B (at most one pair apart).
struct Item {
    int q0, span_start, n_span, n_units, n_pairs, end_a, next_a, first_b, sel;
    bool has_b, use_a, use_b;                            // the item has a tile B; the tiles this block works on
};

// selection block of span unit u, relative to the first one of the span (a span touches at most four)
__device__ __forceinline__ int span_block(int u, int cpb) { return (u >= cpb) + (u >= 2 * cpb) + (u >= 3 * cpb); }
// Whether the 32 rows of warp w of tile x see the 32-key chunk c of pair j (attn_walk.cuh: visible(); everything in it but
// s <= t is the same for 32 aligned rows and 32 aligned keys, and rows past the end are not stored).
__device__ __forceinline__ bool chunk_seen(const Item& t, int x, int w, int j, int c, int cpb, int nbs, int own_chunk) {
    const int u = 2 * j + (c >> 1), row = t.q0 + x * ATT_BM + 32 * w;
    if (u >= t.n_span) return u < t.n_units;
    const int rb = span_block(u, cpb), blk_end = t.span_start + (rb + 1) * nbs;
    const bool selb = (t.sel >> rb) & 1;
    return own_chunk ? t.span_start + u * ATT_BN + 32 * (c & 1) <= row && (selb || row < blk_end) : selb && row >= blk_end;
}
// (the whole warp)  Bit 4w + c: chunk c of tile A's pair ja is seen by its warp w; the upper half the same for tile B and jb.
__device__ __forceinline__ uint32_t seen_chunks(const Item& t, int ja, int jb, int lane, int cpb, int nbs, int own_chunk) {
    const int x = lane >> 4;
    return __ballot_sync(0xffffffffu, chunk_seen(t, x, (lane >> 2) & 3, x ? jb : ja, lane & 3, cpb, nbs, own_chunk));
}
__device__ __forceinline__ int span_units(int q0, int span_start, bool has_b, int T) {
    return (min(q0 + (has_b ? AT_ITEM : ATT_BM), T) - span_start + ATT_BN - 1) / ATT_BN;
}
__device__ __forceinline__ Item make_item(int q0, int span_start, int n_past_blocks, int sel, int T, int q_end, int only,
                                          int nbs, int own_chunk, int lane) {
    Item t;
    const int cpb = nbs / ATT_BN;
    t.q0 = q0;
    t.sel = sel;
    t.has_b = q0 + ATT_BM < q_end;
    t.use_a = only != 2;
    t.use_b = t.has_b && only != 1;
    t.span_start = span_start;
    t.n_span = span_units(q0, span_start, t.has_b, T);
    t.n_units = t.n_span + n_past_blocks * cpb;
    t.n_pairs = (t.n_units + 1) >> 1;
    const int a_units = min((q0 + ATT_BM - span_start) / ATT_BN, t.n_span);
    t.end_a = (a_units + 1) >> 1;
    t.next_a = max(t.end_a, t.n_units > t.n_span ? t.n_span >> 1 : t.n_pairs);
    t.first_b = t.has_b && own_chunk && (seen_chunks(t, 0, 0, lane, cpb, nbs, 1) >> 16) == 0;
    return t;
}
__device__ __forceinline__ bool uses_a(const Item& t, int j) { return t.use_a && (j < t.end_a || j >= t.next_a); }
__device__ __forceinline__ bool uses_b(const Item& t, int j) { return t.use_b && j >= t.first_b; }

// What one tile does in a step: flags, ring stages and phases of its pair, as one word.
enum : uint32_t {
    ST_VALID = 1, ST_USE0 = 2, ST_USE1 = 4,              // the tile takes part; some row sees the first / second unit
    ST_FIRST = 8, ST_LAST = 16,                          // first / last pair of the item
    ST_ALONE = 32, ST_TWO = 64,                          // the other tile does not use the pair; the second unit is loaded
    ST_K = 8, ST_KPAR = 10, ST_V = 11, ST_VPAR = 13,     // shifts: K stage, its phase parity, V stage, its phase parity
    ST_CHUNK_LAST = 1u << 14, ST_STOP = 1u << 15,        // (word of tile A)
};

template <int DK, int DV>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_kr,
                   const __grid_constant__ CUtensorMap map_vr, int k_split, int B_rem, const int* __restrict__ rem_base,
                   int rem_slots, const int* __restrict__ types_i, const int* __restrict__ indices,
                   const int* __restrict__ attn_n_iters, __nv_bfloat16* __restrict__ o, float* __restrict__ lse, int T,
                   int Tq, int q_off, int HQ, int HKV, int HN, int TN, int nbs, float scale_log2, int own_chunk,
                   const Order od, int* status) {
    // T = number of keys (and the length the tables were built for); the Tq queries are the tokens
    // [q_off, q_off + Tq) of that sequence (q_off = 0, Tq = T except under sequence parallelism).
    // Keys [0, k_split) live in a second pair of tensors (map_kr / map_vr, batch index b % B_rem: the
    // gathered blocks of other segments, shared by the local segments), keys [k_split, T) in map_k / map_v.
    // With rem_base the gathered tensors are [B_rem, tokens, 1, D]: the selected (block, head) pairs of every
    // gathered segment packed back to back; virtual block g * rem_slots + j of head hkv is pair
    // rem_base[(b % B_rem, g, hkv)] + j.
    using L = AtSmem<DK, DV>;
    constexpr int KST = L::KST, VST = L::VST, LEAD = L::LEAD;
    constexpr uint32_t P_COL = LEAD == 1 ? 0 : 384, P_STRIDE = LEAD == 1 ? 128 : 64;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sbase = smem_u32(smem);
    if ((sbase & 1023u) != 0) {                       // swizzled tiles need 1024-byte alignment
        if (tid == 0) atomicExch(status, 2);
        return;
    }
    const uint32_t s_q = sbase + L::q, s_k = sbase + L::k, s_v = sbase + L::v, s_clc = sbase + L::clc;
    volatile int* items = reinterpret_cast<volatile int*>(smem + L::items);
    int4* steps = reinterpret_cast<int4*>(smem + L::steps);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::tmem);
    const uint32_t bar0 = sbase + L::bars;
    // barrier slots (8 bytes each)
    const uint32_t bar_k_full = bar0, bar_k_empty = bar0 + 32, bar_v_full = bar0 + 64, bar_v_empty = bar0 + 96,
                   bar_q_full = bar0 + 128, bar_q_empty = bar0 + 144, bar_s = bar0 + 160, bar_s_free = bar0 + 176,
                   bar_p = bar0 + 192, bar_o = bar0 + 224, bar_item = bar0 + 240, bar_item_empty = bar0 + 256,
                   bar_clc = bar0 + 272, bar_steps = bar0 + 280, bar_steps_empty = bar0 + 312;
    static_assert(AT_CHUNKS == 4 && KST <= 4 && VST <= 4, "barrier slots");
    const int cpb = nbs / ATT_BN, q_end = q_off + Tq;
    if (tid == 256) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(bar_k_full + 8 * i, 1);
            mbar_init(bar_k_empty + 8 * i, 2);           // one arrival per tile (two of the only one that uses the pair)
            mbar_init(bar_v_full + 8 * i, 1);
            mbar_init(bar_v_empty + 8 * i, 2);
            mbar_init(bar_p + 8 * i, 4);                 // (tile, half): one arrival per softmax warp
            mbar_init(bar_steps + 8 * i, 1);
            mbar_init(bar_steps_empty + 8 * i, 10);      // eight softmax warps and two issuers are through with the chunk
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_item + 8 * i, 1);
            mbar_init(bar_item_empty + 8 * i, 1);
            mbar_init(bar_q_full + 8 * i, 1);
            mbar_init(bar_q_empty + 8 * i, 1);
            mbar_init(bar_s + 8 * i, 1);
            mbar_init(bar_s_free + 8 * i, 4);
            mbar_init(bar_o + 8 * i, 1);
        }
        mbar_init(bar_clc, 1);
        mbar_fence_init();
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        if (k_split > 0) {
            prefetch_tensormap(&map_kr);
            prefetch_tensormap(&map_vr);
        }
    }
    if (warp == 9) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;

    // registers: 2 x 128 x 200 + 128 x 104 = 384 x 168, what the block is launched with
    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        if (warp == 8) {
            // -------------------------------------------------------- TMA producer
            int kc = 0, vc = 0;                          // pairs loaded so far
            int nq[2] = {0, 0};                          // query tiles loaded so far
#pragma unroll 1
            for (int n = 0; ok; ++n) {
                const int slot = n & 1;
                // use: bit x = tile x; skip: one tile alone leaves out the pairs [skip, next_a) (A) or [0, skip) (B)
                int q0, hq, b, span_start, n_span, n_units = -1, use, skip = 0;
                auto take = [&]() {
                    ok = warp_wait(bar_item + slot * 8, (n >> 1) & 1);
                    q0 = items[slot * 8];
                    hq = items[slot * 8 + 1];
                    b = items[slot * 8 + 2];
                    span_start = items[slot * 8 + 3];
                    n_span = items[slot * 8 + 4];
                    n_units = items[slot * 8 + 5];
                    use = items[slot * 8 + 6];
                    skip = items[slot * 8 + 7];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_item_empty + slot * 8);
                };
                if (n > 0) {
                    take();
                    if (!ok || q0 < 0) break;            // no items left
                } else {                                 // tile A's first loads depend on no table
                    int only;
                    locate(od, blockIdx.x, HQ, q_off, q0, only, hq, b);
                    span_start = (uint32_t)q0 / (uint32_t)nbs * nbs;
                    n_span = span_units(q0, span_start, q0 + ATT_BM < q_end, T);
                    use = only ? only : q0 + ATT_BM < q_end ? 3 : 1;
                }
                const int hkv = (uint32_t)hq / od.q_per_kv, hn = (uint32_t)hq / od.q_per_sel, b_rem = (uint32_t)b % (uint32_t)B_rem;
                const int* idx = indices + ((long)b * TN * HN + hn) * 2;
                const long tstride = (long)HN * 2;
                RemoteKeys rk;
                rk.k_split = k_split;
                rk.slots = rem_slots;
                rk.stride = HKV;
                rk.base = rem_base ? rem_base + ((long)b_rem * od.rem_segments) * HKV + hkv : nullptr;
                const int rem_head = rem_base ? 0 : hkv;         // packed pairs have no head axis
                // token coordinate of unit u in the tensor it is loaded from; bit 31 = gathered keys
                auto unit = [&](int u) -> uint32_t {
                    if (u >= (n_units < 0 ? n_span : n_units)) return 0;
                    int s0;
                    if (u < n_span) {
                        s0 = span_start + u * ATT_BN;
                    } else {
                        const uint32_t up = u - n_span, blk = up / (uint32_t)cpb;
                        s0 = __ldg(idx + (long)blk * tstride) * nbs + (int)(up - blk * cpb) * ATT_BN;
                    }
                    if (s0 >= rk.k_split) return (uint32_t)(s0 - rk.k_split);
                    int coord = s0;
                    if (rk.base) {
                        const int vb = (uint32_t)s0 / (uint32_t)nbs, g = (uint32_t)vb / (uint32_t)rk.slots;
                        coord = (rk.base[(long)g * rk.stride] + (vb - g * rk.slots)) * nbs + (s0 - vb * nbs);
                    }
                    return (uint32_t)coord | 0x80000000u;
                };
                auto load_q = [&](int x) {
                    if (nq[x] > 0) ok = warp_wait(bar_q_empty + x * 8, (nq[x] - 1) & 1);
                    if (ok && lane == 0) {
                        mbar_expect_tx(bar_q_full + x * 8, 128 * DK * 2);
#pragma unroll
                        for (int sub = 0; sub < DK / 64; ++sub)
                            tma_load_4d(s_q + x * (128 * DK * 2) + sub * 16384, &map_q, sub * 64, hq, q0 - q_off + x * ATT_BM, b,
                                        bar_q_full + x * 8);
                    }
                    __syncwarp();
                    if (ok) ++nq[x];
                };
                auto load_pair = [&](uint32_t dst, uint32_t full, const CUtensorMap* own, const CUtensorMap* rem, int subs,
                                     uint32_t u0, uint32_t u1, bool two) {            // lane 0 only
                    mbar_expect_tx(full, (two ? 2 : 1) * subs * 8192);
#pragma unroll 1
                    for (int e = 0; e < (two ? 2 : 1); ++e) {
                        const uint32_t u = e ? u1 : u0;
                        const bool r = (u >> 31) != 0;
#pragma unroll 1
                        for (int sub = 0; sub < subs; ++sub)
                            tma_load_4d(dst + sub * 16384 + e * 8192, r ? rem : own, sub * 64, r ? rem_head : hkv,
                                        (int)(u & 0x7fffffffu), r ? b_rem : b, full);
                    }
                };
                if (use & 1) load_q(0);
                uint32_t mine = 0;                       // lane l: unit l of the 32 that hold the pair at hand
#pragma unroll 1
                for (int j = 0; ok; ++j) {
                    const bool now = n_units < 0 && (j > 0 || n_span < 2 || use == 2);
                    if (now) take();
                    if (!ok || (n_units >= 0 && 2 * j >= n_units)) break;
                    if ((j & 15) == 0 || now) mine = unit(2 * (j & ~15) + lane);
                    const uint32_t u0 = __shfl_sync(0xffffffffu, mine, (2 * j) & 31), u1 = __shfl_sync(0xffffffffu, mine, (2 * j + 1) & 31);
                    const bool two = 2 * j + 1 < (n_units < 0 ? n_span : n_units);
                    if (j == 0 && use == 2) load_q(1);
                    if (!ok) break;
                    if (skip > 0 && (use == 2 ? j < skip : j >= skip && 2 * j < n_span && !(2 * j + 1 == n_span && n_units > n_span)))
                        continue;                        // only the other tile uses it
                    const int ks = kc % KST;
                    if (kc >= KST) ok = warp_wait(bar_k_empty + ks * 8, (kc / KST - 1) & 1);
                    if (!ok) break;
                    if (lane == 0) load_pair(s_k + ks * (128 * DK * 2), bar_k_full + ks * 8, &map_k, &map_kr, DK / 64, u0, u1, two);
                    __syncwarp();
                    ++kc;
                    // behind the first keys, not before: tile A may already go on while the last scores of the previous item's
                    // tile B, which still read the old query tile, have yet to be issued
                    if (j == 0 && use == 3) load_q(1);
                    if (!ok) break;
                    const int vs = vc % VST;
                    if (vc >= VST) ok = warp_wait(bar_v_empty + vs * 8, (vc / VST - 1) & 1);
                    if (!ok) break;
                    if (lane == 0) load_pair(s_v + vs * (128 * DV * 2), bar_v_full + vs * 8, &map_v, &map_vr, DV / 64, u0, u1, two);
                    __syncwarp();
                    ++vc;
                }
            }
            if (!ok) {                                   // nothing may still be on its way into shared memory
#pragma unroll 1
                for (int c = max(0, kc - KST); c < kc; ++c) warp_wait(bar_k_full + (c % KST) * 8, (c / KST) & 1);
#pragma unroll 1
                for (int c = max(0, vc - VST); c < vc; ++c) warp_wait(bar_v_full + (c % VST) * 8, (c / VST) & 1);
                if (nq[0] > 0) warp_wait(bar_q_full, (nq[0] - 1) & 1);
                if (nq[1] > 0) warp_wait(bar_q_full + 8, (nq[1] - 1) & 1);
            }
        } else if (warp != 10) {
            // -------------------------------------------------------- MMA issuer of one tile (the whole warp, converged)
            // One issuing warp per tile: neither waits for the other's softmax.
            constexpr uint32_t idesc_s1 = umma_idesc_bf16(128, 64, false), idesc_s2 = umma_idesc_bf16(128, 128, false);
            constexpr uint32_t idesc_pv = umma_idesc_bf16(128, DV, true);
            const int x = warp == 9 ? 0 : 1;
            const uint32_t qlo = umma_desc_lo(s_q, 16) + x * (128 * DK * 2 >> 4), k_lo = umma_desc_lo(s_k, 16),
                           v_lo = umma_desc_lo(s_v, 16384);
            const uint32_t t_s = tmem + x * 128, t_p = tmem + P_COL + x * P_STRIDE, t_o = tmem + AT_O_COL + x * DV;
            const uint32_t b_s = bar_s + x * 8, b_free = bar_s_free + x * 8, b_p = bar_p + x * 16, b_o = bar_o + x * 8;
            bool more = true;
            uint32_t q_par = 0, p_par = 0, f_par = 1;    // parities of the next query tile / probabilities / release of the scores
            uint32_t acc = 0;                            // O holds a product of this item
            int chunk = 0, pos = 0;
            // The next step, which may be one that this tile takes no part in.  It is never looked for further ahead than LEAD
            // steps: the items behind are only scheduled once the loads of this one, which wait for its products, are through.
            auto next_step = [&]() -> uint32_t {
                if (!more) return ST_STOP;
                const int slot = chunk & (AT_CHUNKS - 1);
                if (pos == 0) ok = warp_wait(bar_steps + slot * 8, (chunk / AT_CHUNKS) & 1);
                const int4 e = steps[(slot * AT_CHUNK + pos) * 2];
                // (through a shuffle: what follows from the words is the same in all lanes, which the compiler then knows)
                const uint32_t fa = __shfl_sync(0xffffffffu, (uint32_t)e.x, 0), fx = __shfl_sync(0xffffffffu, (uint32_t)(x ? e.y : e.x), 0);
                ++pos;
                if (fa & ST_CHUNK_LAST) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_steps_empty + slot * 8);
                    ++chunk;
                    pos = 0;
                }
                more = ok && !(fa & ST_STOP);
                return more ? fx : ST_STOP;
            };
            auto issue_s = [&](uint32_t f) {             // S = Q K^T
                if (!ok || !(f & ST_VALID)) return;
                if (f & ST_FIRST) {
                    ok = warp_wait(bar_q_full + x * 8, q_par);
                    q_par ^= 1;
                }
                const uint32_t st = (f >> ST_K) & 3;
                if (ok) ok = warp_wait(bar_k_full + st * 8, (f >> ST_KPAR) & 1);
                if (LEAD == 2) {                         // the softmax holds the previous scores in registers (first time: free)
                    if (ok) ok = warp_wait(b_free, f_par);
                    f_par ^= 1;
                }
                if (!ok) return;
                tc_fence_after();
                const uint32_t klo = k_lo + st * (128 * DK * 2 >> 4), idesc = (f & ST_TWO) ? idesc_s2 : idesc_s1;
#pragma unroll
                for (int h = 0; h < DK / 64; ++h) umma_ss_x4<2, 2>(t_s, qlo + h * 1024, klo + h * 1024, idesc, h > 0);
                umma_commit(b_s);
                umma_commit(bar_k_empty + st * 8);
                if (f & ST_ALONE) umma_commit(bar_k_empty + st * 8);
                if (f & ST_LAST) umma_commit(bar_q_empty + x * 8);
            };
            auto issue_pv = [&](uint32_t f) {            // O += P V
                if (!ok || !(f & ST_VALID)) return;
                if (f & ST_FIRST) acc = 0;
                const uint32_t st = (f >> ST_V) & 3;
                ok = warp_wait(bar_v_full + st * 8, (f >> ST_VPAR) & 1);
                const uint32_t vlo = v_lo + st * (128 * DV * 2 >> 4), par = p_par;
                p_par ^= 1;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (ok && (e == 0 || LEAD == 1)) ok = warp_wait(b_p + e * 8, par);
                    if (!ok) return;
                    tc_fence_after();
                    if (f & (e ? ST_USE1 : ST_USE0)) {   // a unit that no row sees stays out, whatever its values are
                        umma_ts_x4<128>(t_o, t_p + e * 32, vlo + e * 512, idesc_pv, acc);
                        acc = 1;
                    }
                }
                if (LEAD == 2 || (f & ST_LAST)) umma_commit(b_o);
                umma_commit(bar_v_empty + st * 8);
                if (f & ST_ALONE) umma_commit(bar_v_empty + st * 8);
            };
            uint32_t ring[LEAD];                         // steps whose scores are issued and whose products are not
#pragma unroll
            for (int e = 0; e < LEAD; ++e) ring[e] = 0;
#pragma unroll 1
            while (ok && !(ring[0] & ST_STOP)) {
                const uint32_t f = next_step();
                issue_pv(ring[0]);
                issue_s(f);
#pragma unroll
                for (int e = 0; e + 1 < LEAD; ++e) ring[e] = ring[e + 1];
                ring[LEAD - 1] = f;
            }
        } else {
            // -------------------------------------------------------- scheduler: work items, and their steps, one lane per step
            // (It runs ahead of the loads.  A single warp that works the steps out between two products costs more than the
            // products themselves, and one that does so between two loads makes every item begin with a wait.)
            bool stop = false;
            int asked = -1;                              // request whose answer is outstanding
            int chunk = 0, base = 0;                     // base: pairs of all items before
            int block = blockIdx.x;
            const int NTq = (T + ATT_BM - 1) / ATT_BM;
            auto request = [&](int n) {
                asked = n;
                if (lane == 0) {
                    fence_async_smem();
                    mbar_expect_tx(bar_clc, 16);
                    request_block(s_clc, bar_clc);
                }
                __syncwarp();
            };
#pragma unroll 1
            for (int n = 0; ok; ++n) {
                if (n > 0) {
                    if (asked < 0) {                     // not before the loads of the item before have begun
                        ok = warp_wait(bar_item_empty + ((n - 1) & 1) * 8, ((n - 1) >> 1) & 1);
                        if (!ok) break;
                        request(n - 1);
                    }
                    ok = warp_wait(bar_clc, (n - 1) & 1);
                    if (!ok) break;
                    asked = -1;
                    stop = !taken_block(s_clc, block);
                    __syncwarp();
                }
                const int islot = n & 1;
                if (n >= 2) ok = warp_wait(bar_item_empty + islot * 8, ((n >> 1) - 1) & 1);
                if (!ok) break;
                int q0, only, hq, b;
                locate(od, stop ? 0 : block, HQ, q_off, q0, only, hq, b);
                const int hn = (uint32_t)hq / od.q_per_sel, blk0 = (uint32_t)q0 / (uint32_t)nbs;
                const int* selp = types_i + ((long)b * TN * HN + hn) * 2;
                const int n_past = __ldg(attn_n_iters + ((long)b * NTq + q0 / ATT_BM) * HN + hn);
                // the own span touches at most four selection blocks
                const int s_lane = (lane < 4 && blk0 + lane < TN) ? __ldg(selp + (long)(blk0 + lane) * HN * 2) : 0;
                const int sel = (int)(__ballot_sync(0xffffffffu, s_lane != 0) & 15u);
                const Item it = make_item(q0, blk0 * nbs, n_past, sel, T, q_end, only, nbs, own_chunk, lane);
                if (lane == 0) {
                    items[islot * 8 + 0] = stop ? -1 : q0;
                    items[islot * 8 + 1] = hq;
                    items[islot * 8 + 2] = b;
                    items[islot * 8 + 3] = it.span_start;
                    items[islot * 8 + 4] = it.n_span;
                    items[islot * 8 + 5] = it.n_units;
                    items[islot * 8 + 6] = (it.use_a ? 1 : 0) | (it.use_b ? 2 : 0);
                    items[islot * 8 + 7] = it.use_a && it.use_b ? 0 : it.use_a ? it.end_a : it.first_b;
                    mbar_arrive(bar_item + islot * 8);
                }
                __syncwarp();
                // An item of a few pairs is over before the next one could be taken and planned: ask at once.  Behind a longer
                // one a block is better left to an SM that is free earlier.
                if (!stop && it.n_pairs <= 4) request(n);
                const int n_a = it.use_a ? it.end_a + it.n_pairs - it.next_a : 0, n_b = it.use_b ? it.n_pairs - it.first_b : 0;
                const int n_steps = stop ? 1 : max(n_a, n_b);
#pragma unroll 1
                for (int i0 = 0; ok && i0 < n_steps; i0 += AT_CHUNK) {
                    const int slot = chunk & (AT_CHUNKS - 1), i = i0 + lane;
                    if (chunk >= AT_CHUNKS) ok = warp_wait(bar_steps_empty + slot * 8, (chunk / AT_CHUNKS - 1) & 1);
                    const bool mine = lane < AT_CHUNK && i < n_steps;
                    const int ja = i < it.end_a ? i : i + it.next_a - it.end_a, jb = i + it.first_b;
                    auto masked = [&](int j) { return 2 * j < it.n_span || 2 * j + 1 >= it.n_units; };
                    uint32_t seen = 0xffffffffu;         // seen_chunks() of this lane's step
#pragma unroll 1
                    for (uint32_t todo = __ballot_sync(0xffffffffu, mine && (masked(ja) || masked(jb))); todo; todo &= todo - 1) {
                        const int src = __ffs(todo) - 1;
                        const uint32_t bits = seen_chunks(it, __shfl_sync(0xffffffffu, ja, src), __shfl_sync(0xffffffffu, jb, src),
                                                          lane, cpb, nbs, own_chunk);
                        if (lane == src) seen = bits;
                    }
                    if (ok && mine) {
                        uint32_t f[2] = {0, 0}, mk[2] = {0, 0};
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const int nx = x ? n_b : n_a;
                            if (stop || i >= nx) continue;
                            const int j = x ? jb : ja, c = base + (it.use_a && it.use_b ? j : i);
                            const bool alone = !(uses_a(it, j) && uses_b(it, j));
                            const uint32_t m = (seen >> (16 * x)) & 0xffffu;
                            // the chunk whose keys are the warp's own rows is chunk w + d of the pair
                            const int d = (it.q0 + x * ATT_BM - (it.span_start + 2 * j * ATT_BN)) / 32;
                            const bool own = own_chunk && 2 * j < it.n_span && d > -4 && d < 4;
                            f[x] = ST_VALID | ((m & 0x3333u) ? ST_USE0 : 0) | ((m & 0xccccu) ? ST_USE1 : 0) | (i == 0 ? ST_FIRST : 0) |
                                   (i == nx - 1 ? ST_LAST : 0) | (alone ? ST_ALONE : 0) | (2 * j + 1 < it.n_units ? ST_TWO : 0) |
                                   ((uint32_t)(c % KST) << ST_K) | ((uint32_t)((c / KST) & 1) << ST_KPAR) |
                                   ((uint32_t)(c % VST) << ST_V) | ((uint32_t)((c / VST) & 1) << ST_VPAR);
                            mk[x] = m | (own ? (uint32_t)(d + 4) << 16 : 0u);
                        }
                        if (lane == AT_CHUNK - 1 || i == n_steps - 1) f[0] |= ST_CHUNK_LAST;
                        if (stop) f[0] |= ST_STOP;
                        steps[(slot * AT_CHUNK + lane) * 2] = make_int4((int)f[0], (int)f[1], (int)mk[0], (int)mk[1]);
                        steps[(slot * AT_CHUNK + lane) * 2 + 1] = make_int4(it.q0, hq, b, 0);
                    }
                    __syncwarp();
                    if (ok && lane == 0) mbar_arrive(bar_steps + slot * 8);
                    ++chunk;
                }
                if (stop) break;
                base += it.use_a && it.use_b ? it.n_pairs : n_steps;                  // loaded pairs
            }
            if (asked >= 0) warp_wait(bar_clc, asked & 1);       // (after a failed wait: the answer may still be on its way)
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
        // ------------------------------------------------------------ softmax + epilogue (tile x, one row per thread)
        const int x = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t t_s = lane_base + x * 128, t_o = lane_base + AT_O_COL + x * DV, t_p = lane_base + P_COL + x * P_STRIDE;
        const bool wide = (reinterpret_cast<uintptr_t>(o) & 31) == 0;
        const uint32_t tri = (2u << lane) - 1;           // keys of the row's own 32-key chunk that it sees
        int ns = 0, no = 0;                              // score tiles, phases of bar_o taken so far
        int chunk = 0, pos = 0;
        float m = -INFINITY;
        uint64_t l2a = 0, l2b = 0;                       // two packed partial sums of the row
#pragma unroll 1
        while (ok) {
            const int slot = chunk & (AT_CHUNKS - 1);
            if (pos == 0) ok = warp_wait(bar_steps + slot * 8, (chunk / AT_CHUNKS) & 1);
            if (!ok) break;
            const int4 e0 = steps[(slot * AT_CHUNK + pos) * 2], e1 = steps[(slot * AT_CHUNK + pos) * 2 + 1];
            const uint32_t fa = __shfl_sync(0xffffffffu, (uint32_t)e0.x, 0), f = x ? __shfl_sync(0xffffffffu, (uint32_t)e0.y, 0) : fa,
                           mk = __shfl_sync(0xffffffffu, (uint32_t)(x ? e0.w : e0.z), 0);
            ++pos;
            if (fa & ST_CHUNK_LAST) {
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_steps_empty + slot * 8);
                ++chunk;
                pos = 0;
            }
            if (fa & ST_STOP) break;
            if (!(f & ST_VALID)) continue;
            const int t = e1.x + x * ATT_BM + row, hq = e1.y, b = e1.z;
            if (f & ST_FIRST) {
                m = -INFINITY;
                l2a = l2b = 0;
            }
            ok = warp_wait(bar_s + x * 8, ns & 1);
            ++ns;
            if (!ok) break;
            tc_fence_after();
            uint32_t sr[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(t_s + c * 32, sr[c]);
            tmem_ld_wait();
            if (LEAD == 2) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_s_free + x * 8);
            }
            // Chunks of 32 columns that no row of the warp sees cost nothing below; the one that holds the warp's own rows is
            // masked per element, every other one is seen in full.
            const uint32_t live = (mk >> (4 * (warp & 3))) & 15u;
            if (mk >> 16) {
                const int diag = (warp & 3) + (int)(mk >> 16) - 4;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (c == diag) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) sr[c][e] = (tri & (1u << e)) ? sr[c][e] : 0xff800000u;      // -inf
                    }
            }
            // row maximum of the raw scores (scale > 0, so max(scale * s) = scale * max(s))
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx[c] = -INFINITY;
                if ((live >> c) & 1) {
#pragma unroll
                    for (int e = 0; e < 32; e += 2) mx[c] = fmax3(mx[c], __uint_as_float(sr[c][e]), __uint_as_float(sr[c][e + 1]));
                }
            }
            const float mnew = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]) * scale_log2;
            const bool need = mnew > m + LAZY_RESCALE_LOG2;
            if (__any_sync(0xffffffffu, need)) {
                const float mn = need ? mnew : m;
                const float alpha = mn == -INFINITY ? 1.f : ex2(m - mn);
                if (!(f & ST_FIRST)) {
                    // O must be at rest.  LEAD = 2: the product of the previous P; LEAD = 1: these scores are complete, hence
                    // so is every product issued before them.
                    if (LEAD == 2) {
                        ok = warp_wait(bar_o + x * 8, no & 1);
                        if (!ok) break;
                        tc_fence_after();
                    }
#pragma unroll 1
                    for (int c0 = 0; c0 < DV; c0 += 32) {
                        uint32_t orr[32];
                        tmem_ld32(t_o + c0, orr);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e) orr[e] = __float_as_uint(__uint_as_float(orr[e]) * alpha);
                        tmem_st32(t_o + c0, orr);
                    }
                }
                const uint64_t al2 = pack2(alpha, alpha);
                l2a = fma2(l2a, al2, 0);
                l2b = fma2(l2b, al2, 0);
                m = mn;
            }
            const float neg = m == -INFINITY ? 0.f : -m;
            const uint64_t sc2 = pack2(scale_log2, scale_log2), ng2 = pack2(neg, neg);
            uint64_t ta = 0, tb = 0;                     // sums of the step: one addition to the row's sums per step, not per key
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t pr[32];
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if ((live >> (2 * h + g)) & 1) {
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const uint32_t* s2 = sr[2 * h + g] + 2 * c;
                            float x0, x1;
                            unpack2(fma2(pack2(__uint_as_float(s2[0]), __uint_as_float(s2[1])), sc2, ng2), x0, x1);
                            x0 = ex2(x0);
                            x1 = ex2(x1);
                            if (c & 1) tb = add2(tb, pack2(x0, x1));
                            else ta = add2(ta, pack2(x0, x1));
                            pr[16 * g + c] = pack_bf16(x0, x1);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 16; ++c) pr[16 * g + c] = 0;
                    }
                }
                if (LEAD == 2 && h == 0 && !(f & ST_FIRST)) {     // the previous P has been used
                    ok = warp_wait(bar_o + x * 8, no & 1);
                    ++no;
                    if (!ok) break;
                    tc_fence_after();
                }
                tmem_st32(t_p + h * 32, pr);
                if (LEAD == 1 || h == 1) {               // (LEAD = 1: P V of the first 64 keys starts while the others' P is formed)
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_p + (2 * x + (LEAD == 1 ? h : 0)) * 8);
                }
            }
            if (!ok) break;
            l2a = add2(l2a, ta);
            l2b = add2(l2b, tb);
            if (!(f & ST_LAST)) continue;
            ok = warp_wait(bar_o + x * 8, no & 1);
            ++no;
            if (!ok) break;
            tc_fence_after();
            float l0, l1, l2, l3;
            unpack2(l2a, l0, l1);
            unpack2(l2b, l2, l3);
            const float l = (l0 + l1) + (l2 + l3);
            const bool none = l == 0.f;                  // no visible key: O may never have been written
            const float inv = none ? 0.f : 1.f / l;
            const int tq = t - q_off;
            __nv_bfloat16* orow = o + (((long)b * Tq + tq) * HQ + hq) * DV;
#pragma unroll 1
            for (int c0 = 0; c0 < DV; c0 += 32) {
                uint32_t orr[32], pk[16];
                tmem_ld32(t_o + c0, orr);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    pk[e] = none ? 0u : pack_bf16(__uint_as_float(orr[2 * e]) * inv, __uint_as_float(orr[2 * e + 1]) * inv);
                if (tq < Tq) {
                    if (wide) {                          // whole 32-byte sectors
#pragma unroll
                        for (int e = 0; e < 16; e += 8)
                            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                                         ::"l"(orow + c0 + 2 * e), "r"(pk[e]), "r"(pk[e + 1]), "r"(pk[e + 2]), "r"(pk[e + 3]),
                                           "r"(pk[e + 4]), "r"(pk[e + 5]), "r"(pk[e + 6]), "r"(pk[e + 7])
                                         : "memory");
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; e += 4)
                            *reinterpret_cast<uint4*>(orow + c0 + 2 * e) = make_uint4(pk[e], pk[e + 1], pk[e + 2], pk[e + 3]);
                    }
                }
            }
            if (tq < Tq) lse[((long)b * Tq + tq) * HQ + hq] = l > 0.f ? m + log2f(l) : 0.f;
            tc_fence_before();                           // O is read before the next item's first P is announced
        }
    }
    // ---------------------------------------------------------------- teardown
    if (!ok && lane == 0) atomicExch(status, NATSL_DEV_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem, 512);
}

template <int DK, int DV>
int launch_attn_tc(const void* q, const void* k_rem, const void* v_rem, const void* k, const void* v,
                   const int* rem_base, int rem_slots, int rem_tokens, const int* types_i, const int* indices,
                   const int* n_iters, void* o, float* lse, int B, int B_rem, int T, int Tq, int q_off, int k_split,
                   int HQ, int HKV, int HN, int nbs, float scale, int own_chunk, cudaStream_t st) {
    using L = AtSmem<DK, DV>;
    auto kern = attn_fwd_tc_kernel<DK, DV>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total);
    if (e != cudaSuccess) {
        set_error("natsl_attn_fwd: cannot reserve %d B of shared memory (%s)", L::total, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    CUtensorMap mq, mk, mv, mkr, mvr;
    int rc = encode_bthd_map(&mq, q, B, Tq, HQ, DK, 128, "natsl_attn_fwd(q)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mk, k, B, T - k_split, HKV, DK, 64, "natsl_attn_fwd(k)");
    if (rc == NATSL_OK) rc = encode_bthd_map(&mv, v, B, T - k_split, HKV, DV, 64, "natsl_attn_fwd(v)");
    if (k_split > 0) {
        const int rt = rem_base ? rem_tokens : k_split, rh = rem_base ? 1 : HKV;
        if (rc == NATSL_OK) rc = encode_bthd_map(&mkr, k_rem, B_rem, rt, rh, DK, 64, "natsl_attn_fwd(k_rem)");
        if (rc == NATSL_OK) rc = encode_bthd_map(&mvr, v_rem, B_rem, rt, rh, DV, 64, "natsl_attn_fwd(v_rem)");
    } else {
        mkr = mk;
        mvr = mv;
        B_rem = B;
    }
    int* status = nullptr;
    if (rc == NATSL_OK) rc = status_word_ptr(&status);
    if (rc != NATSL_OK) return rc;
    const int TN = (T + nbs - 1) / nbs;
    Order od;
    od.n_heads = HQ * B;
    od.q_per_kv = HQ / HKV;
    od.q_per_sel = HQ / HN;
    od.rem_segments = k_split > 0 && rem_base ? k_split / (rem_slots * nbs) : 0;
    // The two tiles of an item share the loads of keys and values; where all tiles together do not even fill the SMs once, each
    // gets an SM of its own (128 tiles of 128/128, T = 1024: 15.1 us, 18.9 us in pairs; 64 tiles, T = 512: 11.1 and 12.8).  Up to
    // 222 tiles that would still be faster for this kernel alone (192 tiles, T = 2048: 20.2 against 25.2 us), but it holds SMs that
    // the linear branch beside it waits for: the op at B = 1, T = 2048, 12 heads of 128/128 takes 73.8 instead of 66.5 us.
    // Against CTAs of half an SM (the kernel before), alone, speeds are 0.92 - 1.18 x up to 148 tiles, 0.85 - 1.30 x up to 320 and
    // 1.0 - 1.4 x beyond; whole layers of 64 to 12000 tokens, captured, are 1.04 - 1.22 x as fast.
    const int n_tiles = (Tq + ATT_BM - 1) / ATT_BM;
    od.split = (long)n_tiles * od.n_heads <= AT_SMS;
    od.n_blocks = od.split ? n_tiles : (Tq + AT_ITEM - 1) / AT_ITEM;
    od.group = (uint32_t)std::max<long>(1, std::min<long>(od.n_heads, AT_GROUP_BYTES / ((long)T * (DK + DV) * 2)));
    NATSL_REQUIRE((long)od.n_blocks * (long)od.n_heads <= 0x7fffffffL, NATSL_ERR_TOO_LARGE, "natsl_attn_fwd: too many query tiles");
    kern<<<od.n_blocks * od.n_heads, AT_THREADS, L::total, st>>>(
        mq, mk, mv, mkr, mvr, k_split, B_rem, k_split > 0 ? rem_base : nullptr, rem_slots, types_i, indices, n_iters,
        reinterpret_cast<__nv_bfloat16*>(o), lse, T, Tq, q_off, HQ, HKV, HN, TN, nbs, scale * 1.44269504f, own_chunk, od, status);
    return check_launch("natsl_attn_fwd");
}

}  // namespace
}  // namespace natsl

extern "C" int natsl_attn_fwd_split(const void* q, const void* k_rem, const void* v_rem, const int32_t* rem_base,
                                    int rem_slots, int rem_tokens, const void* k, const void* v, const int32_t* types_i,
                                    const int32_t* indices, const int32_t* attn_n_iters, void* o, float* lse, int B,
                                    int B_rem, int T, int Tq, int q_off, int k_split, int HQ, int HKV, int HN, int DK,
                                    int DV, int nbs, float scale, int flags, void* stream) {
    using namespace natsl;
    NATSL_REQUIRE(q && k && v && types_i && indices && attn_n_iters && o && lse, NATSL_ERR_NULL,
                  "natsl_attn_fwd: null pointer");
    NATSL_REQUIRE(B > 0 && T > 0 && HQ > 0 && HKV > 0 && HN > 0 && HQ % HKV == 0 && HQ % HN == 0, NATSL_ERR_BAD_SHAPE,
                  "natsl_attn_fwd: bad shape B=%d T=%d HQ=%d HKV=%d HN=%d", B, T, HQ, HKV, HN);
    NATSL_REQUIRE(Tq > 0 && q_off >= 0 && q_off + Tq <= T, NATSL_ERR_BAD_SHAPE,
                  "natsl_attn_fwd: queries [%d, %d) do not lie inside the %d keys", q_off, q_off + Tq, T);
    NATSL_REQUIRE(HQ <= 65535 && B <= 65535, NATSL_ERR_TOO_LARGE, "natsl_attn_fwd: B and HQ must be <= 65535");
    NATSL_REQUIRE(nbs >= 64 && nbs % 64 == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_attn_fwd: nats_block_size must be a multiple of 64 (got %d)", nbs);
    NATSL_REQUIRE(q_off % 128 == 0 && q_off % nbs == 0, NATSL_ERR_UNSUPPORTED,
                  "natsl_attn_fwd: the query offset must be a multiple of 128 and of nats_block_size (got %d)", q_off);
    NATSL_REQUIRE(k_split >= 0 && k_split <= q_off && k_split % nbs == 0, NATSL_ERR_BAD_SHAPE,
                  "natsl_attn_fwd: the key split %d must be a multiple of nats_block_size and <= the query offset %d",
                  k_split, q_off);
    NATSL_REQUIRE(k_split == 0 || (k_rem && v_rem && B_rem > 0 && B % B_rem == 0), NATSL_ERR_BAD_SHAPE,
                  "natsl_attn_fwd: a key split needs k_rem, v_rem and a batch B_rem that divides B");
    NATSL_REQUIRE(k_split == 0 || !rem_base || (rem_slots > 0 && k_split % (rem_slots * nbs) == 0 && rem_tokens > 0),
                  NATSL_ERR_BAD_SHAPE, "natsl_attn_fwd: packed gathered keys need rem_slots dividing the key split");
    const int own = (flags & NATSL_FLAG_ATTN_OWN_CHUNK) ? 1 : 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (flags & NATSL_FLAG_ATTN_MMA_SYNC) {
        NATSL_REQUIRE(q_off == 0 && Tq == T && k_split == 0, NATSL_ERR_UNSUPPORTED,
                      "natsl_attn_fwd: the mma.sync comparison kernel has no query offset or key split");
        return attn_fwd_mma_sync(q, k, v, types_i, indices, attn_n_iters, o, lse, B, T, HQ, HKV, HN, DK, DV, nbs, scale,
                                 own, st);
    }
#define NATSL_ATT_ARGS                                                                                                 \
    q, k_rem, v_rem, k, v, rem_base, rem_slots, rem_tokens, types_i, indices, attn_n_iters, o, lse, B, B_rem, T, Tq, q_off, \
        k_split, HQ, HKV, HN, nbs, scale, own, st
#define NATSL_ATT_CASE(KK, VV) \
    if (DK == KK && DV == VV) return launch_attn_tc<KK, VV>(NATSL_ATT_ARGS);
    NATSL_ATT_CASE(64, 64)
    NATSL_ATT_CASE(64, 128)
    NATSL_ATT_CASE(128, 64)
    NATSL_ATT_CASE(128, 128)
#undef NATSL_ATT_CASE
#undef NATSL_ATT_ARGS
    set_error("natsl_attn_fwd: unsupported head dims DK=%d DV=%d (each 64 or 128)", DK, DV);
    return NATSL_ERR_UNSUPPORTED;
}

extern "C" int natsl_attn_fwd_ex(const void* q, const void* k, const void* v, const int32_t* types_i,
                                 const int32_t* indices, const int32_t* attn_n_iters, void* o, float* lse, int B,
                                 int T, int Tq, int q_off, int HQ, int HKV, int HN, int DK, int DV, int nbs, float scale,
                                 int flags, void* stream) {
    return natsl_attn_fwd_split(q, nullptr, nullptr, nullptr, 0, 0, k, v, types_i, indices, attn_n_iters, o, lse, B, B, T,
                                Tq, q_off, 0, HQ, HKV, HN, DK, DV, nbs, scale, flags, stream);
}

extern "C" int natsl_attn_fwd(const void* q, const void* k, const void* v, const int32_t* types_i,
                              const int32_t* indices, const int32_t* attn_n_iters, void* o, float* lse, int B, int T,
                              int HQ, int HKV, int HN, int DK, int DV, int nbs, float scale, int flags, void* stream) {
    return natsl_attn_fwd_ex(q, k, v, types_i, indices, attn_n_iters, o, lse, B, T, T, 0, HQ, HKV, HN, DK, DV, nbs, scale,
                             flags, stream);
}
