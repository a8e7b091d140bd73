// Dequant GEMM with exact-class operands on the 5th-generation tensor cores: y[m, n] = sum_k x[m, k] * W[n, k] (+ bias,
// + residual) from the tile-repacked ggml blocks (gemv_imma.cuh) for steps of DQ_MIN_M rows and more: batched decode,
// mixed steps, prompts.
//
// What is multiplied. Activation rows are scaled by a power of two into (-1, 1) and split into an fp16 leading part and the
// fp16 of what that rounding dropped (dq_rows.cu). Weights are never rounded:
//   Q4_K  w = d * (sc * q) - dmin * m. sc * q <= 945 is an exact fp16 integer: ONE operand plane, two products per column
//         (X_hi, X_lo). The minimum term is a product with the sums of 32 activations, see below.
//   Q6_K  w = d * (sc * (q - 32)), |sc * (q - 32)| <= 4096: two planes, the integer rounded to fp16 and the exact remainder.
//   Q8_0  w = d * q (19 bits): two planes, product rounded to fp16 and the exact remainder.
// Two planes take three products (W_hi X_hi, W_lo X_hi, W_hi X_lo). The tensor core sums 256 columns at a time; the block scale
// d is applied in f32 when a sum leaves tensor memory, so no f32 rounding chain is longer than that and the K-quant scales
// cost nothing per weight.
//
// Why this shape. What bounded the kernel that this one replaced was not the tensor pipe (13 % busy) nor DRAM (7 %) but its
// 16 producer warps: weights were rebuilt in f32 and split there, 376 warp instructions per 1024 weights, their raw words one
// register set ahead. Here a pair of 4-bit weights costs a mask and one half-pair multiply-add (about 60 instructions per 1024),
// and raw tiles arrive by bulk copies through a ring of up to 150 KB per SM, requested before the previous kernel has ended.
// A block owns 128 weight rows x up to 128 activation rows:
//   warp 0      one thread issues tcgen05.mma (A: weights in tensor memory, B: activations in shared memory)
//   warp 1      bulk copies of raw weight tiles; warp 2: TMA of activation boxes (64 columns, both planes) and 32-sums
//   warps 4-11  producers: a 16-row tile each, raw words -> fp16 planes -> tensor memory
//   warps 12-19 drains: after 256 columns a sum is read from tensor memory (two accumulator buffers), multiplied by d and
//               added to f32 registers; for Q4_K the minimum term m * (32-sums) is an mma.sync of 8 columns (leading parts and
//               remainders of the sums, minima exact) times dmin, which costs a quarter instruction per element.
// Columns are stored in the order 0 2 1 3 within groups of four, in activations and weights alike: the order in which masks
// pick bytes out of a word, so that no weight is moved.
// What holds it is the serial work of its single warps -- the one that issues the products, the one that asks for activations -- whose
// instructions wait for those of 16 busy others: copies of activations are one box for both planes and all columns of a stage (four at
// 32 rows before), roles branch on a warp number that is uniform to the compiler, and drains take the minimum term before
// they wait for the sums. Q4_K 28672 x 4096 32 rows 48.5 -> 39.5 us, 128 rows 70.5 -> 67.3, 512 rows 214 -> 208; Q6_K 4096 x 14336 37 rows
// 31.0 -> 29.3; Q4_K 17920 x 1536 192 rows 29.7 -> 28.0; Q8_0 28672 x 4096 32 rows 49.8 -> 48.5, 10240 x 2560 389 rows 60.2 -> 60.0.
// Without effect: a second group of eight producers, two warps that issue products for accumulators in turn, a ring of 3 or 5
// activation stages instead of 4, waits that ask without looking first.
// Error against float64 at K = 14336: 5e-7.
// The K range of a tile is shared by the blocks of a cluster when tiles alone leave SMs idle; they meet in distributed shared
// memory and add in part order, so results do not vary from run to run. Every wait on an mbarrier is bounded; after one that ran out
// nothing more is issued, the warps that did issue wait (bounded) for their copies and products in flight, y is left alone.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "gemv_imma.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "plan_common.cuh"
#include "sp_common.cuh"
#include "tc5_ptx.cuh"

namespace sp {

cudaError_t count_launch_and_check();  // kernels.cu

constexpr int DQ_THREADS = 640;
constexpr int DQ_PRODUCERS = 8, DQ_FIRST_PRODUCER = 4, DQ_DRAINS = 8, DQ_FIRST_DRAIN = 12;
constexpr int DQ_BM = 128;                 // weight rows per block
constexpr int DQ_NB = 128;                 // activation rows per block at most
constexpr int DQ_A_SLOTS = 4;              // weight slots in tensor memory, 64 columns each: 128 columns of K of one plane (a half);
                                           // two planes take a pair of slots and go by the second one's barriers
constexpr int DQ_A_COL = 2 * DQ_NB;        // tensor memory: two accumulators of DQ_NB columns, then the weight stages
constexpr int DQ_MAX_B = 8, DQ_MAX_R = 8, DQ_X_STAGES = 3;
constexpr int DQ_SMEM = 224 * 1024;
constexpr int DQ_MAX_PARTS = 8;
constexpr int DQ_P_STRIDE = DQ_BM + 4;     // floats between the columns of a partial tile: no bank conflicts

constexpr int T_Q8_0_HALF = 1000 + T_Q8_0;  // Q8_0 whose width is an odd multiple of 128: tiles of four blocks

struct DqArgs {
    Tc5Seg seg[3];
    int nseg, k, m, ldy;
    const float* res;      // [m][ldres] or null, added to segment 0 (may alias its y)
    int ldres;
    int m_tiles, nb;       // row tiles, rows per tile (a multiple of 16)
    int item0, items;      // tiles of this launch: item0 .. items - 1
    int parts;             // blocks of the cluster that share a tile's K range
    int b_stages, r_stages, r_bytes;  // depth of the activation ring, of the raw ring, bytes of a raw stage
    const float* xscale;   // [m]
    const __half* xsum;    // [k / 256][m][16]: sums of 32 columns as dq_rows.cu leaves them
    int* waits;            // WaitFlags of the launch's owner
};

__device__ __forceinline__ void dq_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 lanes x 32 columns of tensor memory from a warp: words 4 i .. 4 i + 3 of lane (g, t) are columns 8 i + 2 t, + 1 of lanes g
// (first two) and g + 8.
__device__ __forceinline__ void dq_st(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr), "r"(v[0]),
        "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
        "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

// 16 lanes x 8 (16) columns, in the layout of an mma accumulator fragment.
__device__ __forceinline__ void dq_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void dq_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void dq_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Boxes of 64 columns, leading parts and remainders of the rows from m0 on, one after the other: [box][plane][row][64].
__device__ __forceinline__ void dq_box(uint32_t dst, const CUtensorMap* map, int m0, int box, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %2, %4}], [%5];\n" ::"r"(dst), "l"(map), "r"(0),
        "r"(m0), "r"(box), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void dq_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dq_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(tc5_smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ __half2 dq_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t dq_u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 dq_const(float f) { return __float2half2_rn(f); }
__device__ __forceinline__ uint32_t dq_word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// Byte b of v twice, as the half pair (1024 + byte, 1024 + byte).
__device__ __forceinline__ __half2 dq_twice(uint32_t v, int b) { return dq_h2(__byte_perm(v, 0x64646464u, 0x4040 | (b << 8) | b)); }

// The eight 6-bit scales (minima) of a Q4_K block header, one per byte.
__device__ __forceinline__ void q4k_scales(const uint4& hd, uint32_t& lo, uint32_t& hi) {
    lo = hd.y & 0x3F3F3F3Fu;
    hi = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
}
__device__ __forceinline__ void q4k_minima(const uint4& hd, uint32_t& lo, uint32_t& hi) {
    lo = hd.z & 0x3F3F3F3Fu;
    hi = ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
}

// bytes of one 16-row tile's 256 columns
__host__ __device__ constexpr int dq_tile_bytes(int dt) { return dt == T_Q4_K ? Q4_K_TILE_BYTES : dt == T_Q6_K ? Q6_K_TILE_BYTES : 8 * 544; }

// A 16-row tile's weights, 128 columns (a half) at a time: the words of a half are read from shared memory together, then turned
// into operands 64 columns at a time. o is the operand plane (of two planes the leading parts), ol the remainders; words
// 4 c .. 4 c + 3 are lane (g, t)'s columns 16 c + 4 t .. + 3 of rows g and g + 8.
template <int DT>
struct DqTile {
    const uint8_t* tile;   // in shared memory
    int lane;
    uint4 hd[2];           // Q4_K, Q6_K: headers of rows g, g + 8
    uint4 q[4];            // the half's words: Q4_K 2, Q6_K 3, Q8_0 4 pieces
    uint2 d8[2];           // Q8_0: the half's four scales of rows g, g + 8
    __device__ __forceinline__ DqTile(const uint8_t* tile_, int lane_) : tile(tile_), lane(lane_) {
        const int g = lane >> 2;
        constexpr int AT = DT == T_Q4_K ? 2048 : 3072;
        if (DT == T_Q4_K || DT == T_Q6_K) {
            hd[0] = *reinterpret_cast<const uint4*>(tile + AT + g * 16);
            hd[1] = *reinterpret_cast<const uint4*>(tile + AT + (g + 8) * 16);
        }
    }
    __device__ __forceinline__ void load(int half) {
        constexpr int N = DT == T_Q4_K ? 2 : DT == T_Q6_K ? 3 : 4;
        const uint8_t* at = tile + (DT == T_Q8_0_HALF ? half * 2176 : half * N * 512) + lane * 16;
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = *reinterpret_cast<const uint4*>(at + i * 512);
        if (DT == T_Q8_0 || DT == T_Q8_0_HALF) {
            const uint8_t* ds = DT == T_Q8_0 ? tile + 4096 + half * 8 : tile + half * 2176 + 2048;
            constexpr int PITCH = DT == T_Q8_0 ? 16 : 8;
            d8[0] = *reinterpret_cast<const uint2*>(ds + (lane >> 2) * PITCH);
            d8[1] = *reinterpret_cast<const uint2*>(ds + ((lane >> 2) + 8) * PITCH);
        }
    }
    // columns 128 half + 64 e .. + 63
    __device__ __forceinline__ void group(int half, int e, uint32_t (&o)[16], uint32_t (&ol)[16]) {
        if (DT == T_Q4_K) {
            const uint4 w = q[e];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                uint32_t lo, hi;
                q4k_scales(hd[r], lo, hi);
                const uint32_t sc = half ? hi : lo;
                // low nibbles: (1024 + q) sc - 1024 sc; high nibbles stand 16 times higher: (1024 + 16 q) sc / 16 - 64 sc. Both exact.
                const __half2 s0 = __hadd2(dq_twice(sc, 2 * e), dq_const(-1024.f));
                const __half2 s1 = __hfma2(dq_twice(sc, 2 * e + 1), dq_const(0.0625f), dq_const(-64.f));
                const __half2 c0 = __hmul2(s0, dq_const(-1024.f)), c1 = __hmul2(s1, dq_const(-1024.f));
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t v = dq_word(w, 2 * r + h), v8 = v >> 8;
                    o[4 * h + 2 * r] = dq_u(__hfma2(dq_h2((v & 0x000F000Fu) | 0x64006400u), s0, c0));
                    o[4 * h + 2 * r + 1] = dq_u(__hfma2(dq_h2((v8 & 0x000F000Fu) | 0x64006400u), s0, c0));
                    o[8 + 4 * h + 2 * r] = dq_u(__hfma2(dq_h2((v & 0x00F000F0u) | 0x64006400u), s1, c1));
                    o[8 + 4 * h + 2 * r + 1] = dq_u(__hfma2(dq_h2((v8 & 0x00F000F0u) | 0x64006400u), s1, c1));
                }
            }
        } else if (DT == T_Q6_K) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t sw = dq_word(hd[r], 2 * half + e) ^ 0x80808080u;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const int base = 6 * p + 3 * r;
                    const uint32_t qh = dq_word(q[(base + 2) >> 2], (base + 2) & 3);
#pragma unroll
                    for (int ab = 0; ab < 2; ++ab) {
                        const uint32_t ql = dq_word(q[(base + ab) >> 2], (base + ab) & 3);
                        const int quarter = 2 * e + ab;
                        const uint32_t top = quarter == 0 ? qh << 4 : quarter == 1 ? qh << 2 : quarter == 2 ? qh : qh >> 2;
                        const uint32_t v = ((e ? ql >> 4 : ql) & 0x0F0F0F0Fu) | (top & 0xF0F0F0F0u);
                        const __half2 sc = __hadd2(dq_twice(sw, 2 * ab + p), dq_const(-1152.f));
                        const __half2 a = __hadd2(dq_h2((v & 0x003F003Fu) | 0x64006400u), dq_const(-1056.f));
                        const __half2 b = __hadd2(dq_h2(((v >> 8) & 0x003F003Fu) | 0x64006400u), dq_const(-1056.f));
                        const __half2 ah = __hmul2_rn(a, sc), bh = __hmul2_rn(b, sc);
                        const int c = 4 * (2 * ab + p) + 2 * r;
                        o[c] = dq_u(ah);
                        o[c + 1] = dq_u(bh);
                        ol[c] = dq_u(__hfma2(a, sc, __hneg2(ah)));
                        ol[c + 1] = dq_u(__hfma2(b, sc, __hneg2(bh)));
                    }
                }
            }
        } else {
#pragma unroll
            for (int blk = 0; blk < 2; ++blk) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t dw = e ? d8[r].y : d8[r].x;
                    const __half2 d = dq_h2(__byte_perm(dw, 0u, blk ? 0x3232 : 0x1010));
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t v = dq_word(q[2 * e + blk], 2 * r + h);
                        const __half2 a = __hadd2(dq_h2((v & 0x00FF00FFu) ^ 0x64806480u), dq_const(-1152.f));
                        const __half2 b = __hadd2(dq_h2(((v >> 8) & 0x00FF00FFu) ^ 0x64806480u), dq_const(-1152.f));
                        const __half2 ah = __hmul2_rn(a, d), bh = __hmul2_rn(b, d);
                        const int c = 4 * (2 * blk + h) + 2 * r;
                        o[c] = dq_u(ah);
                        o[c + 1] = dq_u(bh);
                        ol[c] = dq_u(__hfma2(a, d, __hneg2(ah)));
                        ol[c + 1] = dq_u(__hfma2(b, d, __hneg2(bh)));
                    }
                }
            }
        }
    }
};

struct DqBars {
    uint64_t full_r[DQ_MAX_R], empty_r[DQ_MAX_R], full_a[DQ_A_SLOTS], empty_a[DQ_A_SLOTS], full_b[DQ_MAX_B], empty_b[DQ_MAX_B];
    uint64_t full_x[DQ_X_STAGES], empty_x[DQ_X_STAGES], full_d[2], empty_d[2], idle;
};

// Where a warp stands in a ring of `n` stages: the stage and how often the ring has wrapped. Carried from tile to tile.
struct DqRing {
    int st = 0;
    uint32_t u = 0;
    __device__ __forceinline__ void next(int n) {
        if (++st == n) { st = 0; ++u; }
    }
    __device__ __forceinline__ bool full(uint64_t* bars) const { return tc5_wait(&bars[st], u & 1); }
    __device__ __forceinline__ bool empty(uint64_t* bars) const { return u == 0 || tc5_wait(&bars[st], (u - 1) & 1); }
};

// A producer warp's walk over the block's K range, a half (128 columns) at a time; all eight warps fill a slot or a pair.
template <int DT>
__device__ __forceinline__ bool dq_produce(DqBars& bars, const uint8_t* raw, int r_bytes, int r_stages, int tile_w, int lane, uint32_t a_base, int n_sb,
                                           int halves_last, DqRing& rr, DqRing& ra, bool ok) {
    constexpr bool TWO = DT != T_Q4_K;
    for (int sb = 0; sb < n_sb; ++sb) {
        ok = ok && rr.full(bars.full_r);
        DqTile<DT> t(raw + (size_t)rr.st * r_bytes + tile_w * dq_tile_bytes(DT), lane);
        const int halves = DT == T_Q8_0_HALF && sb == n_sb - 1 ? halves_last : 2;
        t.load(0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (DT == T_Q8_0_HALF && h >= halves) break;
            const uint32_t at = a_base + 64u * (uint32_t)ra.st;
            uint32_t o[16], o1[16];
            t.group(h, 0, o, o1);
            if (!TWO) t.group(h, 1, o1, o1);
            if (TWO) ra.next(DQ_A_SLOTS);  // (a pair's second slot)
            ok = ok && ra.empty(bars.empty_a);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            dq_st(at, o);
            dq_st(at + (TWO ? 64u : 32u), o1);
            if (TWO) {
                t.group(h, 1, o, o1);
                dq_st(at + 32u, o);
                dq_st(at + 96u, o1);
            }
            if (h + 1 < halves) {
                t.load(1);
            } else {  // the raw words have been read
                __syncwarp();
                if (lane == 0) tc5_arrive(&bars.empty_r[rr.st]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (TWO) tc5_arrive(&bars.full_a[ra.st - 1]);
                tc5_arrive(&bars.full_a[ra.st]);
            }
            ra.next(DQ_A_SLOTS);
        }
        rr.next(r_stages);
    }
    return ok;
}

// Tiles of up to 64 activation rows have both planes of the activations side by side in one product (its N is twice the rows) and
// in the accumulator; the drain adds them. Wider tiles multiply the planes one after the other into the same columns.
constexpr int DQ_SIDE_NJT = 4;
// 64-column boxes of an activation stage: two, so that there are fewer hand-overs; one for tall tiles, whose boxes of up to 32 KB
// would leave a ring of two stages.
__host__ __device__ constexpr int dq_boxes(int njt) { return njt <= DQ_SIDE_NJT ? 2 : 1; }

// A drain warp's walk: acc[tile][j] holds rows 16 tile + g (+ 8) of the warp's 32, columns 8 j + 2 t (+ 1) of its NJT 8-column tiles.
template <int DT, int NJT>
__device__ __forceinline__ bool dq_drain(DqBars& bars, const uint8_t* raw, int r_bytes, int r_stages, const uint8_t* xs, int x_bytes, int plane, int quarter,
                                         int half, int lane, uint32_t tmem, int n_sb, DqRing& rr, DqRing& rx, DqRing& rd, float (&acc)[2][NJT][4], bool ok) {
    constexpr bool SIDE = NJT <= DQ_SIDE_NJT;
    const int g = lane >> 2, t = lane & 3;
    for (int sb = 0; sb < n_sb; ++sb) {
        float d[2][2], dm[2][2];
        uint32_t mn[2][2];
        ok = ok && rr.full(bars.full_r);
        if (DT == T_Q4_K || DT == T_Q6_K) {
            const uint8_t* base = raw + (size_t)rr.st * r_bytes + 2 * quarter * dq_tile_bytes(DT);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint8_t* tile = base + i * dq_tile_bytes(DT);
                    if (DT == T_Q4_K) {
                        const uint4 hd = *reinterpret_cast<const uint4*>(tile + 2048 + (g + 8 * r) * 16);
                        d[i][r] = __low2float(dq_h2(hd.x));
                        dm[i][r] = -__high2float(dq_h2(hd.x));
                        uint32_t lo, hi;
                        q4k_minima(hd, lo, hi);
                        // minima 2 t, 2 t + 1 as a half pair
                        const uint32_t two = __byte_perm(t < 2 ? lo : hi, 0x64646464u, (t & 1) ? 0x4342 : 0x4140);
                        mn[i][r] = dq_u(__hadd2(dq_h2(two), dq_const(-1024.f)));
                    } else {
                        d[i][r] = __half2float(*reinterpret_cast<const __half*>(tile + 3328 + 2 * (g + 8 * r)));
                    }
                }
        }
        __syncwarp();
        if (lane == 0) tc5_arrive(&bars.empty_r[rr.st]);
        rr.next(r_stages);
        // (the warp's verdict, not each lane's: what it guards is an instruction of the whole warp)
        if (DT == T_Q4_K) ok = __all_sync(0xFFFFFFFFu, ok && rx.full(bars.full_x));
        const uint8_t* xrow = xs + (size_t)rx.st * x_bytes + (half * NJT * 8 + g) * 32 + t * 8;
        if (DT == T_Q4_K && ok) {
#pragma unroll
            for (int j = 0; j < NJT; ++j) {
                const uint2 x = *reinterpret_cast<const uint2*>(xrow + j * 256);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float p[4];
                    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%4,%5}, {%6,%7}, {%8,%8,%8,%8};\n"
                        : "=f"(p[0]), "=f"(p[1]), "=f"(p[2]), "=f"(p[3])
                        : "r"(mn[i][0]), "r"(mn[i][1]), "r"(x.x), "r"(x.y), "f"(0.f));
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][j][e] = fmaf(dm[i][e >> 1], p[e], acc[i][j][e]);
                }
            }
        }
        ok = ok && rd.full(bars.full_d);
        ok = __all_sync(0xFFFFFFFFu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t from = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(rd.st * DQ_NB + half * NJT * 8);
        // batches of two 8-column tiles, the next one requested before the current one is added
        constexpr int NB2 = NJT >= 2 ? NJT / 2 : 1, W = NJT >= 2 ? 2 : 1, PL = SIDE ? 2 : 1;
        uint32_t v[2][PL][4 * W];
        auto fetch = [&](int b, uint32_t (&dst)[PL][4 * W]) {
#pragma unroll
            for (int p = 0; p < PL; ++p) {
                const uint32_t a = from + ((uint32_t)(16 * (b / NB2)) << 16) + (uint32_t)((b % NB2) * 8 * W + p * plane);
                if (W == 2) dq_ld16(a, dst[p]);
                else dq_ld8(a, dst[p]);
            }
        };
        fetch(0, v[0]);
#pragma unroll
        for (int b = 0; b < 2 * NB2; ++b) {
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            uint32_t(&c)[PL][4 * W] = v[b & 1];
#pragma unroll
            for (int e = 0; e < PL * 4 * W; ++e) asm volatile("" : "+r"(c[e / (4 * W)][e % (4 * W)]));  // not to be used before the wait
            if (b + 1 < 2 * NB2) fetch(b + 1, v[(b + 1) & 1]);
            const int i = b / NB2;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                float* const a = acc[i][(b % NB2) * W + w];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float f = __uint_as_float(c[0][4 * w + e]);
                    if (SIDE) f += __uint_as_float(c[PL - 1][4 * w + e]);
                    a[e] = DT == T_Q4_K || DT == T_Q6_K ? fmaf(d[i][e >> 1], f, a[e]) : a[e] + f;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            tc5_arrive(&bars.empty_d[rd.st]);
            if (DT == T_Q4_K) tc5_arrive(&bars.empty_x[rx.st]);
        }
        rd.next(2);
        if (DT == T_Q4_K) rx.next(DQ_X_STAGES);
    }
    return ok;
}

// The MMA warp's walk, an activation stage (BOXES boxes of 64 columns) at a time. The whole warp takes part and one elected thread
// issues: control flow and operands are uniform then, as the tensor instructions want them. Issuing is the serial part of the
// pipeline (a wait that is already over costs 100 to 250 cycles on a busy SM), so the barriers of the next stage are looked at ahead of
// a stage's products and only waited for if they were not over by then; with two weight planes half of the products go first, so
// that the tensor pipe has work under the looks (Q8_0 28672 x 4096, 96 rows 84 -> 79 us; with one plane it costs 2 %).
template <bool TWO, bool SIDE, int BOXES>
__device__ __forceinline__ bool dq_issue(DqBars& bars, uint32_t tm, uint64_t bd0, uint32_t b16, int b_stages, uint32_t idesc, uint32_t idesc_side, int n_sb,
                                         int halves_last, bool leader, DqRing& ra, DqRing& rb, DqRing& rd, bool& seen, bool ok) {
    constexpr int STEPS = 2 / BOXES;  // activation stages of a half
    const uint32_t box16 = b16 / BOXES, plane16 = box16 >> 1;  // a box of 64 columns: both planes
    for (int sb = 0; sb < n_sb; ++sb) {
        const int halves = sb == n_sb - 1 ? halves_last : 2;
        for (int h = 0; h < halves; ++h) {
            const uint32_t At = tm + (uint32_t)DQ_A_COL + 64u * (uint32_t)ra.st;
            if (TWO) ra.next(DQ_A_SLOTS);  // (a pair's second slot)
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const bool first = h == 0 && s == 0, a_last = s == STEPS - 1, last = a_last && h == halves - 1;
                if (!seen && ok) {
                    bool w = true;
                    if (first) w = rd.empty(bars.empty_d);
                    if (s == 0) w = w && ra.full(bars.full_a);
                    w = w && rb.full(bars.full_b);
                    ok = __all_sync(0xFFFFFFFFu, w);
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t dt = tm + (uint32_t)(rd.st * DQ_NB);
                const uint64_t b0 = bd0 + (uint64_t)((uint32_t)rb.st * b16);  // (the address field: no carry out of the low word)
                uint64_t* const e_b = &bars.empty_b[rb.st];
                uint64_t* const e_a = &bars.empty_a[ra.st];
                uint64_t* const f_d = &bars.full_d[rd.st];
                rb.next(b_stages);
                if (a_last) ra.next(DQ_A_SLOTS);
                if (last) rd.next(2);
                auto multiply = [&](int from, int to) {
#pragma unroll
                    for (int i = from; i < to; ++i) {
                        const uint32_t more = i > 0 || s > 0 ? 1u : (uint32_t)(h > 0), Ai = At + 32u * s + 8u * i;
                        const uint64_t bh = b0 + (i >> 2) * box16 + 2u * (i & 3);
                        if (SIDE) {
                            dq_mma(dt, Ai, bh, idesc_side, more);                  // W [X_hi | X_lo]
                        } else {
                            dq_mma(dt, Ai, bh + plane16, idesc, more);             // W X_lo
                            dq_mma(dt, Ai, bh, idesc, 1u);                         // W X_hi
                        }
                        if (TWO) dq_mma(dt, Ai + 64u, bh, idesc, 1u);              // W_lo X_hi
                    }
                };
                constexpr int AHEAD = TWO ? 2 * BOXES : 0;  // columns / 16 multiplied before the looks
                if (AHEAD > 0 && leader && ok) multiply(0, AHEAD);
                bool next = tc5_peek(&bars.full_b[rb.st], rb.u & 1);
                // (where the next tile's format is another one, the other slot of the pair says the same: slots are filled in order)
                if (a_last) next = tc5_peek(&bars.full_a[ra.st + (TWO ? 1 : 0)], ra.u & 1) && next;
                if (last && rd.u > 0) next = tc5_peek(&bars.empty_d[rd.st], (rd.u - 1) & 1) && next;
                if (leader && ok) {
                    multiply(AHEAD, 4 * BOXES);
                    tc5_commit(e_b);
                    if (a_last) {
                        if (TWO) tc5_commit(e_a - 1);
                        tc5_commit(e_a);
                    }
                    if (last) tc5_commit(f_d);
                }
                seen = __all_sync(0xFFFFFFFFu, next);
            }
        }
    }
    return ok;
}

// The end of a tile: a lane's rows of y (row0, + 1, + 8, ..; left of them are there) at the columns n, + 8, + 16, + 24. Short straight
// code: all that a warp does once per tile is fetched from far away, an instruction in some ten cycles, and with an address and
// two bounds for each value a tile's end took 10 000 cycles (96 rows), twice what the two accumulators bridge (in shared memory first,
// for stores of 128 bytes, it took as long). Q8_0 17920 x 1536, 192 rows 41.4 -> 33.7 us, 512 rows 80 -> 68.
template <int NJT, bool WHOLE, bool RES>
__device__ __forceinline__ void dq_store(const float (&acc)[2][NJT][4], const DqArgs& a, const Tc5Seg& sg, int64_t row0, int left, int n) {
    float bias[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) bias[i] = sg.bias && (WHOLE || n + 8 * i < sg.n) ? sg.bias[n + 8 * i] : 0.f;
    const float* xs = a.xscale + row0;
    float sc[2 * NJT];  // (ahead of the stores, which the compiler takes for possible changes of them)
#pragma unroll
    for (int j = 0; j < 2 * NJT; ++j) sc[j] = (j >> 1) * 8 + (j & 1) < left ? xs[(j >> 1) * 8 + (j & 1)] : 0.f;
    float* y = sg.y + row0 * a.ldy + n;
    const float* r = RES ? a.res + row0 * a.ldres + n : nullptr;
#pragma unroll
    for (int j = 0; j < 2 * NJT; ++j) {
        if ((j >> 1) * 8 + (j & 1) < left) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = fmaf(acc[i >> 1][j >> 1][2 * (i & 1) + (j & 1)], sc[j], bias[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (RES && (WHOLE || n + 8 * i < sg.n)) v[i] += r[8 * i];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (WHOLE || n + 8 * i < sg.n) y[8 * i] = v[i];
        }
        y += (j & 1) ? 7 * (int64_t)a.ldy : (int64_t)a.ldy;
        if (RES) r += (j & 1) ? 7 * (int64_t)a.ldres : (int64_t)a.ldres;
    }
}

// Which matrix and rows a tile is.
struct DqItem {
    int si, dt, n0, m0, rows;
    __device__ __forceinline__ DqItem(const DqArgs& a, int item) {
        int bx = item / a.m_tiles;
        si = 0;
        while (si < a.nseg - 1 && bx >= (a.seg[si].n + DQ_BM - 1) / DQ_BM) { bx -= (a.seg[si].n + DQ_BM - 1) / DQ_BM; ++si; }
        dt = (a.seg[si].dtype == T_Q8_0 && (a.k & 255)) ? T_Q8_0_HALF : a.seg[si].dtype;
        n0 = bx * DQ_BM;
        m0 = (item % a.m_tiles) * a.nb;
        rows = min(a.nb, a.m - m0);
    }
};

// NJT: 8-column tiles of activation rows per drain warp; a tile's rows are at most 16 NJT. A block takes tiles blockIdx.x,
// blockIdx.x + gridDim.x, ..; its warps run from one into the next (the epilogue of a tile under the products of the next one).
template <int NJT>
__global__ void __launch_bounds__(DQ_THREADS, 1) gemm_dq_kernel(const DqArgs a, const __grid_constant__ CUtensorMap tmap_x) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) DqBars bars;
    __shared__ uint32_t tmem_slot;
    constexpr bool SIDE = NJT <= DQ_SIDE_NJT;
    constexpr int BOXES = dq_boxes(NJT);
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    uint8_t* smem = smem_raw + ((1024u - (tc5_smem_u32(smem_raw) & 1023u)) & 1023u);
    const int all_sb = (a.k + 255) / 256, part = blockIdx.z;
    const int sb0 = part * all_sb / a.parts, n_sb = (part + 1) * all_sb / a.parts - sb0;
    const int halves_last = min(2, (a.k - (sb0 + n_sb - 1) * 256) / 128);  // 128-column halves of this block's last 256 columns
    const int b_bytes = BOXES * 2 * a.nb * 128, x_bytes = a.nb * 32;
    uint8_t* const xs = smem + (size_t)a.b_stages * b_bytes;
    uint8_t* const raw = xs + DQ_X_STAGES * x_bytes;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(tc5_smem_u32(&tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 32) {
        tc5_prefetch_map(&tmap_x);
        for (int s = 0; s < a.r_stages; ++s) { dq_init(&bars.full_r[s], 1); dq_init(&bars.empty_r[s], DQ_PRODUCERS + DQ_DRAINS); }
        for (int s = 0; s < DQ_A_SLOTS; ++s) { dq_init(&bars.full_a[s], DQ_PRODUCERS); dq_init(&bars.empty_a[s], 1); }
        for (int s = 0; s < a.b_stages; ++s) { dq_init(&bars.full_b[s], 1); dq_init(&bars.empty_b[s], 1); }
        for (int s = 0; s < DQ_X_STAGES; ++s) { dq_init(&bars.full_x[s], 1); dq_init(&bars.empty_x[s], DQ_DRAINS); }
        for (int s = 0; s < 2; ++s) { dq_init(&bars.full_d[s], 1); dq_init(&bars.empty_d[s], DQ_DRAINS); }
        dq_init(&bars.idle, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_slot, 0);

    bool ok = true;
    if (warp < DQ_FIRST_PRODUCER) {
        if (NJT >= 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");  // 128 x 32 + 256 x 96 + 256 x 128 = 640 x 96
        if (warp == 1) {
            if (lane == 0) {
                // raw tiles: weights, which no kernel writes, so they are requested before the previous kernel has ended
                DqRing r;
                int issued = 0;
                for (int item = a.item0 + blockIdx.x; item < a.items && ok; item += gridDim.x) {
                    const DqItem it(a, item);
                    const int tb = dq_tile_bytes(it.dt), live = min(8, ((a.seg[it.si].n + 15) >> 4) - (it.n0 >> 4));
                    const int64_t row_bytes = (int64_t)(a.k >> 7) * (tb >> 1);
                    const uint8_t* src = a.seg[it.si].wt + (int64_t)(it.n0 >> 4) * row_bytes + (int64_t)sb0 * tb;
                    for (int sb = 0; sb < n_sb; ++sb) {
                        ok = r.empty(bars.empty_r);
                        if (!ok) break;
                        const uint32_t bytes = sb == n_sb - 1 ? (uint32_t)(tb / 2 * halves_last) : (uint32_t)tb;
                        const uint32_t bar = tc5_smem_u32(&bars.full_r[r.st]), dst = tc5_smem_u32(raw + (size_t)r.st * a.r_bytes);
                        dq_expect(bar, bytes * live);
                        for (int i = 0; i < live; ++i) dq_bulk(dst + i * tb, src + i * row_bytes + (int64_t)sb * tb, bytes, bar);
                        r.next(a.r_stages);
                        ++issued;
                    }
                }
                // (all copies land before the block ends, whatever became of their readers)
                for (int i = max(0, issued - a.r_stages); i < issued; ++i) ok = tc5_wait(&bars.full_r[i % a.r_stages], (uint32_t)((i / a.r_stages) & 1)) && ok;
            }
            __syncwarp();
            pdl_wait();
        } else {
            pdl_wait();
            pdl_trigger();
        }
        if (warp == 2 && lane == 0) {
            DqRing r, rx;
            int boxes = 0, sums = 0;
            for (int item = a.item0 + blockIdx.x; item < a.items && ok; item += gridDim.x) {
                const DqItem it(a, item);
                for (int sb = 0; sb < n_sb && ok; ++sb) {
                    const int steps = 2 / BOXES * (sb == n_sb - 1 ? halves_last : 2);
                    for (int h = 0; h < steps; ++h) {
                        ok = r.empty(bars.empty_b);
                        if (!ok) break;
                        const uint32_t bar = tc5_smem_u32(&bars.full_b[r.st]), dst = tc5_smem_u32(smem + (size_t)r.st * b_bytes);
                        dq_expect(bar, (uint32_t)b_bytes);
                        dq_box(dst, &tmap_x, it.m0, (sb0 + sb) * 4 + BOXES * h, bar);
                        r.next(a.b_stages);
                        ++boxes;
                    }
                    if (it.dt == T_Q4_K && ok) {
                        ok = rx.empty(bars.empty_x);
                        if (!ok) break;
                        const uint32_t bar = tc5_smem_u32(&bars.full_x[rx.st]);
                        dq_expect(bar, (uint32_t)(it.rows * 32));
                        dq_bulk(tc5_smem_u32(xs + rx.st * x_bytes), a.xsum + ((int64_t)(sb0 + sb) * a.m + it.m0) * 16, (uint32_t)(it.rows * 32), bar);
                        rx.next(DQ_X_STAGES);
                        ++sums;
                    }
                }
            }
            for (int i = max(0, boxes - a.b_stages); i < boxes; ++i) ok = tc5_wait(&bars.full_b[i % a.b_stages], (uint32_t)((i / a.b_stages) & 1)) && ok;
            for (int i = max(0, sums - DQ_X_STAGES); i < sums; ++i) ok = tc5_wait(&bars.full_x[i % DQ_X_STAGES], (uint32_t)((i / DQ_X_STAGES) & 1)) && ok;
        } else if (warp == 0) {
            const bool leader = tc5_elect();
            // fp16 x fp16 -> f32; N is the tile height, twice that where both planes stand side by side
            const uint32_t idesc = (1u << 4) | ((uint32_t)(a.nb >> 3) << 17) | ((uint32_t)(DQ_BM >> 4) << 24), idesc_side = idesc + ((uint32_t)(a.nb >> 3) << 17);
            const uint64_t bd0 = tc5_desc(tc5_smem_u32(smem));
            DqRing ra, rb, rd;
            bool seen = false;
            for (int item = a.item0 + blockIdx.x; item < a.items; item += gridDim.x) {
                const DqItem it(a, item);
#define SP_DQ_ISSUE(TWO) \
    ok = dq_issue<TWO, SIDE, BOXES>(bars, tmem, bd0, (uint32_t)b_bytes >> 4, a.b_stages, idesc, idesc_side, n_sb, halves_last, leader, ra, rb, rd, seen, ok)
                if (it.dt == T_Q4_K) SP_DQ_ISSUE(false);
                else SP_DQ_ISSUE(true);
#undef SP_DQ_ISSUE
            }
            if (!ok && leader) {  // what has been issued reads shared and writes tensor memory
                tc5_commit(&bars.idle);
                tc5_wait(&bars.idle, 0);
            }
        }
        __syncwarp();
        if (a.parts > 1) { cluster_sync(); cluster_sync(); }
    } else if (warp < DQ_FIRST_DRAIN) {  // (reads and writes nothing of another kernel: its first slots are made before that has ended)
        // Tall tiles gain 0.2 % by that, and lose 2 % on average of Q6_K's products from 30 us on, 7 % of tiles shared after a walk (6144 x
        // 4096, 512 rows 66 -> 71 us): theirs wait.
        if (NJT == 8) pdl_wait();
        const int pw = warp - DQ_FIRST_PRODUCER, tile_w = 2 * (warp & 3) + (pw >> 2);
        const uint32_t a_base = tmem + ((uint32_t)(16 * tile_w) << 16) + (uint32_t)DQ_A_COL;
        DqRing rr, ra;
        for (int item = a.item0 + blockIdx.x; item < a.items; item += gridDim.x) {
            const int dt = DqItem(a, item).dt;
#define SP_DQ_PRODUCE(T) ok = dq_produce<T>(bars, raw, a.r_bytes, a.r_stages, tile_w, lane, a_base, n_sb, halves_last, rr, ra, ok)
            if (dt == T_Q4_K) SP_DQ_PRODUCE(T_Q4_K);
            else if (dt == T_Q6_K) SP_DQ_PRODUCE(T_Q6_K);
            else if (dt == T_Q8_0) SP_DQ_PRODUCE(T_Q8_0);
            else SP_DQ_PRODUCE(T_Q8_0_HALF);
#undef SP_DQ_PRODUCE
        }
        __syncwarp();
        if (a.parts > 1) { cluster_sync(); cluster_sync(); }
    } else {
        if (NJT >= 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 128;\n");
        pdl_wait();
        const int quarter = warp & 3, half = (warp - DQ_FIRST_DRAIN) >> 2, g = lane >> 2, t = lane & 3;
        DqRing rr, rx, rd;
        for (int item = a.item0 + blockIdx.x; item < a.items; item += gridDim.x) {
            const DqItem it(a, item);
            const Tc5Seg& sg = a.seg[it.si];
            float acc[2][NJT][4];
#pragma unroll
            for (int i = 0; i < 2 * NJT * 4; ++i) acc[i / (NJT * 4)][(i / 4) % NJT][i & 3] = 0.f;
#define SP_DQ_DRAIN(T) \
    ok = dq_drain<T, NJT>(bars, raw, a.r_bytes, a.r_stages, xs, x_bytes, a.nb, quarter, half, lane, tmem, n_sb, rr, rx, rd, acc, ok)
            if (it.dt == T_Q4_K) SP_DQ_DRAIN(T_Q4_K);
            else if (it.dt == T_Q6_K) SP_DQ_DRAIN(T_Q6_K);
            else SP_DQ_DRAIN(T_Q8_0);
#undef SP_DQ_DRAIN
            const float* res = it.si == 0 ? a.res : nullptr;
            if (a.parts == 1) {
                if (ok) {
                    const int left = it.rows - half * NJT * 8 - 2 * t, n = it.n0 + 32 * quarter + g;
                    const bool whole = it.n0 + 32 * quarter + 32 <= sg.n;
                    const int64_t row0 = it.m0 + half * NJT * 8 + 2 * t;
                    if (whole && res) dq_store<NJT, true, true>(acc, a, sg, row0, left, n);
                    else if (whole) dq_store<NJT, true, false>(acc, a, sg, row0, left, n);
                    else if (res) dq_store<NJT, false, true>(acc, a, sg, row0, left, n);
                    else dq_store<NJT, false, false>(acc, a, sg, row0, left, n);
                }
                continue;
            }
            // (a block of a cluster takes one tile)
            asm volatile("bar.sync 1, 256;\n" ::: "memory");  // nobody reads raw tiles or sums any more: their memory takes the partial tile
            float* const partial = reinterpret_cast<float*>(smem);
            static_assert(DQ_NB * DQ_P_STRIDE * 4 <= DQ_SMEM - 1024, "a partial tile of any height");
            // (rows that are not there too: nobody reads them)
            float* const mine_at = partial + (half * NJT * 8 + 2 * t) * DQ_P_STRIDE + 32 * quarter + g;
#pragma unroll
            for (int j = 0; j < 2 * NJT; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    mine_at[((j >> 1) * 8 + (j & 1)) * DQ_P_STRIDE + 16 * (i >> 1) + 8 * (i & 1)] = acc[i >> 1][j >> 1][2 * (i & 1) + (j & 1)];
            __syncwarp();
            cluster_sync();
            // the cluster's blocks share out the activation rows; each adds its rows' partials in part order
            const int idx = tid - 32 * DQ_FIRST_DRAIN, nl = idx & 127, n = it.n0 + nl;
            if (n < sg.n && ok) {
                const float bias = sg.bias ? sg.bias[n] : 0.f;
                const uint32_t mine = tc5_smem_u32(partial + nl);
                constexpr int NC = 4;
                for (int c0 = part + a.parts * (idx >> 7); c0 < it.rows; c0 += 2 * NC * a.parts) {
                    float f[NC], r[NC], sc[NC];
#pragma unroll
                    for (int j = 0; j < NC; ++j) {
                        const int c = c0 + 2 * j * a.parts;
                        f[j] = 0.f;
                        sc[j] = c < it.rows ? a.xscale[it.m0 + c] : 0.f;
                        r[j] = res && c < it.rows ? res[(int64_t)(it.m0 + c) * a.ldres + n] : 0.f;
                    }
                    for (int p = 0; p < a.parts; ++p) {
                        const uint32_t peer = peer_smem(mine, p);
#pragma unroll
                        for (int j = 0; j < NC; ++j) {
                            const int c = c0 + 2 * j * a.parts;
                            if (c < it.rows) f[j] += ld_peer(peer + (uint32_t)(c * DQ_P_STRIDE) * 4);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < NC; ++j) {
                        const int c = c0 + 2 * j * a.parts;
                        if (c < it.rows) sg.y[(int64_t)(it.m0 + c) * a.ldy + n] = fmaf(f[j], sc[j], bias) + r[j];
                    }
                }
            }
            __syncwarp();
            cluster_sync();  // nobody leaves while its partials are being read
        }
    }
    if (!ok) report_wait(a.waits, WAIT_GEMM);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

// How many clusters of 1 .. DQ_MAX_PARTS blocks the device holds at once (a block fills an SM, and a cluster lies within one GPC).
struct DqClusters { std::atomic<int> of[DQ_MAX_PARTS + 1]; };
static const DqClusters& dq_clusters() {
    static DqClusters cache[SP_MAX_DEVICES];
    DqClusters& c = cache[current_device_index()];
    for (int parts = 1; parts <= DQ_MAX_PARTS; ++parts) {  // (each for itself: another thread may be half through)
        if (c.of[parts].load(std::memory_order_relaxed) != 0) continue;
        int n = device_sm_count() / parts;
        if (parts > 1) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1, 1, (unsigned)parts);
            cfg.blockDim = dim3(DQ_THREADS);
            cfg.dynamicSmemBytes = DQ_SMEM;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = (unsigned)parts;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int got = 0;
            if (cudaOccupancyMaxActiveClusters(&got, gemm_dq_kernel<2>, &cfg) == cudaSuccess && got > 0) n = got;
            else cudaGetLastError();
        }
        c.of[parts].store(std::max(n, 1), std::memory_order_relaxed);
    }
    return c;
}

cudaError_t launch_gemm_dq(const Tc5Seg* segs, int nseg, int k, const DqInput& in, int m, int ldy, const float* res, int ldres, cudaStream_t st) {
    if (m <= 0 || nseg <= 0) return cudaSuccess;
    if (nseg > 3 || k % 128 != 0 || !in.waits) return cudaErrorInvalidValue;
    DqArgs a{};
    int tiles = 0, one_plane = 0, tb = 0;
    for (int i = 0; i < nseg; ++i) {
        if (!tc5_supported(segs[i].dtype, k) || segs[i].n <= 0) return cudaErrorInvalidValue;
        a.seg[i] = segs[i];
        tiles += (segs[i].n + DQ_BM - 1) / DQ_BM;
        if (segs[i].dtype == T_Q4_K) one_plane += (segs[i].n + DQ_BM - 1) / DQ_BM;
        tb = std::max(tb, dq_tile_bytes(segs[i].dtype));
    }
    a.nseg = nseg; a.k = k; a.m = m; a.ldy = ldy; a.res = res; a.ldres = ldres;
    a.xscale = in.xscale; a.xsum = in.xsum; a.waits = in.waits;
    static PerDeviceOnce attr_once;  // (ahead of the plan, which asks how many clusters fit)
    cudaError_t le = attr_once.run([] {
        for (auto f : {gemm_dq_kernel<1>, gemm_dq_kernel<2>, gemm_dq_kernel<4>, gemm_dq_kernel<8>}) {
            const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM);
            if (e != cudaSuccess) return e;
        }
        // the register split of the tall variants draws on what their blocks are launched with
        for (auto f : {gemm_dq_kernel<4>, gemm_dq_kernel<8>}) {
            cudaFuncAttributes fa;
            const cudaError_t e = cudaFuncGetAttributes(&fa, f);
            if (e != cudaSuccess) return e;
            if (fa.numRegs * DQ_THREADS < 128 * 32 + 256 * 96 + 256 * 128) return cudaErrorLaunchOutOfResources;
        }
        return cudaSuccess;
    });
    if (le != cudaSuccess) return le;
    // How high the tiles are and how they are dealt out, by a model of the time in us, fitted to 30,000 forced choices (21 matrices x 24 row
    // counts x 3 formats; 4 % off). SPAN: 256 columns of a tile by its height; a low tile's take less time, if more for each row. One block per
    // SM walks over tiles, or clusters share a tile's K range, where every wave pays for its start and for the parts that are added, and the
    // last clusters that fit start late (3000 x 2048, 112 rows, 72 of 74 pairs 15.5, as four parts of one tile 14.1); where tiles go over whole
    // rounds of the SMs, those that do may have a launch of their own. Q4_K 6144 x 4096, 512 rows (192 tiles) walked 74.7, clusters of two 84.5, a
    // walk and 44 tiles shared by two 70.6; 20000 x 14336, 20 rows (157 tiles) 160, clusters of four 121, nine tiles shared by eight 97; 8960 x
    // 1536, 300 rows (210 tiles) 37 walked, 39 in two launches.
    // Tiles lower than need be are for SMs that would be idle, and taken where they promise 3 %: 0.96 of the time of the fewest tiles over those
    // sizes. Q8_0, 389 rows: 2560 x 2560 80 tiles of 112 rows 25.4 us, 140 of 64 21.1; 2560 x 10240 71.9 and 66.1; 1152 x 896, 300 rows 10.9
    // and 8.6; Q4_K 2048 x 1536, 192 rows 12.0 and 11.0.
    const int all_sb = (k + 255) / 256, sms = device_sm_count(), fewest = (m + DQ_NB - 1) / DQ_NB;
    const DqClusters& clusters = dq_clusters();
    int items = 0, walk = 0, parts = 1;  // tiles; those that are walked over; the rest is shared by `parts` blocks each
    double best = 0.0;
    bool lower = false;
    for (int low = fewest, last = 0; last != 16; ++low) {
        const int h = ((m + low - 1) / low + 15) & ~15, m_tiles = (m + h - 1) / h, n = tiles * m_tiles;
        if (h == last) continue;
        if (last && n > 8 * sms) break;
        if (last && !lower) best *= 0.97;
        lower = last != 0;
        static constexpr double SPAN[2][8] = {{1.26, 1.36, 1.48, 1.54, 1.81, 1.84, 1.89, 2.00}, {1.12, 1.10, 1.26, 1.27, 1.66, 1.68, 1.72, 1.77}};
        const double span = (SPAN[0][h / 16 - 1] * (tiles - one_plane) + SPAN[1][h / 16 - 1] * one_plane) / tiles;
        const int whole = n / sms * sms;
        auto walked = [&](int count) { return ((count + sms - 1) / sms) * (all_sb * span + 0.013 * h); };
        auto take = [&](double us, int w, int p) {
            if (best == 0.0 || us < best) { best = us; a.nb = h; a.m_tiles = m_tiles; items = n; walk = w; parts = p; }
        };
        take(walked(n), n, 1);
        for (int p = 2; p <= std::min(DQ_MAX_PARTS, all_sb); ++p) {
            const int places = clusters.of[p].load(std::memory_order_relaxed);
            const double wave = ((all_sb + p - 1) / p) * span + 3.92 + 0.037 * h - 0.017 * p;
            auto shared = [&](int first, double launch) {
                const int count = n - first;
                const double filled = std::min(1.0, (double)count / places), late = filled * filled;
                if (count > 0) take(((count + places - 1) / places) * wave + 1.37 * late * late + launch, first, p);
            };
            shared(0, -3.05);  // (its start lies under the kernel before)
            if (whole > 0) shared(whole, walked(whole) + 0.80);
        }
        last = h;
    }
    // shared memory: at most half for activations (each box serves 64 columns), the rest for raw tiles
    const int njt = a.nb <= 16 ? 1 : a.nb <= 32 ? 2 : a.nb <= 64 ? 4 : 8;
    const int b_bytes = dq_boxes(njt) * 2 * a.nb * 128, x_bytes = DQ_X_STAGES * a.nb * 32;
    a.r_bytes = 8 * tb;
    a.b_stages = std::min(DQ_MAX_B, 128 * 1024 / b_bytes);
    a.r_stages = std::min(DQ_MAX_R, (DQ_SMEM - 1024 - a.b_stages * b_bytes - x_bytes) / a.r_bytes);
    const PFN_encodeTiled encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    CUtensorMap tmap;
    {
        const cuuint64_t gdim[4] = {64u, (cuuint64_t)m, 2u, (cuuint64_t)(k / 64)};
        const cuuint64_t gstride[3] = {(cuuint64_t)k * sizeof(__half), (cuuint64_t)m * k * sizeof(__half), 64 * sizeof(__half)};
        const cuuint32_t box[4] = {64u, (cuuint32_t)a.nb, 2u, (cuuint32_t)dq_boxes(njt)};
        const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
        if (encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, in.xh, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    auto kernel = njt == 1 ? gemm_dq_kernel<1> : njt == 2 ? gemm_dq_kernel<2> : njt == 4 ? gemm_dq_kernel<4> : gemm_dq_kernel<8>;
    auto launch = [&](int from, int to, int parts) {
        a.item0 = from; a.items = to; a.parts = parts;
        const int n = to - from;
        if (n == 0) return cudaSuccess;
        const dim3 grid((unsigned)(parts == 1 ? std::min(n, sms) : n), 1, (unsigned)parts);
        const cudaError_t e = launch_pdl_cluster(kernel, grid, dim3(DQ_THREADS), DQ_SMEM, st, parts, a, tmap);
        return e != cudaSuccess ? e : count_launch_and_check();
    };
    le = launch(0, walk, 1);
    return le != cudaSuccess ? le : launch(walk, items, parts);
}

}  // namespace sp
