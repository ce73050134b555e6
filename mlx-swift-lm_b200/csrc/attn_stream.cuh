// Decode attention over every pair of K / V representations a 16-bit caller can hold (raw rows, affine
// 4- / 8-bit codes, 2- / 3- / 4-bit codebook indices, mixed: raw or affine keys with index values, index
// keys with affine values; raw keys with raw values have kernels of their own), head dims 64 / 128 / 256, up to 64 query
// rows per KV head, and lists of calls of one shape.
//
// What bounds it: instruction issue and the shared-memory pipe for the packed layouts, HBM for the wide ones.
// Split: every WARP is on its own. It walks 16-token blocks of the CTA's token range (every fifth to twelfth:
// as many as the CTA has warps),
// keeps a private ring of packed blocks in shared memory that its own lanes fill with 16-byte cp.async copies
// (a block of 16 rows is one contiguous piece of each array; bytes past the last token are zero-filled, so no
// padding of the arrays is asked for), and no barrier is taken until the segment ends. The token side sits on
// the 16-row side of mma.sync.m16n8k16 (S^T = K Q^T, O^T = V^T P^T), the query rows on its 8 columns, so a
// group of up to eight rows costs half the MMAs and accumulators of the row-major orientation.
//   * Keys go from the packed words into A fragments in registers: the order of the head dims inside an MMA
//     is free as long as the query fragments use the same one, so lane (g, c) reads a contiguous piece of rows
//     g and g + 8. Affine codes enter as exact integers around zero and the scale / bias of a group is applied to the
//     group's fp32 score (s * (q . (c - m)) + (b + m s) * sum q); index keys enter as centroids (pair lookups in a table
//     replicated per lane, no bank conflicts) and the row norm multiplies the fp32 score.
//   * Values need no transpose either: a register of the A operand of O^T = V^T P^T holds one dim of two tokens, so
//     a lane reads the same run of dims of its four tokens and interleaves the codes of two tokens with a few logic
//     operations; the pair is an index of the same table (codebook indices) or one logic operation away from two f16
//     (affine codes). The row norm / group scale goes into P in fp32, the affine bias is accumulated beside the MMAs
//     in fp32. Before, the rows went through a private f16 tile and came back with ldmatrix: two thirds
//     of the shared-memory wavefronts of the value side, and a wait between the lookups and the products.
//   * A table entry holds the high and the low halves of a centroid pair, eight bytes a lane: one load for both.
//   * Nothing fp32 is cut to one f16: P * factor, rotated queries and centroids are pairs (high half, low half, 22
//     bits) and a product is the three MMAs hi hi + lo hi + hi lo (two where one side is exact). The MMAs are not what
//     bounds the kernel; the second table lookup of each centroid pair is the price.
//     8 layers x 4 sequences x 4099 tokens, 32/8 heads, D 128, 8-bit keys / 4-bit values, f16: 2521 us on the general
//     kernel, 89 us here (114 with the values through the tile and a load for each half); with single f16 operands the
//     outputs no longer err by the store's rounding alone.
//   * The running reference is only moved when a score (with its value factor) passes it by more than 2^3.
// Work is cut into ranges of 64-token tiles, equal ones or ones that end where units end (plan_units); units that cross a CTA
// boundary are merged by segment_epilogue.
#pragma once

#include "attn_common.cuh"

#include <algorithm>
#include <type_traits>

namespace kvc {

namespace stream {

using namespace dev;

constexpr int ST_TILE = 64;        // tokens per tile of the flat plan
constexpr int ST_STAGES = 2;       // packed 16-token blocks per warp: one in use, one on its way
constexpr int ST_SEGMENT = 8;      // what a segment costs beside its tiles, in tiles
constexpr int ST_COUNTER_BYTES = 64 * 1024;
constexpr float ST_LAZY = 3.f;     // log2 of how far a score may pass the running maximum
constexpr float ST_PSCALE = 1024.f;  // P * factor (at most 2^3) is carried 2^10 up: its low half stays clear of f16 subnormals
constexpr int ST_SMEM = 227 * 1024;
constexpr float ST_NONE = -1e30f;

enum { SK_RAW = 0, SK_A4, SK_A8, SK_T2, SK_T3, SK_T4 };

template <int KIND, int D>
struct Kind {
    static constexpr bool RAW = KIND == SK_RAW, AFFINE = KIND == SK_A4 || KIND == SK_A8, TURBO = !RAW && !AFFINE;
    static constexpr int BITS = RAW ? 16 : KIND == SK_A4 ? 4 : KIND == SK_A8 ? 8 : KIND == SK_T2 ? 2 : KIND == SK_T3 ? 3 : 4;
    static constexpr int RB = D * BITS / 8;                       // bytes per row
    static constexpr int BLOCK = 16 * RB;                         // bytes per 16-token block
    static constexpr int SIDE = RAW ? 0 : AFFINE ? 16 * (D / 32) * 2 : 64;   // scales (and as much again for biases) or norms
    static constexpr int STAGE = BLOCK + (AFFINE ? 2 : 1) * SIDE;
    static constexpr int TABLE = TURBO ? (1 << (2 * BITS)) * 256 : 0;   // high and low halves of a centroid pair, per lane
    static constexpr int CH = RB / 16;                            // 16-byte chunks per row (where whole)
    static constexpr bool POW2 = RB % 16 == 0 && (CH & (CH - 1)) == 0;
};

struct StreamSource {
    const void *data, *scales, *biases;   // rows or words; scales, biases or norms
    int64_t sb, sh, gsb, gsh;             // BYTE strides over batch and head
};

// One call of a list (a layer of a batched step, a sequence of a ragged one): its own arrays and length, the
// shape in common.
struct StreamSeq {
    const void *q;
    void *out;
    StreamSource k, v;
    const float *q_signs, *q_calib, *o_signs;
    int64_t q_sb, o_sb, tile_first;       // flat tiles of the calls before this one
    int32_t T, tiles;                     // tiles per unit
    int64_t causal_offset;
};
struct StreamList {
    int32_t n;
    StreamSeq seq[KVC_LIST_MAX];
};
struct StreamNoList {};

struct StreamParams {
    const void *q;
    void *out;
    int64_t q_sb, q_sh, q_sl, o_sb, o_sh, o_sl;
    StreamSource k, v;
    const float *q_signs, *q_calib, *o_signs;
    float kcb[16], vcb[16];               // times a power of two that brings the largest near 8
    float kcb_undo, vcb_undo;
    float *o_part;
    float2 *ml_part;
    int *counters;
    UnitPlan flat;
    int32_t B, Hq, Hkv, L, T;
    int32_t groups_k, groups_v;           // affine groups per row
    int32_t chunks;                       // row blocks per KV head
    int32_t v_table;                      // byte offset of the value table (0: first, or the keys' own)
    int *status;
    int32_t out_dtype, causal;
    int64_t causal_offset;
    float scale_log2;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r) : "r"(a) : "memory");
    return r;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t r;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(r) : "r"(a) : "memory");
    return r;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 r;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(a) : "memory");
    return r;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 r;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a) : "memory");
    return r;
}
__device__ __forceinline__ void sts64(uint32_t a, uint2 v) {
    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(a), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// What an f16 pair leaves of the two floats it was rounded from.
__device__ __forceinline__ uint32_t low_half2(uint32_t hi, float a, float b) {
    const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    return pack_h2(a - h.x, b - h.y);
}
// e with |x| < 2^e, kept to a range in which the weights that are carried relative to it stay clear of both ends.
__device__ __forceinline__ float exponent_above(float x) {
    return (float)min(max((int)((__float_as_uint(x) >> 23) & 255u) - 126, -64), 100);
}

// Where 16-byte chunk `ch` of token `tok` sits in a staged block: the key side is read by lanes (token, quarter
// of a piece), the value side by lanes that hold eight consecutive tokens at one chunk; both orders then spread
// over the 32 banks.
template <int KIND, int D, int UNIT>
__device__ __forceinline__ int key_xor(int tok) {
    constexpr int CH = Kind<KIND, D>::CH;
    if (KIND == SK_RAW) return CH >= 8 ? (tok & 1) << 2 : 0;
    if (KIND == SK_A8 && UNIT == 64) return CH >= 8 ? (tok & 1) << 2 : 0;
    if (KIND == SK_A8) return CH >= 8 ? (tok & 3) << 1 : ((tok >> 1) & 1) << 1;
    if (KIND == SK_A4 && UNIT == 64) return CH >= 8 ? (tok & 3) << 1 : CH == 4 ? ((tok >> 1) & 1) << 1 : 0;
    if (KIND == SK_A4) return CH >= 8 ? tok & 7 : CH == 4 ? (tok >> 1) & 3 : (tok >> 2) & 1;
    if (KIND == SK_T4 && CH == 8) return tok & 1;
    return 0;
}
// Values are read by lanes (run of dims g, tokens 2c and 2c + 1, then 8 tokens on): the four tokens of a load lie
// next to each other, their chunks turned so that the runs of eight (sixteen byte loads: two) lanes fill all banks.
template <int KIND, int D>
__device__ __forceinline__ int value_xor(int c) {
    constexpr int CH = Kind<KIND, D>::CH;
    if (!Kind<KIND, D>::POW2) return 0;
    return CH >= 8 ? 2 * c : CH == 4 ? c & 2 : 0;
}
template <int KIND, int D>
__device__ __forceinline__ int value_slot(int tok) {
    return Kind<KIND, D>::POW2 ? (tok & 8) | (tok & 1) << 2 | ((tok >> 1) & 3) : tok;
}

// Byte offset of the table entry that field n (2 * BITS bits) of a run of words names; `lane_const` holds the lane's
// place in the entry and, above the fields' bits, which table it is.
template <int BITS, int NW>
__device__ __forceinline__ uint32_t entry_offset(const uint32_t (&w)[NW], int n, uint32_t lane_const) {
    constexpr int B2 = 2 * BITS;
    if constexpr (BITS == 4) return __byte_perm(w[n >> 2], lane_const, 0x7604 | ((n & 3) << 4));
    constexpr uint32_t MASK = ((1u << B2) - 1u) << 8;
    const int bit = B2 * n, k = bit >> 5, s = bit & 31;
    uint32_t x;
    if (s + B2 <= 32) x = (s >= 8) ? (w[k] >> (s - 8)) : (w[k] << (8 - s));
    else x = __funnelshift_r(w[k], w[(k + 1 < NW) ? k + 1 : k], s - 8);
    return (x & MASK) | lane_const;
}
// Dynamic shared memory starts here in a block's window (what the driver reserves lies in front; the host asks the device
// before it launches), so that the tables' place is part of the load.
constexpr uint32_t ST_WINDOW = 1024;
// Tables do not change after the barrier behind their making: these loads may be moved freely.
__device__ __forceinline__ uint2 table_entry(uint32_t offset) {
    uint2 r;
    asm("ld.shared.v2.b32 {%0,%1}, [%2+%3];" : "=r"(r.x), "=r"(r.y) : "r"(offset), "n"(ST_WINDOW));
    return r;
}

// Bits of word k of a run of 3-bit codes that belong to codes of even places.
__host__ __device__ constexpr uint32_t even3(int k) {
    uint32_t m = 0;
    for (int i = 0; i < 32; ++i)
        if ((32 * k + i) % 6 < 3) m |= 1u << i;
    return m;
}
// The codes of one run of dims of tokens a and b as pairs: field n of `even` (`odd`) has dim 2n (2n + 1) of a in its
// lower BITS bits and of b in its upper ones.
template <int BITS, int NW>
__device__ __forceinline__ void pair_tokens(const uint32_t (&a)[NW], const uint32_t (&b)[NW], uint32_t (&even)[NW], uint32_t (&odd)[NW]) {
#pragma unroll
    for (int k = 0; k < NW; ++k) {
        const uint32_t m = BITS == 4 ? 0x0F0F0F0Fu : BITS == 2 ? 0x33333333u : even3(k);
        const uint32_t up = BITS == 3 && k > 0 ? __funnelshift_l(b[k > 0 ? k - 1 : 0], b[k], BITS) : b[k] << BITS;
        const uint32_t down = BITS == 3 && k + 1 < NW ? __funnelshift_r(a[k], a[k + 1 < NW ? k + 1 : k], BITS) : a[k] >> BITS;
        even[k] = (a[k] & m) | (up & ~m);
        odd[k] = (down & m) | (b[k] & ~m);
    }
}

// Two codes n as the f16 pair n - 8 or n - 128, exact: 1024 + n (+ 16 n for the upper nibble of a byte) by one logic
// operation or byte permute, then one f16 addition or fma. 4-bit words give the dims (i, i + 4), i odd from the upper
// nibbles; 8-bit words (0, 1) and (2, 3). Codes left as the subnormals n * 2^-24 save the second instruction, but the
// MMA aligns its products by their operands' exponents and cut the small ones short: with 4-bit values and 4 000 .. 8 000
// keys f16 outputs erred by 0.06 .. 0.11 % more than those of the general kernel. Around zero, the codes' part of a sum
// is no larger than the sum.
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, float b, float c) {
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&a), __float2half2_rn(b), __float2half2_rn(c));
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t code4(uint32_t w, int i) {
    const uint32_t x = (((i & 2) ? w >> 8 : w) & ((i & 1) ? 0x00F000F0u : 0x000F000Fu)) | 0x64006400u;
    return (i & 1) ? h2_fma(x, 0.0625f, -72.f) : h2_fma(x, 1.f, -1032.f);
}
__device__ __forceinline__ uint32_t code8(uint32_t w, int i) { return h2_fma(__byte_perm(w, 0x64646464u, i ? 0x4342 : 0x4140), 1.f, -1152.f); }
template <int KIND> constexpr float code_middle() { return KIND == SK_A4 ? 8.f : 128.f; }

template <typename T> __device__ __forceinline__ float ld16(uint32_t a) {
    uint16_t r;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(r) : "r"(a) : "memory");
    return to_f32<T>(*reinterpret_cast<const T *>(&r));
}

template <typename T, int D, int KK, int VK, int UNIT, int NB, bool LIST>
struct StreamShape {
    using K = Kind<KK, D>;
    using V = Kind<VK, D>;
    static constexpr int STAGE = K::STAGE + V::STAGE;
    static constexpr int WARP_BYTES = ST_STAGES * STAGE;
    static constexpr int ROWS = 8 * NB;
    static constexpr int RED_STRIDE = D + 4;
    static constexpr int QS = ROWS * D * 4;                       // staged query rows
    static constexpr int HEAD = 32 + ROWS * 4 > 128 ? 256 : 128;  // merge flag, one factor per query row
    static constexpr int fixed(int warps) {
        const int red = warps * ROWS * (RED_STRIDE + 2) * 4 + ROWS * D * 4, rings = warps * WARP_BYTES;
        return (rings > red ? rings : red) + QS + HEAD;           // the merge buffers reuse the ring
    }
    // Eight warps where two CTAs fit an SM; where the tables leave room for one, twelve that share them if they fit:
    // 168 registers keep a step's loads in flight (sixteen warps of 128 registers: 99 us
    // where this takes 90, the shape above).
    static constexpr int MOST_TABLES = K::TABLE + V::TABLE;
    static constexpr bool WIDE = NB == 1 && D <= 128;
    static constexpr bool PAIR = WIDE && 2 * (MOST_TABLES + fixed(8) + 1024) <= 228 * 1024;
    static constexpr bool fits(int warps) { return MOST_TABLES + fixed(warps) <= ST_SMEM; }
    static constexpr int WARPS = PAIR ? 8 : WIDE && fits(12) ? 12 : fits(8) ? 8 : fits(6) ? 6 : 5;
    static_assert(fits(WARPS), "the rings and tables of this pair do not fit shared memory");
    static constexpr int RESIDENT = PAIR ? 2 : 1;
    static constexpr int THREADS = WARPS * 32;
    static constexpr int FIXED = fixed(WARPS);
    // A table lies at a multiple of its size, so that an entry's offset and the table's are joined by a logic operation:
    // the larger one first.
    static constexpr int K_AT = K::TURBO && V::TABLE > K::TABLE ? V::TABLE : 0;
    static constexpr int tables(int v_table) {
        const int k = K_AT + K::TABLE, v = V::TURBO ? v_table + V::TABLE : 0;
        return k > v ? k : v;
    }
};

// Token range and place of one segment: `x` flat tiles in, at most `left` tiles.
struct Segment {
    int seq, unit, b, hk, chunk, tile, tiles, unit_tiles, T;
    int64_t unit_x;
};

template <typename T, int D, int KK, int VK, int UNIT, int NB, bool LIST>
__global__ void __launch_bounds__(StreamShape<T, D, KK, VK, UNIT, NB, LIST>::THREADS, StreamShape<T, D, KK, VK, UNIT, NB, LIST>::RESIDENT)
attn_stream_kernel(const __grid_constant__ StreamParams p,
                   const __grid_constant__ std::conditional_t<LIST, StreamList, StreamNoList> list) {
    using SH = StreamShape<T, D, KK, VK, UNIT, NB, LIST>;
    using K = Kind<KK, D>;
    using V = Kind<VK, D>;
    using KT = std::conditional_t<K::RAW, T, __half>;             // operand type of the score MMAs
    static_assert(!V::RAW, "raw values have kernels of their own");
    constexpr int ST_WARPS = SH::WARPS, ST_THREADS = SH::THREADS;
    constexpr int KSTEPS = D / 16, MT = D / 16;
    constexpr int KU = K::AFFINE ? UNIT : K::RAW ? 32 : D;        // dims that share a fragment order
    constexpr int NU = D / KU, UK = KU / 16;                      // units, k-steps per unit
    constexpr int NG = V::AFFINE ? D / UNIT : 1;                  // value groups kept apart (128-wide ones twice)
    constexpr int VU = V::AFFINE ? UNIT : D, VM = VU / 16;        // value dims under one factor, their MMAs
    constexpr int VRUN = VU / 8, VRB = VRUN * V::BITS, VW = (VRB + 31) / 32;   // a lane's run of them: dims, bits, words
    constexpr int QP = K::TURBO ? 2 : 1;                          // query fragments: high and low halves where the rows are rotated

    extern __shared__ __align__(1024) unsigned char smem[];
    // tables first (constant offsets), then the merge flag, the query rows and the rings
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const uint32_t s0 = smem_u32(smem);
    if (s0 != ST_WINDOW) {                                        // (asked before; uniform over the grid)
        pdl_wait();
        if (tid == 0) atomicExch(p.status, 36);
        return;
    }
    const int tab_end = SH::tables(p.v_table);
    int *flag = (int *)(smem + tab_end);
    float *rowf = (float *)(smem + tab_end + 32);                 // what a score of the row is multiplied by in the end
    float *qs = (float *)(smem + tab_end + SH::HEAD);
    unsigned char *body = smem + tab_end + SH::HEAD + SH::QS;
    const uint32_t ring = smem_u32(body) + warp * SH::WARP_BYTES;
    const uint32_t k_lane_bits = (uint32_t)lane << 3 | SH::K_AT, v_lane_bits = (uint32_t)lane << 3 | (uint32_t)p.v_table;

    // Pair tables, 32 equal (high, low) pairs of words per entry: a warp takes an entry, the centroids sit in its lanes.
    auto build_table = [&](auto bits, const float *cb, uint2 *dst) {
        constexpr int BITS = decltype(bits)::value;
        const float mine = lane < (1 << BITS) ? cb[lane] : 0.f;
#pragma unroll 4
        for (int j = warp; j < (1 << (2 * BITS)); j += ST_WARPS) {
            const float a = __shfl_sync(0xffffffffu, mine, j & ((1 << BITS) - 1)), b = __shfl_sync(0xffffffffu, mine, j >> BITS);
            const uint32_t hi = pack_h2(a, b);
            dst[j * 32 + lane] = make_uint2(hi, low_half2(hi, a, b));
        }
    };
    if constexpr (K::TURBO) build_table(std::integral_constant<int, K::BITS>{}, p.kcb, (uint2 *)(smem + SH::K_AT));
    if constexpr (V::TURBO)
        if (!K::TURBO || SH::K_AT || p.v_table) build_table(std::integral_constant<int, V::BITS>{}, p.vcb, (uint2 *)(smem + p.v_table));
    pdl_wait();
    pdl_trigger();

    const UnitPlan fp = p.flat;
    const int rep = p.Hq / p.Hkv, rows_all = rep * p.L;
    int64_t x = flat_lo(fp, blockIdx.x);
    const int64_t x_end = flat_lo(fp, blockIdx.x + 1);
    while (x < x_end) {
        Segment sg;
        int64_t in = x;
        sg.seq = 0; sg.unit = 0; sg.unit_tiles = fp.tiles; sg.T = p.T;
        if constexpr (LIST) {
            while (sg.seq + 1 < list.n && list.seq[sg.seq + 1].tile_first <= x) ++sg.seq;
            in -= list.seq[sg.seq].tile_first;
            sg.T = list.seq[sg.seq].T;
            sg.unit_tiles = list.seq[sg.seq].tiles;
            sg.unit = sg.seq * p.B * p.Hkv * p.chunks;
        }
        const int u_in = flat_div(in, sg.unit_tiles);
        sg.unit += u_in;
        sg.tile = flat_mod(in, sg.unit_tiles, u_in);
        sg.chunk = u_in % p.chunks;
        sg.hk = (u_in / p.chunks) % p.Hkv;
        sg.b = u_in / p.chunks / p.Hkv;
        sg.unit_x = x - sg.tile;
        sg.tiles = (int)min((int64_t)(sg.unit_tiles - sg.tile), x_end - x);
        const int row0 = sg.chunk * SH::ROWS, R = min(SH::ROWS, rows_all - row0);
        const int t_lo = sg.tile * ST_TILE, t_hi = min(sg.T, (sg.tile + sg.tiles) * ST_TILE);
        const int nblk = (t_hi - t_lo + 15) / 16;

        StreamSource ks = p.k, vs = p.v;
        const T *qp = (const T *)p.q + sg.b * p.q_sb;
        const float *q_signs = p.q_signs, *q_calib = p.q_calib;
        int64_t causal_offset = p.causal_offset;
        if constexpr (LIST) {
            const StreamSeq &sq = list.seq[sg.seq];
            ks = sq.k; vs = sq.v;
            qp = (const T *)sq.q + sg.b * sq.q_sb;
            q_signs = sq.q_signs; q_calib = sq.q_calib;
            causal_offset = sq.causal_offset;
        }
        const int64_t bi = sg.b;
        const char *kd = (const char *)ks.data + bi * ks.sb + sg.hk * ks.sh;
        const char *vd = (const char *)vs.data + bi * vs.sb + sg.hk * vs.sh;
        const char *ksc = K::RAW ? nullptr : (const char *)ks.scales + bi * ks.gsb + sg.hk * ks.gsh;
        const char *vsc = (const char *)vs.scales + bi * vs.gsb + sg.hk * vs.gsh;
        const char *kbi = K::AFFINE ? (const char *)ks.biases + bi * ks.gsb + sg.hk * ks.gsh : nullptr;
        const char *vbi = V::AFFINE ? (const char *)vs.biases + bi * vs.gsb + sg.hk * vs.gsh : nullptr;
        const int k_side = K::AFFINE ? 2 * p.groups_k : 4, v_side = V::AFFINE ? 2 * p.groups_v : 4;   // bytes per token

        // ---- one 16-token block into a stage ----
        // Rows are contiguous, so a block is one run of 16-byte chunks per array; this lane's chunks are 32 apart.
        // The scale / bias / norm arrays are a few chunks each: they are laid end to end over the lanes.
        auto key_place = [](int i) {
            if constexpr (K::RB % 16 != 0 || KK == SK_T3) return i << 4;
            else {
                const int tok = i / K::CH, ch = i % K::CH;
                return (tok * K::CH + (ch ^ key_xor<KK, D, UNIT>(tok))) << 4;
            }
        };
        auto value_place = [](int i) {
            if constexpr (!V::POW2) return i << 4;
            else {
                const int tok = i / V::CH, ch = i % V::CH, slot = value_slot<VK, D>(tok);
                return (slot * V::CH + (ch ^ value_xor<VK, D>(slot & 3))) << 4;
            }
        };
        constexpr int KC = K::BLOCK / 16, VC = V::BLOCK / 16, KI = (KC + 31) / 32, VI = (VC + 31) / 32;
        constexpr int SIDES = (K::AFFINE ? 2 : K::TURBO) + (V::AFFINE ? 2 : V::TURBO);
        constexpr int SI = (SIDES * ((K::AFFINE || V::AFFINE) ? D / 16 : 4) + 31) / 32;   // most rounds of side chunks
        const char *side_src[SI];
        int side_dst[SI], side_step[SI], side_row[SI];
#pragma unroll
        for (int r = 0; r < SI; ++r) {
            int i = lane + 32 * r;
            side_dst[r] = -1; side_src[r] = nullptr; side_step[r] = 0; side_row[r] = 0;
            auto claim = [&](const char *src, int per_token, int dst) {
                if (i >= 0 && i < per_token) {       // 16 tokens * per_token bytes = per_token chunks
                    side_src[r] = src + (int64_t)t_lo * per_token + i * 16;
                    side_dst[r] = dst + i * 16;
                    side_step[r] = 16 * per_token;
                    side_row[r] = i * 16;
                }
                i -= per_token;
            };
            if (!K::RAW) claim(ksc, k_side, K::BLOCK);
            if (K::AFFINE) claim(kbi, k_side, K::BLOCK + K::SIDE);
            claim(vsc, v_side, K::STAGE + V::BLOCK);
            if (V::AFFINE) claim(vbi, v_side, K::STAGE + V::BLOCK + V::SIDE);
        }
        const char *k_lane = kd + (int64_t)t_lo * K::RB + lane * 16, *v_lane = vd + (int64_t)t_lo * V::RB + lane * 16;
        auto fetch = [&](int blk, int st) {
            const uint32_t dst = ring + st * SH::STAGE;
            const char *ksrc = k_lane + (int64_t)blk * K::BLOCK, *vsrc = v_lane + (int64_t)blk * V::BLOCK;
            const int live = sg.T - t_lo - blk * 16;
            if (live >= 16) {
#pragma unroll
                for (int r = 0; r < KI; ++r)
                    if (KC % 32 == 0 || lane + 32 * r < KC) cp_async16(dst + key_place(lane + 32 * r), ksrc + 512 * r, 16);
#pragma unroll
                for (int r = 0; r < VI; ++r)
                    if (VC % 32 == 0 || lane + 32 * r < VC) cp_async16(dst + K::STAGE + value_place(lane + 32 * r), vsrc + 512 * r, 16);
#pragma unroll
                for (int r = 0; r < SI; ++r)
                    if (side_dst[r] >= 0) cp_async16(dst + side_dst[r], side_src[r] + (int64_t)blk * side_step[r], 16);
            } else {       // the last block of the unit: bytes of tokens past the end become zero
#pragma unroll 1
                for (int i = lane; i < KC; i += 32) {
                    const int n = min(16, max(0, live * K::RB - i * 16));
                    cp_async16(dst + key_place(i), n > 0 ? ksrc + (i - lane) * 16 : kd, n);
                }
#pragma unroll 1
                for (int i = lane; i < VC; i += 32) {
                    const int n = min(16, max(0, live * V::RB - i * 16));
                    cp_async16(dst + K::STAGE + value_place(i), n > 0 ? vsrc + (i - lane) * 16 : vd, n);
                }
#pragma unroll
                for (int r = 0; r < SI; ++r)
                    if (side_dst[r] >= 0) {
                        const int n = min(16, max(0, live * (side_step[r] >> 4) - side_row[r]));
                        cp_async16(dst + side_dst[r], n > 0 ? side_src[r] + (int64_t)blk * side_step[r] : kd, n);
                    }
            }
        };
        if (warp < nblk) fetch(warp, 0);
        cp_commit();

        // ---- query rows: f32 in shared memory (rotated for index keys), then B fragments ----
        for (int i = tid; i < SH::ROWS * D; i += ST_THREADS) {
            const int r = i / D, d = i % D;
            float v = 0.f;
            if (r < R) {
                int h, l;
                split_row(row0 + r, p.L, h, l);
                v = to_f32<T>(qp[(sg.hk * rep + h) * p.q_sh + l * p.q_sl + d]);
                if (K::TURBO) v *= q_signs[d];
            }
            qs[i] = v;
        }
        __syncthreads();
        if constexpr (!K::RAW) {
            // A warp takes a row. Index keys: Walsh-Hadamard over the lanes (D / 32 dims each), 1 / sqrt(D), calibration.
            // Then the row goes to [2^11, 2^12) by a power of two, which its scores get back: no query overflows f16, and
            // what 16 bits of a row lose is relative to the row's largest element.
            constexpr int E = D / 32;
            for (int r = warp; r < SH::ROWS; r += ST_WARPS) {
                float e[E];
#pragma unroll
                for (int j = 0; j < E; ++j) e[j] = qs[r * D + E * lane + j];
                if constexpr (K::TURBO) {
#pragma unroll
                    for (int h = 1; h < E; h <<= 1)
#pragma unroll
                        for (int i = 0; i < E; ++i)
                            if ((i & h) == 0) {
                                const float a = e[i], b = e[i + h];
                                e[i] = a + b;
                                e[i + h] = a - b;
                            }
#pragma unroll
                    for (int m = 1; m < 32; m <<= 1)
#pragma unroll
                        for (int j = 0; j < E; ++j) {
                            const float y = __shfl_xor_sync(0xffffffffu, e[j], m);
                            e[j] = (lane & m) ? y - e[j] : e[j] + y;
                        }
                    const float f = rsqrtf((float)D);
#pragma unroll
                    for (int j = 0; j < E; ++j) e[j] *= f * (q_calib ? q_calib[E * lane + j] : 1.f);
                }
                uint32_t top = 0;       // the largest magnitude: bit patterns of non-negative floats order like the floats
#pragma unroll
                for (int j = 0; j < E; ++j) top = max(top, __float_as_uint(e[j]) & 0x7fffffffu);
                top = __reduce_max_sync(0xffffffffu, top);
                const int ex = top ? max((int)(top >> 23), 27) - 127 : 0;         // the row is below 2^(ex + 1)
                const float up = __uint_as_float((uint32_t)(127 + 11 - ex) << 23);
#pragma unroll
                for (int j = 0; j < E; ++j) qs[r * D + E * lane + j] = e[j] * up;
                if (lane == 0) rowf[r] = __uint_as_float((uint32_t)(127 - 11 + ex) << 23) * p.scale_log2 * (K::TURBO ? p.kcb_undo : 1.f);
            }
            __syncthreads();
        }
        uint32_t qb[NB][QP][KSTEPS][2];
        float rf[NB][2];
        float qsum[NB][K::AFFINE ? NU : 1][2];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            const float *qr = qs + (8 * nb + g) * D;
#pragma unroll
            for (int u = 0; u < NU; ++u)
#pragma unroll
                for (int s = 0; s < UK; ++s) {
                    const int base = u * KU + c * (KU / 4);
                    int e[4];
                    if (KK == SK_A4) {
                        const int w = base + 8 * (s >> 1), i = 2 * (s & 1);
                        e[0] = w + i; e[1] = w + i + 4; e[2] = w + i + 1; e[3] = w + i + 5;
                    } else {
                        for (int j = 0; j < 4; ++j) e[j] = base + 4 * s + j;
                    }
                    qb[nb][0][u * UK + s][0] = MmaType<KT>::pack(qr[e[0]], qr[e[1]]);
                    qb[nb][0][u * UK + s][1] = MmaType<KT>::pack(qr[e[2]], qr[e[3]]);
                    if constexpr (QP == 2) {
                        qb[nb][1][u * UK + s][0] = low_half2(qb[nb][0][u * UK + s][0], qr[e[0]], qr[e[1]]);
                        qb[nb][1][u * UK + s][1] = low_half2(qb[nb][0][u * UK + s][1], qr[e[2]], qr[e[3]]);
                    }
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) rf[nb][h] = K::RAW ? p.scale_log2 : rowf[8 * nb + 2 * c + h];
            if (K::AFFINE) {
#pragma unroll
                for (int u = 0; u < NU; ++u)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // sum over the unit's dims of row 8 nb + 2 c + h, spread over the eight lanes g
                        float a = 0.f;
                        for (int d = g; d < KU; d += 8) a += qs[(8 * nb + 2 * c + h) * D + u * KU + d];
                        a += __shfl_xor_sync(0xffffffffu, a, 4);
                        a += __shfl_xor_sync(0xffffffffu, a, 8);
                        a += __shfl_xor_sync(0xffffffffu, a, 16);
                        qsum[nb][u][h] = a;
                    }
            }
        }
        int lim[NB][2], lim_min = sg.T - 1;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int rr = row0 + 8 * nb + 2 * c + h;
                lim[nb][h] = sg.T - 1;
                if (p.causal && rr < rows_all)
                    lim[nb][h] = (int)min((int64_t)(sg.T - 1), causal_offset + rr % p.L);
                lim_min = min(lim_min, lim[nb][h]);
            }
        lim_min = min(lim_min, __shfl_xor_sync(0xffffffffu, lim_min, 1));
        lim_min = min(lim_min, __shfl_xor_sync(0xffffffffu, lim_min, 2));

        float m_run[NB][2], l_run[NB][2], acc[NB][MT][4], vbias[NB][NG][2];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            m_run[nb][0] = m_run[nb][1] = ST_NONE;
            l_run[nb][0] = l_run[nb][1] = 0.f;
#pragma unroll
            for (int i = 0; i < MT; ++i) acc[nb][i][0] = acc[nb][i][1] = acc[nb][i][2] = acc[nb][i][3] = 0.f;
#pragma unroll
            for (int i = 0; i < NG; ++i) vbias[nb][i][0] = vbias[nb][i][1] = 0.f;
        }

        int stage = 0;
        for (int blk = warp; blk < nblk; blk += ST_WARPS) {
            if (blk + ST_WARPS < nblk) fetch(blk + ST_WARPS, stage ^ 1);
            cp_commit();
            cp_wait<1>();
            __syncwarp();
            const uint32_t kst = ring + stage * SH::STAGE, vst = kst + K::STAGE;
            const int t0 = t_lo + blk * 16;

            // ---- scores: s[nb] = {(g, 2c), (g, 2c + 1), (g + 8, 2c), (g + 8, 2c + 1)} of (token, row), log2 domain ----
            // A chain of MMAs rounds towards zero at every step: raw rows take two short chains, index keys one for the
            // high halves and one (s2) for the small products.
            float s[NB][4], s2[NB][4];
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                s[nb][0] = s[nb][1] = s[nb][2] = s[nb][3] = 0.f;
                s2[nb][0] = s2[nb][1] = s2[nb][2] = s2[nb][3] = 0.f;
            }
            auto mma_k = [&](float (&d)[NB][4], int ks, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
                const uint32_t a[4] = {a0, a1, a2, a3};
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    MmaType<KT>::mma(d[nb], a, qb[nb][0][ks][0], qb[nb][0][ks][1]);
                    if constexpr (QP == 2) MmaType<KT>::mma(s2[nb], a, qb[nb][1][ks][0], qb[nb][1][ks][1]);
                }
            };
            if constexpr (K::RAW) {
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    const int ch = u * 4 + c;
                    const uint4 x0 = lds128(kst + ((g * K::CH + (ch ^ key_xor<KK, D, UNIT>(g))) << 4));
                    const uint4 x1 = lds128(kst + (((g + 8) * K::CH + (ch ^ key_xor<KK, D, UNIT>(g + 8))) << 4));
                    mma_k(s, 2 * u, x0.x, x1.x, x0.y, x1.y);
                    mma_k(s2, 2 * u + 1, x0.z, x1.z, x0.w, x1.w);
                }
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[nb][e] += s2[nb][e];
            } else if constexpr (K::AFFINE) {
                constexpr int PB = KU / 4 * K::BITS / 8;      // bytes of a lane's piece: 4, 8 or 16
                constexpr int PW = PB / 4;
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    uint32_t w[2][PW];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int tok = g + 8 * i, off = u * 4 * PB + c * PB;
                        const uint32_t ad = kst + tok * K::RB + ((((off >> 4) ^ key_xor<KK, D, UNIT>(tok)) << 4) | (off & 15));
                        if constexpr (PW == 4) { const uint4 v = lds128(ad); w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w; }
                        else if constexpr (PW == 2) { const uint2 v = lds64(ad); w[i][0] = v.x; w[i][1] = v.y; }
                        else w[i][0] = lds32(ad);
                    }
                    float d[NB][4];
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) d[nb][0] = d[nb][1] = d[nb][2] = d[nb][3] = 0.f;
#pragma unroll
                    for (int q = 0; q < UK; ++q) {
                        if constexpr (KK == SK_A4)
                            mma_k(d, u * UK + q, code4(w[0][q >> 1], 2 * (q & 1)), code4(w[1][q >> 1], 2 * (q & 1)),
                                  code4(w[0][q >> 1], 2 * (q & 1) + 1), code4(w[1][q >> 1], 2 * (q & 1) + 1));
                        else
                            mma_k(d, u * UK + q, code8(w[0][q], 0), code8(w[1][q], 0), code8(w[0][q], 1), code8(w[1][q], 1));
                    }
                    const int gr = (u * p.groups_k) / NU;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t ad = kst + K::BLOCK + ((g + 8 * i) * p.groups_k + gr) * 2;
                        const float sc = ld16<T>(ad), bb = fmaf(sc, code_middle<KK>(), ld16<T>(ad + K::SIDE));
#pragma unroll
                        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                s[nb][2 * i + h] = fmaf(sc, d[nb][2 * i + h], fmaf(bb, qsum[nb][u][h], s[nb][2 * i + h]));
                    }
                }
            } else {
                constexpr int QW = (D / 4 * K::BITS + 31) / 32;   // words of a quarter row
                uint32_t w[2][QW];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int tok = g + 8 * i;
                    if constexpr (KK == SK_T3 && D == 64) {       // quarters of 48 bits: from a half word on
                        const uint32_t ad = kst + tok * K::RB + ((3 * c) >> 1) * 4;
                        const uint32_t lo = lds32(ad), hi = lds32(ad + 4);
                        w[i][0] = (c & 1) ? __funnelshift_r(lo, hi, 16) : lo;
                        w[i][1] = (c & 1) ? hi >> 16 : hi;
                    } else if constexpr (KK == SK_T3) {
#pragma unroll
                        for (int j = 0; j < QW; ++j) w[i][j] = lds32(kst + tok * K::RB + (c * QW + j) * 4);
                    } else if constexpr (QW == 1) {
                        w[i][0] = lds32(kst + tok * K::RB + c * 4);
                    } else if constexpr (QW == 2) {
                        const uint2 v = lds64(kst + tok * K::RB + c * 8);
                        w[i][0] = v.x; w[i][1] = v.y;
                    } else {
#pragma unroll
                        for (int j = 0; j < QW / 4; ++j) {
                            const uint4 v = lds128(kst + tok * K::RB + (((c * (QW / 4) + j) ^ key_xor<KK, D, UNIT>(tok)) << 4));
                            w[i][4 * j] = v.x; w[i][4 * j + 1] = v.y; w[i][4 * j + 2] = v.z; w[i][4 * j + 3] = v.w;
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < KSTEPS; ++q) {
                    const uint2 x0 = table_entry(entry_offset<K::BITS, QW>(w[0], 2 * q, k_lane_bits)), x1 = table_entry(entry_offset<K::BITS, QW>(w[1], 2 * q, k_lane_bits));
                    const uint2 x2 = table_entry(entry_offset<K::BITS, QW>(w[0], 2 * q + 1, k_lane_bits)), x3 = table_entry(entry_offset<K::BITS, QW>(w[1], 2 * q + 1, k_lane_bits));
                    mma_k(s, q, x0.x, x1.x, x2.x, x3.x);
                    const uint32_t lo[4] = {x0.y, x1.y, x2.y, x3.y};
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) MmaType<KT>::mma(s2[nb], lo, qb[nb][0][q][0], qb[nb][0][q][1]);
                }
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[nb][e] += s2[nb][e];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float f = __uint_as_float(lds32(kst + K::BLOCK + (g + 8 * i) * 4));
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        s[nb][2 * i] *= f;
                        s[nb][2 * i + 1] *= f;
                    }
                }
            }
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[nb][e] *= rf[nb][e & 1];
            if (t0 + 15 > lim_min) {
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (t0 + g + 8 * (e >> 1) > lim[nb][e & 1]) s[nb][e] = -INFINITY;
            }
            // ---- probabilities ----
            // The running reference bounds score + log2(value factor): what P * factor needs to fit f16 whatever the
            // norms and scales are. The sums of exp2(score - reference) are fp32 and only meet each other.
            float vf[2][NG], ve[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float big = 0.f;
#pragma unroll
                for (int u = 0; u < NG; ++u) {
                    if constexpr (V::TURBO) vf[i][u] = __uint_as_float(lds32(vst + V::BLOCK + (g + 8 * i) * 4));
                    else vf[i][u] = ld16<T>(vst + V::BLOCK + ((g + 8 * i) * p.groups_v + (u * p.groups_v) / NG) * 2);
                    big = fmaxf(big, fabsf(vf[i][u]));
                }
                ve[i] = exponent_above(big);
            }
            bool moved = false;
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int h = 0; h < 2; ++h) moved |= fmaxf(s[nb][h] + ve[0], s[nb][2 + h] + ve[1]) > m_run[nb][h] + ST_LAZY;
            if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    float alpha[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float mx = fmaxf(s[nb][h] + ve[0], s[nb][2 + h] + ve[1]);
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                        mx = fmaxf(mx, m_run[nb][h]);
                        alpha[h] = fast_exp2(m_run[nb][h] - mx);
                        m_run[nb][h] = mx;
                        l_run[nb][h] *= alpha[h];
#pragma unroll
                        for (int i = 0; i < NG; ++i) vbias[nb][i][h] *= alpha[h];
                    }
#pragma unroll
                    for (int i = 0; i < MT; ++i) {
                        acc[nb][i][0] *= alpha[0]; acc[nb][i][1] *= alpha[1];
                        acc[nb][i][2] *= alpha[0]; acc[nb][i][3] *= alpha[1];
                    }
                }
            }
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[nb][e] = fast_exp2(s[nb][e] - m_run[nb][e & 1]);
                    l_run[nb][e & 1] += s[nb][e];
                }
            // ---- values ----
            uint32_t pb[NB][2][2];                    // [high, low half][k half]
            auto pack_p = [&](float f0, float f1) {   // P^T fragments with the tokens' factors folded in
                f0 *= ST_PSCALE; f1 *= ST_PSCALE;
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float f = i ? f1 : f0, x = s[nb][2 * i] * f, y = s[nb][2 * i + 1] * f;
                        const uint32_t hi = pack_h2(x, y);
                        pb[nb][0][i] = movmatrix_free(hi);
                        pb[nb][1][i] = movmatrix_free(low_half2(hi, x, y));
                    }
            };
            // this lane's run of unit u of token 2c + j + 8h
            auto load_run = [&](int u, int j, int h, uint32_t (&w)[VW]) {
                if constexpr (V::POW2) {
                    const int off = u * (VU * V::BITS / 8) + g * (VRB / 8);
                    const uint32_t ad = vst + (8 * h + 4 * j + c) * V::RB + ((((off >> 4) ^ value_xor<VK, D>(c)) << 4) | (off & 15));
                    if constexpr (VRB == 16) w[0] = lds16(ad);
                    else if constexpr (VRB == 32) w[0] = lds32(ad);
                    else if constexpr (VRB == 64) { const uint2 v = lds64(ad); w[0] = v.x; w[1] = v.y; }
                    else { const uint4 v = lds128(ad); w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
                } else {                              // 3-bit indices: runs of 24, 48 and 96 bits
                    const int byte = g * (VRB / 8);
                    const uint32_t ad = vst + (2 * c + j + 8 * h) * V::RB + (byte & ~3);
                    if constexpr (VRB == 96) {
                        w[0] = lds32(ad); w[1] = lds32(ad + 4); w[2] = lds32(ad + 8);
                    } else {                          // (the word behind a run may be the next row's: its bits are not used)
                        const uint32_t lo = lds32(ad), hi = lds32(ad + 4);
                        w[0] = __funnelshift_r(lo, hi, 8 * (byte & 3));
                        if constexpr (VRB == 48) w[1] = hi >> (8 * (byte & 3));
                    }
                }
            };
            // the high halves of the centroids (or the exact codes) meet both halves of P, the low ones the high half
            auto mma_v = [&](int mt, const uint32_t (&a)[4]) {
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    mma_f16(acc[nb][mt], a, pb[nb][0][0], pb[nb][0][1]);
                    mma_f16(acc[nb][mt], a, pb[nb][1][0], pb[nb][1][1]);
                }
            };
            if constexpr (V::TURBO) {
                uint32_t even[2][VW], odd[2][VW];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t wa[VW], wb[VW];
                    load_run(0, 0, h, wa);
                    load_run(0, 1, h, wb);
                    pair_tokens<V::BITS, VW>(wa, wb, even[h], odd[h]);
                }
                pack_p(vf[0][0], vf[1][0]);
#pragma unroll
                for (int n = 0; n < VM; ++n) {
                    const uint2 x0 = table_entry(entry_offset<V::BITS, VW>(even[0], n, v_lane_bits)), x1 = table_entry(entry_offset<V::BITS, VW>(odd[0], n, v_lane_bits));
                    const uint2 x2 = table_entry(entry_offset<V::BITS, VW>(even[1], n, v_lane_bits)), x3 = table_entry(entry_offset<V::BITS, VW>(odd[1], n, v_lane_bits));
                    const uint32_t hi[4] = {x0.x, x1.x, x2.x, x3.x}, lo[4] = {x0.y, x1.y, x2.y, x3.y};
                    mma_v(n, hi);
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) mma_f16(acc[nb][n], lo, pb[nb][0][0], pb[nb][0][1]);
                }
            } else {
#pragma unroll
                for (int u = 0; u < NG; ++u) {
                    uint32_t w[2][2][VW];             // [token pair][token]
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        load_run(u, 0, h, w[h][0]);
                        load_run(u, 1, h, w[h][1]);
                    }
                    const int gr = (u * p.groups_v) / NG;
                    const uint32_t a0 = vst + V::BLOCK + V::SIDE + (g * p.groups_v + gr) * 2, a1 = a0 + 16 * p.groups_v;
                    pack_p(vf[0][u], vf[1][u]);
                    const float b0 = fmaf(vf[0][u], code_middle<VK>(), ld16<T>(a0)), b1 = fmaf(vf[1][u], code_middle<VK>(), ld16<T>(a1));
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            vbias[nb][u][h] = fmaf(s[nb][h], b0, fmaf(s[nb][2 + h], b1, vbias[nb][u][h]));
#pragma unroll
                    for (int n = 0; n < VM; n += 2) { // four dims: half a word of 4-bit codes, a word of 8-bit ones
                        uint32_t a[2][4];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if constexpr (VK == SK_A4) {
                                const uint32_t x = __byte_perm(w[h][0][0], w[h][1][0], (n & 2) ? 0x7632 : 0x5410);
                                a[0][2 * h] = code4(x, 0); a[0][2 * h + 1] = code4(x, 1);
                                a[1][2 * h] = code4(x, 2); a[1][2 * h + 1] = code4(x, 3);
                            } else {
                                const uint32_t x = __byte_perm(w[h][0][n >> 1], w[h][1][n >> 1], 0x5140), y = __byte_perm(w[h][0][n >> 1], w[h][1][n >> 1], 0x7362);
                                a[0][2 * h] = code8(x, 0); a[0][2 * h + 1] = code8(x, 1);
                                a[1][2 * h] = code8(y, 0); a[1][2 * h + 1] = code8(y, 1);
                            }
                        }
                        mma_v(u * VM + n, a[0]);
                        mma_v(u * VM + n + 1, a[1]);
                    }
                }
            }
            __syncwarp();   // this stage may be refilled
            stage ^= 1;
        }
        cp_wait<0>();

        // ---- end of the segment ----
        const int rr_n = fp.red_rows;
        float *red_o = (float *)body;
        float *red_ml = red_o + ST_WARPS * rr_n * SH::RED_STRIDE;
        float *work = red_ml + ((ST_WARPS * rr_n * 2 + 3) & ~3);      // 16-byte aligned for any row count
        __syncthreads();        // every warp has left the ring that the merge buffers overlay
        const float undo = (V::AFFINE ? 1.f : p.vcb_undo) / ST_PSCALE;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float l = l_run[nb][h];
#pragma unroll
                for (int o = 4; o <= 16; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
                float vb[NG];
#pragma unroll
                for (int i = 0; i < NG; ++i) {
                    vb[i] = 0.f;
                    if (V::AFFINE) {
                        vb[i] = vbias[nb][i][h];
#pragma unroll
                        for (int o = 4; o <= 16; o <<= 1) vb[i] += __shfl_xor_sync(0xffffffffu, vb[i], o);
                    }
                }
                const int r = 8 * nb + 2 * c + h;
                if (r < R) {
                    float *dst = red_o + (warp * rr_n + r) * SH::RED_STRIDE;
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        const int u = mt / VM;
                        const float b = vb[V::AFFINE ? u : 0];
                        *(float2 *)&dst[u * VU + g * VRUN + 2 * (mt % VM)] = make_float2(fmaf(acc[nb][mt][h], undo, b), fmaf(acc[nb][mt][2 + h], undo, b));
                    }
                    if (g == 0) {
                        red_ml[(warp * rr_n + r) * 2] = l > 0.f ? m_run[nb][h] : -INFINITY;
                        red_ml[(warp * rr_n + r) * 2 + 1] = l;
                    }
                }
            }
        UnitOut uo;
        uo.o_part = p.o_part; uo.ml_part = p.ml_part; uo.counters = p.counters;
        uo.out = p.out;
        uo.out_dtype = p.out_dtype;
        uo.o_sb = p.o_sb; uo.o_sh = p.o_sh; uo.o_sl = p.o_sl;
        uo.o_signs = p.o_signs;
        int b_row = sg.b;         // row of the partials: the batches of a list are laid end to end
        if constexpr (LIST) {
            b_row += sg.seq * p.B;
            uo.o_sb = list.seq[sg.seq].o_sb;
            uo.out = (T *)list.seq[sg.seq].out - (int64_t)sg.seq * p.B * uo.o_sb;
            uo.o_signs = list.seq[sg.seq].o_signs;
        }
        uo.splits = 0; uo.Hq = p.Hq; uo.L = p.L;
        segment_epilogue<D, ST_WARPS>(uo, fp, red_o, red_ml, SH::RED_STRIDE, work, flag, sg.unit, b_row, sg.hk, rep, R,
                                      sg.unit_x, sg.unit_tiles, row0, min(ST_WARPS, nblk));
        x += sg.tiles;
    }
}

template <typename T, int D, int KK, int VK, int UNIT, int NB, bool LIST>
void launch_stream_typed(const StreamParams &p, const void *list, int ctas, cudaStream_t stream) {
    using SH = StreamShape<T, D, KK, VK, UNIT, NB, LIST>;
    using LT = std::conditional_t<LIST, StreamList, StreamNoList>;
    auto kernel = attn_stream_kernel<T, D, KK, VK, UNIT, NB, LIST>;
    const size_t tables = SH::tables(p.v_table);
    const size_t smem = tables + SH::FIXED;
    static size_t configured[64] = {0};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && configured[dev] < smem) {
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured[dev] = smem;
    }
    static const LT none = {};
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(kernel, dim3(ctas), dim3(SH::THREADS), smem, stream, p, list ? *(const LT *)list : none));
    timer.stop();
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

struct StreamPick {
    int kk, vk, unit;
};

// The flat plan over `work` tiles, `max_tiles` in the longest unit; false when the partials need too many slots.
inline bool stream_plan(const AttnArgs &a, int64_t units, int64_t work, int64_t max_tiles, int resident, int rows, StreamParams *p,
                 int64_t qrows, cudaStream_t stream, int *ctas) {
    if (units * (int64_t)sizeof(int) > ST_COUNTER_BYTES || !flat_fits(2 * units * max_tiles)) return false;
    const int64_t slots = (int64_t)sm_count(a.device) * resident;
    int64_t n;
    if (work == units * max_tiles) {
        n = plan_units(&p->flat, units, max_tiles, slots, ST_SEGMENT);
    } else {
        n = std::min(slots, work);
        p->flat.tiles = (int)max_tiles;
        p->flat.step = 1;
        p->flat.per = (int)(work / n);
        p->flat.rem = (int)(work % n);
        p->flat.nslots = (int)((max_tiles + p->flat.per - 1) / p->flat.per + 1);
    }
    p->flat.red_rows = rows;
    const size_t o_bytes = (size_t)qrows * p->flat.nslots * a.D * sizeof(float);
    char *scratch = (char *)scratch_get(a.device, o_bytes + (size_t)qrows * p->flat.nslots * sizeof(float2) + 256, stream);
    p->o_part = (float *)scratch;
    p->ml_part = (float2 *)(scratch + ((o_bytes + 255) / 256) * 256);
    p->counters = counters_get(a.device, stream, ST_COUNTER_BYTES);
    *ctas = (int)n;
    return true;
}

// The tiles of a list's calls where the plan has rounded them up (then all calls have as many).
template <typename Seq>
inline void stream_list_tiles(Seq *seq, int n, int64_t units, const UnitPlan &f) {
    if (f.step == 1) return;
    for (int i = 0; i < n; ++i) {
        seq[i].tiles = f.tiles;
        seq[i].tile_first = i * units * f.tiles;
    }
}

// One call (list null) or a list of calls of one shape in one launch.
template <typename T, int D, int KK, int VK, int UNIT, int NB>
int run_stream(const AttnArgs &a, StreamParams p, StreamList *list, cudaStream_t stream) {
    const int rows = a.Hq / a.Hkv * a.L;
    p.chunks = (rows + 8 * NB - 1) / (8 * NB);
    const int64_t units = (int64_t)a.B * a.Hkv * p.chunks;
    const int n = list ? list->n : 1;
    int64_t work = 0, most = 0;
    if (list)
        for (int i = 0; i < n; ++i) {
            StreamSeq &sq = list->seq[i];
            sq.tiles = (sq.T + ST_TILE - 1) / ST_TILE;
            sq.tile_first = work;
            work += units * sq.tiles;
            most = std::max<int64_t>(most, sq.tiles);
        }
    else work = units * (most = (a.T + ST_TILE - 1) / ST_TILE);
    int ctas;
    if (!stream_plan(a, n * units, work, most, StreamShape<T, D, KK, VK, UNIT, NB, false>::RESIDENT, std::min(rows, 8 * NB), &p,
                     (int64_t)n * a.B * a.Hq * a.L, stream, &ctas))
        return 0;
    if constexpr (NB <= 2) {   // lists hold up to sixteen rows
        if (list) {
            stream_list_tiles(list->seq, n, units, p.flat);
            launch_stream_typed<T, D, KK, VK, UNIT, NB, true>(p, list, ctas, stream);
            return 1;
        }
    }
    launch_stream_typed<T, D, KK, VK, UNIT, NB, false>(p, nullptr, ctas, stream);
    return 1;
}

// Up to eight rows per KV head: one column block. More: two column blocks share one unpacking where the
// accumulators fit the registers (D <= 128), else units of eight rows. At head dim 64 four blocks, but only where a CTA
// walks many tiles (the line: 128 an SM): a verify round of 28 rows over 30 x 17 642 tokens, 3-bit keys and 4-bit values, takes
// 460 us in units of sixteen rows and 399 in units of 32; over 4 x 1 500 tokens the longer start of a segment costs more
// than the second unpacking (two layers: 38 us and 45).
template <typename T, int D, int KK, int VK, int UNIT>
int run_stream_rows(const AttnArgs &a, const StreamParams &p, StreamList *list, cudaStream_t stream) {
    if constexpr (D == 64) {
        const int64_t tiles = (int64_t)a.B * a.Hkv * ((a.T + ST_TILE - 1) / ST_TILE);
        if (!list && a.Hq / a.Hkv * a.L > 16 && tiles >= 128 * (int64_t)sm_count(a.device))
            return run_stream<T, D, KK, VK, UNIT, 4>(a, p, nullptr, stream);
    }
    if constexpr (D <= 128)
        if (a.Hq / a.Hkv * a.L > 8) return run_stream<T, D, KK, VK, UNIT, 2>(a, p, list, stream);
    return run_stream<T, D, KK, VK, UNIT, 1>(a, p, list, stream);
}

template <typename T, int D>
int run_stream_kinds(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream) {
#define KVC_ST(KK, VK)                                                                             \
    if (pk.kk == KK && pk.vk == VK) return run_stream_rows<T, D, KK, VK, 64>(a, p, list, stream);
#define KVC_STA(KK, VK)                                                                            \
    if (pk.kk == KK && pk.vk == VK)                                                                \
        return pk.unit == 32 ? run_stream_rows<T, D, KK, VK, 32>(a, p, list, stream) : run_stream_rows<T, D, KK, VK, 64>(a, p, list, stream);
    KVC_STA(SK_A4, SK_A4) KVC_STA(SK_A8, SK_A8)
    KVC_ST(SK_T2, SK_T2) KVC_ST(SK_T3, SK_T3) KVC_ST(SK_T4, SK_T4) KVC_ST(SK_T3, SK_T4) KVC_ST(SK_T4, SK_T2)
    KVC_ST(SK_RAW, SK_T2) KVC_ST(SK_RAW, SK_T3) KVC_ST(SK_RAW, SK_T4)
    KVC_STA(SK_A8, SK_T2) KVC_STA(SK_A8, SK_T3) KVC_STA(SK_A8, SK_T4)
    KVC_STA(SK_T3, SK_A4) KVC_STA(SK_T4, SK_A4)
#undef KVC_ST
#undef KVC_STA
    return 0;
}

}  // namespace stream

}  // namespace kvc
