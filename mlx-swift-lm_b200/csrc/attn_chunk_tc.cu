// Prefill / long verify chunks over raw K/V on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// attentionWithCacheUpdate's scaledDotProductAttention call (AttentionUtils.swift:87-93) for a chunk
// of L query positions per head. The query rows of a KV head's group are cut into tiles of up to 128
// rows, position-major (a tile is `lb` positions x `hb` heads of the group: an odd group wastes no row
// block and a tile's causal limits lie close together). A unit is TWO neighbouring row tiles, A and B,
// which share every K and V tile, or, where the tiles do not fill the SMs (SINGLE), one.
//
//   warps 0..3  softmax of tile A, warps 4..7 of tile B: thread = query row = TMEM lane. The 128 scores of a
//               key tile come out of TMEM in one round trip, row maximum, exponentials, and P goes back into
//               TMEM over the scores' own columns, where the O product reads it as its A operand
//   warp 8 (4)  TMA producer: Q tiles per unit, K and V tiles into one ring
//   warp 9 (5)  owns the TMEM allocation and issues the MMAs in the order
//                 O_A += P_A(j) V_j | S_A = Q_A K_{j+1}^T | O_B += P_B(j) V_j | S_B = Q_B K_{j+1}^T
//               so that one tile's products run while the other tile's softmax does. A single row tile has B's buffer for
//               its scores too, S of tile j + 1 comes before O += P(j) V(j), and there are no warps 4..7
//
// O accumulates in TMEM, in the reference that the row's exponents are taken against. The scores of tile j + 1 are
// issued behind the O product of tile j, so when they arrive O is settled and the softmax threads may multiply it; they
// do so under their exponentials, which wait for the special-function unit. Two forms:
//   the reference is the row's running maximum, which moves at most once per 128 keys (PARTS = 1);
//   it is the largest score of every 128 / PARTS keys, also where that is below the row's (PARTS = 2 or 4): the largest
//   probability of each part is exactly 1 and loses nothing to the 16-bit store, so the errors against 64-bit sums are
//   4 ... 10 % smaller (bf16 and f16, 128 ... 16 000 keys), for O products in parts with a rescale between them.
//
// The tensor core adds towards zero: a sum of n keys in one accumulator loses 6e-9 n of itself (values of one sign), which
// outgrows the rounding of an f16 output within a few thousand keys. After `fold` key tiles the softmax threads therefore add
// O to fp32 sums of their own, behind O in TMEM or, for pairs at head dim 128, in memory, and the next O product starts from
// nothing.
//
// Units are handed out whole, in rounds of one per SM; what is left over is laid end to end and cut into equal ranges,
// or few units are cut into pieces (a cut unit leaves fp32 partials, and the CTA that finishes it merges them).
//
// TMEM columns: S_A / P_A at 0, S_B / P_B at 128, O_A at 256, O_B at 384. (Single: S_0 / P_0, S_1 / P_1, O, folded sums.)
//
// Shared-memory operand layout (what TMA's 128-byte swizzle writes): a box is 128 rows x 128 bytes
// (64 elements), 16-byte chunk c of row r at chunk c ^ (r & 7); a 128 x 128 tile is two boxes (Q, K and
// V tiles at head dim 64 are one box, the O product then has 64 columns).
// Matrix descriptors: K-major operands advance 32 bytes per 16-element k-step inside the row, 8-row
// groups are 1024 bytes apart; the MN-major V tile advances 2048 bytes per 16 keys, its two 64-dim
// halves are 16384 bytes apart (leading offset) and its 8-key groups 1024 bytes (stride offset).
//
// Every wait is bounded; a wait that runs out sets the device status word, the CTA waits (bounded too) for its copies and
// products in flight and frees its TMEM.
#include <atomic>
#include <climits>
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "attn_common.cuh"
#include "common.h"
#include "tc_common.cuh"

namespace kvc {
namespace {

using namespace dev;

using namespace tc;

// Pairs: registers a thread: 384 * 168 at launch = 256 * 216 (softmax) + 128 * 72 (the warps that issue copies and MMAs). A single
// row tile has half the softmax warps, and registers enough as launched.
template <bool SINGLE> constexpr int ct_threads() { return SINGLE ? 192 : 384; }
constexpr int CT_REGS_SOFTMAX = 216, CT_REGS_ISSUE = 72;
// The reference of a part is never further below the row's largest score than this, so that O and the sums stay far
// from overflow.
constexpr float CT_SPAN_LOG2 = 24.f;

struct ChunkTcParams {
    void *out;
    int64_t o_sb, o_sh, o_sl;
    int32_t rep, Hkv, L;
    int64_t T;
    int32_t wide;               // row tiles a unit
    int32_t hb, lb;             // heads and positions of a row tile (hb * lb <= 128)
    int32_t head_tiles;         // row tiles side by side over the group's heads
    int32_t row_tiles;          // row tiles of a (batch, KV head)
    int32_t units;              // ... and units of one or two row tiles
    int32_t causal;
    int64_t causal_offset;
    float scale_log2;
    // units end to end over all (batch, KV head): CTA c walks units c, c + grid, ... of the first waves * grid, then the
    // key tiles [c * per + min(c, rem), ...) of the rest (the tail), whose units are cut where the ranges end
    int32_t all_units, waves;
    int32_t ranges, per, rem;   // ranges = 0: no tail
    int32_t pieces;             // not 0: every unit is cut into this many pieces, one CTA each (no rounds, no tail)
    int32_t group_tiles;        // key tiles of the units of a (batch, KV head)
    int32_t tail_base;          // ... of those before the tail's first unit in its own group
    int32_t fold;               // key tiles of a segment between two folds
    float *o_fold;              // [CTA][A / B][D / 4][128 rows][4] (pairs at head dim 128)
    float *o_part;              // [CTA][first / last segment][A / B][D / 4][128 rows][4]
    float2 *ml_part;            // [CTA][first / last segment][A / B][128 rows] (reference, sum)
    int *tickets;               // [unit of the tail][A / B], zeroed before the launch
    int *status;
};

template <int D> constexpr int ct_stages() { return D == 128 ? 5 : 10; }

template <int STAGES> struct Bars {
    enum : int {
        Q_FULL = 0,                        // [2] row tile A / B
        Q_EMPTY = Q_FULL + 2,              // [2] free once the unit's last S product has read the tile
        RING_FULL = Q_EMPTY + 2,           // [STAGES] K_0, V_0, K_1, V_1, ...
        RING_EMPTY = RING_FULL + STAGES,   // [STAGES]
        S_FULL = RING_EMPTY + STAGES,      // [2]
        P_FULL = S_FULL + 2,               // [4][2] the probabilities of a part of the tile, O in their reference
        O_PART = P_FULL + 8,               // [2] the O product of a part other than the last is done
        O_FULL = O_PART + 2,               // [2] the segment's last O product is done
        GROUP = O_FULL + 2,                // [2] the 128 threads of a softmax group meet
        DRAIN = GROUP + 2,                 // the products of a CTA that gave up are done
        COUNT = DRAIN + 1
    };
};

// The first row tile of a unit, and its key tiles. Units of a (batch, KV head) are counted from the last positions
// to the first: with a causal mask the long units go first.
__device__ __host__ inline int ct_first_of(const ChunkTcParams &p, int unit) { return p.wide * (p.units - 1 - unit % p.units); }
__device__ __host__ inline int ct_unit_tiles(const ChunkTcParams &p, int unit) {
    if (!p.causal) return (int)((p.T + TC_KEYS - 1) / TC_KEYS);
    const int first = ct_first_of(p, unit), last_tile = first + p.wide <= p.row_tiles ? first + p.wide - 1 : p.row_tiles - 1;
    const int64_t end = (int64_t)(last_tile / p.head_tiles + 1) * p.lb;
    const int64_t keys = p.causal_offset + (end < p.L ? end : p.L);
    return (int)(((keys < p.T ? keys : p.T) + TC_KEYS - 1) / TC_KEYS);
}

// A CTA's work in segments, one per unit it touches. (What takes divisions is worked out once, before the wait for the launch
// ahead: on short calls the producer's first copy and the stores waited for it.)
struct CtSegment {
    int unit;
    int t0, t1, n;     // its key tiles, and the unit's
    int has_b;         // the unit has two row tiles
    int hk, b;         // KV head and sequence
    int l0[2], h0[2];  // first position and head of the row tiles
};
constexpr int CT_MAX_SEGMENTS = 40;

template <typename T, int D, int PARTS, bool SINGLE>
__global__ void __launch_bounds__(ct_threads<SINGLE>(), 1)
attn_chunk_tc_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                     const __grid_constant__ CUtensorMap vmap, const __grid_constant__ ChunkTcParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    // parts in which a tile's probabilities are handed over; with one reference for all of them, the first 96 keys and the
    // rest (their O product runs under the other exponentials; 64 keys: 3 % slower)
    constexpr int HANDS = PARTS == 1 ? 2 : PARTS;
    auto key_of = [](int part) constexpr { return PARTS == 1 ? (part == 0 ? 0 : part == 1 ? 96 : TC_KEYS) : part * (TC_KEYS / PARTS); };
    constexpr int STAGES = ct_stages<D>();
    using BAR = Bars<STAGES>;
    constexpr int NBOX = D / 64;                               // boxes of 64 head dims per Q / K / V tile
    constexpr int TILE = NBOX * TC_BOX;                        // bytes of a 128-row tile of D head dims
    unsigned char *sq = base;                                  // Q tiles A, B
    unsigned char *ring = sq + 2 * TILE;
    uint64_t *bars = (uint64_t *)(ring + STAGES * TILE);
    uint32_t *tmem_slot = (uint32_t *)(bars + BAR::COUNT);
    int *s_segments = (int *)(tmem_slot + 1);
    int *s_ticket = s_segments + 1;                            // [2]
    CtSegment *s_seg = (CtSegment *)(s_ticket + 2);            // [CT_MAX_SEGMENTS]

    constexpr int THREADS = ct_threads<SINGLE>(), PRODUCER = SINGLE ? 4 : 8, ISSUER = PRODUCER + 1;   // (warps)
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // known to be the same in all lanes: a role's addresses stay in uniform registers

    if (tid == 0) {
        for (int w = 0; w < 2; ++w) {
            mbar_init(&bars[BAR::Q_FULL + w], 1);
            mbar_init(&bars[BAR::Q_EMPTY + w], 1);
            mbar_init(&bars[BAR::S_FULL + w], 1);
            for (int h = 0; h < 4; ++h) mbar_init(&bars[BAR::P_FULL + 2 * h + w], 128);
            mbar_init(&bars[BAR::O_PART + w], 1);
            mbar_init(&bars[BAR::O_FULL + w], 1);
            mbar_init(&bars[BAR::GROUP + w], 128);
        }
        mbar_init(&bars[BAR::DRAIN], 1);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&bars[BAR::RING_FULL + s], 1);
            mbar_init(&bars[BAR::RING_EMPTY + s], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        // the segments of the CTA
        if (lane < 3) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)(lane == 0 ? &qmap : lane == 1 ? &kmap : &vmap)) : "memory");
        const int c = blockIdx.x;
        int segments = 0;
        auto add = [&](int unit, int t0, int t1, int n) {
            if (lane == 0) {
                CtSegment &g = s_seg[segments];
                g.unit = unit;
                g.t0 = t0; g.t1 = t1; g.n = n;
                const int group = unit / p.units, rt = ct_first_of(p, unit);
                g.has_b = !SINGLE && rt + 1 < p.row_tiles;
                g.b = group / p.Hkv;
                g.hk = group - g.b * p.Hkv;
                for (int i = 0; i < (SINGLE ? 1 : 2); ++i) {
                    const int row_block = (rt + i) / p.head_tiles;
                    g.l0[i] = row_block * p.lb;
                    g.h0[i] = (rt + i - row_block * p.head_tiles) * p.hb;
                }
            }
            ++segments;
        };
        if (p.pieces > 0) {
            const int unit = c / p.pieces, piece = c % p.pieces, n = ct_unit_tiles(p, unit);
            add(unit, n * piece / p.pieces, n * (piece + 1) / p.pieces, n);
        }
        for (int r = 0; r < p.waves; ++r) {
            const int unit = r * (int)gridDim.x + c;
            if (unit < p.all_units) {
                const int n = ct_unit_tiles(p, unit);
                add(unit, 0, n, n);
            }
        }
        if (c < p.ranges) {
            // the unit of the range's first tile: its group by division, the unit by a scan over the group's
            const int pos = p.tail_base + c * p.per + min(c, p.rem);
            int unit = (p.waves * (int)gridDim.x / p.units + pos / p.group_tiles) * p.units, t = pos % p.group_tiles;
            for (int e = 0; e < p.units; e += 32) {
                const int n = e + lane < p.units ? ct_unit_tiles(p, unit + e + lane) : 0;
                int upto = n;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int o = __shfl_up_sync(0xffffffffu, upto, d);
                    if (lane >= d) upto += o;
                }
                const unsigned past = __ballot_sync(0xffffffffu, upto > t);
                if (past) {
                    const int at = __ffs(past) - 1;
                    unit += e + at;
                    t -= __shfl_sync(0xffffffffu, upto - n, at);
                    break;
                }
                t -= __shfl_sync(0xffffffffu, upto, 31);
            }
            int left = p.per + (c < p.rem ? 1 : 0);
            while (left > 0 && segments < CT_MAX_SEGMENTS) {
                const int n = ct_unit_tiles(p, unit);
                add(unit, t, min(n, t + left), n);
                left -= n - t;
                t = 0;
                ++unit;
            }
        }
        if (lane == 0) *s_segments = segments;
    }
    // rows of a Q tile that no copy writes are zero
    for (int i = tid; i < 2 * NBOX * (TC_ROWS - p.hb * p.lb) * 8; i += THREADS) {
        const int chunk = i & 7, box = (i >> 3) % (2 * NBOX), row = (i >> 3) / (2 * NBOX) + p.hb * p.lb;
        *(uint4 *)(sq + box * TC_BOX + row * 128 + chunk * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    // the first copies are on their way while the others wait for the TMEM columns
    if (warp == ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp != PRODUCER) {
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(THREADS - 32) : "memory");
        tc_fence_after();
    }
    const uint32_t tmem = warp == PRODUCER ? 0u : *tmem_slot;       // (nothing of the producer's)
    const int segments = *s_segments;
    pdl_wait();  // everything below reads what earlier kernels on the stream wrote

    if (warp >= PRODUCER) {
        if constexpr (!SINGLE) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CT_REGS_ISSUE));
        if (warp == PRODUCER && lane == 0) {
            // ---------------- producer ----------------
            bool ok = true;
            uint32_t slot = 0, round = 0, q_used[2] = {0, 0};
            auto load_tile = [&](const CUtensorMap *map, int t, int hk, int b) {
                if (round > 0 && !mbar_wait(&bars[BAR::RING_EMPTY + slot], (round - 1) & 1)) return false;
                unsigned char *dst = ring + (size_t)slot * TILE;
                mbar_expect_tx(&bars[BAR::RING_FULL + slot], TILE);
#pragma unroll
                for (int bx = 0; bx < NBOX; ++bx) tma_load_4d(dst + bx * TC_BOX, map, &bars[BAR::RING_FULL + slot], bx * 64, t * TC_KEYS, hk, b);
                if (++slot == STAGES) {
                    slot = 0;
                    ++round;
                }
                return true;
            };
            for (int sg = 0; ok && sg < segments; ++sg) {
                const CtSegment &g = s_seg[sg];
                const int hk = g.hk, b = g.b;
                ok = load_tile(&kmap, g.t0, hk, b);
                for (int i = 0; ok && i <= g.has_b; ++i) {
                    if (q_used[i] > 0) ok = mbar_wait(&bars[BAR::Q_EMPTY + i], (q_used[i] - 1) & 1);
                    if (!ok) break;
                    ++q_used[i];
                    mbar_expect_tx(&bars[BAR::Q_FULL + i], (uint32_t)(p.hb * p.lb * 128 * NBOX));
#pragma unroll
                    for (int bx = 0; bx < NBOX; ++bx)
                        tma_load_5d(sq + i * TILE + bx * TC_BOX, &qmap, &bars[BAR::Q_FULL + i], bx * 64, g.h0[i], g.l0[i], hk, b);
                }
                for (int t = g.t0; ok && t < g.t1; ++t) {
                    if (t > g.t0) ok = load_tile(&kmap, t, hk, b);
                    if (ok) ok = load_tile(&vmap, t, hk, b);
                }
            }
            if (!ok) {
                atomicExch(p.status, 21);
                drain_copies(&bars[BAR::RING_FULL], STAGES, slot, round);
#pragma unroll 1
                for (int i = 0; i < 2; ++i)
                    if (q_used[i] > 0) (void)mbar_wait(&bars[BAR::Q_FULL + i], (q_used[i] - 1) & 1);
            }
        } else if (warp == ISSUER) {
            // ---------------- MMA issue ----------------
            // instruction descriptor: f32 accumulator (bits 4-5 = 1), A and B formats (bits 7-9 and 10-12:
            // 0 = f16, 1 = bf16), B major at bit 16 (1 = MN-major), N / 8 at bits 17-22, M / 16 at 24-28
            constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
            constexpr uint32_t IDESC = (1u << 4) | (FMT << 7) | (FMT << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
            // the O product has N = D columns
            constexpr uint32_t IDESC_PV = (1u << 4) | (FMT << 7) | (FMT << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((128u >> 4) << 24);
            // Descriptors differ only in the start-address field (16-byte units): a box is 1024 units, a
            // k-step inside a box row 2, 16 keys of the MN-major V tile 128.
            const uint64_t q_desc = umma_desc(smem_u32(sq), 16, 1024);
            const uint64_t k_desc = umma_desc(smem_u32(ring), 16, 1024);
            const uint64_t v_desc = umma_desc(smem_u32(ring), 16384, 1024);
            bool ok = true;
            uint32_t k_slot = 0, k_par = 0, v_slot = 1, v_par = 0;   // ring entries of the next K and V tile
            uint32_t q_par = 0, p_par = 0;                           // bit i: row tile i
            auto step2 = [](uint32_t &slot, uint32_t &par) {
                slot += 2;
                if (slot >= (uint32_t)STAGES) {
                    slot -= STAGES;
                    par ^= 1;
                }
            };
            if constexpr (SINGLE) {
                // One step takes the S product of a key tile, into the buffer its predecessor does not use, and the O product of
                // that predecessor.
                int sg = 0, left = 0, since = 0;     // the segment of the next S product, its tiles still to come; S products behind the last fold
                bool o_here = false, o_first = false;
                for (uint32_t n = 0; ok; ++n) {
                    const bool opens = left == 0 && sg < segments;
                    if (opens) {
                        left = s_seg[sg].t1 - s_seg[sg].t0;
                        ++sg;
                    }
                    const bool s_here = left > 0, o_last = o_here && (opens || !s_here);
                    if (!o_here && !s_here) break;
                    if (s_here) {
                        ok = warp_wait(&bars[BAR::RING_FULL + k_slot], k_par);
                        if (ok && opens) {
                            ok = warp_wait(&bars[BAR::Q_FULL], q_par);
                            q_par ^= 1;
                        }
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t kd = k_desc + (uint64_t)(k_slot * (TILE / 16));
                        if (elect_one()) {
#pragma unroll
                            for (int ks = 0; ks < D / 16; ++ks) {
                                const uint64_t off = (uint64_t)((ks >> 2) * (TC_BOX / 16) + (ks & 3) * 2);
                                umma_f16(tmem + (n & 1) * 128u, q_desc + off, kd + off, IDESC, ks > 0 ? 1u : 0u);
                            }
                            umma_commit(&bars[BAR::S_FULL + (n & 1)]);
                            if (left == 1) umma_commit(&bars[BAR::Q_EMPTY]);
                            umma_commit(&bars[BAR::RING_EMPTY + k_slot]);
                        }
                        __syncwarp();
                        step2(k_slot, k_par);
                    }
                    if (o_here) {
                        const uint32_t buf = (n - 1) & 1, par = ((n - 1) >> 1) & 1;
                        ok = warp_wait(&bars[BAR::RING_FULL + v_slot], v_par);
                        const uint64_t vd = v_desc + (uint64_t)(v_slot * (TILE / 16));
                        auto o_part = [&](auto which) {
                            constexpr int h = decltype(which)::value, FROM = key_of(h) / 16, TO = key_of(h + 1) / 16;
                            if (ok) ok = warp_wait(&bars[BAR::P_FULL + 2 * h + buf], par);
                            if (!ok) return;
                            tc_fence_after();
                            if (elect_one()) {
#pragma unroll
                                for (int ks = FROM; ks < TO; ++ks)
                                    umma_f16_ts(tmem + 256u, tmem + buf * 128u + (uint32_t)ks * 8u, vd + (uint64_t)(ks * 128), IDESC_PV,
                                                (o_first && ks == 0) ? 0u : 1u);
                                if (PARTS > 1 || h == HANDS - 1) umma_commit(&bars[BAR::O_PART]);
                                if (h == HANDS - 1) {
                                    if (o_last) umma_commit(&bars[BAR::O_FULL]);
                                    umma_commit(&bars[BAR::RING_EMPTY + v_slot]);
                                }
                            }
                            __syncwarp();
                        };
                        o_part(std::integral_constant<int, 0>());
                        o_part(std::integral_constant<int, 1>());
                        if constexpr (HANDS == 4) {
                            o_part(std::integral_constant<int, 2>());
                            o_part(std::integral_constant<int, 3>());
                        }
                        step2(v_slot, v_par);
                    }
                    o_here = s_here;
                    since = opens || since == p.fold - 1 ? 0 : since + 1;
                    o_first = since == 0;
                    if (s_here) --left;
                }
            }
            // One step takes the O products of a key tile and the S products of the next one, which may open the next segment.
            int sg = 0, left = 0;                    // the segment of the next S products, and its tiles still to come
            int since = 0;                           // S products behind the last fold
            bool o_here = false, o_first = false, o_b = false, b = false;   // *b: the unit has a row tile B
            while (!SINGLE && ok) {
                const bool opens = left == 0 && sg < segments;
                o_b = b;
                if (opens) {
                    left = s_seg[sg].t1 - s_seg[sg].t0;
                    b = s_seg[sg].has_b != 0;
                    ++sg;
                }
                const bool s_here = left > 0, s_last = left == 1, o_last = o_here && (opens || !s_here);
                if (!o_here && !s_here) break;
                if (o_here) ok = warp_wait(&bars[BAR::RING_FULL + v_slot], v_par);
                if (ok && s_here) ok = warp_wait(&bars[BAR::RING_FULL + k_slot], k_par);
                const uint64_t kd = k_desc + (uint64_t)(k_slot * (TILE / 16)), vd = v_desc + (uint64_t)(v_slot * (TILE / 16));
                auto o_part = [&](uint32_t i, auto which) {
                    constexpr int h = decltype(which)::value, FROM = key_of(h) / 16, TO = key_of(h + 1) / 16;
                    if (ok) ok = warp_wait(&bars[BAR::P_FULL + 2 * h + i], (p_par >> i) & 1);
                    if (!ok) return;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int ks = FROM; ks < TO; ++ks)
                            umma_f16_ts(tmem + 256u + i * 128u, tmem + i * 128u + (uint32_t)ks * 8u, vd + (uint64_t)(ks * 128), IDESC_PV,
                                        (o_first && ks == 0) ? 0u : 1u);
                        if (PARTS > 1) umma_commit(&bars[BAR::O_PART + i]);
                    }
                    __syncwarp();
                };
                // (a part waits for the rescale behind the one before: the other row tile's part runs meanwhile)
                if (PARTS > 1 && o_here) {
                    o_part(0, std::integral_constant<int, 0>());
                    if (o_b) o_part(1, std::integral_constant<int, 0>());
                }
                if (PARTS == 4 && o_here) {
                    o_part(0, std::integral_constant<int, 1>());
                    if (o_b) o_part(1, std::integral_constant<int, 1>());
                    o_part(0, std::integral_constant<int, 2>());
                    if (o_b) o_part(1, std::integral_constant<int, 2>());
                }
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    if (!ok) break;
                    const bool o_i = o_here && (i == 0 || o_b), s_i = s_here && (i == 0 || b);
                    if (s_i && opens) {
                        ok = warp_wait(&bars[BAR::Q_FULL + i], (q_par >> i) & 1);
                        q_par ^= 1u << i;
                    }
                    if (o_i) {
                        if (PARTS == 1) o_part(i, std::integral_constant<int, 0>());
                        if (ok) ok = warp_wait(&bars[BAR::P_FULL + 2 * (HANDS - 1) + i], (p_par >> i) & 1);
                        p_par ^= 1u << i;
                    }
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t s_addr = tmem + i * 128u;
                        if (o_i) {
#pragma unroll
                            for (int ks = key_of(HANDS - 1) / 16; ks < TC_KEYS / 16; ++ks)
                                umma_f16_ts(tmem + 256u + i * 128u, s_addr + (uint32_t)ks * 8u, vd + (uint64_t)(ks * 128), IDESC_PV, 1u);
                            if (o_last) umma_commit(&bars[BAR::O_FULL + i]);
                        }
                        if (s_i) {
                            const uint64_t qd = q_desc + (uint64_t)(i * (TILE / 16));
#pragma unroll
                            for (int ks = 0; ks < D / 16; ++ks) {
                                const uint64_t off = (uint64_t)((ks >> 2) * (TC_BOX / 16) + (ks & 3) * 2);
                                umma_f16(s_addr, qd + off, kd + off, IDESC, ks > 0 ? 1u : 0u);
                            }
                            umma_commit(&bars[BAR::S_FULL + i]);
                            if (s_last) umma_commit(&bars[BAR::Q_EMPTY + i]);
                        }
                        if (i == 1) {
                            if (o_here) umma_commit(&bars[BAR::RING_EMPTY + v_slot]);
                            if (s_here) umma_commit(&bars[BAR::RING_EMPTY + k_slot]);
                        }
                    }
                    __syncwarp();
                }
                if (o_here) step2(v_slot, v_par);
                if (s_here) step2(k_slot, k_par);
                o_here = s_here;
                since = opens || since == p.fold - 1 ? 0 : since + 1;
                o_first = since == 0;
                if (s_here) --left;
            }
            if (!ok) {
                atomicExch(p.status, 22);
                drain_products(&bars[BAR::DRAIN]);
            }
        }
    } else {
        // ---------------- softmax and output: thread = row ----------------
        if constexpr (!SINGLE) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CT_REGS_SOFTMAX));
        const int i = warp >> 2;                            // row tile A / B
        const int quarter = warp & 3;                       // the TMEM lanes this warp may touch
        const int row = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16), o_addr = lanes + 256u + (uint32_t)i * 128u;
        uint32_t buf = i, s_addr = lanes + buf * 128u;       // S / P buffer: the row tile's own, or both in turn
        const int row_l = row / p.hb, row_h = row % p.hb;
        const uint64_t scale2 = pack_f2(p.scale_log2, p.scale_log2);
        uint32_t s_par = 0, o_par = 0, g_par = 0, h_par = 0;
        bool ok = true;
        for (int sg = 0; ok && sg < segments; ++sg) {
            const CtSegment &w = s_seg[sg];
            if (i == 1 && !w.has_b) continue;
            const int l0 = w.l0[i], l = l0 + row_l, h = w.h0[i] + row_h;
            const bool valid = row < p.hb * p.lb && l < p.L && h < p.rep;
            const int limit = (int)(p.causal ? min(p.T - 1, p.causal_offset + l) : p.T - 1);     // last visible key
            const int tile_limit = (int)(p.causal ? min(p.T - 1, p.causal_offset + l0) : p.T - 1);
            float m_top = -INFINITY, m_ref = -INFINITY, l_run = 0.f;   // largest score, reference of O and of l_run
            int since = -1;                                            // tiles behind the last fold
            using Sums = FoldedSums<D, SINGLE || D == 64>;
            Sums sums(o_addr, (float4 *)p.o_fold + ((int64_t)blockIdx.x * 2 + i) * (D / 4) * TC_ROWS + row);
            for (int t = w.t0; t < w.t1; ++t) {
                ok = warp_wait(&bars[BAR::S_FULL + buf], s_par);
                if (!ok) break;
                if (!SINGLE) s_par ^= 1;
                tc_fence_after();
                // one row tile: the scores come while the O product of the tile before may be under way
                bool settled = !SINGLE || t == w.t0;
                auto settle = [&] {
                    ok = warp_wait(&bars[BAR::O_PART], h_par);
                    h_par ^= 1;
                    tc_fence_after();
                    settled = true;
                };
                typename Sums::Form fold = Sums::DONE;
                float fold_f = 1.f;
                if (++since == p.fold) {
                    if (!settled) settle();
                    if (!ok) break;
                    fold = sums.begin(m_ref, fold_f);
                    since = 0;
                }
                uint32_t raw[TC_KEYS];
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) tmem_ld32_issue(s_addr + cb * 32, raw + cb * 32);
                tmem_ld_wait();
                if (t * TC_KEYS + TC_KEYS - 1 > tile_limit) {   // some row of the tile loses keys here
                    const int last = limit - t * TC_KEYS;
#pragma unroll
                    for (int k = 0; k < TC_KEYS; ++k)
                        if (k > last) raw[k] = 0xff800000u;   // -inf
                }
                float ref[PARTS], alpha[PARTS];
#pragma unroll
                for (int part = 0; part < PARTS; ++part) {
                    constexpr int KEYS = TC_KEYS / PARTS;
                    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int k = part * KEYS; k < (part + 1) * KEYS; k += 2)
                        mx4[(k >> 1) & 3] = fmaxf(mx4[(k >> 1) & 3], fmaxf(__uint_as_float(raw[k]), __uint_as_float(raw[k + 1])));
                    const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
                    m_top = fmaxf(m_top, mx);
                    ref[part] = PARTS > 1 ? fmaxf(mx, m_top - CT_SPAN_LOG2) : m_top;
                    alpha[part] = m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - ref[part]);
                    m_ref = ref[part];
                }
                // O is settled when the scores of a pair are there: they came behind the O products of the tile before
                auto hand_over = [&](auto which) {
                    constexpr int h = decltype(which)::value, FROM = key_of(h), TO = key_of(h + 1), part = PARTS == 1 ? 0 : h;
                    const bool first = h == 0, lay = first && fold != Sums::DONE;
                    const bool move = (first ? since > 0 : PARTS > 1) && __any_sync(0xffffffffu, alpha[part] != 1.f);
                    const uint64_t alpha2 = pack_f2(alpha[part], alpha[part]);
                    constexpr int CH = PARTS == 1 ? 32 : 16;   // columns of O at a time (16: 3 % slower with one reference)
                    uint32_t o[CH];
                    auto o_load = [&](int cb) {
                        if constexpr (CH == 32) tmem_ld32_issue(o_addr + cb * CH, o);
                        else tmem_ld16_issue(o_addr + cb * CH, o);
                    };
                    auto o_store = [&](int cb) {
                        tmem_ld_wait();
                        if (lay) {
                            sums.put(fold, cb * CH / 4, o, fold_f);
                            return;
                        }
#pragma unroll
                        for (int k = 0; k < CH; k += 2) {
                            float lo, hi;
                            unpack_f2(mul_f2(pack_f2(__uint_as_float(o[k]), __uint_as_float(o[k + 1])), alpha2), lo, hi);
                            o[k] = __float_as_uint(lo);
                            o[k + 1] = __float_as_uint(hi);
                        }
                        if constexpr (CH == 32) tmem_st32_issue(o_addr + cb * CH, o);
                        else tmem_st16_issue(o_addr + cb * CH, o);
                    };
                    const float neg_m = ref[part] == -INFINITY ? 0.f : -ref[part];   // exp2(-inf) = 0
                    const uint64_t neg2 = pack_f2(neg_m, neg_m);
                    uint64_t sum[2] = {0, 0};
                    if (SINGLE && first && !settled) settle();
#pragma unroll
                    for (int k0 = FROM; k0 < TO; k0 += CH) {
                        // a rescale of O, or a fold, runs under the exponentials: they wait for the special-function unit
                        if (first && (move || lay) && k0 < D) o_load(k0 / CH);
#pragma unroll
                        for (int k = k0; k < k0 + CH; k += 2) {
                            float e0, e1;
                            unpack_f2(fma_f2(pack_f2(__uint_as_float(raw[k]), __uint_as_float(raw[k + 1])), scale2, neg2), e0, e1);
                            e0 = fast_exp2(e0);
                            e1 = fast_exp2(e1);
                            sum[(k >> 1) & 1] = add_f2(sum[(k >> 1) & 1], pack_f2(e0, e1));
                            // the probabilities as pairs, kept in the registers the scores came in
                            raw[k >> 1] = pack_pair<T>(e0, e1);
                        }
                        if (first && (move || lay) && k0 < D) o_store(k0 / CH);
                    }
                    if (!first && PARTS > 1) {
                        if (ok) ok = warp_wait(&bars[BAR::O_PART + i], h_par);
                        h_par ^= 1;
                        tc_fence_after();
                    }
                    if (move || lay)
#pragma unroll
                        for (int cb = first ? TO / CH : 0; cb < D / CH; ++cb) {
                            o_load(cb);
                            o_store(cb);
                        }
#pragma unroll
                    for (int c = FROM / 2; c < TO / 2; c += 16) tmem_st16_issue(s_addr + c, raw + c);
                    tmem_st_wait();
                    tc_fence_before();
                    mbar_arrive(&bars[BAR::P_FULL + 2 * h + buf]);
                    float s0, s1, s2, s3;
                    unpack_f2(sum[0], s0, s1);
                    unpack_f2(sum[1], s2, s3);
                    l_run = fmaf(l_run, first || PARTS > 1 ? alpha[part] : 1.f, (s0 + s1) + (s2 + s3));
                };
                hand_over(std::integral_constant<int, 0>());
                hand_over(std::integral_constant<int, 1>());
                if (PARTS == 4) {
                    hand_over(std::integral_constant<int, PARTS == 4 ? 2 : 0>());
                    hand_over(std::integral_constant<int, PARTS == 4 ? 3 : 0>());
                }
                if (!ok) break;
                if (SINGLE) {
                    s_par ^= buf;
                    buf ^= 1;
                    s_addr = lanes + buf * 128u;
                }
            }
            if (!ok) break;
            if (SINGLE) h_par ^= 1;                          // (the last O product: the wait below)
            ok = warp_wait(&bars[BAR::O_FULL + i], o_par);
            if (!ok) break;
            o_par ^= 1;
            tc_fence_after();
            T *dst = (T *)p.out + w.b * p.o_sb + (int64_t)(w.hk * p.rep + h) * p.o_sh + (int64_t)l * p.o_sl;
            if (w.t0 == 0 && w.t1 == w.n) {
                const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll 1
                for (int cb = 0; cb < D / 32; ++cb) {
                    float o[32];
                    sums.total(cb, m_ref, o);
                    if (valid) store_row32<T>(dst + cb * 32, o, inv);
                }
                continue;
            }
            // ---- the unit is cut: leave a partial; the CTA that leaves the last one merges them ----
            const int c = blockIdx.x;
            {
                const int64_t slot = ((int64_t)c * 2 + (sg == p.waves ? 0 : 1)) * 2 + i;
                sums.leave(m_ref, (float4 *)p.o_part + slot * (D / 4) * TC_ROWS + row);
                p.ml_part[slot * TC_ROWS + row] = make_float2(m_ref, l_run);
            }
            __threadfence();
            mbar_arrive(&bars[BAR::GROUP + i]);
            ok = warp_wait(&bars[BAR::GROUP + i], g_par);
            if (!ok) break;
            g_par ^= 1;
            // the CTAs c0 ... c1 that own pieces of the unit: [x, x + n) of the tail
            int c0, c1;
            bool starts = true;   // the unit opens its first CTA's range
            if (p.pieces > 0) {
                c0 = w.unit * p.pieces;
                c1 = c0 + p.pieces - 1;
            } else {
                int x = c * p.per + min(c, p.rem) - s_seg[p.waves].t0;
                for (int k = p.waves; k < sg; ++k) x += s_seg[k].n;
                const int big = p.rem * (p.per + 1);
                auto cta_of = [&](int f) { return f < big ? f / (p.per + 1) : p.rem + (f - big) / p.per; };
                c0 = cta_of(x);
                c1 = cta_of(x + w.n - 1);
                starts = x == c0 * p.per + min(c0, p.rem);
            }
            if (row == 0) s_ticket[i] = atomicAdd(&p.tickets[(w.unit - p.waves * (int)gridDim.x) * 2 + i], 1);
            mbar_arrive(&bars[BAR::GROUP + i]);
            ok = warp_wait(&bars[BAR::GROUP + i], g_par);
            if (!ok) break;
            g_par ^= 1;
            if (s_ticket[i] != c1 - c0) continue;
            __threadfence();
            auto slot_of = [&](int cc) { return ((int64_t)cc * 2 + (cc == c0 && !starts ? 1 : 0)) * 2 + i; };
            // two partials at a time: sixteen vectors of a thread in flight
            constexpr int AT_ONCE = 2;
            float m = -INFINITY, l_sum = 0.f;
            auto ml_of = [&](int cc) {
                return cc <= c1 ? __ldcg(&p.ml_part[slot_of(cc) * TC_ROWS + row]) : make_float2(-INFINITY, 0.f);
            };
            for (int cc = c0; cc <= c1; cc += AT_ONCE) {
                float2 ml[AT_ONCE];
#pragma unroll
                for (int j = 0; j < AT_ONCE; ++j) ml[j] = ml_of(cc + j);
#pragma unroll
                for (int j = 0; j < AT_ONCE; ++j) {
                    const float m_new = fmaxf(m, ml[j].x);
                    if (m_new != -INFINITY) l_sum = l_sum * fast_exp2(m - m_new) + ml[j].y * fast_exp2(ml[j].x - m_new);
                    m = m_new;
                }
            }
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
#pragma unroll 1
            for (int cb = 0; cb < D / 32; ++cb) {
                float acc[32];
#pragma unroll
                for (int k = 0; k < 32; ++k) acc[k] = 0.f;
#pragma unroll 1
                for (int cc = c0; cc <= c1; cc += AT_ONCE) {
                    float4 v[AT_ONCE][8];
                    float f[AT_ONCE];
#pragma unroll
                    for (int j = 0; j < AT_ONCE; ++j) {
                        const float4 *po = (const float4 *)p.o_part + slot_of(cc + j) * (D / 4) * TC_ROWS + row;
                        f[j] = ml_of(cc + j).x;
#pragma unroll
                        for (int c4 = 0; c4 < 8; ++c4) v[j][c4] = cc + j <= c1 ? __ldcg(&po[(cb * 8 + c4) * TC_ROWS]) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < AT_ONCE; ++j) {
                        f[j] = f[j] == -INFINITY ? 0.f : fast_exp2(f[j] - m);
#pragma unroll
                        for (int c4 = 0; c4 < 8; ++c4) {
                            acc[c4 * 4 + 0] = fmaf(v[j][c4].x, f[j], acc[c4 * 4 + 0]);
                            acc[c4 * 4 + 1] = fmaf(v[j][c4].y, f[j], acc[c4 * 4 + 1]);
                            acc[c4 * 4 + 2] = fmaf(v[j][c4].z, f[j], acc[c4 * 4 + 2]);
                            acc[c4 * 4 + 3] = fmaf(v[j][c4].w, f[j], acc[c4 * 4 + 3]);
                        }
                    }
                }
                if (valid) store_row32<T>(dst + cb * 32, acc, inv);
            }
        }
        if (!ok) atomicExch(p.status, 23);
    }
    // all roles meet here; TMEM goes back whatever happened
    tc_fence_before();
    __syncthreads();
    if (warp == ISSUER) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
    }
}

template <typename T, int D, int PARTS, bool SINGLE>
bool launch_tc_as(const CUtensorMap &qmap, const CUtensorMap &kmap, const CUtensorMap &vmap, const ChunkTcParams &p, int ctas,
                  cudaStream_t stream) {
    const size_t smem = (size_t)(D / 64) * TC_BOX * (2 + ct_stages<D>()) + Bars<ct_stages<D>()>::COUNT * sizeof(uint64_t) + 16 +
                        CT_MAX_SEGMENTS * sizeof(CtSegment) + 1024;
    static_assert((D / 64) * TC_BOX * (2 + ct_stages<D>()) + Bars<ct_stages<D>()>::COUNT * 8 + 16 + CT_MAX_SEGMENTS * sizeof(CtSegment) + 1024 <= 232448,
                  "more shared memory than a CTA may have");
    // 0 = not yet, 1 = ready, -1 = refused; distinct handles may call from distinct host threads
    static std::atomic<int> configured[64];
    const int dev = current_device();
    if (dev < 0 || dev >= 64) return false;
    int state = configured[dev].load(std::memory_order_acquire);
    if (state == 0) {
        // setting the attribute twice from two racing threads is harmless; the result is the same
        const cudaError_t e = cudaFuncSetAttribute(attn_chunk_tc_kernel<T, D, PARTS, SINGLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) (void)cudaGetLastError();
        state = e == cudaSuccess ? 1 : -1;
        configured[dev].store(state, std::memory_order_release);
    }
    if (state < 0) return false;
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(attn_chunk_tc_kernel<T, D, PARTS, SINGLE>, dim3(ctas), dim3(ct_threads<SINGLE>()), smem, stream, qmap, kmap, vmap, p));
    timer.stop();
    ++g_launch_count;
    return true;
}

template <typename T, int D, bool SINGLE>
bool launch_tc_parts(const CUtensorMap &qmap, const CUtensorMap &kmap, const CUtensorMap &vmap, const ChunkTcParams &p, int ctas, int parts,
                     cudaStream_t stream) {
    if (parts == 4) return launch_tc_as<T, D, 4, SINGLE>(qmap, kmap, vmap, p, ctas, stream);
    return parts == 2 ? launch_tc_as<T, D, 2, SINGLE>(qmap, kmap, vmap, p, ctas, stream) : launch_tc_as<T, D, 1, SINGLE>(qmap, kmap, vmap, p, ctas, stream);
}

template <typename T, int D>
bool launch_tc_typed(const CUtensorMap &qmap, const CUtensorMap &kmap, const CUtensorMap &vmap, const ChunkTcParams &p, int ctas, int parts,
                     cudaStream_t stream) {
    return p.wide == 1 ? launch_tc_parts<T, D, true>(qmap, kmap, vmap, p, ctas, parts, stream)
                       : launch_tc_parts<T, D, false>(qmap, kmap, vmap, p, ctas, parts, stream);
}

// 128-row blocks of the call's query rows, head by head.
int64_t row_blocks_of(const AttnArgs &a) { return (int64_t)a.B * a.Hq * ((a.L + TC_ROWS - 1) / TC_ROWS); }

// Fewer blocks than half the part holds, or few positions.
bool few_blocks(const AttnArgs &a) { return row_blocks_of(a) < sm_count(a.device) / 2 || a.L < 64; }

}  // namespace

// Returns 1 when the call was taken (head dim 64 or 128, f16 / bf16 raw K and V, no array mask), 0 otherwise.
// KVC_CHUNK_TC=0 turns the path off.
bool attention_chunk_tc_accepts(const AttnArgs &a) {
    static const bool off = [] {
        const char *e = std::getenv("KVC_CHUNK_TC");
        return e && e[0] == '0';
    }();
    if (off) return false;
    if ((a.D != 128 && a.D != 64) || (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16)) return false;
    if (a.k.kind != SRC_RAW || a.v.kind != SRC_RAW || a.k.dtype != a.q_dtype || a.v.dtype != a.q_dtype) return false;
    if (a.mask.mode == KVC_MASK_ARRAY || a.q_signs || a.o_signs || a.q_calib || a.new_k || a.q_rot || a.o_rot) return false;
    if (a.B < 1 || a.L < 1 || a.Hq < 1 || a.Hkv <= 0 || a.Hq % a.Hkv || a.T < 1 || a.T > (int64_t)1 << 30) return false;
    // hidden keys are -inf before the scale meets them, and the maximum is taken there too: positive scales only (the mma.sync
    // chunk kernel multiplies first)
    if (!(a.scale > 0.f)) return false;
    // Up to 64 rows of a KV head's group the decode and verify kernels do less work on rows that are not there; from there on
    // (8 of 32 heads, D 128, behind 4 096 keys) 64 positions take 38 us here and 82 on the mma.sync chunk kernel, 128 of 16
    // sequences 0.6 of its time. (More than 128 heads of a group at few positions leave a row tile nearly empty.)
    const int64_t rep = a.Hq / a.Hkv;
    if (a.L < 64 && (rep * a.L <= 64 || rep > TC_ROWS)) return false;
    // (one tile of that kernel's keys: its maximum per 16 of them is the more precise one, and little is left to gain)
    if (few_blocks(a) && a.T <= 64) return false;
    if (a.mask.mode == KVC_MASK_CAUSAL && a.mask.causal_offset < 0) return false;
    if (row_blocks_of(a) > (int64_t)1 << 30) return false;
    if (!strides_fit(a.q, a.D, a.q_sl, a.q_sh, a.q_sb, a.Hq, a.B)) return false;
    if (!strides_fit(a.k.data, a.D, a.k.st, a.k.sh, a.k.sb, a.Hkv, a.B) || !strides_fit(a.v.data, a.D, a.v.st, a.v.sh, a.v.sb, a.Hkv, a.B))
        return false;
    if (((uintptr_t)a.out & 15) != 0 || (a.o_sl * 2) % 16 || (a.o_sh * 2) % 16 || (a.o_sb * 2) % 16) return false;
    return true;
}

int launch_attention_chunk_tc(const AttnArgs &a, cudaStream_t stream) {
    if (!attention_chunk_tc_accepts(a)) return 0;
    int *status = device_status_word(a.device);
    if (!status) return 0;
    ChunkTcParams p = {};
    p.out = a.out;
    p.o_sb = a.o_sb; p.o_sh = a.o_sh; p.o_sl = a.o_sl;
    p.rep = a.Hq / a.Hkv; p.Hkv = a.Hkv; p.L = a.L; p.T = a.T;
    p.causal = a.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
    p.causal_offset = a.mask.causal_offset;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.status = status;
    // a row tile holds all heads of the group at 128 / rep positions, or 128 positions of one head: the one with fewer tiles
    const int64_t one_head = (int64_t)p.rep * ((a.L + TC_ROWS - 1) / TC_ROWS);
    p.hb = 1; p.lb = TC_ROWS;
    if (p.rep <= TC_ROWS && (a.L + TC_ROWS / p.rep - 1) / (TC_ROWS / p.rep) <= one_head) {
        p.hb = p.rep;
        p.lb = TC_ROWS / p.rep;
    }
    p.head_tiles = p.rep / p.hb;
    const int64_t row_tiles = (int64_t)p.head_tiles * ((a.L + p.lb - 1) / p.lb);
    if (row_tiles > (int64_t)1 << 20) return 0;
    p.row_tiles = (int)row_tiles;
    const int64_t groups = (int64_t)a.B * a.Hkv;
    if (groups * p.row_tiles > (int64_t)1 << 28) return 0;

    CUtensorMap qmap, kmap, vmap;
    if (!make_query_map(&qmap, a, p.rep, p.hb, p.lb)) return 0;
    if (!make_map_tc(&kmap, a.k.data, a.k.dtype, a.D, a.T, a.Hkv, a.B, a.k.st, a.k.sh, a.k.sb)) return 0;
    if (!make_map_tc(&vmap, a.v.data, a.v.dtype, a.D, a.T, a.Hkv, a.B, a.v.st, a.v.sh, a.v.sb)) return 0;

    // Small calls take a finer reference: the mma.sync chunk kernel that takes them otherwise errs by little (a running maximum per
    // 16 keys, in up to 64 splits of 64 keys and up: four references are as precise below 16 384 keys, two from there on; behind
    // 4 000 keys two err by 3 % more).
    const int parts = few_blocks(a) ? (a.T < 16384 ? 4 : 2) : 1;

    // How the units are handed out, judged by the key tiles of the busiest SM (a CTA's start takes about three tiles' time,
    // the change of a unit one or two, writing a partial two, merging one a half, the memory for them and its cleared tickets
    // three, or two of the longer ones with finer references):
    //   whole units in rounds, one per SM, or, where units differ much, a CTA for each;
    //   few units: all cut into the same number of pieces, a CTA for each piece;
    //   equal ranges of all units end to end: evenest, but the CTAs are spread over all of K and V at once, so only where
    //     those stay in L2 (8 x 8 heads of 8 704 keys, 285 MB: 2.1 GB came from HBM in a launch);
    //   whole units in rounds, so that neighbours share their K and V tiles, and equal ranges of what is left.
    // (D 128, 160 units of 1 ... 3 tiles: 19 us whole, 34 in ranges; 48 of 5 or 6, D 64: 17 whole, 21 in pieces; 40 of 16: 38
    // whole, 33 in pieces, 37 in ranges; 64 of 254: 494, 261, 236.)
    // All of it for units of two row tiles and of one, whose key tiles take 0.6 of the time, or more where the references of a tile
    // follow one another (D 128, us in pairs and one by one: 8 heads x 400 positions behind 695 keys 29.1, 19.5; 512 behind 1 024
    // 31.2, 22.9; 1 024 of 1 024 23.5, 29.8; four references, 64 positions behind 448 20.1, 14.9).
    constexpr int64_t L2_BYTES = (int64_t)64 << 20;
    const int64_t sms = sm_count(a.device);
    const bool settled = groups * a.T * a.D * 4 <= L2_BYTES;
    struct Plan {
        double cost;
        int64_t units, group_tiles, rounds, waves, pieces, ranges, tail_tiles;
        int most;
        bool even;
    };
    auto plan_of = [&](int wide) {
        Plan g = {};
        p.wide = wide;
        p.units = (p.row_tiles + wide - 1) / wide;
        int least = INT_MAX;
        for (int u = 0; u < p.units; ++u) {
            const int n = ct_unit_tiles(p, u);
            g.group_tiles += n;
            g.most = std::max(g.most, n);
            least = std::min(least, n);
        }
        g.units = groups * p.units;
        const double tile = wide == 2 ? 1.0 : parts == 1 ? 0.6 : parts == 2 ? 0.8 : 0.9;
        const int64_t flat = groups * g.group_tiles, average = (flat + g.units - 1) / g.units;
        g.rounds = (g.units + sms - 1) / sms;
        g.even = least * 4 >= g.most * 3 && g.rounds <= CT_MAX_SEGMENTS;
        g.waves = settled ? 0 : g.units / sms;
        const int64_t tail = settled ? flat : (g.units - g.waves * sms) * average, per = std::max<int64_t>(4, (tail + sms - 1) / sms);   // (exact length below)
        g.pieces = std::min<int64_t>(sms / g.units, least / 2);
        const int set_up = 3 + (parts == 1 ? 3 : 2);
        const double whole = g.even ? 3 + g.rounds * (average * tile + 1) : std::max<int64_t>(g.most, g.rounds * average) * tile + 3 * g.rounds;
        const double cut = set_up + g.waves * (g.most * tile + 1) + per * tile + 2 * (per / average) + 3 + (g.most / per + 2) / 2;
        const double apart = g.pieces > 1 ? set_up + (g.most + g.pieces - 1) / g.pieces * tile + 2 + g.pieces / 2 : INFINITY;
        g.cost = whole;
        if (apart < whole && apart <= cut) {
            g.ranges = g.units * g.pieces;
            g.cost = apart;
        } else if (cut < whole && g.waves + 2 < CT_MAX_SEGMENTS) {
            g.tail_tiles = flat;
            for (int64_t u = 0; u < g.waves * sms; ++u) g.tail_tiles -= ct_unit_tiles(p, (int)(u % p.units));
            g.ranges = std::max<int64_t>(1, std::min<int64_t>(sms, g.tail_tiles / 4));
            g.cost = cut;
            if (g.tail_tiles < 1 || g.tail_tiles > (int64_t)1 << 29 || g.group_tiles > (int64_t)1 << 29 ||
                g.tail_tiles / g.ranges / least + 2 > CT_MAX_SEGMENTS - g.waves) {
                g.tail_tiles = g.ranges = 0;
                g.cost = whole;
            }
        }
        return g;
    };
    Plan g = plan_of(1);
    if (p.row_tiles > 1) {
        const Plan pairs = plan_of(2);
        if (pairs.cost <= g.cost) g = pairs;
        else (void)plan_of(1);
    }
    p.all_units = (int)g.units;
    int64_t ctas, longest;                                       // ... and the most key tiles of a segment
    size_t o_bytes, ml_bytes, t_bytes, fold_bytes;
    auto lay_out = [&] {
        if (g.tail_tiles > 0) {
            ctas = g.waves > 0 ? sms : g.ranges;
            p.waves = (int)g.waves;
            p.ranges = (int)g.ranges;
            p.per = (int)(g.tail_tiles / g.ranges);
            p.rem = (int)(g.tail_tiles % g.ranges);
            p.group_tiles = (int)g.group_tiles;
            for (int64_t u = g.waves * sms / p.units * p.units; u < g.waves * sms; ++u) p.tail_base += ct_unit_tiles(p, (int)u);
            longest = g.waves > 0 ? g.most : std::min(g.most, p.per + 1);
        } else if (g.ranges > 0) {
            ctas = g.ranges;
            p.pieces = (int)g.pieces;
            longest = (g.most + g.pieces - 1) / g.pieces;
        } else {
            ctas = g.even ? std::min(g.units, sms) : g.units;
            p.waves = g.even ? (int)g.rounds : 1;
            longest = g.most;
        }
        // (in memory a fold costs half a key tile's time, under the exponentials, a whole one ahead of them: every 768 keys 282 and 300
        // us where no folds take 262; the kernel that folded every tile in registers took 312. 512 x 8 x 32 f16 heads behind 3 584 keys)
        const bool in_memory = a.D == 128 && p.wide == 2;
        p.fold = fold_keys(a.q_dtype) * (in_memory ? 3 : 2) / 2 / TC_KEYS;
        if (in_memory) {                                         // even stretches: no fold for a last tile or two
            const int64_t stretches = std::max<int64_t>(1, (2 * longest + p.fold) / (2 * p.fold));
            p.fold = (int)((longest + stretches - 1) / stretches);
        }
        const size_t part = (size_t)g.ranges * 4 * TC_ROWS;
        o_bytes = part * a.D * sizeof(float);
        ml_bytes = part * sizeof(float2);
        t_bytes = g.ranges > 0 ? (size_t)(g.tail_tiles > 0 ? g.units - g.waves * sms : g.units) * 2 * sizeof(int) : 0;
        fold_bytes = in_memory && longest > p.fold ? (size_t)ctas * 2 * TC_ROWS * a.D * sizeof(float) : 0;
        return fold_bytes + o_bytes + ml_bytes + t_bytes;
    };
    const ChunkTcParams uncut = p;
    CallMemory mem(lay_out(), stream);
    if (!mem.ptr && g.ranges > 0) {                              // no room: whole units
        p = uncut;
        g.tail_tiles = g.ranges = 0;
        lay_out();
    }
    if (!mem.ptr && fold_bytes > 0) return 0;
    p.o_fold = (float *)mem.ptr;
    p.o_part = (float *)((char *)mem.ptr + fold_bytes);
    p.ml_part = (float2 *)((char *)p.o_part + o_bytes);
    p.tickets = (int *)((char *)p.ml_part + ml_bytes);
    if (g.ranges > 0) KVC_CUDA(cudaMemsetAsync(p.tickets, 0, t_bytes, stream));
    bool taken;
    if (a.D == 128)
        taken = a.q_dtype == KVC_BF16 ? launch_tc_typed<__nv_bfloat16, 128>(qmap, kmap, vmap, p, (int)ctas, parts, stream)
                                      : launch_tc_typed<__half, 128>(qmap, kmap, vmap, p, (int)ctas, parts, stream);
    else
        taken = a.q_dtype == KVC_BF16 ? launch_tc_typed<__nv_bfloat16, 64>(qmap, kmap, vmap, p, (int)ctas, parts, stream)
                                      : launch_tc_typed<__half, 64>(qmap, kmap, vmap, p, (int)ctas, parts, stream);
    if (taken && trace_dispatch())
        fprintf(stderr, "[kvc] chunk_tc: %lld units of %d row tiles (%d heads x %d positions), %lld CTAs, %d rounds, ranges of %d tiles, %d pieces, %d references a tile\n",
                (long long)g.units, p.wide, p.hb, p.lb, (long long)ctas, p.waves, p.per, p.pieces, parts);
    return taken ? 1 : 0;
}

}  // namespace kvc
