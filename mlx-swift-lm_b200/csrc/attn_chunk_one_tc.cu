// Chunks over raw K/V whose probabilities are kept as pairs of 16-bit values, on the 5th-generation tensor cores:
// boolean array masks (prompt chunks through sliding-window layers, KVCache.swift:834-871 with
// AttentionUtils.swift:87-93) at head dim 64, 128 and 256, and head dim 256 under any causal mask or none.
//
// One CTA takes one tile of up to 128 query rows (all heads of a KV head's group at 128 / rep positions) and walks
// 64-key tiles:
//   warps 0..3  softmax: thread = query row = TMEM lane; scores out of TMEM, mask, running maximum, exponentials; P goes
//               back over the scores' columns as two 16-bit values, its high half and what that leaves (the O product
//               adds both: P has 16 or 22 significant bits, as on the mma.sync kernel that took these calls)
//   warp 4      TMA producer: Q, then K_0, K_1, V_0, K_2, V_1, ... into one ring
//   warp 5      owns the TMEM allocation and issues the MMAs: S of tile j + 1 (two S buffers) before O += P(j) V(j), so
//               that the tensor cores have the next scores ready while the softmax runs
// Key tiles of 64 because at head dim 256 a K or V tile of 128 keys is 64 KB: two stages beside the queries. At head dim
// 64 and 128 two CTAs share an SM (256 TMEM columns each) and one's products run under the other's softmax.
//
// Where there are few row tiles a unit is cut into pieces, one CTA each; piece i takes every pieces-th key tile from i
// on, so that a window's run of visible tiles is shared evenly. Under an array mask the CTA first reads the mask of its
// rows and tiles and leaves out the tiles no row sees.
//
// Every `fold` tiles O goes on in fp32 sums, as in attn_chunk_tc.cu (masked f16 outputs: errors against 64 bits + 0.5 % at 32 000
// keys without it, in eight pieces).
//
// A hidden key has weight zero, which an infinite or NaN value turns into NaN: in all rows of a tile that some row sees, as in
// softmax times V.
//
// What bounds it: the chain S -> softmax -> O of one row tile; the two products take 1 800 cycles of a tile at head dim
// 256 (768 for S, whose 64 columns are bound by shared-memory reads, 1 024 for both halves of P).
//
// TMEM columns: S_0 / P_0 at 0, S_1 / P_1 at 64, O behind them. Operand layouts as in attn_chunk_tc.cu, with K / V boxes
// of 64 rows (8 192 bytes).
//
// Every wait is bounded; a wait that runs out sets the device status word, the CTA waits (bounded too) for its copies and
// products in flight and frees its TMEM.
#include <atomic>
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "attn_common.cuh"
#include "common.h"
#include "tc_common.cuh"

namespace kvc {
namespace {

using namespace dev;

using namespace tc;

constexpr int ON_THREADS = 192;
constexpr int ON_KEYS = 64;
constexpr int ON_BOX = ON_KEYS * 128;      // bytes of a 64-element-wide box of 64 keys
constexpr int ON_LIVE_WORDS = 64;          // key tiles of a CTA, a bit each

struct ChunkOneParams {
    void *out;
    int64_t o_sb, o_sh, o_sl;
    int32_t rep, Hkv, L;
    int64_t T;
    int32_t hb, lb, head_tiles, row_tiles;   // as in attn_chunk_tc.cu
    int32_t pieces;                          // CTAs of a unit (a row tile)
    int32_t causal;
    int64_t causal_offset;
    float scale_log2;
    MaskDesc mask;
    int32_t fold;                            // key tiles of a CTA between two folds
    float *o_part;                           // [unit][piece][D / 4][128 rows][4]: partials, and (head dim 128 and 256) the folded sums until then
    float2 *ml_part;                         // [unit][piece][128 rows] (reference, sum)
    int *tickets;                            // [unit], zeroed before the launch
    int *status;
};

template <int D> constexpr int on_stages() { return D == 256 ? 5 : D == 128 ? 4 : 6; }
template <int D> constexpr int on_columns() { return D == 256 ? 512 : 256; }

template <int STAGES> struct OneBars {
    enum : int {
        Q_FULL = 0,
        RING_FULL = 1,
        RING_EMPTY = RING_FULL + STAGES,
        S_FULL = RING_EMPTY + STAGES,    // [2]
        P_FULL = S_FULL + 2,             // [2]
        O_DONE = P_FULL + 2,             // every O product
        O_LAST = O_DONE + 1,             // the last one
        GROUP = O_LAST + 1,              // the softmax threads meet
        DRAIN = GROUP + 1,               // the products of a CTA that gave up are done
        COUNT = DRAIN + 1
    };
};

template <typename T> __device__ __forceinline__ float2 unpack_pair(uint32_t w);
template <> __device__ __forceinline__ float2 unpack_pair<__half>(uint32_t w) { return MmaType<__half>::unpack(w); }
template <> __device__ __forceinline__ float2 unpack_pair<__nv_bfloat16>(uint32_t w) { return MmaType<__nv_bfloat16>::unpack(w); }

template <typename T, int D, bool MASKED, bool FOLDS>
__global__ void __launch_bounds__(ON_THREADS, D == 256 ? 1 : 2)
attn_chunk_one_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                      const __grid_constant__ CUtensorMap vmap, const __grid_constant__ ChunkOneParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int STAGES = on_stages<D>(), COLUMNS = on_columns<D>(), O_COL = D == 256 ? 256 : 128;
    using BAR = OneBars<STAGES>;
    constexpr int NBOX = D / 64, TILE = NBOX * ON_BOX;
    // f16 probabilities are at most 1024, so that their low halves stay normal numbers
    constexpr float P_UP = std::is_same<T, __half>::value ? 1024.f : 1.f;
    unsigned char *sq = base;
    unsigned char *ring = sq + NBOX * TC_BOX;
    uint64_t *bars = (uint64_t *)(ring + STAGES * TILE);
    uint32_t *tmem_slot = (uint32_t *)(bars + BAR::COUNT);
    int *s_ticket = (int *)(tmem_slot + 1);
    uint32_t *s_live = (uint32_t *)(s_ticket + 1);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int piece = blockIdx.x % p.pieces, unit = blockIdx.x / p.pieces;
    // late positions first: under a causal mask they see the most keys
    const int rt = p.row_tiles - 1 - unit % p.row_tiles, group = unit / p.row_tiles, hk = group % p.Hkv, b = group / p.Hkv;
    const int l0 = (rt / p.head_tiles) * p.lb, h0 = (rt % p.head_tiles) * p.hb;
    const int64_t keys = p.causal ? min(p.T, p.causal_offset + min(p.L, l0 + p.lb)) : p.T;
    const int tiles = (int)((keys + ON_KEYS - 1) / ON_KEYS);
    const int mine = piece < tiles ? (tiles - piece + p.pieces - 1) / p.pieces : 0;   // tile piece + c * pieces, c < mine

    if (tid == 0) {
        mbar_init(&bars[BAR::Q_FULL], 1);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&bars[BAR::RING_FULL + s], 1);
            mbar_init(&bars[BAR::RING_EMPTY + s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars[BAR::S_FULL + s], 1);
            mbar_init(&bars[BAR::P_FULL + s], 128);
        }
        mbar_init(&bars[BAR::O_DONE], 1);
        mbar_init(&bars[BAR::O_LAST], 1);
        mbar_init(&bars[BAR::GROUP], 128);
        mbar_init(&bars[BAR::DRAIN], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 && lane < 3) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)(lane == 0 ? &qmap : lane == 1 ? &kmap : &vmap)) : "memory");
    for (int i = tid; i < NBOX * (TC_ROWS - p.hb * p.lb) * 8; i += ON_THREADS) {   // rows no copy writes are zero
        const int chunk = i & 7, box = (i >> 3) % NBOX, row = (i >> 3) / NBOX + p.hb * p.lb;
        *(uint4 *)(sq + box * TC_BOX + row * 128 + chunk * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (MASKED)
        for (int i = tid; i < ON_LIVE_WORDS; i += ON_THREADS) s_live[i] = 0u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)COLUMNS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();  // everything below reads what earlier kernels on the stream wrote
    auto mask_row = [&](int h, int l) {
        return (const uint8_t *)p.mask.data + b * p.mask.sb + (int64_t)(hk * p.rep + h) * p.mask.sh + (int64_t)l * p.mask.sl;
    };
    if (MASKED) {
        const int heads = p.mask.sh == 0 ? 1 : min(p.hb, p.rep - h0), rows = min(p.lb, p.L - l0);
        for (int64_t i = tid; i < (int64_t)heads * rows * mine; i += ON_THREADS) {
            const int c = (int)(i % mine), r = (int)(i / mine), key0 = (piece + c * p.pieces) * ON_KEYS;
            const uint8_t *row = mask_row(h0 + r % heads, l0 + r / heads) + key0;
            const int n = (int)min((int64_t)ON_KEYS, p.T - key0);
            if (mask_bits32(row, n) | mask_bits32(row + 32, n - 32)) atomicOr(&s_live[c >> 5], 1u << (c & 31));
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto live = [&](int c) { return !MASKED || ((s_live[c >> 5] >> (c & 31)) & 1u); };

    if (warp == 4) {
        if (lane == 0) {
            // ---------------- producer ----------------
            bool ok = true;
            uint32_t slot = 0, round = 0;
            auto load_tile = [&](const CUtensorMap *map, int t) {
                if (round > 0 && !mbar_wait(&bars[BAR::RING_EMPTY + slot], (round - 1) & 1)) return false;
                unsigned char *dst = ring + (size_t)slot * TILE;
                mbar_expect_tx(&bars[BAR::RING_FULL + slot], TILE);
#pragma unroll
                for (int bx = 0; bx < NBOX; ++bx) tma_load_4d(dst + bx * ON_BOX, map, &bars[BAR::RING_FULL + slot], bx * 64, t * ON_KEYS, hk, b);
                if (++slot == STAGES) {
                    slot = 0;
                    ++round;
                }
                return true;
            };
            int before = -1;
            bool q_loaded = false;
            for (int c = 0; ok && c < mine; ++c) {
                if (!live(c)) continue;
                const int t = piece + c * p.pieces;
                ok = load_tile(&kmap, t);
                if (before < 0) {
                    q_loaded = true;
                    mbar_expect_tx(&bars[BAR::Q_FULL], (uint32_t)(p.hb * p.lb * 128 * NBOX));
#pragma unroll
                    for (int bx = 0; bx < NBOX; ++bx) tma_load_5d(sq + bx * TC_BOX, &qmap, &bars[BAR::Q_FULL], bx * 64, h0, l0, hk, b);
                } else if (ok) {
                    ok = load_tile(&vmap, before);
                }
                before = t;
            }
            if (ok && before >= 0) ok = load_tile(&vmap, before);
            if (!ok) {
                atomicExch(p.status, 16);
                drain_copies(&bars[BAR::RING_FULL], STAGES, slot, round);
                if (q_loaded) (void)mbar_wait(&bars[BAR::Q_FULL], 0);
            }
        }
    } else if (warp == 5) {
        // ---------------- MMA issue (descriptors: attn_chunk_tc.cu) ----------------
        constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
        constexpr uint32_t IDESC = (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(ON_KEYS >> 3) << 17) | ((128u >> 4) << 24);
        constexpr uint32_t IDESC_PV = (1u << 4) | (FMT << 7) | (FMT << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t q_desc = umma_desc(smem_u32(sq), 16, 1024);
        const uint64_t k_desc = umma_desc(smem_u32(ring), 16, 1024);
        const uint64_t v_desc = umma_desc(smem_u32(ring), ON_BOX, 1024);
        bool ok = true;
        uint32_t slot = 0, par = 0, n = 0;   // ring entry; S products issued
        int since = 0;                       // O products behind the last fold
        auto next = [&] {
            if (++slot == (uint32_t)STAGES) {
                slot = 0;
                par ^= 1;
            }
        };
        auto issue_o = [&](uint32_t j, bool last) {
            ok = warp_wait(&bars[BAR::RING_FULL + slot], par);
            if (ok) ok = warp_wait(&bars[BAR::P_FULL + (j & 1)], (j >> 1) & 1);
            if (!ok) return;
            tc_fence_after();
            const uint64_t vd = v_desc + (uint64_t)(slot * (TILE / 16));
            const uint32_t p_addr = tmem + (j & 1) * 64u;
            if (elect_one()) {
#pragma unroll
                for (int low = 1; low >= 0; --low)   // what the high halves leave comes first
#pragma unroll
                    for (int ks = 0; ks < ON_KEYS / 16; ++ks)
                        umma_f16_ts(tmem + O_COL, p_addr + (uint32_t)(low * 32 + ks * 8), vd + (uint64_t)(ks * 128), IDESC_PV,
                                    (since == 0 && low == 1 && ks == 0) ? 0u : 1u);
                umma_commit(&bars[BAR::O_DONE]);
                if (last) umma_commit(&bars[BAR::O_LAST]);
                umma_commit(&bars[BAR::RING_EMPTY + slot]);
            }
            __syncwarp();
            since = FOLDS && since == p.fold - 1 ? 0 : since + 1;
            next();
        };
        for (int c = 0; ok && c < mine; ++c) {
            if (!live(c)) continue;
            if (n == 0) ok = warp_wait(&bars[BAR::Q_FULL], 0);
            if (ok) ok = warp_wait(&bars[BAR::RING_FULL + slot], par);
            if (!ok) break;
            tc_fence_after();
            const uint64_t kd = k_desc + (uint64_t)(slot * (TILE / 16));
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_f16(tmem + (n & 1) * 64u, q_desc + (uint64_t)((ks >> 2) * (TC_BOX / 16) + (ks & 3) * 2),
                             kd + (uint64_t)((ks >> 2) * (ON_BOX / 16) + (ks & 3) * 2), IDESC, ks > 0 ? 1u : 0u);
                umma_commit(&bars[BAR::S_FULL + (n & 1)]);
                umma_commit(&bars[BAR::RING_EMPTY + slot]);
            }
            __syncwarp();
            next();
            if (n > 0) issue_o(n - 1, false);
            ++n;
        }
        if (ok && n > 0) issue_o(n - 1, true);
        if (!ok) {
            atomicExch(p.status, 17);
            drain_products(&bars[BAR::DRAIN]);
        }
    } else {
        // ---------------- softmax and output: thread = row ----------------
        const int row = warp * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16), o_addr = lane_addr + O_COL;
        const int l = l0 + row / p.hb, h = h0 + row % p.hb;
        const bool valid = row < p.hb * p.lb && l < p.L && h < p.rep;
        const int limit = (int)(p.causal ? min(p.T - 1, p.causal_offset + l) : p.T - 1);   // last visible key
        const uint8_t *mrow = MASKED && valid ? mask_row(h, l) : nullptr;
        float m_run = -INFINITY, l_run = 0.f;
        uint32_t n = 0;
        int since = -1;                      // tiles behind the last fold
        bool ok = true;
        auto own_part = [&] { return (float4 *)p.o_part + ((int64_t)unit * p.pieces + piece) * (D / 4) * TC_ROWS + row; };
        FoldedSums<D, D == 64> sums(o_addr, FOLDS ? own_part() : nullptr);
        for (int c = 0; c < mine; ++c) {
            if (!live(c)) continue;
            const int key0 = (piece + c * p.pieces) * ON_KEYS;
            uint32_t seen[2] = {0u, 0u};                 // read while the scores are on their way
            if (MASKED && valid) {
                const int in = (int)min((int64_t)ON_KEYS, p.T - key0);
                seen[0] = mask_bits32(mrow + key0, in);
                seen[1] = mask_bits32(mrow + key0 + 32, in - 32);
            }
            ok = warp_wait(&bars[BAR::S_FULL + (n & 1)], (n >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint32_t s_addr = lane_addr + (n & 1) * 64u;
            uint32_t raw[ON_KEYS];
            tmem_ld32_issue(s_addr, raw);
            tmem_ld32_issue(s_addr + 32, raw + 32);
            tmem_ld_wait();
            if (MASKED) {
#pragma unroll
                for (int k = 0; k < ON_KEYS; ++k)
                    if (!((seen[k >> 5] >> (k & 31)) & 1u)) raw[k] = 0xff800000u;   // -inf
            } else if (key0 + ON_KEYS - 1 > limit) {
#pragma unroll
                for (int k = 0; k < ON_KEYS; ++k)
                    if (key0 + k > limit) raw[k] = 0xff800000u;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int k = 0; k < ON_KEYS; k += 2)
                mx4[(k >> 1) & 3] = fmaxf(mx4[(k >> 1) & 3], fmaxf(__uint_as_float(raw[k]), __uint_as_float(raw[k + 1])));
            const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2);
            const float alpha = m_run == m_new ? 1.f : fast_exp2(m_run - m_new);   // exp2(-inf) = 0
            const float m_old = m_run;
            m_run = m_new;
            const float neg_m = m_new == -INFINITY ? 0.f : -m_new;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t low[ON_KEYS / 2];
#pragma unroll
            for (int k = 0; k < ON_KEYS; k += 2) {
                const float e0 = fast_exp2(fmaf(__uint_as_float(raw[k]), p.scale_log2, neg_m));
                const float e1 = fast_exp2(fmaf(__uint_as_float(raw[k + 1]), p.scale_log2, neg_m));
                sum4[k & 2] += e0;
                sum4[(k & 2) + 1] += e1;
                const uint32_t high = pack_pair<T>(e0 * P_UP, e1 * P_UP);
                const float2 f = unpack_pair<T>(high);
                low[k >> 1] = pack_pair<T>(e0 * P_UP - f.x, e1 * P_UP - f.y);
                raw[k >> 1] = high;
            }
            const bool fold = FOLDS && ++since == p.fold;
            if (n > 0 && (fold || __any_sync(0xffffffffu, alpha != 1.f))) {
                ok = warp_wait(&bars[BAR::O_DONE], (n - 1) & 1);   // (not a phase too early: the product before
                                                                     // it was done when these scores came)
                if (!ok) break;
                tc_fence_after();
                if (fold) {
                    sums.fold(m_old);
                    since = 0;
                } else
#pragma unroll 2
                for (int cb = 0; cb < D / 32; ++cb) {
                    uint32_t o[32];
                    tmem_ld32_issue(o_addr + cb * 32, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                    tmem_st32_issue(o_addr + cb * 32, o);
                }
            }
            tmem_st32_issue(s_addr, raw);
            tmem_st32_issue(s_addr + 32, low);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&bars[BAR::P_FULL + (n & 1)]);
            l_run = fmaf(l_run, alpha, (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            ++n;
        }
        if (ok && n > 0) ok = warp_wait(&bars[BAR::O_LAST], 0);
        if (ok) {
            tc_fence_after();
            T *dst = (T *)p.out + b * p.o_sb + (int64_t)(hk * p.rep + h) * p.o_sh + (int64_t)l * p.o_sl;
            auto o_of = [&](int cb, float (&o)[32]) {
                if (n > 0) {
                    if constexpr (FOLDS) sums.total(cb, m_run, o);
                    else tmem_ld32(o_addr + cb * 32, o);
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k) o[k] = 0.f;
                }
            };
            if (p.pieces == 1) {
                const float inv = l_run > 0.f ? 1.f / (l_run * P_UP) : 0.f;
#pragma unroll 1
                for (int cb = 0; cb < D / 32; ++cb) {
                    float o[32];
                    o_of(cb, o);
                    if (valid) store_row32<T>(dst + cb * 32, o, inv);
                }
            } else {
                // ---- leave a partial; the CTA that leaves the last one of the unit merges them ----
                float4 *part = own_part();
#pragma unroll 1
                for (int cb = 0; cb < D / 32; ++cb) {
                    float o[32];
                    o_of(cb, o);
#pragma unroll
                    for (int c4 = 0; c4 < 8; ++c4) part[(cb * 8 + c4) * TC_ROWS] = make_float4(o[c4 * 4], o[c4 * 4 + 1], o[c4 * 4 + 2], o[c4 * 4 + 3]);
                }
                p.ml_part[((int64_t)unit * p.pieces + piece) * TC_ROWS + row] = make_float2(m_run, l_run);
                __threadfence();
                mbar_arrive(&bars[BAR::GROUP]);
                ok = warp_wait(&bars[BAR::GROUP], 0);
                if (ok) {
                    if (row == 0) *s_ticket = atomicAdd(&p.tickets[unit], 1);
                    mbar_arrive(&bars[BAR::GROUP]);
                    ok = warp_wait(&bars[BAR::GROUP], 1);
                }
                if (ok && *s_ticket == p.pieces - 1) {
                    __threadfence();
                    const float2 *ml = p.ml_part + (int64_t)unit * p.pieces * TC_ROWS + row;
                    const float4 *parts = (const float4 *)p.o_part + (int64_t)unit * p.pieces * (D / 4) * TC_ROWS + row;
                    float m = -INFINITY, l_sum = 0.f;
                    for (int i = 0; i < p.pieces; ++i) {
                        const float2 x = __ldcg(&ml[i * TC_ROWS]);
                        const float m_new = fmaxf(m, x.x);
                        if (m_new != -INFINITY) l_sum = l_sum * fast_exp2(m - m_new) + x.y * fast_exp2(x.x - m_new);
                        m = m_new;
                    }
                    const float inv = l_sum > 0.f ? 1.f / (l_sum * P_UP) : 0.f;
#pragma unroll 1
                    for (int cb = 0; cb < D / 32; ++cb) {
                        float acc[32];
#pragma unroll
                        for (int k = 0; k < 32; ++k) acc[k] = 0.f;
#pragma unroll 2
                        for (int i = 0; i < p.pieces; ++i) {
                            const float mi = __ldcg(&ml[i * TC_ROWS]).x, f = mi == -INFINITY ? 0.f : fast_exp2(mi - m);
                            float4 v[8];
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) v[c4] = __ldcg(&parts[((int64_t)i * (D / 4) + cb * 8 + c4) * TC_ROWS]);
#pragma unroll
                            for (int c4 = 0; c4 < 8; ++c4) {
                                acc[c4 * 4 + 0] = fmaf(v[c4].x, f, acc[c4 * 4 + 0]);
                                acc[c4 * 4 + 1] = fmaf(v[c4].y, f, acc[c4 * 4 + 1]);
                                acc[c4 * 4 + 2] = fmaf(v[c4].z, f, acc[c4 * 4 + 2]);
                                acc[c4 * 4 + 3] = fmaf(v[c4].w, f, acc[c4 * 4 + 3]);
                            }
                        }
                        if (valid) store_row32<T>(dst + cb * 32, acc, inv);
                    }
                }
            }
        }
        if (!ok) atomicExch(p.status, 18);
    }
    // all roles meet here; TMEM goes back whatever happened
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)COLUMNS) : "memory");
    }
}

template <typename T, int D, bool MASKED, bool FOLDS>
bool launch_one_as(const CUtensorMap &qmap, const CUtensorMap &kmap, const CUtensorMap &vmap, const ChunkOneParams &p, int ctas,
                   cudaStream_t stream) {
    constexpr size_t smem = (size_t)(D / 64) * (TC_BOX + on_stages<D>() * ON_BOX) + OneBars<on_stages<D>()>::COUNT * sizeof(uint64_t) + 8 +
                            ON_LIVE_WORDS * sizeof(uint32_t) + 1024;
    static_assert(smem <= (D == 256 ? 232448 : 115200), "more shared memory than there is");
    // 0 = not yet, 1 = ready, -1 = refused (attn_chunk_tc.cu)
    static std::atomic<int> configured[64];
    const int dev = current_device();
    if (dev < 0 || dev >= 64) return false;
    int state = configured[dev].load(std::memory_order_acquire);
    if (state == 0) {
        const cudaError_t e = cudaFuncSetAttribute(attn_chunk_one_kernel<T, D, MASKED, FOLDS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) (void)cudaGetLastError();
        state = e == cudaSuccess ? 1 : -1;
        configured[dev].store(state, std::memory_order_release);
    }
    if (state < 0) return false;
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(attn_chunk_one_kernel<T, D, MASKED, FOLDS>, dim3(ctas), dim3(ON_THREADS), smem, stream, qmap, kmap, vmap, p));
    timer.stop();
    ++g_launch_count;
    return true;
}

template <typename T, bool FOLDS>
bool launch_one(const CUtensorMap &qmap, const CUtensorMap &kmap, const CUtensorMap &vmap, const ChunkOneParams &p, int D, bool masked,
                int ctas, cudaStream_t stream) {
    if (D == 256)
        return masked ? launch_one_as<T, 256, true, FOLDS>(qmap, kmap, vmap, p, ctas, stream)
                      : launch_one_as<T, 256, false, FOLDS>(qmap, kmap, vmap, p, ctas, stream);
    return D == 128 ? launch_one_as<T, 128, true, FOLDS>(qmap, kmap, vmap, p, ctas, stream)
                    : launch_one_as<T, 64, true, FOLDS>(qmap, kmap, vmap, p, ctas, stream);
}

}  // namespace

// Returns 1 when the call was taken (f16 / bf16 raw K and V; a boolean mask with contiguous rows at head dim 64, 128 or
// 256, or head dim 256 under a causal mask or none), 0 otherwise. KVC_CHUNK_TC=0 turns the path off.
int launch_attention_chunk_one(const AttnArgs &a, cudaStream_t stream) {
    static const bool off = [] {
        const char *e = std::getenv("KVC_CHUNK_TC");
        return e && e[0] == '0';
    }();
    if (off) return 0;
    if ((a.D != 256 && a.D != 128 && a.D != 64) || (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16)) return 0;
    if (a.k.kind != SRC_RAW || a.v.kind != SRC_RAW || a.k.dtype != a.q_dtype || a.v.dtype != a.q_dtype) return 0;
    if (a.q_signs || a.o_signs || a.q_calib || a.new_k || a.q_rot || a.o_rot) return 0;
    const bool masked = a.mask.mode == KVC_MASK_ARRAY;
    if (masked ? (a.mask.dtype != KVC_BOOL || a.mask.st != 1 || !a.mask.data) : a.D != 256) return 0;
    if (a.mask.mode == KVC_MASK_CAUSAL && a.mask.causal_offset < 0) return 0;
    if (!(a.scale > 0.f)) return 0;   // as in attn_chunk_tc.cu: hidden keys are -inf before the scale meets them
    // up to 64 keys: one tile of the mma.sync chunk kernel, whose maximum per 16 of them is as precise
    if (a.B < 1 || a.L < 1 || a.Hq < 1 || a.Hkv <= 0 || a.Hq % a.Hkv || a.T <= 64 || a.T > (int64_t)1 << 30) return 0;
    const int64_t rep = a.Hq / a.Hkv;
    if (a.L < 64 && (rep * a.L <= 64 || rep > TC_ROWS)) return 0;
    if (!strides_fit(a.q, a.D, a.q_sl, a.q_sh, a.q_sb, a.Hq, a.B)) return 0;
    if (!strides_fit(a.k.data, a.D, a.k.st, a.k.sh, a.k.sb, a.Hkv, a.B) || !strides_fit(a.v.data, a.D, a.v.st, a.v.sh, a.v.sb, a.Hkv, a.B)) return 0;
    if (((uintptr_t)a.out & 15) != 0 || (a.o_sl * 2) % 16 || (a.o_sh * 2) % 16 || (a.o_sb * 2) % 16) return 0;
    int *status = device_status_word(a.device);
    if (!status) return 0;
    ChunkOneParams p = {};
    p.out = a.out;
    p.o_sb = a.o_sb; p.o_sh = a.o_sh; p.o_sl = a.o_sl;
    p.rep = (int)rep; p.Hkv = a.Hkv; p.L = a.L; p.T = a.T;
    p.causal = a.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
    p.causal_offset = a.mask.causal_offset;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.mask = a.mask;
    p.status = status;
    p.hb = rep <= TC_ROWS ? (int)rep : 1;
    p.lb = TC_ROWS / p.hb;
    p.head_tiles = p.rep / p.hb;
    const int64_t row_tiles = (int64_t)p.head_tiles * ((a.L + p.lb - 1) / p.lb), units = (int64_t)a.B * a.Hkv * row_tiles;
    if (row_tiles > (int64_t)1 << 20 || units > (int64_t)1 << 24) return 0;
    p.row_tiles = (int)row_tiles;
    // Pieces where places are free for them and they pay, in tiles' time (1.7 us): a partial costs the merging CTA two and a half
    // to write and 1.2 to merge at head dim 256 (0.3 at 64). A mask is taken to hide half of the tiles. Two CTAs on an SM take 1.6
    // times as long for a tile. (64 row tiles of 10 visible tiles, D 256: 25 us whole, 30 as two pieces. One row tile of four heads
    // behind 40 000 keys, all visible: 149 us in 8 pieces, 62 in 32 at D 64; 178 in 8, 118 in 16, 104 in 24 at D 256. 8 row tiles
    // behind 16 000, D 64: 64 us in 8, 40 in 16, 48 in 24.)
    const int64_t sms = sm_count(a.device), slots = sms * (a.D == 256 ? 1 : 2), n = (a.T + ON_KEYS - 1) / ON_KEYS;
    const double visible = masked ? 0.5 * n : n;
    int64_t pieces = 1;
    double least = visible;
    for (int64_t s = 2; s <= 64 && units * s <= slots && s * 3 <= n; ++s) {
        const double time = visible / s * (units * s > sms ? 1.6 : 1.0) + 2.5 + 1.2 * s * a.D / 256;
        if (time < least) {
            least = time;
            pieces = s;
        }
    }
    const int64_t most = masked ? ON_LIVE_WORDS * 32 : n;   // a bit for every tile under a mask
    if ((n + pieces - 1) / pieces > most) return 0;

    CUtensorMap qmap, kmap, vmap;
    if (!make_query_map(&qmap, a, p.rep, p.hb, p.lb)) return 0;
    if (!make_map_tc(&kmap, a.k.data, a.k.dtype, a.D, a.T, a.Hkv, a.B, a.k.st, a.k.sh, a.k.sb, ON_KEYS)) return 0;
    if (!make_map_tc(&vmap, a.v.data, a.v.dtype, a.D, a.T, a.Hkv, a.B, a.v.st, a.v.sh, a.v.sb, ON_KEYS)) return 0;

    p.fold = fold_keys(a.q_dtype) / ON_KEYS;
    const bool folds = (n + pieces - 1) / pieces > p.fold;
    const size_t part = (size_t)units * pieces * TC_ROWS;
    const size_t o_bytes = part * a.D * sizeof(float), ml_bytes = part * sizeof(float2), t_bytes = (size_t)units * sizeof(int);
    CallMemory mem(pieces > 1 ? o_bytes + ml_bytes + t_bytes : folds && a.D > 64 ? o_bytes : 0, stream);
    if (!mem.ptr && (pieces > 1 || (folds && a.D > 64))) {   // no room: whole units that need no sums in memory, or the mma.sync kernel
        if (n > most || (n > p.fold && a.D > 64)) return 0;
        pieces = 1;
    }
    p.pieces = (int)pieces;
    p.o_part = (float *)mem.ptr;
    if (pieces > 1) {
        p.ml_part = (float2 *)((char *)mem.ptr + o_bytes);
        p.tickets = (int *)((char *)p.ml_part + ml_bytes);
        KVC_CUDA(cudaMemsetAsync(p.tickets, 0, t_bytes, stream));
    }
    const int ctas = (int)(units * p.pieces);
    // (the test for a fold costs a call of ten tiles 0.7 %)
    const bool long_sums = (n + pieces - 1) / pieces > p.fold;
    const bool taken = a.q_dtype == KVC_BF16
        ? (long_sums ? launch_one<__nv_bfloat16, true>(qmap, kmap, vmap, p, a.D, masked, ctas, stream)
                     : launch_one<__nv_bfloat16, false>(qmap, kmap, vmap, p, a.D, masked, ctas, stream))
        : (long_sums ? launch_one<__half, true>(qmap, kmap, vmap, p, a.D, masked, ctas, stream)
                     : launch_one<__half, false>(qmap, kmap, vmap, p, a.D, masked, ctas, stream));
    if (taken && trace_dispatch())
        fprintf(stderr, "[kvc] chunk_one: %lld row tiles (%d heads x %d positions), %d pieces%s\n", (long long)units, p.hb, p.lb, p.pieces,
                masked ? ", array mask" : "");
    return taken ? 1 : 0;
}

}  // namespace kvc
