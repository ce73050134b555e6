// Split-K flash decoding for raw f16/bf16 caches on sm_100a.
//
// Work unit = (batch, KV head, token split). A CTA of one producer warp and
// four consumer warps streams its token range through a ring of shared-memory
// stages: the producer issues tiled TMA loads (cp.async.bulk.tensor, 128-byte
// swizzle) of K and V tiles straight from the cache arrays and signals an
// mbarrier per stage; each consumer warp owns 16 of a tile's 64 tokens, scores
// all query rows of the GQA group against them with m16n8k16 tensor-core MMAs
// (queries are the 16-row A operand, so every K/V byte is read from HBM and
// from shared memory exactly once for the whole group), keeps an online
// softmax in registers and accumulates P.V with a second MMA. The four warps'
// states are merged in shared memory into one un-normalised partial per unit.
// The last unit of a (batch, head) to finish - found with a ticket counter -
// merges the partials of all splits with a log-sum-exp reduction and writes
// the output row, so no second kernel is needed.
//
// Shared-memory layout of a tile: boxes of [64 tokens][64 elements] (128 bytes
// per row), 16-byte chunk c of row r stored at chunk c ^ (r & 7).
//   * K operand (B fragment, "col-major"): a lane reads whole 16-byte chunks of
//     its token's row; the k-slot <-> head-dim assignment of the MMAs is a
//     permutation (shared with the Q fragments) chosen so that a quarter-warp
//     touches all eight chunk columns: no bank conflicts, no shuffles.
//   * V operand: ldmatrix.trans over eight consecutive token rows, which the
//     swizzle spreads over all eight chunk columns as well.
//
// Every wait on an mbarrier is bounded; a wait that runs out records an error
// code in a device status word and the CTA leaves its loops.
#include "attn_common.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

namespace kvc {

namespace {

using namespace dev;

constexpr int CONSUMER_WARPS = 4;
constexpr int DEC_THREADS = (CONSUMER_WARPS + 1) * 32;
constexpr int TILE_T = 64;  // tokens per tile: one 16-token block per consumer warp
constexpr int BOX_BYTES = TILE_T * 128;
constexpr int COUNTER_BYTES = 64 * 1024;  // ticket counters at the start of the scratch arena

struct DecodeParams {
    const void *q;
    void *out;
    int64_t q_sb, q_sh, q_sl, o_sb, o_sh, o_sl;
    float *o_part;
    float2 *ml_part;
    int *counters;
    int *status;
    int32_t B, Hq, Hkv, L;
    int64_t T;
    int32_t splits;       // units per (batch, head)
    int32_t tiles_base;   // tiles per unit; the first tiles_rem units take one more
    int32_t tiles_rem;
    int32_t causal;
    int32_t out_dtype;
    int32_t debug_skip;  // measurement aid: 1 = consumers release tiles without computing
    int32_t row_blocks;  // chunk kernel: 64-row blocks per (batch, head)
    int32_t tiles_all;   // chunk kernel: tiles covering all T tokens
    FlatPlan flat;       // flat kernel
    int32_t q_bulk;      // flat kernel: the unit's query rows are one contiguous 16-byte aligned block
    // cache arrays as plain pointers (byte strides): fused append target, and the measurement aid
    // debug_skip & 2 (linear bulk copies of the same bytes instead of the tiled TMA loads)
    unsigned char *k_base, *v_base;
    int64_t kv_sb, kv_sh, kv_st;
    // fused append: the new rows [B, Hkv, D] of this step (null = the cache already holds them)
    const void *new_k, *new_v;
    int32_t early_tiles;  // flat kernel: the stored rows may be streamed before the preceding kernel has finished
    // flat kernel, fused append of unturned rows: pairs that turn (0: rows come turned), their layout and the position
    int32_t rope_pairs, rope_traditional;
    double rope_log2;
    float rope_scale;
    int64_t rope_position;
    int64_t new_slot;     // flat kernel, fused append: token index the new row is stored at (T - 1, or a ring slot)
    int64_t nk_sb, nk_sh, nv_sb, nv_sh;  // element strides
    int64_t causal_offset;
    float scale_log2;  // scale * log2(e)
    MaskDesc mask;     // chunk kernel with an array mask
    // chunk kernel on operand pairs: what the 16-bit rows of q leave of the exact ones (same strides; null: nothing),
    // whether the keys have such a half too, and the factors that give the scaled operands their size back (per query
    // row, per (batch, KV head) of the keys and of the values; null: 1)
    const void *q_low;
    const float *q_undo, *k_undo, *v_undo;
    int32_t k_low;
};

template <typename T, int D, int NSTAGE>
__global__ void __launch_bounds__(DEC_THREADS, (D <= 128 ? 2 : 1))
attn_decode_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                   const DecodeParams p) {
    constexpr int TILE_BYTES = TILE_T * D * 2;     // one K (or V) tile
    constexpr int BOXES = D / 64;                  // [64 tokens][64 elements] boxes per tile
    constexpr int KSTEPS = D / 16;
    constexpr int NT_O = D / 8;                    // output n-tiles (8 head dims each)
    constexpr int RED_STRIDE = D + 8;              // padded row of the cross-warp merge buffer
    static_assert(TILE_T == 16 * CONSUMER_WARPS, "one 16-token block per consumer warp");
    static_assert(CONSUMER_WARPS * 16 * RED_STRIDE * 4 + 512 + 16 * 64 * 4 <= NSTAGE * 2 * TILE_BYTES, "merge buffers must fit");

    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // pointer + offset (no integer round trip) so that loads through it stay ld.shared
    unsigned char *stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t *full = (uint64_t *)(stages + (size_t)NSTAGE * 2 * TILE_BYTES);
    uint64_t *empty = full + NSTAGE;
    int *is_last = (int *)(empty + NSTAGE);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = blockIdx.x % p.splits;
    const int bh = blockIdx.x / p.splits;
    const int hk = bh % p.Hkv, b = bh / p.Hkv;
    const int rep = p.Hq / p.Hkv;
    const int R = rep * p.L;

    // balanced split of the tile range
    const int tile_begin = split * p.tiles_base + min(split, p.tiles_rem);
    const int ntiles = p.tiles_base + (split < p.tiles_rem ? 1 : 0);

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CONSUMER_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();  // everything below reads what earlier kernels on the stream wrote

    bool ok = true;
    const int g = lane >> 2, c = lane & 3;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float o_acc[NT_O][4];
#pragma unroll
    for (int i = 0; i < NT_O; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;

    if (warp == CONSUMER_WARPS) {
        // ---------------- producer ----------------
        if (lane == 0) {
            for (int it = 0; it < ntiles && ok; ++it) {
                const int s = it % NSTAGE;
                if (it >= NSTAGE) ok = mbar_wait(&empty[s], ((it / NSTAGE) - 1) & 1);
                if (!ok) break;
                unsigned char *kt = stages + (size_t)s * 2 * TILE_BYTES;
                unsigned char *vt = kt + TILE_BYTES;
                mbar_expect_tx(&full[s], 2 * TILE_BYTES);
                const int t0 = (tile_begin + it) * TILE_T;
#pragma unroll
                for (int bx = 0; bx < BOXES; ++bx) {
                    tma_load_4d(kt + bx * BOX_BYTES, &kmap, &full[s], bx * 64, t0, hk, b);
                    tma_load_4d(vt + bx * BOX_BYTES, &vmap, &full[s], bx * 64, t0, hk, b);
                }
            }
            if (!ok) atomicExch(p.status, 1);
        }
    } else {
        // ---------------- consumers ----------------
        // Query fragments: rows r < R of this KV head's group; row r <-> (rep index r / L, position r % L).
        // k-step ks = (box bx, pass ps, half h): lane c covers chunk 2c + ps of the box, elements 4h..4h+3.
        uint32_t qa[KSTEPS][4];
        int64_t row_limit[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = g + 8 * half;
            const int l = r % p.L;
            row_limit[half] = (r < R) ? (p.causal ? min(p.T - 1, p.causal_offset + l) : p.T - 1) : -1;
        }
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
            const int bx = ks / 4, ps = (ks >> 1) & 1, h = ks & 1;
            const int d0 = bx * 64 + (2 * c + ps) * 8 + 4 * h;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = g + 8 * half;
                uint32_t w0 = 0, w1 = 0;
                if (r < R) {
                    const int hq = hk * rep + r / p.L, l = r % p.L;
                    const T *qp = (const T *)p.q + b * p.q_sb + hq * p.q_sh + l * p.q_sl + d0;
                    w0 = *(const uint32_t *)qp;
                    w1 = *(const uint32_t *)(qp + 2);
                }
                qa[ks][half] = w0;      // a0 / a1: k-slots 2c, 2c+1
                qa[ks][2 + half] = w1;  // a2 / a3: k-slots 2c+8, 2c+9
            }
        }
        // Lane-constant byte offsets inside a box.
        //   K: token row (16*warp + 8*j + g), chunk (2c + ps) ^ g
        //   V (ldmatrix): lane supplies the row of matrix i = lane / 8: token 16*warp + 8*(i & 1) + (lane & 7),
        //                 chunk (2*cp + (i >> 1)) ^ (lane & 7) for chunk pair cp
        const int blk = warp;
        uint32_t k_off[2];
#pragma unroll
        for (int ps = 0; ps < 2; ++ps) k_off[ps] = (uint32_t)((blk * 16 + g) * 128 + (((2 * c + ps) ^ g) << 4));
        uint32_t v_off[4];
        {
            const int mi = lane >> 3, rr = lane & 7;
#pragma unroll
            for (int cp = 0; cp < 4; ++cp)
                v_off[cp] = (uint32_t)((blk * 16 + (mi & 1) * 8 + rr) * 128 + (((2 * cp + (mi >> 1)) ^ rr) << 4));
        }

        for (int it = 0; it < ntiles && ok; ++it) {
            const int s = it % NSTAGE;
            ok = mbar_wait(&full[s], (it / NSTAGE) & 1);
            if (!ok) break;
            if (KVC_SKIP_BITS(p)) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);
                continue;
            }
            const unsigned char *kt = stages + (size_t)s * 2 * TILE_BYTES;
            const uint32_t vt_addr = smem_u32(kt + TILE_BYTES);
            const int64_t t_blk = (int64_t)(tile_begin + it) * TILE_T + blk * 16;

            // ---- S = Q K^T for 16 tokens (two n-tiles of 8), the two accumulator chains interleaved ----
            float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                for (int ps = 0; ps < 2; ++ps) {
                    const uint4 k0 = *(const uint4 *)(kt + bx * BOX_BYTES + k_off[ps]);
                    const uint4 k1 = *(const uint4 *)(kt + bx * BOX_BYTES + k_off[ps] + 8 * 128);
                    const int ks = bx * 4 + ps * 2;
                    MmaType<T>::mma(sc[0], qa[ks], k0.x, k0.y);
                    MmaType<T>::mma(sc[1], qa[ks], k1.x, k1.y);
                    MmaType<T>::mma(sc[0], qa[ks + 1], k0.z, k0.w);
                    MmaType<T>::mma(sc[1], qa[ks + 1], k1.z, k1.w);
                }
            }
            // ---- online softmax (log2 domain) ----
            float tmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int half = e >> 1;
                    const int64_t t = t_blk + j * 8 + 2 * c + (e & 1);
                    float v = sc[j][e] * p.scale_log2;
                    v = (t <= row_limit[half]) ? v : -INFINITY;
                    sc[j][e] = v;
                    tmax[half] = fmaxf(tmax[half], v);
                }
            }
            float alpha[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 1));
                tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 2));
                const float m_new = fmaxf(m_run[half], tmax[half]);
                alpha[half] = (m_new == -INFINITY) ? 1.f : fast_exp2(m_run[half] - m_new);
                m_run[half] = m_new;
            }
            uint32_t pa[4];
            {
                float pr[2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int half = e >> 1;
                        pr[j][e] = (m_run[half] == -INFINITY) ? 0.f : fast_exp2(sc[j][e] - m_run[half]);
                    }
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    l_run[half] = l_run[half] * alpha[half] + pr[0][2 * half] + pr[0][2 * half + 1] +
                                  pr[1][2 * half] + pr[1][2 * half + 1];
                pa[0] = MmaType<T>::pack(pr[0][0], pr[0][1]);  // row g,   k-slots 2c, 2c+1   (tokens 0..7)
                pa[1] = MmaType<T>::pack(pr[0][2], pr[0][3]);  // row g+8
                pa[2] = MmaType<T>::pack(pr[1][0], pr[1][1]);  // row g,   k-slots 2c+8, 2c+9 (tokens 8..15)
                pa[3] = MmaType<T>::pack(pr[1][2], pr[1][3]);  // row g+8
            }
            // ---- O = O * alpha + P V (rescale only when some row's maximum moved) ----
            if (__any_sync(0xffffffffu, (alpha[0] != 1.f) | (alpha[1] != 1.f))) {
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt) {
                    o_acc[nt][0] *= alpha[0];
                    o_acc[nt][1] *= alpha[0];
                    o_acc[nt][2] *= alpha[1];
                    o_acc[nt][3] *= alpha[1];
                }
            }
#pragma unroll
            for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                for (int cp = 0; cp < 4; ++cp) {
                    // four 8x8 matrices: (tokens 0..7 | 8..15) x (chunk 2cp | 2cp+1) of this box
                    uint32_t vf[4];
                    ldmatrix_x4_trans(vf, vt_addr + bx * BOX_BYTES + v_off[cp]);
                    MmaType<T>::mma(o_acc[bx * 8 + 2 * cp], pa, vf[0], vf[1]);
                    MmaType<T>::mma(o_acc[bx * 8 + 2 * cp + 1], pa, vf[2], vf[3]);
                }
            }
            release_fenced(&empty[s], lane);
        }
        if (!ok && lane == 0) atomicExch(p.status, 2);
    }

    // ---------------- merge the four consumer warps ----------------
    __syncthreads();
    float *red_o = (float *)stages;                                  // [4][16][RED_STRIDE]
    float *red_ml = red_o + CONSUMER_WARPS * 16 * RED_STRIDE;        // [4][16][2]
    if (warp < CONSUMER_WARPS) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 1);
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 2);
        }
        float *wo = red_o + warp * 16 * RED_STRIDE;
#pragma unroll
        for (int nt = 0; nt < NT_O; ++nt) {
            // n-tile nt: C columns 2c, 2c+1 <-> head dims 8*nt + 2c, 8*nt + 2c + 1
            *(float2 *)&wo[g * RED_STRIDE + 8 * nt + 2 * c] = make_float2(o_acc[nt][0], o_acc[nt][1]);
            *(float2 *)&wo[(g + 8) * RED_STRIDE + 8 * nt + 2 * c] = make_float2(o_acc[nt][2], o_acc[nt][3]);
        }
        if (c == 0) {
            red_ml[(warp * 16 + g) * 2 + 0] = m_run[0];
            red_ml[(warp * 16 + g) * 2 + 1] = l_run[0];
            red_ml[(warp * 16 + g + 8) * 2 + 0] = m_run[1];
            red_ml[(warp * 16 + g + 8) * 2 + 1] = l_run[1];
        }
    }
    __syncthreads();
    UnitOut u;
    u.o_part = p.o_part; u.ml_part = p.ml_part; u.counters = p.counters;
    u.out = p.out; u.out_dtype = p.out_dtype;
    u.o_sb = p.o_sb; u.o_sh = p.o_sh; u.o_sl = p.o_sl;
    u.o_signs = nullptr;
    u.splits = p.splits; u.Hq = p.Hq; u.L = p.L;
    // work area behind the cross-warp buffers (the stage ring is idle by now)
    float *work = red_ml + CONSUMER_WARPS * 16 * 2;
    unit_epilogue<D, CONSUMER_WARPS>(u, red_o, red_ml, RED_STRIDE, work, is_last, b, hk, rep, R, split, bh);
}

// ---------------------------------------------------------------------
// Flat tile decomposition of the same decode computation. All (batch, head) units have
// the same number of tiles, so the launch is one wave of resident CTAs and CTA c simply
// owns the flat tile range [c W / G, (c + 1) W / G) of the W = units x tiles tiles. A
// range that crosses a unit boundary is processed as consecutive segments: the producer
// keeps streaming through the boundary, the consumers finish a segment (cross-warp
// merge, partial to scratch, ticket) and start the next with fresh state. Every CTA does
// the same amount of streaming whatever the shape, and the ramp at both ends of the
// launch is paid once. The cross-warp buffer sits beside the ring (the ring stays live),
// and the consumer warps synchronise among themselves with a named barrier that every
// warp reaches whether or not one of its bounded waits has run out.
// ---------------------------------------------------------------------
//
// LIST runs the calls of one shape (the layers of a batched step, whose inputs are all in hand) as one
// launch: a step of small layers is otherwise a chain of launches that each cost their ramp, merge and tail
// (26 layers of the Gemma-3-1B shape: 383 us as 26 launches). Each call keeps the ranges it has as a launch of its
// own, dealt to the resident CTAs in turn, so its outputs are the same bits: P is rounded to 16 bits, tokens that are
// a range's maximum are exact, and longer ranges have fewer of those (one range per CTA over all calls: the error
// against 64-bit sums rises by 3 .. 5 %). With several ranges per CTA a range must end without a wait: every warp
// leaves its state in memory and walks on, and flat_list_merge_kernel does the merges of all units behind it. 26 layers
// of the Gemma-3-1B shape (4 x 2048 tokens, rings of 512) and 8 layers of 8 x 8192 tokens, 32/8 heads, D 128, bf16:
// 160 and 436 us with the merges inside (ticket, last CTA of the unit), 61 and 379 behind, 47 and 350 with the
// descriptors handed over (FlatWork); one launch per call took 391 and 402.
constexpr int FLAT_AHEAD = 4;   // segments of a list the producer may be ahead
struct FlatLayer {
    CUtensorMap kmap, vmap;
    const void *q;
    void *out;
    int64_t q_sb, o_sb;
    unsigned char *k_base, *v_base;
    int64_t kv_sb, kv_sh, kv_st;
    const void *new_k, *new_v;
    int64_t new_slot, nk_sb, nk_sh, nv_sb, nv_sh, T;
    int64_t part_first;        // row slots of the partials before this layer's
    int32_t tiles, per, rem;   // tiles per unit; tiles per range of the call's own plan
    int32_t nslots, first;     // partial slots per row; ranges of the layers before this one
};
struct FlatList {
    int32_t n, ranges;
    FlatLayer layer[KVC_LIST_MAX];
};
struct FlatSingle {
    CUtensorMap kmap, vmap;
};

// The range and the unit a CTA is at, and the unit's arrays.
struct FlatSeg {
    FlatPlan plan;
    const CUtensorMap *kmap, *vmap;
    const void *q, *new_k, *new_v;
    void *out;
    int64_t q_sb, o_sb;
    unsigned char *k_base, *v_base;
    int64_t kv_sb, kv_sh, kv_st, new_slot, nk_sb, nk_sh, nv_sb, nv_sh, T, part_first;
    int cta, layer, unit, hk, b, t0, n;
};

// Range `r` of the launch: its call and its tiles [x_lo, x_hi) of that call.
template <bool LIST, typename LT>
__device__ __forceinline__ void flat_range(FlatSeg &g, const DecodeParams &p, const LT &list, int r, int64_t &x_lo, int64_t &x_hi) {
    g.plan = p.flat;
    g.cta = r;
    if constexpr (LIST) {
        while (g.layer + 1 < list.n && list.layer[g.layer + 1].first <= r) ++g.layer;
        const FlatLayer &l = list.layer[g.layer];
        g.cta = r - l.first;
        g.plan.tiles = l.tiles; g.plan.per = l.per; g.plan.rem = l.rem; g.plan.nslots = l.nslots;
        g.part_first = l.part_first;
        g.kmap = &l.kmap; g.vmap = &l.vmap;
        g.q = l.q; g.out = l.out; g.q_sb = l.q_sb; g.o_sb = l.o_sb;
        g.k_base = l.k_base; g.v_base = l.v_base;
        g.kv_sb = l.kv_sb; g.kv_sh = l.kv_sh; g.kv_st = l.kv_st;
        g.new_k = l.new_k; g.new_v = l.new_v; g.new_slot = l.new_slot;
        g.nk_sb = l.nk_sb; g.nk_sh = l.nk_sh; g.nv_sb = l.nv_sb; g.nv_sh = l.nv_sh;
        g.T = l.T;
    } else {
        g.kmap = &list.kmap; g.vmap = &list.vmap;
        g.q = p.q; g.out = p.out; g.q_sb = p.q_sb; g.o_sb = p.o_sb;
        g.k_base = p.k_base; g.v_base = p.v_base;
        g.kv_sb = p.kv_sb; g.kv_sh = p.kv_sh; g.kv_st = p.kv_st;
        g.new_k = p.new_k; g.new_v = p.new_v; g.new_slot = p.new_slot;
        g.nk_sb = p.nk_sb; g.nk_sh = p.nk_sh; g.nv_sb = p.nv_sb; g.nv_sh = p.nv_sh;
        g.T = p.T;
    }
    x_lo = flat_lo(g.plan, g.cta);
    x_hi = flat_lo(g.plan, g.cta + 1);
}

// The unit that tile `x` of the call falls in (32-bit: a tile is 16 KB at least).
__device__ __forceinline__ void flat_locate(FlatSeg &g, const DecodeParams &p, int64_t x, int64_t x_hi) {
    const int u = (int)((uint32_t)x / (uint32_t)g.plan.tiles);
    g.t0 = (int)x - u * g.plan.tiles;
    g.n = (int)min((int64_t)(g.plan.tiles - g.t0), x_hi - x);
    g.b = u / p.Hkv;
    g.hk = u - g.b * p.Hkv;
    g.unit = u;
}

// What the consumers need of a segment.
struct FlatWork {
    const unsigned char *q, *new_k, *new_v;   // the unit's query rows, and its new rows (null: stored already)
    unsigned char *k_row, *v_row;             // where the new rows go
    int64_t T, new_slot, part;                // part: first row slot of the segment's partials (lists)
    int32_t t0, n, nslots, more;              // more: 0 ends a list
    int32_t unit, hk, b, last;                // last: the segment ends its unit
};
// Its new rows and where they go (read by the warp that appends, at the segment's end).
template <typename T>
__device__ __forceinline__ void flat_new_rows(FlatWork &w, const FlatSeg &g) {
    w.new_k = (const unsigned char *)((const T *)g.new_k + g.b * g.nk_sb + g.hk * g.nk_sh);
    w.new_v = (const unsigned char *)((const T *)g.new_v + g.b * g.nv_sb + g.hk * g.nv_sh);
    const int64_t row = g.b * g.kv_sb + g.hk * g.kv_sh + g.new_slot * g.kv_st;
    w.k_row = g.k_base + row;
    w.v_row = g.v_base + row;
}
template <typename T>
__device__ __forceinline__ FlatWork flat_work(const FlatSeg &g, const DecodeParams &p) {
    FlatWork w;
    const int rep = p.Hq / p.Hkv;
    w.q = (const unsigned char *)((const T *)g.q + g.b * g.q_sb + (int64_t)g.hk * rep * p.q_sh);
    w.new_k = (const unsigned char *)g.new_k;
    w.T = g.T; w.new_slot = g.new_slot;
    w.t0 = g.t0; w.n = g.n;
    w.unit = g.unit; w.hk = g.hk; w.b = g.b;
    w.last = g.t0 + g.n == g.plan.tiles;
    w.more = 1;
    return w;
}

// The queries of a chat step come unturned (ROPE): a launch of its own for their rotary positions cost more than the turns.
// The angles are worked out before the wait on the kernel before; the consumers turn the unit's query rows where the bulk
// copy puts them, the warp that appends turns the new key row, and the tiles are drawn towards L2 before the wait. A layer
// of 32/8 heads, D 128, 1 031 tokens: 8.8 us in two launches, 8.1 in one. The bits are those of the two launches.
template <typename T, int D>
__device__ __forceinline__ void rope_row(T *row, const float2 *tab, const DecodeParams &p, int i) {
    const int i0 = p.rope_traditional ? 2 * i : i, i1 = p.rope_traditional ? 2 * i + 1 : i + p.rope_pairs;
    float y0, y1;
    rope_turn(to_f32<T>(row[i0]), to_f32<T>(row[i1]), tab[i].x, tab[i].y, y0, y1);
    MmaType<T>::store(row, i0, y0);
    MmaType<T>::store(row, i1, y1);
}

template <typename T, int D, int NSTAGE, bool LIST, bool ROPE>
__global__ void __launch_bounds__(DEC_THREADS, (D <= 128 ? 2 : 1))
attn_decode_flat_kernel(const __grid_constant__ std::conditional_t<LIST, FlatList, FlatSingle> list,
                        const __grid_constant__ DecodeParams p) {
    constexpr int TILE_BYTES = TILE_T * D * 2;
    constexpr int BOXES = D / 64;
    constexpr int KSTEPS = D / 16;
    constexpr int NT_O = D / 8;
    constexpr int RED_STRIDE = D + 8;

    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t *full = (uint64_t *)(stages + (size_t)NSTAGE * 2 * TILE_BYTES);
    uint64_t *empty = full + NSTAGE;
    int *is_last = (int *)(empty + NSTAGE);
    const FlatPlan &fp = p.flat;
    float *red_o = (float *)(is_last + 4);                                   // [4][red_rows][RED_STRIDE]
    float *red_ml = red_o + CONSUMER_WARPS * fp.red_rows * RED_STRIDE;       // [4][red_rows][2]
    // Query rows of a segment's unit, brought in by the producer with one bulk copy (two buffers):
    // plain loads issued by the consumers while the tile stream saturates the memory system cost
    // several microseconds per segment.
    // Lists have no cross-warp buffer, and the producer hands the consumers a segment's descriptor with its query rows:
    // worked out by every warp at a segment's start it was constant-cache misses and divisions between two tiles.
    constexpr int NQ = LIST ? FLAT_AHEAD : 2;
    uint64_t *qfull = LIST ? (uint64_t *)red_o : (uint64_t *)(red_ml + CONSUMER_WARPS * fp.red_rows * 2);   // (qbuf stays 16-byte aligned)
    uint64_t *qempty = qfull + NQ;
    unsigned char *qbuf = (unsigned char *)(qempty + NQ);                     // [NQ][red_rows][D] elements
    float2 *rope_tab = (float2 *)(qbuf + (size_t)NQ * (p.Hq / p.Hkv) * p.L * D * 2);   // [D / 2] cosines and sines (ROPE), then
    T *rope_k = (T *)(rope_tab + D / 2);                                      // [D] the new key row
    FlatWork *works = (FlatWork *)(qbuf + (size_t)NQ * (p.Hq / p.Hkv) * p.L * D * 2);   // [NQ] (lists)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rep = p.Hq / p.Hkv;
    const int R = rep * p.L;
    const uint32_t q_bytes = (uint32_t)R * D * 2;
    int ranges = gridDim.x;
    if constexpr (LIST) ranges = list.ranges;

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CONSUMER_WARPS);
        }
        for (int s = 0; s < NQ; ++s) {
            mbar_init(&qfull[s], 1);
            mbar_init(&qempty[s], CONSUMER_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (ROPE && tid < p.rope_pairs) {
        float cs, sn;
        rope_angle(tid, p.rope_log2, p.rope_position, p.rope_scale, cs, sn);
        rope_tab[tid] = make_float2(cs, sn);
    }
    __syncthreads();
    // Everything read below was written by earlier kernels on the stream, so it comes after the wait
    // on the preceding kernel. One exception, early_tiles: the producer streams its first tiles of
    // stored rows before that wait. The host vouches that the preceding kernel does not write them (it
    // is a layer of the same batched call, working on another cache), and every kernel before that one
    // has completed, because kernels release their successor only after their own wait.
    const bool early = p.early_tiles != 0 && warp == CONSUMER_WARPS, ahead = early || (ROPE && warp == CONSUMER_WARPS);
    if (!ahead) {
        pdl_wait();
        pdl_trigger();
    }

    bool ok = true;
    if (warp == CONSUMER_WARPS) {
        // ---------------- producer: one stream of tiles across the segments ----------------
        if (lane == 0) {
            int it = 0, sg = 0;
            bool waited = !ahead;
            FlatSeg gs;
            gs.layer = 0;
            int r = blockIdx.x;
            for (int64_t x = 0, x_hi = 0; ok; ++sg) {
                if (x == x_hi) {
                    if (r >= ranges) break;
                    flat_range<LIST>(gs, p, list, r, x, x_hi);
                    r += gridDim.x;
                }
                flat_locate(gs, p, x, x_hi);
                const int t0 = gs.t0, n = gs.n, hk = gs.hk, b = gs.b;
                int j_first = 0;
                if (ROPE && !waited && !early) {
                    for (int j = 0; j < n && j < NSTAGE; ++j)
#pragma unroll
                        for (int bx = 0; bx < BOXES; ++bx) {
                            tma_prefetch_4d(gs.kmap, bx * 64, (t0 + j) * TILE_T, hk, b);
                            tma_prefetch_4d(gs.vmap, bx * 64, (t0 + j) * TILE_T, hk, b);
                        }
                    pdl_wait();
                    pdl_trigger();
                    waited = true;
                }
                if (!waited) {
                    // the ring is empty: up to NSTAGE tiles go out before the wait
                    for (; j_first < n && j_first < NSTAGE; ++j_first, ++it) {
                        unsigned char *kt = stages + (size_t)it * 2 * TILE_BYTES;
                        unsigned char *vt = kt + TILE_BYTES;
                        mbar_expect_tx(&full[it], 2 * TILE_BYTES);
                        const int tok = (t0 + j_first) * TILE_T;
#pragma unroll
                        for (int bx = 0; bx < BOXES; ++bx) {
                            tma_load_4d(kt + bx * BOX_BYTES, gs.kmap, &full[it], bx * 64, tok, hk, b);
                            tma_load_4d(vt + bx * BOX_BYTES, gs.vmap, &full[it], bx * 64, tok, hk, b);
                        }
                    }
                    pdl_wait();
                    pdl_trigger();
                    waited = true;
                }
                if (LIST || p.q_bulk) {
                    const int qb = sg % NQ;
                    if (sg >= NQ) ok = mbar_wait(&qempty[qb], ((sg / NQ) - 1) & 1);
                    if (!ok) break;
                    if constexpr (LIST) {
                        FlatWork w = flat_work<T>(gs, p);
                        if (gs.new_k) flat_new_rows<T>(w, gs);
                        w.nslots = gs.plan.nslots;
                        w.part = gs.part_first + ((int64_t)b * p.Hq + hk * rep) * w.nslots + gs.cta - flat_cta_of(gs.plan, x - t0);
                        works[qb] = w;
                    }
                    if (p.q_bulk) mbar_expect_tx(&qfull[qb], q_bytes);
                    else mbar_arrive(&qfull[qb]);
                }
                if (p.q_bulk) {
                    const int qb = sg % NQ;
                    bulk_load(qbuf + (size_t)qb * q_bytes, (const T *)gs.q + b * gs.q_sb + (int64_t)hk * rep * p.q_sh, q_bytes,
                              &qfull[qb]);
                }
                for (int j = j_first; j < n && ok; ++j, ++it) {
                    const int s = it % NSTAGE;
                    if (it >= NSTAGE) {
                        // measurement aid (debug_skip & 4): the producer alone recycles the ring
                        if (KVC_SKIP_BITS(p) & 4) ok = mbar_wait(&full[s], ((it / NSTAGE) - 1) & 1);
                        else ok = mbar_wait(&empty[s], ((it / NSTAGE) - 1) & 1);
                    }
                    if (!ok) break;
                    unsigned char *kt = stages + (size_t)s * 2 * TILE_BYTES;
                    unsigned char *vt = kt + TILE_BYTES;
                    mbar_expect_tx(&full[s], 2 * TILE_BYTES);
                    const int tok = (t0 + j) * TILE_T;
                    if (KVC_SKIP_BITS(p) & 2) {
                        const int64_t off = b * gs.kv_sb + hk * gs.kv_sh + (int64_t)tok * gs.kv_st;
                        bulk_load(kt, gs.k_base + off, TILE_BYTES, &full[s]);
                        bulk_load(vt, gs.v_base + off, TILE_BYTES, &full[s]);
                        continue;
                    }
#pragma unroll
                    for (int bx = 0; bx < BOXES; ++bx) {
                        tma_load_4d(kt + bx * BOX_BYTES, gs.kmap, &full[s], bx * 64, tok, hk, b);
                        tma_load_4d(vt + bx * BOX_BYTES, gs.vmap, &full[s], bx * 64, tok, hk, b);
                    }
                }
                x += n;
            }
            if constexpr (LIST) {
                const int qb = sg % NQ;
                if (ok && sg >= NQ) ok = mbar_wait(&qempty[qb], ((sg / NQ) - 1) & 1);
                if (ok) {
                    works[qb].more = 0;
                    mbar_arrive(&qfull[qb]);
                }
            }
            if (!ok) atomicExch(p.status, 9);
        }
        return;
    }

    // ---------------- consumers ----------------
    if (KVC_SKIP_BITS(p) & 8) return;  // measurement aid: no consumer work at all (with 4: producer-only streaming)
    const int g = lane >> 2, c = lane & 3;
    const int blk = warp;
    uint32_t k_off[2];
#pragma unroll
    for (int ps = 0; ps < 2; ++ps) k_off[ps] = (uint32_t)((blk * 16 + g) * 128 + (((2 * c + ps) ^ g) << 4));
    uint32_t v_off[4];
    {
        const int mi = lane >> 3, rr = lane & 7;
#pragma unroll
        for (int cp = 0; cp < 4; ++cp)
            v_off[cp] = (uint32_t)((blk * 16 + (mi & 1) * 8 + rr) * 128 + (((2 * cp + (mi >> 1)) ^ rr) << 4));
    }

    const uint32_t none = gridDim.y - 1;
    int it = 0, sg = 0;
    FlatSeg gs;
    gs.layer = 0;
    int64_t x = 0, x_hi = 0;
    if constexpr (!LIST) flat_range<LIST>(gs, p, list, blockIdx.x, x, x_hi);
    for (;; ++sg) {
        FlatWork own;
        const int qb = sg % NQ;
        if constexpr (LIST) {
            ok = ok && mbar_wait(&qfull[qb], (sg / NQ) & 1);
            if (!ok) {
                if (lane == 0) atomicExch(p.status, 13);
                break;                                // no barrier is shared with the other warps here
            }
            if (!works[qb].more) break;
        } else {
            if (x >= x_hi) break;
            flat_locate(gs, p, x, x_hi);
            own = flat_work<T>(gs, p);
        }
        const FlatWork &w = LIST ? works[qb] : own;
        const int t0 = w.t0, n = w.n;
        // Fused append: token T - 1 is not in the cache yet; the tiles are masked up to T - 2 and the
        // new row is scored from its source by warp 0 of the CTA that owns the unit's last tile.
        const bool fused = w.new_k != nullptr;
        // Appending at the end: the tiles are simply cut one token short. Replacing a row inside a
        // wrapped ring: every token is visible except that slot, which still holds the row it loses.
        const bool ring = fused && w.new_slot != w.T - 1;
        const int64_t t_cached = w.T - ((fused && !ring) ? 2 : 1);
        const int64_t hole = ring ? w.new_slot : -1;
        int64_t row_limit[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = g + 8 * half;
            const int l = r % p.L;
            row_limit[half] = (r < R) ? (p.causal ? min(t_cached, p.causal_offset + l) : t_cached) : -1;
        }
        if (ROPE && fused && warp == 0 && w.last) {
            // the new key row, turned as the queries are; its last reads lie behind the barriers of the segment before
            FlatWork rows;
            flat_new_rows<T>(rows, gs);
            if (lane < D / 8) *(uint4 *)(rope_k + 8 * lane) = *(const uint4 *)(rows.new_k + 16 * lane);
            __syncwarp();
            for (int i = lane; i < p.rope_pairs; i += 32) rope_row<T, D>(rope_k, rope_tab, p, i);
            __syncwarp();
        }
        if (fused && warp == 0 && w.last && lane < 4) {
            // the new rows are consumed at the end of the segment: pull them towards L2 now
            FlatWork rows;
            if constexpr (!LIST) flat_new_rows<T>(rows, gs);
            const FlatWork &nr = LIST ? w : rows;
            const unsigned char *line = ((lane & 1) ? nr.new_v : nr.new_k) + (lane >> 1) * 128;
            if ((lane >> 1) * 128 < D * 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
        }
        uint32_t qa[KSTEPS][4];
        if (p.q_bulk) {
            if (!LIST && ok) {
                ok = mbar_wait(&qfull[qb], (sg / NQ) & 1);
                if (!ok && lane == 0) atomicExch(p.status, 13);
            }
            const unsigned char *qs = qbuf + (size_t)qb * q_bytes;
            if constexpr (ROPE) {
                // (consumer threads alone; every one of them is here for every segment)
                for (int i = tid; i < R * p.rope_pairs; i += CONSUMER_WARPS * 32) {
                    const int r = i / p.rope_pairs;
                    rope_row<T, D>((T *)(qbuf + (size_t)qb * q_bytes) + (size_t)r * D, rope_tab, p, i - r * p.rope_pairs);
                }
                consumer_bar<CONSUMER_WARPS>();
            }
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
                const int bx = ks / 4, ps = (ks >> 1) & 1, h = ks & 1;
                const int d0 = bx * 64 + (2 * c + ps) * 8 + 4 * h;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int r = g + 8 * half;
                    uint2 w = make_uint2(0u, 0u);
                    if (r < R && ok) w = *(const uint2 *)(qs + ((size_t)r * D + d0) * 2);
                    qa[ks][half] = w.x;
                    qa[ks][2 + half] = w.y;
                }
            }
            // (the rows turned in place above are stores that the next copy into the slot comes after, too)
            if (!LIST && ok) release_fenced(&qempty[qb], lane);
        } else
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
            const int bx = ks / 4, ps = (ks >> 1) & 1, h = ks & 1;
            const int d0 = bx * 64 + (2 * c + ps) * 8 + 4 * h;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = g + 8 * half;
                uint32_t w0 = 0, w1 = 0;
                if (r < R && !(KVC_SKIP_BITS(p) & 32)) {
                    const T *qp = (const T *)w.q + (int64_t)(r / p.L) * p.q_sh + (r % p.L) * p.q_sl + d0;
                    w0 = *(const uint32_t *)qp;
                    w1 = *(const uint32_t *)(qp + 2);
                }
                qa[ks][half] = w0;
                qa[ks][2 + half] = w1;
            }
        }
        float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
        float o_acc[NT_O][4];
#pragma unroll
        for (int i = 0; i < NT_O; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;

        for (int j = 0; j < n; ++j, ++it) {
            if (!ok || (KVC_SKIP_BITS(p) & 4)) continue;  // a wait ran out earlier: walk on to the barriers below
            const int s = it % NSTAGE;
            ok = mbar_wait(&full[s], (it / NSTAGE) & 1);
            if (!ok) {
                if (lane == 0) atomicExch(p.status, 10);
                continue;
            }
            if (KVC_SKIP_BITS(p) & 1) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);
                continue;
            }
            const unsigned char *kt = stages + (size_t)s * 2 * TILE_BYTES;
            const uint32_t vt_addr = smem_u32(kt + TILE_BYTES);
            const int64_t t_blk = (int64_t)(t0 + j) * TILE_T + blk * 16;

            float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                for (int ps = 0; ps < 2; ++ps) {
                    const uint4 k0 = *(const uint4 *)(kt + bx * BOX_BYTES + k_off[ps]);
                    const uint4 k1 = *(const uint4 *)(kt + bx * BOX_BYTES + k_off[ps] + 8 * 128);
                    const int ks = bx * 4 + ps * 2;
                    MmaType<T>::mma(sc[0], qa[ks], k0.x, k0.y);
                    MmaType<T>::mma(sc[1], qa[ks], k1.x, k1.y);
                    MmaType<T>::mma(sc[0], qa[ks + 1], k0.z, k0.w);
                    MmaType<T>::mma(sc[1], qa[ks + 1], k1.z, k1.w);
                }
            }
            float tmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int half = e >> 1;
                    const int64_t t = t_blk + jj * 8 + 2 * c + (e & 1);
                    float v = sc[jj][e] * p.scale_log2;
                    v = (t <= row_limit[half] && t != hole) ? v : -INFINITY;
                    sc[jj][e] = v;
                    tmax[half] = fmaxf(tmax[half], v);
                }
            }
            float alpha[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 1));
                tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 2));
                const float m_new = fmaxf(m_run[half], tmax[half]);
                alpha[half] = (m_new == -INFINITY) ? 1.f : fast_exp2(m_run[half] - m_new);
                m_run[half] = m_new;
            }
            uint32_t pa[4];
            {
                float pr[2][4];
#pragma unroll
                for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int half = e >> 1;
                        pr[jj][e] = (m_run[half] == -INFINITY) ? 0.f : fast_exp2(sc[jj][e] - m_run[half]);
                    }
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    l_run[half] = l_run[half] * alpha[half] + pr[0][2 * half] + pr[0][2 * half + 1] +
                                  pr[1][2 * half] + pr[1][2 * half + 1];
                pa[0] = MmaType<T>::pack(pr[0][0], pr[0][1]);
                pa[1] = MmaType<T>::pack(pr[0][2], pr[0][3]);
                pa[2] = MmaType<T>::pack(pr[1][0], pr[1][1]);
                pa[3] = MmaType<T>::pack(pr[1][2], pr[1][3]);
            }
            if (__any_sync(0xffffffffu, (alpha[0] != 1.f) | (alpha[1] != 1.f))) {
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt) {
                    o_acc[nt][0] *= alpha[0];
                    o_acc[nt][1] *= alpha[0];
                    o_acc[nt][2] *= alpha[1];
                    o_acc[nt][3] *= alpha[1];
                }
            }
            uint32_t read = 0;   // the last word of the tile
#pragma unroll
            for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                for (int cp = 0; cp < 4; ++cp) {
                    uint32_t vf[4];
                    ldmatrix_x4_trans(vf, vt_addr + bx * BOX_BYTES + v_off[cp]);
                    read = vf[3];
                    MmaType<T>::mma(o_acc[bx * 8 + 2 * cp], pa, vf[0], vf[1]);
                    MmaType<T>::mma(o_acc[bx * 8 + 2 * cp + 1], pa, vf[2], vf[3]);
                }
            }
            // (6 layers of 13 sequences, 16/16 heads, D 64, 512 and 1 833 tokens: 50.9 us, 51.9 with the fence)
            release_after(&empty[s], lane, read, none);
        }

        if (fused && warp == 0 && w.last && !(KVC_SKIP_BITS(p) & 32)) {
            // ---- the step's new token: score q . k_new, fold it into this warp's state, store the rows ----
            FlatWork rows;
            if constexpr (!LIST) flat_new_rows<T>(rows, gs);
            const FlatWork &nr = LIST ? w : rows;
            const T *kn = ROPE ? rope_k : (const T *)nr.new_k, *vn = (const T *)nr.new_v;
            float dot[2] = {0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
                const int bx = ks / 4, ps = (ks >> 1) & 1, h = ks & 1;
                const int d0 = bx * 64 + (2 * c + ps) * 8 + 4 * h;
                const uint2 kw = *(const uint2 *)(kn + d0);
                const float2 k01 = MmaType<T>::unpack(kw.x), k23 = MmaType<T>::unpack(kw.y);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float2 q01 = MmaType<T>::unpack(qa[ks][half]), q23 = MmaType<T>::unpack(qa[ks][2 + half]);
                    dot[half] += q01.x * k01.x + q01.y * k01.y + q23.x * k23.x + q23.y * k23.y;
                }
            }
            float pn[2], alpha[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                dot[half] += __shfl_xor_sync(0xffffffffu, dot[half], 1);
                dot[half] += __shfl_xor_sync(0xffffffffu, dot[half], 2);
                const float sc_new = (g + 8 * half < R) ? dot[half] * p.scale_log2 : -INFINITY;
                const float m_new = fmaxf(m_run[half], sc_new);
                alpha[half] = (m_new == -INFINITY) ? 1.f : fast_exp2(m_run[half] - m_new);
                pn[half] = (m_new == -INFINITY) ? 0.f : fast_exp2(sc_new - m_new);
                m_run[half] = m_new;
                l_run[half] = l_run[half] * alpha[half] + (c == 0 ? pn[half] : 0.f);  // once per row
            }
#pragma unroll
            for (int nt = 0; nt < NT_O; ++nt) {
                const float2 vv = MmaType<T>::unpack(*(const uint32_t *)(vn + 8 * nt + 2 * c));
                o_acc[nt][0] = o_acc[nt][0] * alpha[0] + pn[0] * vv.x;
                o_acc[nt][1] = o_acc[nt][1] * alpha[0] + pn[0] * vv.y;
                o_acc[nt][2] = o_acc[nt][2] * alpha[1] + pn[1] * vv.x;
                o_acc[nt][3] = o_acc[nt][3] * alpha[1] + pn[1] * vv.y;
            }
            // the append itself: rows of D elements, 16 bytes per lane
            constexpr int CHUNKS = D * 2 / 16;
            for (int i = lane; i < 2 * CHUNKS; i += 32) {
                const bool is_v = i >= CHUNKS;
                const int ch = is_v ? i - CHUNKS : i;
                const uint4 x = *(const uint4 *)((const unsigned char *)(is_v ? vn : kn) + ch * 16);
                *(uint4 *)((is_v ? nr.v_row : nr.k_row) + ch * 16) = x;
            }
        }

        // ---- end of the segment ----
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 1);
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 2);
        }
        if constexpr (LIST) {
            // this warp's state goes to its place in the partials; the merge kernel reads it
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = g + 8 * half;
                if (r >= R) continue;
                const int64_t at = (w.part + (int64_t)r * w.nslots) * CONSUMER_WARPS + warp;
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt)
                    __stcg((float2 *)&p.o_part[at * D + 8 * nt + 2 * c], make_float2(o_acc[nt][2 * half], o_acc[nt][2 * half + 1]));
                if (c == 0) __stcg(&p.ml_part[at], make_float2(m_run[half], l_run[half]));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&qempty[qb]);      // descriptor and query rows may be replaced
        } else {
            // merge the four warps, publish the partial, maybe merge the unit
            float *wo = red_o + warp * fp.red_rows * RED_STRIDE;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = g + 8 * half;
                if (r >= R) continue;
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt)
                    *(float2 *)&wo[r * RED_STRIDE + 8 * nt + 2 * c] = make_float2(o_acc[nt][2 * half], o_acc[nt][2 * half + 1]);
                if (c == 0) {
                    red_ml[(warp * fp.red_rows + r) * 2 + 0] = m_run[half];
                    red_ml[(warp * fp.red_rows + r) * 2 + 1] = l_run[half];
                }
            }
            UnitOut u;
            u.o_part = p.o_part; u.ml_part = p.ml_part; u.counters = p.counters;
            u.out = p.out; u.out_dtype = p.out_dtype;
            u.o_sb = p.o_sb; u.o_sh = p.o_sh; u.o_sl = p.o_sl;
            u.o_signs = nullptr;
            u.splits = 0; u.Hq = p.Hq; u.L = p.L;
            if (!(KVC_SKIP_BITS(p) & 16))
                segment_epilogue<D, CONSUMER_WARPS>(u, fp, red_o, red_ml, RED_STRIDE, nullptr, is_last, w.unit, w.b, w.hk, rep, R);
        }
        x += n;
    }
}

// The merges of a list launch: x = unit over all calls, one thread an output element (latency is all there is to it).
// First the warps of every range, then the ranges of the unit in
// batches of eight: the operations and their order are those of segment_epilogue.
template <typename T, int D>
__global__ void __launch_bounds__(128)
flat_list_merge_kernel(const __grid_constant__ FlatList list, const __grid_constant__ DecodeParams p) {
    pdl_wait();
    pdl_trigger();
    const int units = p.B * p.Hkv, u = blockIdx.x % units, hk = u % p.Hkv, b = u / p.Hkv, rep = p.Hq / p.Hkv;
    const FlatLayer &l = list.layer[blockIdx.x / units];
    FlatPlan plan = p.flat;
    plan.tiles = l.tiles; plan.per = l.per; plan.rem = l.rem;
    const int64_t x = (int64_t)u * l.tiles;
    const int expected = flat_cta_of(plan, x + l.tiles - 1) - flat_cta_of(plan, x) + 1;
    const int i = blockIdx.y * 128 + threadIdx.x;
    if (i < rep * D) {
        const int r = i / D, d = i % D;
        const int64_t at = (l.part_first + ((int64_t)b * p.Hq + hk * rep + r) * l.nslots) * CONSUMER_WARPS;
        float m = -INFINITY, o = 0.f, lsum = 0.f;
        for (int s0 = 0; s0 < expected; s0 += 8) {
            float2 ml[8];
            float ov[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool in = s0 + j < expected;
                float2 wml[CONSUMER_WARPS];
                float wo[CONSUMER_WARPS], wm = -INFINITY;
#pragma unroll
                for (int w = 0; w < CONSUMER_WARPS; ++w) {
                    const int64_t a = at + (s0 + j) * CONSUMER_WARPS + w;
                    wml[w] = in ? __ldcg(&p.ml_part[a]) : make_float2(-INFINITY, 0.f);
                    wo[w] = in ? __ldcg(&p.o_part[a * D + d]) : 0.f;
                    wm = fmaxf(wm, wml[w].x);
                }
                ov[j] = 0.f;
                ml[j] = make_float2(wm, 0.f);
#pragma unroll
                for (int w = 0; w < CONSUMER_WARPS; ++w) {
                    const float fw = (wml[w].x == -INFINITY) ? 0.f : fast_exp2(wml[w].x - wm);
                    ov[j] = fmaf(wo[w], fw, ov[j]);
                    ml[j].y = fmaf(wml[w].y, fw, ml[j].y);
                }
            }
            float mb = m;
#pragma unroll
            for (int j = 0; j < 8; ++j) mb = fmaxf(mb, (ml[j].y > 0.f) ? ml[j].x : -INFINITY);
            const float keep = (m == -INFINITY) ? 0.f : fast_exp2(m - mb);
            o *= keep;
            lsum *= keep;
            m = mb;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float fw = (ml[j].x == -INFINITY || ml[j].y <= 0.f) ? 0.f : fast_exp2(ml[j].x - m);
                lsum = fmaf(ml[j].y, fw, lsum);
                o = fmaf(ov[j], fw, o);
            }
        }
        store_out(l.out, p.out_dtype, b * l.o_sb + (hk * rep + r) * p.o_sh + d, lsum > 0.f ? o / lsum : 0.f);
    }
}

// ---------------------------------------------------------------------
// Multi-token chunks (prefill chunks, speculative verify rounds): more than 16 query
// rows per KV head. Same ring, tiles and fragment layouts as above, but the consumer
// warps split the QUERY ROWS instead of the tokens: a CTA owns a block of 64 rows of one
// (batch, KV head) group (row r <-> head r / L of the group, position r % L), warp w owns
// rows 16w .. 16w+15 with their own softmax state and output accumulators, and every
// warp walks all four 16-token blocks of each tile. Under a causal mask a CTA only
// streams the tiles some row of its block can see. With one split per block the rows are
// normalised and written straight to the output; otherwise partials go to scratch and the
// last CTA of the block merges them.
//
// MASKED takes an array mask (a sliding-window layer's chunk, a caller's own). A boolean mask of a
// warp's 16 rows x 64 tokens is 32 bytes per lane: read as aligned words whatever the row pitch (a
// window mask has an odd one), squeezed to one bit per token while the tile is on its way, and handed
// to the fragment rows with four shuffles. A 16-token block no row of the warp may see costs no MMA.
// Additive masks are read where the scores are, and their scores stay in the natural domain (a row whose mask
// is the type's lowest value throughout is a uniform average; times log2(e) that value would be -inf). These calls
// ran in fp32 before, so P is a pair (its 16-bit rounding and what that leaves) and meets V in two MMAs. f16 pairs are carried
// 2^10 up, clear of subnormals, and FOLD adds a step's tokens to the running sums by fp32 instructions: the MMA's own
// accumulation rounds towards zero, and errors against 64-bit sums grew with the number of keys, by 0.02 % for f16
// outputs at 30 000 (for bf16, whose store is eight times coarser, by 0.0006 % at 16 000: no fold there, it costs a fifth
// of the time at D 256).
// Boolean masks come here only with up to 64 rows of a group or up to 64 keys (else attn_chunk_one_tc.cu), masks that are added
// with any number. Six 512-token chunks of the Gemma-3-1B shape (4 x 4 heads, D 256, five rings of 512 and a global layer) under
// boolean masks took 20.4 ms on the general kernel, 0.407 ms here (0.487 with one 16-token block at a time) and take 0.233 there.
//
// PAIRS takes q, K and V as pairs of arrays, high and low halves of fp32 values that were brought into the range of f16
// by powers of two: products of 22 significant bits (hi hi + lo hi + hi lo; the small ones are summed apart), for rows
// that are decoded from codes. T: f16, or bf16 for raw bf16 keys and their queries, which are exact as they are.
// ---------------------------------------------------------------------

__device__ __forceinline__ float mask_value(const MaskDesc &m, int64_t i) {
    switch (m.dtype) {
        case KVC_BOOL: return ((const uint8_t *)m.data)[i] ? 0.f : -INFINITY;
        case KVC_F32: return ((const float *)m.data)[i];
        case KVC_F16: return __half2float(((const __half *)m.data)[i]);
        default: return __bfloat162float(((const __nv_bfloat16 *)m.data)[i]);
    }
}

struct ChunkMaps {
    CUtensorMap k, v;
};
struct ChunkPairMaps {
    CUtensorMap k, v, k_low, v_low;
};

template <typename T, int D, int NSTAGE, bool MASKED, bool PAIRS>
__global__ void __launch_bounds__(DEC_THREADS, (D <= 128 ? 2 : 1))
attn_chunk_kernel(const __grid_constant__ std::conditional_t<PAIRS, ChunkPairMaps, ChunkMaps> maps, const DecodeParams p) {
    constexpr bool P_PAIR = MASKED || PAIRS;
    using VT = std::conditional_t<PAIRS, __half, T>;               // values and probabilities
    constexpr bool FOLD = P_PAIR && std::is_same_v<VT, __half>;
    constexpr float P_UP = P_PAIR && std::is_same_v<VT, __half> ? 1024.f : 1.f;
    constexpr int TILE_BYTES = TILE_T * D * 2;
    constexpr int BOXES = D / 64;
    constexpr int KSTEPS = D / 16;
    constexpr int NT_O = D / 8;

    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int STAGE_BYTES = (PAIRS ? 4 : 2) * TILE_BYTES;      // K, V (, low halves of K, of V)
    // Query fragments in shared memory where registers are short (bytes of one half); NBK: 16-token blocks a warp
    // takes at a time. At D 256 an SM holds one warp per scheduler, so the chains of a step have to hide one another:
    // two blocks give twice the independent MMAs. SMX: blocks that share a maximum and a rescale. One, where P is a
    // single 16-bit value: tokens that are the maximum of their block are exact, and a maximum per 32 tokens leaves half
    // as many (error against 64-bit sums + 0.4 % at 500 keys).
    constexpr bool Q_SHARED = PAIRS || D == 256;
    constexpr int QF_BYTES = Q_SHARED ? CONSUMER_WARPS * KSTEPS * 32 * 16 : 0;
    constexpr int NBK = D == 256 && !PAIRS ? 2 : 1, SMX = P_PAIR ? NBK : 1;
    unsigned char *qf = stages + (size_t)NSTAGE * STAGE_BYTES;
    uint64_t *full = (uint64_t *)(qf + (PAIRS ? 2 : 1) * QF_BYTES);
    uint64_t *empty = full + NSTAGE;
    int *is_last = (int *)(empty + NSTAGE);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = blockIdx.x % p.splits;
    const int unit = blockIdx.x / p.splits;
    const int rb = unit % p.row_blocks;
    const int bh = unit / p.row_blocks;
    const int hk = bh % p.Hkv, b = bh / p.Hkv;
    const int rep = p.Hq / p.Hkv;
    const int R = rep * p.L;
    const int r_lo = rb * 64, r_hi = min(R, r_lo + 64) - 1;

    // tiles some row of the block can see, then this split's share of them
    int tiles_needed = p.tiles_all;
    if (p.causal) {
        const int max_l = (r_lo / p.L == r_hi / p.L) ? (r_hi % p.L) : (p.L - 1);
        const int64_t lim = min(p.T - 1, p.causal_offset + max_l);
        tiles_needed = (int)min((int64_t)p.tiles_all, lim / TILE_T + 1);
    }
    const int t_base = tiles_needed / p.splits, t_rem = tiles_needed % p.splits;
    const int tile_begin = split * t_base + min(split, t_rem);
    const int ntiles = t_base + (split < t_rem ? 1 : 0);

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CONSUMER_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();  // everything below reads what earlier kernels on the stream wrote

    bool ok = true;
    const int g = lane >> 2, c = lane & 3;
    // scores: log2 domain, or natural (log2_unit turns differences into log2) where values of a mask are added
    const bool bits_mask = MASKED && p.mask.dtype == KVC_BOOL && p.mask.st == 1;
    const float log2_unit = MASKED && !bits_mask ? 1.4426950408889634f : 1.f;
    float score_scale = MASKED && !bits_mask ? p.scale_log2 * 0.6931471805599453f : p.scale_log2;
    float out_scale = 1.f / P_UP;
    if constexpr (PAIRS) {
        if (p.k_undo) score_scale *= p.k_undo[b * p.Hkv + hk];
        out_scale *= p.v_undo[b * p.Hkv + hk];
    }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float o_acc[NT_O][4];
#pragma unroll
    for (int i = 0; i < NT_O; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;

    if (warp == CONSUMER_WARPS) {
        if (lane == 0) {
            for (int it = 0; it < ntiles && ok; ++it) {
                const int s = it % NSTAGE;
                if (it >= NSTAGE) ok = mbar_wait(&empty[s], ((it / NSTAGE) - 1) & 1);
                if (!ok) break;
                unsigned char *kt = stages + (size_t)s * STAGE_BYTES;
                unsigned char *vt = kt + TILE_BYTES;
                mbar_expect_tx(&full[s], (2 + (PAIRS ? 1 + p.k_low : 0)) * TILE_BYTES);
                const int t0 = (tile_begin + it) * TILE_T;
#pragma unroll
                for (int bx = 0; bx < BOXES; ++bx) {
                    tma_load_4d(kt + bx * BOX_BYTES, &maps.k, &full[s], bx * 64, t0, hk, b);
                    tma_load_4d(vt + bx * BOX_BYTES, &maps.v, &full[s], bx * 64, t0, hk, b);
                    if constexpr (PAIRS) {
                        if (p.k_low) tma_load_4d(kt + 2 * TILE_BYTES + bx * BOX_BYTES, &maps.k_low, &full[s], bx * 64, t0, hk, b);
                        tma_load_4d(kt + 3 * TILE_BYTES + bx * BOX_BYTES, &maps.v_low, &full[s], bx * 64, t0, hk, b);
                    }
                }
            }
            if (!ok) atomicExch(p.status, 3);
        }
    } else {
        const int r_warp = r_lo + 16 * warp;
        uint32_t qa[Q_SHARED ? 1 : KSTEPS][4];
        uint4 *qh = (uint4 *)qf + (warp * KSTEPS) * 32 + lane, *ql = qh + QF_BYTES / 16;
        int row_limit[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = r_warp + g + 8 * half;
            const int l = r % p.L;
            row_limit[half] = (r < R) ? (int)(p.causal ? min(p.T - 1, p.causal_offset + l) : p.T - 1) : -1;
        }
        // the warp's widest and narrowest limits (rows past R excluded from the narrowest)
        int lim_max = max(row_limit[0], row_limit[1]);
        int lim_min = min(row_limit[0] < 0 ? 0x7fffffff : row_limit[0], row_limit[1] < 0 ? 0x7fffffff : row_limit[1]);
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
            lim_max = max(lim_max, __shfl_xor_sync(0xffffffffu, lim_max, o));
            lim_min = min(lim_min, __shfl_xor_sync(0xffffffffu, lim_min, o));
        }
        float row_scale[2] = {score_scale, score_scale};
        if (PAIRS && p.q_undo) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = min(r_warp + g + 8 * half, R - 1);
                row_scale[half] *= p.q_undo[((int64_t)b * p.Hq + hk * rep + r / p.L) * p.L + r % p.L];
            }
        }
        auto load_q = [&](const void *q, int ks, uint32_t (&f)[4]) {
            const int bx = ks / 4, ps = (ks >> 1) & 1, h = ks & 1;
            const int d0 = bx * 64 + (2 * c + ps) * 8 + 4 * h;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = r_warp + g + 8 * half;
                uint32_t w0 = 0, w1 = 0;
                if (r < R) {
                    const int hq = hk * rep + r / p.L, l = r % p.L;
                    const T *qp = (const T *)q + b * p.q_sb + hq * p.q_sh + l * p.q_sl + d0;
                    w0 = *(const uint32_t *)qp;
                    w1 = *(const uint32_t *)(qp + 2);
                }
                f[half] = w0;
                f[2 + half] = w1;
            }
        };
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
            load_q(p.q, ks, qa[Q_SHARED ? 0 : ks]);
            if constexpr (Q_SHARED) {      // read back by the lane that wrote them
                qh[ks * 32] = make_uint4(qa[0][0], qa[0][1], qa[0][2], qa[0][3]);
                if (PAIRS && p.q_low) {
                    load_q(p.q_low, ks, qa[0]);
                    ql[ks * 32] = make_uint4(qa[0][0], qa[0][1], qa[0][2], qa[0][3]);
                }
            }
        }
        uint32_t k_off[2];
#pragma unroll
        for (int ps = 0; ps < 2; ++ps) k_off[ps] = (uint32_t)(g * 128 + (((2 * c + ps) ^ g) << 4));
        uint32_t v_off[4];
        {
            const int mi = lane >> 3, rr = lane & 7;
#pragma unroll
            for (int cp = 0; cp < 4; ++cp)
                v_off[cp] = (uint32_t)(((mi & 1) * 8 + rr) * 128 + (((2 * cp + (mi >> 1)) ^ rr) << 4));
        }

        // MASKED: this lane reads the mask of row lane / 2 of the warp, 32 tokens from 32 * (lane & 1) on; mask
        // element (row half, token) of a score sits at row_mask[half] + token * st
        const uint8_t *lane_mask = nullptr;
        int64_t row_mask[2] = {0, 0};
        if (MASKED) {
            auto at = [&](int r) {
                const int rr = min(r, R - 1);
                return b * p.mask.sb + (int64_t)(hk * rep + rr / p.L) * p.mask.sh + (int64_t)(rr % p.L) * p.mask.sl;
            };
            lane_mask = (const uint8_t *)p.mask.data + at(r_warp + (lane >> 1)) + 32 * (lane & 1);
            row_mask[0] = at(r_warp + g);
            row_mask[1] = at(r_warp + g + 8);
        }

        for (int it = 0; it < ntiles && ok; ++it) {
            const int s = it % NSTAGE;
            uint32_t vis[2][2] = {{~0u, ~0u}, {~0u, ~0u}};   // [row half][32-token half of the tile]
            uint32_t live = 15;                              // 16-token blocks some row of the warp sees
            if (MASKED && bits_mask) {
                const int t0 = (tile_begin + it) * TILE_T;
                uint32_t mine = mask_bits32(lane_mask + t0, (int)min((int64_t)64, p.T - t0) - 32 * (lane & 1));
                if (r_warp + (lane >> 1) >= R) mine = 0;
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int q = 0; q < 2; ++q) vis[half][q] = __shfl_sync(0xffffffffu, mine, 2 * (g + 8 * half) + q);
                const uint32_t some = ((mine & 0xffffu) ? 1u : 0u) | ((mine >> 16) ? 2u : 0u);
                live = __reduce_or_sync(0xffffffffu, some << (2 * (lane & 1)));
            }
            ok = mbar_wait(&full[s], (it / NSTAGE) & 1);
            if (!ok) break;
            const unsigned char *kt = stages + (size_t)s * STAGE_BYTES;
            const uint32_t vt_addr = smem_u32(kt + TILE_BYTES);
#pragma unroll 1
            for (int blk = 0; blk < 4; blk += NBK) {
                const int t_blk = (tile_begin + it) * TILE_T + blk * 16;
                if (t_blk > lim_max) break;  // warp-uniform: nothing further in this tile is visible
                if (MASKED && !((live >> blk) & ((1u << NBK) - 1u))) continue;
                const uint32_t boff = blk * 16 * 128;
                float sc[2 * NBK][4], rest[PAIRS ? 2 * NBK : 1][4];      // rest: the products with a low half
#pragma unroll
                for (int j = 0; j < 2 * NBK; ++j) {
                    sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
                    if constexpr (PAIRS) rest[j][0] = rest[j][1] = rest[j][2] = rest[j][3] = 0.f;
                }
#pragma unroll(PAIRS ? 1 : BOXES)
                for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                    for (int ps = 0; ps < 2; ++ps) {
                        const int ks = bx * 4 + ps * 2;
                        const unsigned char *kp = kt + bx * BOX_BYTES + boff + k_off[ps];
                        auto score = [&](float (&d)[2 * NBK][4], const uint32_t (&f0)[4], const uint32_t (&f1)[4], const unsigned char *rows) {
                            uint4 x[2 * NBK];
#pragma unroll
                            for (int j = 0; j < 2 * NBK; ++j) x[j] = *(const uint4 *)(rows + j * 8 * 128);
#pragma unroll
                            for (int j = 0; j < 2 * NBK; ++j) MmaType<T>::mma(d[j], f0, x[j].x, x[j].y);
#pragma unroll
                            for (int j = 0; j < 2 * NBK; ++j) MmaType<T>::mma(d[j], f1, x[j].z, x[j].w);
                        };
                        if constexpr (Q_SHARED) {
                            const uint4 a0 = qh[ks * 32], a1 = qh[ks * 32 + 32];
                            const uint32_t f0[4] = {a0.x, a0.y, a0.z, a0.w}, f1[4] = {a1.x, a1.y, a1.z, a1.w};
                            score(sc, f0, f1, kp);
                            if constexpr (PAIRS) {
                                if (p.k_low) score(rest, f0, f1, kp + 2 * TILE_BYTES);
                                if (p.q_low) {
                                    const uint4 b0 = ql[ks * 32], b1 = ql[ks * 32 + 32];
                                    const uint32_t e0[4] = {b0.x, b0.y, b0.z, b0.w}, e1[4] = {b1.x, b1.y, b1.z, b1.w};
                                    score(rest, e0, e1, kp);
                                }
                            }
                        } else {
                            score(sc, qa[ks], qa[ks + 1], kp);
                        }
                    }
                }
                if constexpr (PAIRS) {
#pragma unroll
                    for (int j = 0; j < 2 * NBK; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) sc[j][e] += rest[j][e];
                }
                const bool edge = t_blk + 16 * NBK - 1 > lim_min;  // warp-uniform
#pragma unroll
                for (int u0 = 0; u0 < NBK; u0 += SMX) {
                    float tmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
                    for (int j = 2 * u0; j < 2 * (u0 + SMX); ++j) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int half = e >> 1;
                            float v = sc[j][e] * row_scale[half];
                            const int t = t_blk + j * 8 + 2 * c + (e & 1);
                            if (MASKED) {
                                if (bits_mask) {
                                    const int bit = (blk & 1) * 16 + j * 8 + 2 * c + (e & 1);
                                    if (!(((blk & 2 ? vis[half][1] : vis[half][0]) >> bit) & 1)) v = -INFINITY;
                                } else if (t <= row_limit[half]) {
                                    v += mask_value(p.mask, row_mask[half] + t * p.mask.st);
                                }
                            }
                            if (edge) v = (t <= row_limit[half]) ? v : -INFINITY;
                            sc[j][e] = v;
                            tmax[half] = fmaxf(tmax[half], v);
                        }
                    }
                    float alpha[2];
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 1));
                        tmax[half] = fmaxf(tmax[half], __shfl_xor_sync(0xffffffffu, tmax[half], 2));
                        const float m_new = fmaxf(m_run[half], tmax[half]);
                        alpha[half] = (m_new == -INFINITY) ? 1.f : fast_exp2((m_run[half] - m_new) * log2_unit);
                        m_run[half] = m_new;
                    }
                    uint32_t pa[SMX][4], pl[SMX][4];       // P, and what its rounding leaves
#pragma unroll
                    for (int j = 2 * u0; j < 2 * (u0 + SMX); ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int half = e >> 1;
                            sc[j][e] = (m_run[half] == -INFINITY) ? 0.f : fast_exp2((sc[j][e] - m_run[half]) * log2_unit);
                        }
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        l_run[half] = fmaf(l_run[half], alpha[half], sc[2 * u0][2 * half]) + sc[2 * u0][2 * half + 1];
#pragma unroll
                        for (int j = 2 * u0 + 1; j < 2 * (u0 + SMX); ++j) l_run[half] = l_run[half] + sc[j][2 * half] + sc[j][2 * half + 1];
                    }
#pragma unroll
                    for (int u = 0; u < SMX; ++u)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int j = 2 * (u0 + u) + (i >> 1);
                            const float x = sc[j][2 * (i & 1)] * P_UP, y = sc[j][2 * (i & 1) + 1] * P_UP;
                            pa[u][i] = MmaType<VT>::pack(x, y);
                            if constexpr (P_PAIR) {
                                const float2 hi = MmaType<VT>::unpack(pa[u][i]);
                                pl[u][i] = MmaType<VT>::pack(x - hi.x, y - hi.y);
                            }
                        }
                    if constexpr (!FOLD) {
                        if (__any_sync(0xffffffffu, (alpha[0] != 1.f) | (alpha[1] != 1.f))) {
#pragma unroll
                            for (int nt = 0; nt < NT_O; ++nt) {
                                o_acc[nt][0] *= alpha[0];
                                o_acc[nt][1] *= alpha[0];
                                o_acc[nt][2] *= alpha[1];
                                o_acc[nt][3] *= alpha[1];
                            }
                        }
                    }
#pragma unroll
                    for (int bx = 0; bx < BOXES; ++bx) {
#pragma unroll
                        for (int cp = 0; cp < 4; ++cp) {
                            const int nt = bx * 8 + 2 * cp;
                            uint32_t vf[4];
                            if constexpr (FOLD) {
                                float part[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};   // this step's tokens
#pragma unroll
                                for (int u = 0; u < SMX; ++u) {
                                    const uint32_t va = vt_addr + bx * BOX_BYTES + boff + (u0 + u) * 16 * 128 + v_off[cp];
                                    if constexpr (PAIRS) {
                                        ldmatrix_x4_trans(vf, va + 2 * TILE_BYTES);
                                        MmaType<VT>::mma(part[0], pa[u], vf[0], vf[1]);
                                        MmaType<VT>::mma(part[1], pa[u], vf[2], vf[3]);
                                    }
                                    ldmatrix_x4_trans(vf, va);
                                    MmaType<VT>::mma(part[0], pl[u], vf[0], vf[1]);
                                    MmaType<VT>::mma(part[1], pl[u], vf[2], vf[3]);
                                    MmaType<VT>::mma(part[0], pa[u], vf[0], vf[1]);
                                    MmaType<VT>::mma(part[1], pa[u], vf[2], vf[3]);
                                }
#pragma unroll
                                for (int i = 0; i < 2; ++i)
#pragma unroll
                                    for (int e = 0; e < 4; ++e) o_acc[nt + i][e] = fmaf(o_acc[nt + i][e], alpha[e >> 1], part[i][e]);
                            } else {
#pragma unroll
                                for (int u = 0; u < SMX; ++u) {
                                    ldmatrix_x4_trans(vf, vt_addr + bx * BOX_BYTES + boff + (u0 + u) * 16 * 128 + v_off[cp]);
                                    MmaType<T>::mma(o_acc[nt], pa[u], vf[0], vf[1]);
                                    MmaType<T>::mma(o_acc[nt + 1], pa[u], vf[2], vf[3]);
                                    if constexpr (P_PAIR) {
                                        MmaType<T>::mma(o_acc[nt], pl[u], vf[0], vf[1]);
                                        MmaType<T>::mma(o_acc[nt + 1], pl[u], vf[2], vf[3]);
                                    }
                                }
                            }
                        }
                    }
                }
            }
            release_fenced(&empty[s], lane);
        }
        if (!ok && lane == 0) atomicExch(p.status, 4);

        // ---- the warp's 16 rows: straight to the output, or partials for the merge ----
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 1);
            l_run[half] += __shfl_xor_sync(0xffffffffu, l_run[half], 2);
        }
        const int64_t qrow0 = ((int64_t)b * p.Hq + hk * rep) * p.L;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = r_warp + g + 8 * half;
            if (r >= R) continue;
            if (p.splits == 1) {
                const float inv = l_run[half] > 0.f ? out_scale / l_run[half] : 0.f;
                const int hq = hk * rep + r / p.L, lq = r % p.L;
                const int64_t base = b * p.o_sb + hq * p.o_sh + lq * p.o_sl;
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt) {
                    store_out(p.out, p.out_dtype, base + 8 * nt + 2 * c, o_acc[nt][2 * half] * inv);
                    store_out(p.out, p.out_dtype, base + 8 * nt + 2 * c + 1, o_acc[nt][2 * half + 1] * inv);
                }
            } else {
                const int64_t pbase = (qrow0 + r) * p.splits + split;
#pragma unroll
                for (int nt = 0; nt < NT_O; ++nt)
                    __stcg((float2 *)&p.o_part[pbase * D + 8 * nt + 2 * c],
                           make_float2(o_acc[nt][2 * half] * out_scale, o_acc[nt][2 * half + 1] * out_scale));
                if (c == 0) __stcg(&p.ml_part[pbase], make_float2(m_run[half], l_run[half]));
            }
        }
    }
    if (p.splits == 1) return;

    // ---- split merge by the last CTA of this row block ----
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int ticket = atomicAdd(&p.counters[unit], 1);
        const int last = (ticket == p.splits - 1) ? 1 : 0;
        if (last) p.counters[unit] = 0;
        *is_last = last;
    }
    __syncthreads();
    if (!*is_last) return;
    __threadfence();
    float *work = (float *)stages;  // [rows of the block][splits] merge weights (the ring is idle)
    const int64_t qrow0 = ((int64_t)b * p.Hq + hk * rep) * p.L;
    const int nrows = r_hi - r_lo + 1;
    for (int rr = warp; rr < nrows; rr += DEC_THREADS / 32) {
        const int64_t row = qrow0 + r_lo + rr;
        float m = -INFINITY;
        for (int s = lane; s < p.splits; s += 32) m = fmaxf(m, __ldcg(&p.ml_part[row * p.splits + s]).x);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float lsum = 0.f;
        for (int s = lane; s < p.splits; s += 32) {
            const float2 ml = __ldcg(&p.ml_part[row * p.splits + s]);
            const float f = (ml.x == -INFINITY || ml.y <= 0.f) ? 0.f : fast_exp2((ml.x - m) * log2_unit);
            work[rr * p.splits + s] = f;
            lsum += ml.y * f;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
        __syncwarp();
        for (int s = lane; s < p.splits; s += 32) work[rr * p.splits + s] *= inv;
    }
    __syncthreads();
    for (int i = tid; i < nrows * D; i += DEC_THREADS) {
        const int rr = i / D, d = i % D;
        const int r = r_lo + rr;
        float o = 0.f;
        const float *src = p.o_part + ((qrow0 + r) * p.splits) * D + d;
        for (int s = 0; s < p.splits; ++s) o = fmaf(__ldcg(src + (int64_t)s * D), work[rr * p.splits + s], o);
        const int hq = hk * rep + r / p.L, lq = r % p.L;
        store_out(p.out, p.out_dtype, b * p.o_sb + hq * p.o_sh + lq * p.o_sl + d, o);
    }
}

// ---------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres);
        if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess) fn = (EncodeTiledFn)p;
        else (void)cudaGetLastError();
    });
    return fn;
}

bool make_map(CUtensorMap *map, const KVSource &s, int D, int64_t T, int Hkv, int B) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)T, (cuuint64_t)Hkv, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)s.st * 2, (cuuint64_t)(Hkv > 1 ? s.sh : s.st * T) * 2,
                                   (cuuint64_t)(B > 1 ? s.sb : (Hkv > 1 ? s.sh * Hkv : s.st * T)) * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)TILE_T, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = s.dtype == KVC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = fn(map, dt, 4, const_cast<void *>(s.data), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool source_fits(const KVSource &s, int D, int Hkv, int B) {
    if (s.kind != SRC_RAW || (s.dtype != KVC_BF16 && s.dtype != KVC_F16)) return false;
    if (((uintptr_t)s.data & 15) != 0) return false;
    auto ok = [](int64_t st) { return st > 0 && (st * 2) % 16 == 0; };
    if (!ok(s.st) || s.st < D) return false;
    if (Hkv > 1 && !ok(s.sh)) return false;
    if (B > 1 && !ok(s.sb)) return false;
    return true;
}

template <typename T, int D, int NSTAGE>
void launch_typed(const CUtensorMap &kmap, const CUtensorMap &vmap, const DecodeParams &p, int units,
                  cudaStream_t stream) {
    const size_t smem = (size_t)NSTAGE * 2 * (TILE_T * D * 2) + 2 * NSTAGE * sizeof(uint64_t) + 64 + 1024;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        KVC_CUDA(cudaFuncSetAttribute(attn_decode_kernel<T, D, NSTAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        KVC_CUDA(cudaFuncSetAttribute(attn_decode_kernel<T, D, NSTAGE>,
                                      cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured[dev] = true;
    }
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(attn_decode_kernel<T, D, NSTAGE>, dim3(units), dim3(DEC_THREADS), smem, stream, kmap, vmap, p));
    timer.stop();
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

template <typename T, int D, int NSTAGE, bool LIST, bool ROPE>
void launch_flat_typed(const std::conditional_t<LIST, FlatList, FlatSingle> &list, const DecodeParams &p, int ctas, size_t smem,
                       cudaStream_t stream) {
    static size_t configured[64] = {0};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && configured[dev] < smem) {
        KVC_CUDA(cudaFuncSetAttribute(attn_decode_flat_kernel<T, D, NSTAGE, LIST, ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        KVC_CUDA(cudaFuncSetAttribute(attn_decode_flat_kernel<T, D, NSTAGE, LIST, ROPE>,
                                      cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured[dev] = smem;
    }
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(attn_decode_flat_kernel<T, D, NSTAGE, LIST, ROPE>, dim3(ctas), dim3(DEC_THREADS), smem, stream, list, p));
    if constexpr (LIST) {
        const int elems = p.Hq / p.Hkv * D;
        KVC_CUDA(launch_pdl(flat_list_merge_kernel<T, D>, dim3(list.n * p.B * p.Hkv, (elems + 127) / 128), dim3(128), 0, stream, list, p));
        ++g_launch_count;
    }
    timer.stop();
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

template <typename T, int D, int NSTAGE, bool MASKED, bool PAIRS>
void launch_chunk_typed(const std::conditional_t<PAIRS, ChunkPairMaps, ChunkMaps> &maps, const DecodeParams &p, int ctas,
                        cudaStream_t stream) {
    const size_t smem = (size_t)NSTAGE * (PAIRS ? 4 : 2) * (TILE_T * D * 2) + (PAIRS ? 2 : D == 256 ? 1 : 0) * CONSUMER_WARPS * (D / 16) * 32 * 16 +
                        2 * NSTAGE * sizeof(uint64_t) + 64 + 1024;
    auto kernel = attn_chunk_kernel<T, D, NSTAGE, MASKED, PAIRS>;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured[dev] = true;
    }
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(kernel, dim3(ctas), dim3(DEC_THREADS), smem, stream, maps, p));
    timer.stop();
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

}  // namespace

// Whether launch_attention_chunk_pairs takes `a` (raw contiguous rows); the pointers are not judged beyond their
// alignment.
bool attention_chunk_rows_accepts(const AttnArgs &a) {
    if (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16) return false;
    if (a.D != 64 && a.D != 128 && a.D != 256) return false;
    if (a.k.dtype != a.q_dtype || a.v.dtype != a.q_dtype || a.q_signs || a.o_signs || a.q_calib) return false;
    if (a.Hkv <= 0 || a.Hq % a.Hkv || a.T < 1 || a.T > (int64_t)1 << 30) return false;
    const int64_t rows = (int64_t)(a.Hq / a.Hkv) * a.L;
    if ((a.mask.mode != KVC_MASK_ARRAY && rows <= 16) || rows > (int64_t)1 << 24) return false;
    if (!source_fits(a.k, a.D, a.Hkv, a.B) || !source_fits(a.v, a.D, a.Hkv, a.B)) return false;
    if (((uintptr_t)a.q & 3) || (a.q_sb & 1) || (a.q_sh & 1) || (a.q_sl & 1)) return false;
    return (int64_t)a.B * a.Hkv * ((rows + 63) / 64) * (int64_t)sizeof(int) <= COUNTER_BYTES && encode_tiled();
}

namespace {

// Shared memory of the flat kernel: ring, barriers, cross-warp buffers, two units' query rows.
constexpr int flat_stages(int D) { return D == 64 ? 6 : 3; }
constexpr size_t flat_smem(int D, int R) {
    const size_t ring = (size_t)flat_stages(D) * 2 * (TILE_T * D * 2);
    const size_t red = (size_t)CONSUMER_WARPS * R * (D + 8) * 4 + (size_t)CONSUMER_WARPS * R * 8 + 16 + 4 * sizeof(uint64_t) + (size_t)2 * R * D * 2;
    return ring + 2 * flat_stages(D) * sizeof(uint64_t) + 64 + red + 1024;
}
constexpr bool flat_fits_sm(int D, int R) { return flat_smem(D, R) <= (size_t)(D <= 128 ? 112 : 224) * 1024; }

// One wave of CTAs over `work` tiles, and the shared memory of the flat kernel for it.
struct FlatShape {
    int64_t ctas, per, rem, nslots;
    size_t smem;
    bool fits;
};
FlatShape flat_shape(int sms, int D, int R, int64_t work, int64_t most_tiles) {
    FlatShape f;
    f.ctas = std::min<int64_t>((int64_t)sms * (D <= 128 ? 2 : 1), work);
    f.per = work / f.ctas; f.rem = work % f.ctas;
    f.nslots = (most_tiles + f.per - 1) / f.per + 1;
    f.smem = flat_smem(D, R);
    f.fits = flat_fits_sm(D, R);
    return f;
}

// Shared memory of a list launch: ring, barriers, and FLAT_AHEAD segments' query rows and descriptors.
size_t flat_list_smem(int D, int R) {
    const int nstage = D == 64 ? 6 : 3;
    return (size_t)nstage * 2 * (TILE_T * D * 2) + 2 * nstage * sizeof(uint64_t) + 64 + FLAT_AHEAD * (2 * sizeof(uint64_t) + (size_t)R * D * 2 + sizeof(FlatWork)) + 1024;
}
constexpr int64_t LIST_PARTIAL_BYTES = (int64_t)32 << 20;   // of a list launch's partials

bool flat_new_rows_ok(const AttnArgs &a) {
    return a.L == 1 && a.mask.mode != KVC_MASK_CAUSAL && !((uintptr_t)a.new_k & 15) && !((uintptr_t)a.new_v & 15) &&
           (a.nk_sb * 2) % 16 == 0 && (a.nk_sh * 2) % 16 == 0 && (a.nv_sb * 2) % 16 == 0 && (a.nv_sh * 2) % 16 == 0;
}

bool flat_off() {
    static const bool off = [] {
        const char *e = std::getenv("KVC_DECODE_FLAT");
        return e && e[0] == '0';
    }();
    return off;
}

}  // namespace

// Whether one launch may turn, append and attend a step of `rows` query rows per KV head: what the flat kernel asks that
// does not depend on the context's length.
bool attention_decode_takes_rope(int D, int64_t rows, int64_t units) {
    return !flat_off() && rows <= 16 && units * (int64_t)sizeof(int) <= COUNTER_BYTES && flat_fits_sm(D, (int)rows);
}

// The single-token steps of up to KVC_LIST_MAX raw caches of one shape (new rows not yet stored, or all stored)
// in one launch. Returns launches made, 0 when they do not fit.
int launch_attention_decode_list(const AttnArgs *args, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX || flat_off()) return 0;
    const AttnArgs &a0 = args[0];
    if (a0.q_dtype != KVC_BF16 && a0.q_dtype != KVC_F16) return 0;
    if (a0.D != 64 && a0.D != 128 && a0.D != 256) return 0;
    if (a0.Hkv <= 0 || a0.Hq % a0.Hkv || a0.L != 1) return 0;
    const int R = a0.Hq / a0.Hkv;
    const int64_t units = (int64_t)a0.B * a0.Hkv;
    if (R > 16 || n * units * (int64_t)sizeof(int) > COUNTER_BYTES) return 0;
    static thread_local FlatList all, list;
    const int sms = sm_count(a0.device);
    const size_t smem = flat_list_smem(a0.D, R);
    bool q_bulk = true;
    for (int i = 0; i < n; ++i) {
        const AttnArgs &a = args[i];
        if (a.q_dtype != a0.q_dtype || a.k.dtype != a.q_dtype || a.v.dtype != a.q_dtype || a.D != a0.D || a.B != a0.B ||
            a.Hq != a0.Hq || a.Hkv != a0.Hkv || a.L != 1 || a.scale != a0.scale || a.mask.mode != KVC_MASK_NONE ||
            a.q_signs || a.o_signs || a.q_calib || a.q_rot || a.o_rot || a.device != a0.device)
            return 0;
        if (a.q_sh != a0.q_sh || a.q_sl != a0.q_sl || a.o_sh != a0.o_sh || a.o_sl != a0.o_sl) return 0;
        if (a.T < 1 || a.T > (int64_t)1 << 30 || (a.new_k != nullptr) != (a0.new_k != nullptr)) return 0;
        if (!source_fits(a.k, a.D, a.Hkv, a.B) || !source_fits(a.v, a.D, a.Hkv, a.B)) return 0;
        if (a.k.sb != a.v.sb || a.k.sh != a.v.sh || a.k.st != a.v.st) return 0;
        if (((uintptr_t)a.q & 3) || (a.q_sb & 1) || (a.q_sh & 1) || (a.q_sl & 1)) return 0;
        if (a.new_k && !flat_new_rows_ok(a)) return 0;
        FlatLayer &l = all.layer[i];
        if (!make_map(&l.kmap, a.k, a.D, a.T, a.Hkv, a.B) || !make_map(&l.vmap, a.v, a.D, a.T, a.Hkv, a.B)) return 0;
        l.q = a.q; l.out = a.out; l.q_sb = a.q_sb; l.o_sb = a.o_sb;
        l.k_base = (unsigned char *)a.k.data; l.v_base = (unsigned char *)a.v.data;
        l.kv_sb = a.k.sb * 2; l.kv_sh = a.k.sh * 2; l.kv_st = a.k.st * 2;
        l.new_k = a.new_k; l.new_v = a.new_v;
        l.new_slot = (a.new_slot >= 0 && a.new_slot < a.T) ? a.new_slot : a.T - 1;
        l.nk_sb = a.nk_sb; l.nk_sh = a.nk_sh; l.nv_sb = a.nv_sb; l.nv_sh = a.nv_sh;
        l.T = a.T;
        l.tiles = (int32_t)((a.T + TILE_T - 1) / TILE_T);
        const FlatShape own = flat_shape(sms, a.D, R, units * l.tiles, l.tiles);
        if (!own.fits) return 0;
        l.per = (int32_t)own.per; l.rem = (int32_t)own.rem;
        l.nslots = (int32_t)own.nslots;
        q_bulk = q_bulk && a.q_sh == a.D && ((uintptr_t)a.q & 15) == 0 && (a.q_sb * 2) % 16 == 0;
    }
    int *status = device_status_word(a0.device);
    if (!status) return 0;
    DecodeParams p = {};
    p.out_dtype = a0.q_dtype;
    p.q_sh = a0.q_sh; p.q_sl = a0.q_sl; p.o_sh = a0.o_sh; p.o_sl = a0.o_sl;
    p.status = status;
    p.B = a0.B; p.Hq = a0.Hq; p.Hkv = a0.Hkv; p.L = 1;
    p.splits = 1; p.row_blocks = 1;
    p.debug_skip = measure_skip_bits();
    p.scale_log2 = a0.scale * 1.4426950408889634f;
    p.flat.red_rows = R;   // the rest of the plan is each call's own
    p.q_bulk = q_bulk ? 1 : 0;
    // as many calls a launch as the partials have room for
    int launches = 0;
    for (int from = 0; from < n;) {
        int64_t ranges = 0, row_slots = 0;
        list.n = 0;
        for (; from < n; ++from) {
            FlatLayer l = all.layer[from];
            const int64_t rows = (int64_t)a0.B * a0.Hq * l.nslots;
            if (list.n && (row_slots + rows) * CONSUMER_WARPS * a0.D * (int64_t)sizeof(float) > LIST_PARTIAL_BYTES) break;
            l.first = (int32_t)ranges;
            l.part_first = row_slots;
            ranges += std::min<int64_t>((int64_t)sms * (a0.D <= 128 ? 2 : 1), units * l.tiles);
            row_slots += rows;
            list.layer[list.n++] = l;
        }
        list.ranges = (int32_t)ranges;
        const int ctas = (int)std::min<int64_t>(ranges, (int64_t)sms * (a0.D <= 128 ? 2 : 1));
        const size_t o_bytes = (size_t)row_slots * CONSUMER_WARPS * a0.D * sizeof(float);
        char *scratch = (char *)scratch_get(a0.device, o_bytes + (size_t)row_slots * CONSUMER_WARPS * sizeof(float2) + 256, stream);
        p.o_part = (float *)scratch;
        p.ml_part = (float2 *)(scratch + ((o_bytes + 255) / 256) * 256);
#define KVC_FLATL(TT, DD, NS) launch_flat_typed<TT, DD, NS, true, false>(list, p, ctas, smem, stream)
        if (a0.q_dtype == KVC_BF16) {
            if (a0.D == 64) KVC_FLATL(__nv_bfloat16, 64, 6);
            else if (a0.D == 128) KVC_FLATL(__nv_bfloat16, 128, 3);
            else KVC_FLATL(__nv_bfloat16, 256, 3);
        } else {
            if (a0.D == 64) KVC_FLATL(__half, 64, 6);
            else if (a0.D == 128) KVC_FLATL(__half, 128, 3);
            else KVC_FLATL(__half, 256, 3);
        }
#undef KVC_FLATL
        launches += 2;
    }
    g_last_chained_launch = g_launch_count;
    return launches;
}

namespace {


int launch_rows(const AttnArgs &a, const ChunkLow *low, cudaStream_t stream) {
    if (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16) return 0;
    if (a.D != 64 && a.D != 128 && a.D != 256) return 0;
    if (a.k.dtype != a.q_dtype || a.v.dtype != a.q_dtype) return 0;
    const bool masked = a.mask.mode == KVC_MASK_ARRAY;   // array masks: the row-split kernel, whatever the row count
    if (masked && a.new_k) return 0;
    if (a.q_signs || a.o_signs || a.q_calib) return 0;
    if (a.Hkv <= 0 || a.Hq % a.Hkv) return 0;
    const int rep = a.Hq / a.Hkv;
    if (a.T < 1 || a.T > (int64_t)1 << 30) return 0;
    if (!source_fits(a.k, a.D, a.Hkv, a.B) || !source_fits(a.v, a.D, a.Hkv, a.B)) return 0;
    if (((uintptr_t)a.q & 3) || (a.q_sb & 1) || (a.q_sh & 1) || (a.q_sl & 1)) return 0;
    const int64_t bh = (int64_t)a.B * a.Hkv;
    const bool chunk = masked || low || rep * a.L > 16;  // more rows than one MMA row block: rows split across warps
    const int64_t row_blocks = chunk ? ((int64_t)rep * a.L + 63) / 64 : 1;
    if (bh * row_blocks * (int64_t)sizeof(int) > COUNTER_BYTES) return 0;
    if (chunk && (int64_t)rep * a.L > (int64_t)1 << 24) return 0;

    CUtensorMap kmap, vmap;
    if (!make_map(&kmap, a.k, a.D, a.T, a.Hkv, a.B) || !make_map(&vmap, a.v, a.D, a.T, a.Hkv, a.B)) return 0;
    int *status = device_status_word(a.device);
    int *counters = counters_get(a.device, stream, COUNTER_BYTES);
    if (!status || !counters) return 0;

    const int64_t tiles = (a.T + TILE_T - 1) / TILE_T;
    const int slots = sm_count(a.device) * (a.D <= 128 ? 2 : 1);

    // Decode (one MMA row block): flat decomposition over one wave of CTAs when its cross-warp
    // buffer fits beside the ring; KVC_DECODE_FLAT=0 keeps the per-unit split kernel.
    if (!chunk) {
        const int R = rep * a.L;
        const FlatShape f = flat_shape(sm_count(a.device), a.D, R, bh * tiles, tiles);
        const int64_t ctas = f.ctas, per = f.per, rem = f.rem, nslots = f.nslots;
        const size_t smem = f.smem;
        if (!flat_off() && f.fits && (!a.new_k || flat_new_rows_ok(a))) {
            const int64_t qrows_f = (int64_t)a.B * a.Hq * a.L;
            const size_t o_bytes_f = (size_t)qrows_f * nslots * a.D * sizeof(float);
            const size_t ml_bytes_f = (size_t)qrows_f * nslots * sizeof(float2);
            char *scratch_f = (char *)scratch_get(a.device, o_bytes_f + ml_bytes_f + 256, stream);
            DecodeParams p = {};
            p.q = a.q; p.out = a.out; p.out_dtype = a.q_dtype;
            p.q_sb = a.q_sb; p.q_sh = a.q_sh; p.q_sl = a.q_sl;
            p.o_sb = a.o_sb; p.o_sh = a.o_sh; p.o_sl = a.o_sl;
            p.o_part = (float *)scratch_f;
            p.ml_part = (float2 *)(scratch_f + ((o_bytes_f + 255) / 256) * 256);
            p.counters = counters; p.status = status;
            p.B = a.B; p.Hq = a.Hq; p.Hkv = a.Hkv; p.L = a.L; p.T = a.T;
            p.splits = 1; p.tiles_base = 0; p.tiles_rem = 0; p.row_blocks = 1;
            p.causal = a.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
            p.debug_skip = measure_skip_bits();
            p.k_base = (unsigned char *)a.k.data; p.v_base = (unsigned char *)a.v.data;
            p.kv_sb = a.k.sb * 2; p.kv_sh = a.k.sh * 2; p.kv_st = a.k.st * 2;
            p.new_k = a.new_k; p.new_v = a.new_v;
            p.new_slot = (a.new_slot >= 0 && a.new_slot < a.T) ? a.new_slot : a.T - 1;
            {
                // early tiles: fused append only (the kernel's tiles end before the row it writes), the
                // caller's word on the preceding launch, and that launch being a kernel that released
                // this one only after its own wait. KVC_EARLY_TILES=0 turns it off.
                static const bool early_off = [] {
                    const char *e = std::getenv("KVC_EARLY_TILES");
                    return e && e[0] == '0';
                }();
                p.early_tiles = (!early_off && a.new_k && a.stored_rows_settled && g_last_chained_launch == g_launch_count &&
                                 KVC_SKIP_BITS(p) == 0) ? 1 : 0;
            }
            p.nk_sb = a.nk_sb; p.nk_sh = a.nk_sh; p.nv_sb = a.nv_sb; p.nv_sh = a.nv_sh;
            p.causal_offset = a.mask.causal_offset;
            p.scale_log2 = a.scale * 1.4426950408889634f;
            p.tiles_all = (int)tiles;
            p.flat.tiles = (int)tiles;
            p.flat.per = (int)per; p.flat.rem = (int)rem;
            p.flat.nslots = (int)nslots; p.flat.red_rows = R;
            p.q_bulk = (a.L == 1 && a.q_sh == a.D && ((uintptr_t)a.q & 15) == 0 && (a.q_sb * 2) % 16 == 0) ? 1 : 0;
            size_t bytes = smem;
            if (a.rope) {
                // the query rows have to come by the bulk copy, and the row and the table need room behind them
                if (!p.q_bulk || !a.new_k || a.rope->D != a.D || a.rope->dims > a.D) return 0;
                p.rope_pairs = a.rope->dims / 2;
                p.rope_traditional = a.rope->traditional;
                p.rope_log2 = a.rope->log2_base_over_half;
                p.rope_scale = a.rope->scale;
                p.rope_position = a.rope->offset;
                bytes += (size_t)a.D / 2 * sizeof(float2) + (size_t)a.D * 2;
            }
            FlatSingle maps;
            maps.kmap = kmap; maps.vmap = vmap;
#define KVC_FLAT(TT, DD, NS)                                                                                       \
    (a.rope ? launch_flat_typed<TT, DD, NS, false, true>(maps, p, (int)ctas, bytes, stream)                         \
            : launch_flat_typed<TT, DD, NS, false, false>(maps, p, (int)ctas, bytes, stream))
            if (a.q_dtype == KVC_BF16) {
                if (a.D == 64) KVC_FLAT(__nv_bfloat16, 64, 6);
                else if (a.D == 128) KVC_FLAT(__nv_bfloat16, 128, 3);
                else KVC_FLAT(__nv_bfloat16, 256, 3);
            } else {
                if (a.D == 64) KVC_FLAT(__half, 64, 6);
                else if (a.D == 128) KVC_FLAT(__half, 128, 3);
                else KVC_FLAT(__half, 256, 3);
            }
#undef KVC_FLAT
            g_last_chained_launch = g_launch_count;
            return 1;
        }
    }

    if (a.new_k) return 0;  // only the flat decode kernel appends by itself; the caller appends and comes back

    // Units per (batch, head): minimise waves x (tiles per unit + fixed cost), with
    // `slots` CTAs resident at once; ties go to fewer splits.
    int64_t best_s = 1;
    double best_cost = 1e30;
    const int64_t max_s = std::min<int64_t>(tiles, 64);
    for (int64_t s = 1; s <= max_s; ++s) {
        const int64_t units = bh * row_blocks * s;
        const int64_t waves = (units + slots - 1) / slots;
        const int64_t per = (tiles + s - 1) / s;
        const double cost = (double)waves * ((double)per + 2.5);
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best_s = s;
        }
    }
    const int64_t splits = best_s;

    const int64_t qrows = (int64_t)a.B * a.Hq * a.L;
    const size_t o_bytes = (size_t)qrows * splits * a.D * sizeof(float);
    const size_t ml_bytes = (size_t)qrows * splits * sizeof(float2);
    char *scratch = (char *)scratch_get(a.device, o_bytes + ml_bytes + 256, stream);
    float *o_part = (float *)scratch;
    float2 *ml_part = (float2 *)(scratch + ((o_bytes + 255) / 256) * 256);

    DecodeParams p = {};
    p.q = a.q; p.out = a.out; p.out_dtype = a.q_dtype;
    p.q_sb = a.q_sb; p.q_sh = a.q_sh; p.q_sl = a.q_sl;
    p.o_sb = a.o_sb; p.o_sh = a.o_sh; p.o_sl = a.o_sl;
    p.o_part = o_part; p.ml_part = ml_part; p.counters = counters; p.status = status;
    p.B = a.B; p.Hq = a.Hq; p.Hkv = a.Hkv; p.L = a.L; p.T = a.T;
    p.splits = (int)splits;
    p.tiles_base = (int)(tiles / splits);
    p.tiles_rem = (int)(tiles % splits);
    p.causal = a.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
    p.debug_skip = measure_skip_bits();
    p.causal_offset = a.mask.causal_offset;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.row_blocks = (int)row_blocks;
    p.tiles_all = (int)tiles;
    p.mask = a.mask;
    if (low) {
        p.out_dtype = low->out_dtype;
        p.q_low = low->q;
        p.k_low = low->k ? 1 : 0;
        p.q_undo = low->q_undo; p.k_undo = low->k_undo; p.v_undo = low->v_undo;
    }
    const int units = (int)(bh * splits);

    if (chunk) {
        const int ctas = (int)(bh * row_blocks * splits);
        if (trace_dispatch())
            fprintf(stderr, "[kvc] chunk_mma: %lld row blocks in %lld splits%s%s\n", (long long)(bh * row_blocks), (long long)splits,
                    masked ? ", array mask" : "", low ? ", pairs" : "");
        if (low) {
            ChunkPairMaps pm;
            KVSource kl = a.k, vl = a.v;
            kl.data = low->k ? low->k : a.k.data;
            vl.data = low->v;
            if (!source_fits(kl, a.D, a.Hkv, a.B) || !source_fits(vl, a.D, a.Hkv, a.B) || !make_map(&pm.k_low, kl, a.D, a.T, a.Hkv, a.B) ||
                !make_map(&pm.v_low, vl, a.D, a.T, a.Hkv, a.B))
                return 0;
            pm.k = kmap; pm.v = vmap;
            // stages: two CTAs an SM up to D 128 (four 8 / 16 KB tiles a stage beside 16 / 32 KB of query fragments)
#define KVC_CHP(TT, DD, NS)                                                               \
    (masked ? launch_chunk_typed<TT, DD, NS, true, true>(pm, p, ctas, stream)             \
            : launch_chunk_typed<TT, DD, NS, false, true>(pm, p, ctas, stream))
            if (a.q_dtype == KVC_BF16) {
                if (a.D == 64) KVC_CHP(__nv_bfloat16, 64, 2);
                else if (a.D == 128) KVC_CHP(__nv_bfloat16, 128, 1);
                else KVC_CHP(__nv_bfloat16, 256, 1);
            } else {
                if (a.D == 64) KVC_CHP(__half, 64, 2);
                else if (a.D == 128) KVC_CHP(__half, 128, 1);
                else KVC_CHP(__half, 256, 1);
            }
#undef KVC_CHP
            return 1;
        }
        ChunkMaps maps;
        maps.k = kmap; maps.v = vmap;
#define KVC_CHK(TT, DD, NS)                                                                  \
    (masked ? launch_chunk_typed<TT, DD, NS, true, false>(maps, p, ctas, stream)             \
            : launch_chunk_typed<TT, DD, NS, false, false>(maps, p, ctas, stream))
        if (a.q_dtype == KVC_BF16) {
            if (a.D == 64) KVC_CHK(__nv_bfloat16, 64, 6);
            else if (a.D == 128) KVC_CHK(__nv_bfloat16, 128, 3);
            else KVC_CHK(__nv_bfloat16, 256, 3);
        } else {
            if (a.D == 64) KVC_CHK(__half, 64, 6);
            else if (a.D == 128) KVC_CHK(__half, 128, 3);
            else KVC_CHK(__half, 256, 3);
        }
#undef KVC_CHK
        return 1;
    }

#define KVC_DEC(TT, DD, NS) launch_typed<TT, DD, NS>(kmap, vmap, p, units, stream)
    if (a.q_dtype == KVC_BF16) {
        if (a.D == 64) KVC_DEC(__nv_bfloat16, 64, 6);
        else if (a.D == 128) KVC_DEC(__nv_bfloat16, 128, 3);
        else KVC_DEC(__nv_bfloat16, 256, 3);
    } else {
        if (a.D == 64) KVC_DEC(__half, 64, 6);
        else if (a.D == 128) KVC_DEC(__half, 128, 3);
        else KVC_DEC(__half, 256, 3);
    }
#undef KVC_DEC
    return 1;
}

}  // namespace

// Returns the number of kernels launched, or 0 when the call does not fit this path.
int launch_attention_decode(const AttnArgs &a, cudaStream_t stream) { return launch_rows(a, nullptr, stream); }

// A chunk over 16-bit rows that are the high halves of exact ones (attention_chunk_rows_accepts has been asked).
int launch_attention_chunk_pairs(const AttnArgs &a, const ChunkLow &low, cudaStream_t stream) { return launch_rows(a, &low, stream); }

}  // namespace kvc
