// Decode attention over affine-quantised caches of single-precision callers (4- / 8-bit codes, f32 scales and
// biases), head dims 64 / 128 / 256, up to eight query rows per unit, one call or a list of calls of one shape.
//
// Everything is fp32 (the codes become scale * code + bias before they are multiplied), two dims an instruction
// (f32x2.cuh). A unit holds two, four or eight rows, as many as the group has: rows that are not there cost as much as
// those that are (2 layers x 3 sequences x 7 876 tokens, 16/8 heads, D 128, 4 bits: 55 us with four rows and single
// products, 43 with two). What bounds small shapes (a few MB of codes per step) is latency. Split as in
// attn_stream.cuh: a warp walks 16-token blocks on its own, with a private two-stage ring filled by 16-byte cp.async copies; no barrier before a segment's end.
//   * scores: lane = (token, half of the head dims); a lane reads its row's chunks (swizzled by the token) and the
//     query rows as broadcasts, the two halves meet in one shuffle.
//   * values: lane = D / 32 neighbouring dims; probabilities are read back as broadcasts.
// Work is cut into ranges of 64-token tiles (plan_units), partials merged by segment_epilogue.
// Before (general kernel + merge kernel): 34 us per layer of the Llama-3.2-1B shape at 1024 tokens.
#include "attn_stream.cuh"
#include "f32x2.cuh"

namespace kvc {

namespace {

using namespace stream;

constexpr int ST_WARPS = 8;
constexpr int ST_THREADS = ST_WARPS * 32;

struct F32Seq {
    const float *q;
    float *out;
    StreamSource k, v;
    int64_t q_sb, o_sb, tile_first;
    int64_t causal_offset;
    int32_t T, tiles;
};
struct F32List {
    int32_t n;
    F32Seq seq[KVC_LIST_MAX];
};
struct F32Params {
    int64_t q_sh, q_sl, o_sh, o_sl;
    float *o_part;
    float2 *ml_part;
    int *counters;
    UnitPlan flat;
    int32_t B, Hq, Hkv, L, chunks, groups, causal;
    float scale_log2;
};

template <int D, int BITS>
struct F32Shape {
    static constexpr int RB = D * BITS / 8, CH = RB / 16;         // bytes and 16-byte chunks per row
    static constexpr int BLOCK = 16 * RB, SIDE = 16 * (D / 32) * 4;
    static constexpr int STAGE = 2 * (BLOCK + 2 * SIDE);
    static constexpr int PROB = 16 * 8 * 4;
    static constexpr int WARP_BYTES = ST_STAGES * STAGE + PROB;
    static constexpr int RED = ST_WARPS * 8 * (D + 4 + 2) * 4;
    static constexpr int RING = ST_WARPS * WARP_BYTES;
    static constexpr int BODY = RING > RED ? RING : RED;
    static constexpr int QROW = D + 8;                            // the second half of a row starts 4 floats late
    static constexpr int SMEM = BODY + 8 * QROW * 4 + 64;
};

template <int CH> __device__ __forceinline__ int row_xor(int tok) {
    return CH >= 8 ? tok & 7 : CH == 4 ? (tok >> 1) & 3 : CH == 2 ? (tok >> 2) & 1 : 0;
}

// Codes k and k + 1 (k even) of a word under a group's scale and bias. A 4-bit code stays where it lies in its half word, so
// it is its integer times 16^(k % 4), of which the scale is rid by a power of two: the products are those of the integers.
template <int BITS> struct GroupScale {
    uint64_t s[BITS == 4 ? 2 : 1], bias;
    __device__ __forceinline__ GroupScale(float scale, float b) {
        if (BITS == 4) {
            s[0] = pack_f2(scale, scale * 0.0625f);
            s[BITS == 4 ? 1 : 0] = pack_f2(scale * 0.00390625f, scale * 0.000244140625f);
        } else {
            s[0] = pack_f2(scale, scale);
        }
        bias = pack_f2(b, b);
    }
    __device__ __forceinline__ uint64_t pair(uint32_t w, int k) const {
        uint32_t a, b;
        if (BITS == 8) {
            a = __byte_perm(w, 0x4B000000u, 0x7440 + k);
            b = __byte_perm(w, 0x4B000000u, 0x7441 + k);
        } else {
            const uint32_t h = k >= 4 ? w >> 16 : w;
            a = (h & (15u << (4 * (k & 3)))) | 0x4B000000u;
            b = (h & (15u << (4 * (k & 3) + 4))) | 0x4B000000u;
        }
        const uint64_t code = add_f2(pack_f2(__uint_as_float(a), __uint_as_float(b)), pack_f2(-8388608.f, -8388608.f));
        return fma_f2(s[BITS == 4 ? (k >> 1) & 1 : 0], code, bias);
    }
};

__device__ __forceinline__ float lds_f32(uint32_t a) { return __uint_as_float(lds32(a)); }
__device__ __forceinline__ void lds_f2x2(uint32_t a, uint64_t &x, uint64_t &y) {
    asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(x), "=l"(y) : "r"(a) : "memory");
}

// RN: query rows a unit carries (2, 4 or 8).
template <int D, int BITS, int RN>
__global__ void __launch_bounds__(ST_THREADS, D <= 128 ? 2 : 1)
attn_f32_kernel(const __grid_constant__ F32Params p, const __grid_constant__ F32List list) {
    using SH = F32Shape<D, BITS>;
    constexpr int CH = SH::CH, E = D / 32, HALF = D / 2;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int *flag = (int *)smem;
    float *qs = (float *)(smem + 64);
    unsigned char *body = smem + 64 + 8 * SH::QROW * 4;
    const uint32_t q0 = smem_u32(qs), ring = smem_u32(body) + warp * SH::WARP_BYTES, prob = ring + ST_STAGES * SH::STAGE;
    pdl_wait();
    pdl_trigger();

    const UnitPlan fp = p.flat;
    const int rep = p.Hq / p.Hkv, rows_all = rep * p.L, side = 4 * p.groups;   // scale bytes per token
    int64_t x = flat_lo(fp, blockIdx.x);
    const int64_t x_end = flat_lo(fp, blockIdx.x + 1);
    int si = 0;
    while (x < x_end) {
        while (si + 1 < list.n && list.seq[si + 1].tile_first <= x) ++si;
        const F32Seq &sq = list.seq[si];
        const int64_t in = x - sq.tile_first;
        const int u_in = flat_div(in, sq.tiles), tile = flat_mod(in, sq.tiles, u_in);
        const int chunk = u_in % p.chunks, hk = (u_in / p.chunks) % p.Hkv, b = u_in / p.chunks / p.Hkv;
        const int tiles = (int)min((int64_t)(sq.tiles - tile), x_end - x);
        const int row0 = chunk * RN, R = min(RN, rows_all - row0), T = sq.T;
        const int t_lo = tile * ST_TILE, t_hi = min(T, (tile + tiles) * ST_TILE), nblk = (t_hi - t_lo + 15) / 16;
        const char *src[6] = {(const char *)sq.k.data + b * sq.k.sb + hk * sq.k.sh, (const char *)sq.v.data + b * sq.v.sb + hk * sq.v.sh,
                              (const char *)sq.k.scales + b * sq.k.gsb + hk * sq.k.gsh, (const char *)sq.k.biases + b * sq.k.gsb + hk * sq.k.gsh,
                              (const char *)sq.v.scales + b * sq.v.gsb + hk * sq.v.gsh, (const char *)sq.v.biases + b * sq.v.gsb + hk * sq.v.gsh};
        // stage: K block | V block | K scales | K biases | V scales | V biases; tokens past the end become zero
        auto fetch = [&](int blk, int st) {
            const int t = t_lo + blk * 16, live = min(16, T - t);
            const uint32_t dst = ring + st * SH::STAGE;
#pragma unroll
            for (int w = 0; w < 2; ++w)
#pragma unroll
                for (int r = 0; r < (SH::BLOCK / 16 + 31) / 32; ++r) {
                    const int i = lane + 32 * r;
                    if (i >= SH::BLOCK / 16) break;
                    const int tok = i / CH, ch = i % CH, n = tok < live ? 16 : 0;
                    cp_async16(dst + w * SH::BLOCK + ((tok * CH + (ch ^ row_xor<CH>(tok))) << 4),
                               src[w] + (n ? (int64_t)t * SH::RB + i * 16 : 0), n);
                }
#pragma unroll
            for (int w = 0; w < 4; ++w)
                for (int i = lane; i < side; i += 32) {          // 16 tokens * side bytes = `side` chunks
                    const int n = min(16, max(0, live * side - i * 16));
                    cp_async16(dst + 2 * SH::BLOCK + w * SH::SIDE + i * 16, src[2 + w] + (n ? (int64_t)t * side + i * 16 : 0), n);
                }
        };
        if (warp < nblk) fetch(warp, 0);
        cp_commit();
        for (int i = tid; i < RN * D; i += ST_THREADS) {
            const int r = i / D, d = i % D;
            float v = 0.f;
            if (r < R) {
                int h, l;
                split_row(row0 + r, p.L, h, l);
                v = sq.q[b * sq.q_sb + (hk * rep + h) * p.q_sh + l * p.q_sl + d];
            }
            qs[r * SH::QROW + d + (d >= HALF ? 4 : 0)] = v;
        }
        __syncthreads();

        const int tok = lane & 15, half = lane >> 4;
        float m_run[RN], l_run[RN];
        uint64_t acc[RN][E / 2];
        int lim[RN];
#pragma unroll
        for (int r = 0; r < RN; ++r) {
            m_run[r] = ST_NONE;
            l_run[r] = 0.f;
            lim[r] = T - 1;
            if (p.causal && row0 + r < rows_all) lim[r] = (int)min((int64_t)(T - 1), sq.causal_offset + (row0 + r) % p.L);
#pragma unroll
            for (int e = 0; e < E / 2; ++e) acc[r][e] = 0;
        }
        int stage = 0;
        for (int blk = warp; blk < nblk; blk += ST_WARPS) {
            if (blk + ST_WARPS < nblk) fetch(blk + ST_WARPS, stage ^ 1);
            cp_commit();
            cp_wait<1>();
            __syncwarp();
            const uint32_t st = ring + stage * SH::STAGE, sides = st + 2 * SH::BLOCK;
            const int t0 = t_lo + blk * 16;

            uint64_t dot[RN];                                      // even and odd dims
#pragma unroll
            for (int r = 0; r < RN; ++r) dot[r] = 0;
            constexpr int PER = 128 / BITS, CPW = 32 / BITS;       // dims per chunk, per word
#pragma unroll
            for (int j = 0; j < CH / 2; ++j) {
                const int ch = half * (CH / 2) + j;
                const uint4 w4 = lds128(st + ((tok * CH + (ch ^ row_xor<CH>(tok))) << 4));
                const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
                const int gr = ch * PER * p.groups / D;
                const GroupScale<BITS> gs(lds_f32(sides + (tok * p.groups + gr) * 4), lds_f32(sides + SH::SIDE + (tok * p.groups + gr) * 4));
#pragma unroll
                for (int i = 0; i < PER; i += 4) {
                    const uint64_t k0 = gs.pair(w[i / CPW], i % CPW), k1 = gs.pair(w[i / CPW], i % CPW + 2);
#pragma unroll
                    for (int r = 0; r < RN; ++r) {
                        uint64_t q01, q23;
                        lds_f2x2(q0 + (r * SH::QROW + half * (HALF + 4) + j * PER + i) * 4, q01, q23);
                        dot[r] = fma_f2(q23, k1, fma_f2(q01, k0, dot[r]));
                    }
                }
            }
            float s[RN];
#pragma unroll
            for (int r = 0; r < RN; ++r) {
                float even, odd;
                unpack_f2(dot[r], even, odd);
                s[r] = even + odd;
            }
            bool moved = false;
#pragma unroll
            for (int r = 0; r < RN; ++r) {
                s[r] = (s[r] + __shfl_xor_sync(0xffffffffu, s[r], 16)) * p.scale_log2;
                if (t0 + tok > lim[r]) s[r] = -INFINITY;
                moved |= s[r] > m_run[r] + ST_LAZY;
            }
            if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                for (int r = 0; r < RN; ++r) {
                    float mx = s[r];
#pragma unroll
                    for (int o = 8; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    mx = fmaxf(mx, m_run[r]);
                    const float alpha = exp2f(m_run[r] - mx);
                    m_run[r] = mx;
                    l_run[r] *= alpha;
#pragma unroll
                    for (int e = 0; e < E / 2; ++e) acc[r][e] = mul_f2(acc[r][e], pack_f2(alpha, alpha));
                }
            }
#pragma unroll
            for (int r = 0; r < RN; ++r) {
                s[r] = exp2f(s[r] - m_run[r]);
                if (half == 0) l_run[r] += s[r];
            }
            if (half == 0) {
                if constexpr (RN == 2) {
                    sts64(prob + tok * 8, make_uint2(__float_as_uint(s[0]), __float_as_uint(s[1])));
                } else {
#pragma unroll
                    for (int r = 0; r < RN; r += 4)
                        sts128(prob + (tok * RN + r) * 4, make_uint4(__float_as_uint(s[r]), __float_as_uint(s[r + 1]),
                                                                     __float_as_uint(s[r + 2]), __float_as_uint(s[r + 3])));
                }
            }
            __syncwarp();
            // ---- values: this lane's E dims of every token ----
            const int off = lane * E * BITS / 8, ch = off >> 4, gr = lane * E * p.groups / D;
            const uint32_t vst = st + SH::BLOCK;
#pragma unroll 4
            for (int t = 0; t < 16; ++t) {
                const uint32_t ad = vst + t * SH::RB + (((ch ^ row_xor<CH>(t)) << 4) | (off & 12));
                uint32_t w[(E * BITS + 31) / 32];
                if constexpr (E * BITS == 64) { const uint2 v = lds64(ad); w[0] = v.x; w[1] = v.y; }
                else w[0] = lds32(ad) >> ((off & 3) * 8);
                const GroupScale<BITS> gs(lds_f32(sides + 2 * SH::SIDE + (t * p.groups + gr) * 4), lds_f32(sides + 3 * SH::SIDE + (t * p.groups + gr) * 4));
                float pr[RN];
                if constexpr (RN == 2) {
                    const uint2 v = lds64(prob + t * 8);
                    pr[0] = __uint_as_float(v.x); pr[1] = __uint_as_float(v.y);
                } else {
#pragma unroll
                    for (int r = 0; r < RN; r += 4) {
                        const uint4 v = lds128(prob + (t * RN + r) * 4);
                        pr[r] = __uint_as_float(v.x); pr[r + 1] = __uint_as_float(v.y);
                        pr[r + 2] = __uint_as_float(v.z); pr[r + 3] = __uint_as_float(v.w);
                    }
                }
#pragma unroll
                for (int e = 0; e < E / 2; ++e) {
                    const uint64_t v = gs.pair(w[2 * e * BITS / 32], 2 * e % (32 / BITS));
#pragma unroll
                    for (int r = 0; r < RN; ++r) acc[r][e] = fma_f2(pack_f2(pr[r], pr[r]), v, acc[r][e]);
                }
            }
            __syncwarp();   // this stage and the probabilities may be overwritten
            stage ^= 1;
        }
        cp_wait<0>();

        const int rr_n = fp.red_rows;
        float *red_o = (float *)body;
        float *red_ml = red_o + ST_WARPS * rr_n * (D + 4);
        __syncthreads();        // every warp has left the ring that the merge buffers overlay
#pragma unroll
        for (int r = 0; r < RN; ++r) {
            float l = l_run[r];
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (r < R) {
#pragma unroll
                for (int e = 0; e < E / 2; ++e) *(uint64_t *)&red_o[(warp * rr_n + r) * (D + 4) + lane * E + 2 * e] = acc[r][e];
                if (lane == 0) {
                    red_ml[(warp * rr_n + r) * 2] = l > 0.f ? m_run[r] : -INFINITY;
                    red_ml[(warp * rr_n + r) * 2 + 1] = l;
                }
            }
        }
        UnitOut uo;
        uo.o_part = p.o_part; uo.ml_part = p.ml_part; uo.counters = p.counters;
        uo.out = sq.out - (int64_t)si * p.B * sq.o_sb;
        uo.out_dtype = KVC_F32;
        uo.o_sb = sq.o_sb; uo.o_sh = p.o_sh; uo.o_sl = p.o_sl;
        uo.o_signs = nullptr;
        uo.splits = 0; uo.Hq = p.Hq; uo.L = p.L;
        segment_epilogue<D, ST_WARPS>(uo, fp, red_o, red_ml, D + 4, nullptr, flag, si * p.B * p.Hkv * p.chunks + u_in, si * p.B + b, hk,
                                      rep, R, x - tile, sq.tiles, row0, min(ST_WARPS, nblk));
        x += tiles;
    }
}

template <int D, int BITS, int RN>
void launch_f32_typed(const F32Params &p, const F32List &list, int ctas, cudaStream_t stream) {
    auto kernel = attn_f32_kernel<D, BITS, RN>;
    const size_t smem = F32Shape<D, BITS>::SMEM;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured[dev] = true;
    }
    KernelTimer timer(stream);
    KVC_CUDA(launch_pdl(kernel, dim3(ctas), dim3(ST_THREADS), smem, stream, p, list));
    timer.stop();
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

bool f32_source(const KVSource &s, int D) {
    if (s.kind != SRC_AFFINE || s.dtype != KVC_F32 || (s.bits != 4 && s.bits != 8)) return false;
    if (s.group != 32 && s.group != 64 && s.group != 128) return false;
    if (D % s.group || s.gst != D / s.group || s.st != (int64_t)D * s.bits / 32) return false;
    for (const void *q : {s.data, s.scales, s.biases})
        if (!q || ((uintptr_t)q & 15)) return false;
    return !((s.sb * 4) & 15) && !((s.sh * 4) & 15) && !((s.gsb * 4) & 15) && !((s.gsh * 4) & 15);
}

bool f32_call(const AttnArgs &a) {
    if (a.q_dtype != KVC_F32 || (a.D != 64 && a.D != 128 && a.D != 256)) return false;
    if (a.mask.mode == KVC_MASK_ARRAY || a.q_signs || a.o_signs || a.q_rot || a.o_rot || a.q_calib || a.new_k) return false;
    if (a.Hkv <= 0 || a.Hq % a.Hkv || a.B < 1 || a.L < 1 || a.T < 1 || a.T > (int64_t)1 << 30) return false;
    if ((int64_t)(a.Hq / a.Hkv) * a.L > 64) return false;
    if (!f32_source(a.k, a.D) || !f32_source(a.v, a.D)) return false;
    return a.k.bits == a.v.bits && a.k.group == a.v.group;
}

StreamSource f32_stream_source(const KVSource &s) {
    StreamSource o;
    o.data = s.data; o.scales = s.scales; o.biases = s.biases;
    o.sb = s.sb * 4; o.sh = s.sh * 4; o.gsb = s.gsb * 4; o.gsh = s.gsh * 4;
    return o;
}

}  // namespace

// Up to KVC_LIST_MAX calls of one shape over f32 affine caches in one launch; 0 when they do not fit.
int launch_attention_f32_list(const AttnArgs *args, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX || !f32_call(args[0])) return 0;
    const AttnArgs &a0 = args[0];
    const int rows = a0.Hq / a0.Hkv * a0.L, rn = rows <= 2 ? 2 : rows <= 4 ? 4 : 8;
    F32Params p = {};
    p.chunks = (rows + rn - 1) / rn;
    const int64_t units = (int64_t)a0.B * a0.Hkv * p.chunks;
    static thread_local F32List list;
    list.n = n;
    int64_t work = 0, most = 0;
    for (int i = 0; i < n; ++i) {
        const AttnArgs &a = args[i];
        if (!f32_call(a) || a.B != a0.B || a.Hq != a0.Hq || a.Hkv != a0.Hkv || a.L != a0.L || a.D != a0.D || a.scale != a0.scale ||
            a.mask.mode != a0.mask.mode || a.k.bits != a0.k.bits || a.k.group != a0.k.group || a.q_sh != a0.q_sh ||
            a.q_sl != a0.q_sl || a.o_sh != a0.o_sh || a.o_sl != a0.o_sl || a.device != a0.device)
            return 0;
        F32Seq &sq = list.seq[i];
        sq.q = (const float *)a.q; sq.out = (float *)a.out;
        sq.k = f32_stream_source(a.k); sq.v = f32_stream_source(a.v);
        sq.q_sb = a.q_sb; sq.o_sb = a.o_sb;
        sq.T = (int32_t)a.T;
        sq.tiles = (sq.T + ST_TILE - 1) / ST_TILE;
        sq.tile_first = work;
        sq.causal_offset = a.mask.causal_offset;
        work += units * sq.tiles;
        most = std::max<int64_t>(most, sq.tiles);
    }
    StreamParams plan = {};
    int ctas;
    if (!stream_plan(a0, n * units, work, most, a0.D <= 128 ? 2 : 1, std::min(rows, rn), &plan, (int64_t)n * a0.B * a0.Hq * a0.L, stream, &ctas))
        return 0;
    p.flat = plan.flat;
    stream_list_tiles(list.seq, n, units, p.flat);
    p.o_part = plan.o_part; p.ml_part = plan.ml_part; p.counters = plan.counters;
    p.q_sh = a0.q_sh; p.q_sl = a0.q_sl; p.o_sh = a0.o_sh; p.o_sl = a0.o_sl;
    p.B = a0.B; p.Hq = a0.Hq; p.Hkv = a0.Hkv; p.L = a0.L;
    p.groups = a0.D / a0.k.group;
    p.causal = a0.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
    p.scale_log2 = a0.scale * 1.4426950408889634f;
#define KVC_F32K(DD, BB)                                                    \
    if (a0.D == DD && a0.k.bits == BB) {                                    \
        if (rn == 2) launch_f32_typed<DD, BB, 2>(p, list, ctas, stream);    \
        else if (rn == 4) launch_f32_typed<DD, BB, 4>(p, list, ctas, stream);    \
        else launch_f32_typed<DD, BB, 8>(p, list, ctas, stream);            \
        return 1;                                                           \
    }
    KVC_F32K(64, 4) KVC_F32K(64, 8) KVC_F32K(128, 4) KVC_F32K(128, 8) KVC_F32K(256, 4) KVC_F32K(256, 8)
#undef KVC_F32K
    return 0;
}

}  // namespace kvc
