// Prefill chunks over packed caches that no specialised kernel takes: mixed representations (raw or affine keys with
// index values, index keys with affine values), head dim 256, array masks over any packed cache, and short chunks at
// head dim 64.
//
// These calls are contractions of 4 * rows * keys * D flops and ran in fp32 on the general kernel (about 5 TFLOP/s).
// Here the rows are decoded once in fp32 and written as PAIRS of f16 arrays, the rounding and what it leaves; rotated
// queries likewise; the row-split mma.sync kernel multiplies pairs (attn_chunk_kernel, PAIRS) and, for index values,
// leaves fp32 rows that one more launch rotates back. Decoded rows are brought up against the f16 range by a power of two
// per (batch, KV head), taken from the largest finite element its scales and biases or norms allow (one small launch),
// query rows by one of their own: 22 significant bits on both sides of every product, whatever the size of the data, and
// nothing clips. Raw keys and queries that need no rotation are exact in 16 bits and are used where they are.
// Sixteen bits (pairs of bf16, which need no scaling) were not enough for f16 callers: with outlier channels in the keys
// the error against 64-bit sums rose by 0.4 .. 1.1 % over that of the general kernel.
//
// What bounds it: the tensor pipe at up to six MMAs per 16-bit one. Decoding moves B*Hkv*T*D*8 + B*Hq*L*D*8 bytes, a tenth
// of the time. The rows come from the stream-ordered pool (the row-split kernel's partials own the scratch arena).
#include "attn_common.cuh"

#include <algorithm>
#include <cstdio>

namespace kvc {

// attn_decode.cu
bool attention_chunk_rows_accepts(const AttnArgs &a);
int launch_attention_chunk_pairs(const AttnArgs &a, const ChunkLow &low, cudaStream_t stream);

namespace {

using namespace dev;

constexpr size_t PAIR_SCRATCH_LIMIT = (size_t)3 << 30;   // bytes per slice of the batch

struct PairSource {
    int32_t kind, group, bits;
    const void *data;             // raw rows or packed words
    const void *scales, *biases;  // affine: [B, H, cap, D / group]
    const float *norms;           // turbo: [B, H, cap]
    int64_t sb, sh, st, gsb, gsh, gst;
    float codebook[16];
};
struct PairRows {
    PairSource s[2];              // keys, values
    __half *high[2], *low[2];     // raw rows: copied to high as they are
    uint32_t *top;                // [2][B][H]: the largest magnitude (float bits) a decoded row may hold
    float *undo;                  // [2][B][H]: what a scaled row is multiplied by to have its size back
    int32_t B, H, D, first;       // first: 1 = values only
    int64_t T;
};

// The power of two that brings magnitudes up to `top` below 2^15, and its inverse.
__device__ __forceinline__ float pair_up(uint32_t top, float *undo) {
    const int e = max((int)(top >> 23) - 127, -100);      // top < 2^(e + 1)
    *undo = __uint_as_float((uint32_t)(127 + e - 14) << 23);
    return top ? __uint_as_float((uint32_t)(127 + 14 - e) << 23) : (*undo = 1.f);
}
// Non-finite values keep to themselves: their low half is zero.
__device__ __forceinline__ float pair_rest(float x, float high) { return fabsf(high) <= 65504.f ? x - high : 0.f; }

__device__ __forceinline__ void store_pair(__half *high, __half *low, const float (&x)[8]) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        h[j] = pack_h2(x[2 * j], x[2 * j + 1]);
        const float2 f = MmaType<__half>::unpack(h[j]);
        l[j] = pack_h2(pair_rest(x[2 * j], f.x), pair_rest(x[2 * j + 1], f.y));
    }
    *(uint4 *)high = make_uint4(h[0], h[1], h[2], h[3]);
    *(uint4 *)low = make_uint4(l[0], l[1], l[2], l[3]);
}

// The largest finite magnitude the decoded rows of a (batch, KV head) can hold; z as in pair_rows_kernel.
template <typename T>
__global__ void __launch_bounds__(256) pair_top_kernel(const __grid_constant__ PairRows p) {
    const int per = 2 - p.first, which = p.first + blockIdx.z % per, b = blockIdx.z / per, h = blockIdx.y;
    const PairSource &s = p.s[which];
    if (s.kind == SRC_RAW) return;
    uint32_t top = 0;
    auto take = [&](float x) {
        const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
        if (u < 0x7f800000u) top = max(top, u);
    };
    const int groups = s.kind == SRC_AFFINE ? p.D / s.group : 1;
    float big = 0.f;
    if (s.kind == SRC_TURBO)
        for (int i = 0; i < (1 << s.bits); ++i) big = fmaxf(big, fabsf(s.codebook[i]));
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.T * groups; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t gi = b * s.gsb + h * s.gsh + i / groups * s.gst + i % groups;
        if (s.kind == SRC_TURBO) {
            take(s.norms[gi] * big);
        } else {
            const float sc = to_f32<T>(((const T *)s.scales)[gi]), bi = to_f32<T>(((const T *)s.biases)[gi]);
            take(bi);
            take(fmaf(sc, (float)((1 << s.bits) - 1), bi));
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&p.top[((int64_t)which * p.B + b) * p.H + h], top);
}

// One thread = eight consecutive head dims of one token of K or V. T: type of scales and biases.
template <typename T>
__global__ void __launch_bounds__(256) pair_rows_kernel(const __grid_constant__ PairRows p) {
    const int per = 2 - p.first, which = p.first + blockIdx.z % per, b = blockIdx.z / per, h = blockIdx.y;
    const PairSource &s = p.s[which];
    const int per_row = p.D / 8;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.T * per_row) return;
    const int64_t t = i / per_row, at = b * s.sb + h * s.sh + t * s.st;
    const int d0 = (int)(i % per_row) * 8;
    const int64_t o = (((int64_t)b * p.H + h) * p.T + t) * p.D + d0;
    if (s.kind == SRC_RAW) {
        const uint16_t *e = (const uint16_t *)s.data + at + d0;
        uint16_t *dst = (uint16_t *)p.high[which] + o;
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = e[j];
        return;
    }
    const int64_t head = ((int64_t)which * p.B + b) * p.H + h;
    float undo, x[8];
    const float up = pair_up(p.top[head], &undo);
    if (i == 0) p.undo[head] = undo;
    // eight codes of a low-bit-first stream, from bit d0 * bits on
    const uint32_t *row = (const uint32_t *)s.data + at;
    const int bit0 = d0 * s.bits, w0 = bit0 >> 5, words = (p.D * s.bits + 31) / 32;
    uint64_t win = row[w0];
    if (w0 + 1 < words) win |= (uint64_t)row[w0 + 1] << 32;
    win >>= bit0 & 31;
    const uint32_t m = (1u << s.bits) - 1u;
    if (s.kind == SRC_AFFINE) {
        const int64_t gi = b * s.gsb + h * s.gsh + t * s.gst + d0 / s.group;
        const float sc = to_f32<T>(((const T *)s.scales)[gi]), bi = to_f32<T>(((const T *)s.biases)[gi]);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = fmaf(sc, (float)((uint32_t)(win >> (j * s.bits)) & m), bi) * up;
    } else {
        const float nrm = s.norms[b * s.gsb + h * s.gsh + t * s.gst];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = nrm * s.codebook[(uint32_t)(win >> (j * s.bits)) & m] * up;
    }
    store_pair(p.high[which] + o, p.low[which] + o, x);
}

// out[row] = post * H(pre * in[row]) / sqrt(D), H the Walsh-Hadamard butterfly, or the rows as they are
// (plain); one warp per row, lane l holds dims E*l .. E*l + E - 1. Written in TO, or (undo set) as f16 times a power of
// two that brings the row's largest finite element to [2^14, 2^15), with what that leaves in low unless plain: a 16-bit
// element that came in is exact in the high half.
struct PairTurn {
    const void *in;
    void *out;
    __half *low;
    float *undo;                  // [B, H, L]
    int64_t i_sb, i_sh, i_sl, o_sb, o_sh, o_sl;
    int32_t B, H, L, plain;
    const float *pre, *post;
};
template <typename TI, typename TO, int D>
__global__ void __launch_bounds__(256) pair_turn_kernel(const __grid_constant__ PairTurn p) {
    constexpr int E = D / 32;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= (int64_t)p.B * p.H * p.L) return;
    const int l = (int)(row % p.L), h = (int)((row / p.L) % p.H), b = (int)(row / ((int64_t)p.L * p.H));
    const TI *src = (const TI *)p.in + b * p.i_sb + h * p.i_sh + l * p.i_sl + E * lane;
    float x[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
        if constexpr (sizeof(TI) == 4) x[j] = src[j];
        else x[j] = to_f32<TI>(src[j]);
        if (p.pre) x[j] *= p.pre[E * lane + j];
    }
    if (!p.plain) {
#pragma unroll
        for (int hh = 1; hh < E; hh <<= 1)
#pragma unroll
            for (int i = 0; i < E; ++i)
                if ((i & hh) == 0) {
                    const float a = x[i], c = x[i + hh];
                    x[i] = a + c;
                    x[i + hh] = a - c;
                }
#pragma unroll
        for (int m = 1; m < 32; m <<= 1)
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float y = __shfl_xor_sync(0xffffffffu, x[j], m);
                x[j] = (lane & m) ? y - x[j] : x[j] + y;
            }
        const float f = rsqrtf((float)D);
#pragma unroll
        for (int j = 0; j < E; ++j) x[j] *= f * (p.post ? p.post[E * lane + j] : 1.f);
    }
    if (p.undo) {
        uint32_t top = 0;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t u = __float_as_uint(x[j]) & 0x7fffffffu;
            if (u < 0x7f800000u) top = max(top, u);
        }
        float undo;
        const float up = pair_up(__reduce_max_sync(0xffffffffu, top), &undo);
#pragma unroll
        for (int j = 0; j < E; ++j) x[j] *= up;
        if (lane == 0) p.undo[row] = undo;
    }
    const int64_t o = b * p.o_sb + h * p.o_sh + l * p.o_sl + E * lane;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        MmaType<TO>::store(p.out, o + j, x[j]);
        if (p.low) p.low[o + j] = __float2half_rn(pair_rest(x[j], __half2float(__float2half_rn(x[j]))));
    }
}
template <typename TI, typename TO>
void pair_turn(const PairTurn &p, int D, cudaStream_t stream) {
    const unsigned blocks = (unsigned)(((int64_t)p.B * p.H * p.L + 7) / 8);
    if (D == 256) pair_turn_kernel<TI, TO, 256><<<blocks, 256, 0, stream>>>(p);
    else if (D == 128) pair_turn_kernel<TI, TO, 128><<<blocks, 256, 0, stream>>>(p);
    else pair_turn_kernel<TI, TO, 64><<<blocks, 256, 0, stream>>>(p);
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

bool pair_source_ok(const KVSource &s, const AttnArgs &a) {
    if (s.kind == SRC_RAW) return s.dtype == a.q_dtype && !((uintptr_t)s.data & 1);
    if ((uintptr_t)s.data & 3) return false;
    if (s.kind == SRC_TURBO) return s.bits >= 2 && s.bits <= 4 && s.norms != nullptr;
    if (s.dtype != a.q_dtype || !s.scales || !s.biases || (s.bits != 2 && s.bits != 4 && s.bits != 8)) return false;
    return s.group >= 8 && a.D % s.group == 0 && s.group % 8 == 0;
}

PairSource pair_source(const KVSource &s, int b0) {
    PairSource o = {};
    o.kind = s.kind; o.group = s.group; o.bits = s.bits;
    o.data = (const char *)s.data + b0 * s.sb * (s.kind == SRC_RAW ? 2 : 4);
    o.scales = s.scales ? (const char *)s.scales + b0 * s.gsb * 2 : nullptr;
    o.biases = s.biases ? (const char *)s.biases + b0 * s.gsb * 2 : nullptr;
    o.norms = s.norms ? s.norms + b0 * s.gsb : nullptr;
    o.sb = s.sb; o.sh = s.sh; o.st = s.st; o.gsb = s.gsb; o.gsh = s.gsh; o.gst = s.gst;
    for (int i = 0; i < 16; ++i) o.codebook[i] = s.codebook[i];
    return o;
}

struct PoolRows {
    void *p;
    cudaStream_t s;
    ~PoolRows() { dev_free(p, s); }
};

}  // namespace

// Returns the number of kernels launched, 0 when the call is left to the general kernel.
int launch_attention_chunk_packed_pairs(const AttnArgs &a, cudaStream_t stream) {
    if ((a.D != 256 && a.D != 128 && a.D != 64) || (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16)) return 0;
    if (a.new_k || a.q_rot || a.o_rot || a.T < 1 || a.T > (int64_t)1 << 30 || a.B < 1 || a.L < 1 || a.Hkv > 65535) return 0;
    if (a.v.kind == SRC_RAW) return 0;
    const bool k_turbo = a.k.kind == SRC_TURBO, v_turbo = a.v.kind == SRC_TURBO, k_raw = a.k.kind == SRC_RAW;
    if (k_turbo != (a.q_signs != nullptr) || v_turbo != (a.o_signs != nullptr) || (a.q_calib && !k_turbo)) return 0;
    if (!pair_source_ok(a.k, a) || !pair_source_ok(a.v, a)) return 0;
    if (a.q_sb < 0 || a.q_sh < 0 || a.q_sl < 0) return 0;

    auto even16 = [](const void *p, int64_t x, int64_t y, int64_t z) { return !((uintptr_t)p & 15) && !((x | y | z) & 7); };
    const int32_t kt = k_raw ? a.q_dtype : (int32_t)KVC_F16;     // type of the score products
    const bool bf16 = a.q_dtype == KVC_BF16;
    const bool k_in_place = k_raw && a.k.st >= a.D && even16(a.k.data, a.k.sb, a.k.sh, a.k.st);
    const bool q_in_place = !k_turbo && a.q_dtype == kt && !((uintptr_t)a.q & 3) && !((a.q_sb | a.q_sh | a.q_sl) & 1);
    const bool q_scaled = !q_in_place && !k_raw;
    AttnArgs r = a;
    r.q_dtype = kt;
    r.k = r.v = KVSource();
    r.k.kind = r.v.kind = SRC_RAW;
    r.k.dtype = r.v.dtype = kt;                  // values are f16; only the width of the rows is asked for
    r.k.st = r.v.st = a.D;
    r.k.sh = r.v.sh = a.T * a.D;
    r.k.sb = r.v.sb = (int64_t)a.Hkv * a.T * a.D;
    r.k.data = r.v.data = (const void *)16;      // only the shape is judged here
    if (k_in_place) r.k = a.k;
    r.q_signs = r.o_signs = r.q_calib = nullptr;
    if (!q_in_place) {
        r.q = (const void *)16;
        r.q_sb = (int64_t)a.Hq * a.L * a.D; r.q_sh = (int64_t)a.L * a.D; r.q_sl = a.D;
    }
    if (!attention_chunk_rows_accepts(r)) return 0;

    // bytes of the parts, per sequence: one half of the rows of K or V, of the queries; fp32 output rows; factors
    auto whole = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t kv = whole((size_t)a.Hkv * a.T * a.D * 2), q = whole((size_t)a.Hq * a.L * a.D * 2);
    const size_t heads = whole((size_t)2 * a.Hkv * 4), rows_f = whole((size_t)a.Hq * a.L * 4);
    const size_t per_b = kv * (k_in_place ? 2 : k_raw ? 3 : 4) + (q_in_place ? 0 : k_turbo ? 2 * q : q) + (v_turbo ? 2 * q : 0) + 2 * heads + rows_f;
    if (per_b > PAIR_SCRATCH_LIMIT) return 0;
    const int fit = (int)std::min<size_t>({(size_t)a.B, PAIR_SCRATCH_LIMIT / per_b, (size_t)32767});
    const int nslices = (a.B + fit - 1) / fit;
    int slice = (a.B + nslices - 1) / nslices;
    // a device too full for the rows of one sequence leaves the call to the general kernel, which needs its partials only
    void *memory = dev_try_alloc((size_t)slice * per_b, stream);
    while (!memory && slice > 1) memory = dev_try_alloc((size_t)(slice = (slice + 1) / 2) * per_b, stream);
    if (!memory) return 0;
    const PoolRows rows{memory, stream};
    int launches = 0;
    for (int b0 = 0; b0 < a.B; b0 += slice) {
        const int nb = std::min(slice, a.B - b0);
        char *at = (char *)rows.p;
        auto take = [&](size_t per_sequence) { char *p = at; at += nb * per_sequence; return p; };
        PairRows pr = {};
        pr.B = nb; pr.H = a.Hkv; pr.D = a.D; pr.T = a.T; pr.first = k_in_place ? 1 : 0;
        pr.top = (uint32_t *)take(heads);
        pr.undo = (float *)take(heads);
        float *q_undo = (float *)take(rows_f);
        for (int w = pr.first; w < 2; ++w) {
            pr.s[w] = pair_source(w ? a.v : a.k, b0);
            pr.high[w] = (__half *)take(kv);
            pr.low[w] = w || !k_raw ? (__half *)take(kv) : nullptr;
        }
        KVC_CUDA(cudaMemsetAsync(pr.top, 0, nb * heads, stream));
        const unsigned planes = (unsigned)((2 - pr.first) * nb);
        const dim3 grid((unsigned)((a.T * (a.D / 8) + 255) / 256), (unsigned)a.Hkv, planes);
        const dim3 tops((unsigned)std::min<int64_t>((a.T + 255) / 256, 64), (unsigned)a.Hkv, planes);
        if (bf16) {
            pair_top_kernel<__nv_bfloat16><<<tops, 256, 0, stream>>>(pr);
            pair_rows_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(pr);
        } else {
            pair_top_kernel<__half><<<tops, 256, 0, stream>>>(pr);
            pair_rows_kernel<__half><<<grid, 256, 0, stream>>>(pr);
        }
        KVC_CUDA(cudaGetLastError());
        g_launch_count += 2;
        launches += 2;

        AttnArgs call = r;
        call.B = nb;
        call.k.data = k_in_place ? (const char *)a.k.data + b0 * a.k.sb * 2 : (const char *)pr.high[0];
        call.v.data = pr.high[1];
        call.q = (const char *)a.q + b0 * a.q_sb * 2;
        call.out = (char *)a.out + b0 * a.o_sb * 2;
        if (a.mask.mode == KVC_MASK_ARRAY) call.mask.data = (const char *)a.mask.data + b0 * a.mask.sb * (int64_t)dtype_size(a.mask.dtype);
        ChunkLow low = {k_raw ? nullptr : pr.low[0], pr.low[1], nullptr, q_scaled ? q_undo : nullptr, k_raw ? nullptr : pr.undo,
                        pr.undo + (size_t)nb * a.Hkv, v_turbo ? (int32_t)KVC_F32 : a.q_dtype};
        if (!q_in_place) {
            PairTurn t = {};
            t.in = call.q; t.out = take(q); t.low = k_turbo ? (__half *)take(q) : nullptr;
            t.undo = q_scaled ? q_undo : nullptr;
            t.i_sb = a.q_sb; t.i_sh = a.q_sh; t.i_sl = a.q_sl;
            t.o_sb = r.q_sb; t.o_sh = r.q_sh; t.o_sl = r.q_sl;
            t.B = nb; t.H = a.Hq; t.L = a.L;
            t.pre = a.q_signs; t.post = a.q_calib; t.plain = k_turbo ? 0 : 1;
            if (kt == KVC_BF16) pair_turn<__nv_bfloat16, __nv_bfloat16>(t, a.D, stream);
            else if (bf16) pair_turn<__nv_bfloat16, __half>(t, a.D, stream);
            else pair_turn<__half, __half>(t, a.D, stream);
            ++launches;
            call.q = t.out;
            low.q = t.low;
        }
        if (v_turbo) {
            call.out = take(2 * q);
            call.o_sb = (int64_t)a.Hq * a.L * a.D; call.o_sh = (int64_t)a.L * a.D; call.o_sl = a.D;
        }
        const int n = launch_attention_chunk_pairs(call, low, stream);
        if (n <= 0) fail(KVC_ERR_INTERNAL, "the chunk kernel on operand pairs refused a call it had accepted");
        launches += n;
        if (v_turbo) {
            PairTurn t = {};
            t.in = call.out; t.out = (char *)a.out + b0 * a.o_sb * 2;
            t.i_sb = call.o_sb; t.i_sh = call.o_sh; t.i_sl = call.o_sl;
            t.o_sb = a.o_sb; t.o_sh = a.o_sh; t.o_sl = a.o_sl;
            t.B = nb; t.H = a.Hq; t.L = a.L;
            t.post = a.o_signs;
            if (bf16) pair_turn<float, __nv_bfloat16>(t, a.D, stream);
            else pair_turn<float, __half>(t, a.D, stream);
            ++launches;
        }
    }
    if (trace_dispatch()) fprintf(stderr, "[kvc] chunk_pairs: rows decoded to pairs, %d sequences per slice\n", slice);
    return launches;
}

}  // namespace kvc
