// Group-wise affine quantisation (MLX `quantized` / `dequantized`, affine mode)
// and the TurboQuant fused Walsh-Hadamard encode.
//
// Both produce integer codes that must be bit-identical to the CPU oracle, so
// every floating-point step uses the explicit round-to-nearest intrinsics
// (never contracted into FMAs) and one fixed reduction tree:
//   * a row of D elements is owned by 32 lanes, lane l holding the E = D/32
//     contiguous elements [l*E, l*E+E);
//   * sums run sequentially over a lane's own elements, then over the xor
//     butterfly 16, 8, 4, 2, 1 across lanes.
#include "attn_common.cuh"
#include "common.h"
#include "f32x2.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace kvc {

namespace {

template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// MLX affine quantisation of one group given its min and max:
//   scale = max((max-min)/(2^b-1), 1e-7); the sign of the scale and the
//   anchoring edge follow the larger-magnitude end, the scale is re-derived so
//   that the edge maps to an integer code, and codes are
//   rint((w - bias)/scale) clamped to [0, 2^b-1].
__device__ __forceinline__ void affine_params(float w_min, float w_max, float n_bins,
                                              float &scale, float &bias) {
    scale = fmaxf(__fdiv_rn(__fsub_rn(w_max, w_min), n_bins), 1e-7f);
    const bool side = fabsf(w_min) > fabsf(w_max);
    scale = side ? scale : -scale;
    const float edge = side ? w_min : w_max;
    const float q0 = rintf(__fdiv_rn(edge, scale));
    bias = 0.f;
    if (q0 != 0.f) {
        scale = __fdiv_rn(edge, q0);
        bias = edge;
    }
}

__device__ __forceinline__ uint32_t affine_code(float w, float scale, float bias, float n_bins) {
    float q = rintf(__fdiv_rn(__fsub_rn(w, bias), scale));
    q = fminf(fmaxf(q, 0.f), n_bins);
    return (uint32_t)q;
}

// One row (D = 32 E elements) by one warp: group min/max by shuffles, MLX affine parameters,
// codes packed low bits first. `src` points at the row's first element, `dst` at its first code
// word, `scales` / `biases` at its first group.
template <typename T, int E>
__device__ __forceinline__ void quantize_row_warp(const T *src, int64_t s_sd, uint32_t *dst, T *scales, T *biases,
                                                  int group, int bits, int lane) {
    float v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = to_float<T>(src[(int64_t)(lane * E + i) * s_sd]);

    float w_min = v[0], w_max = v[0];
#pragma unroll
    for (int i = 1; i < E; ++i) {
        w_min = fminf(w_min, v[i]);
        w_max = fmaxf(w_max, v[i]);
    }
    const int lanes_per_group = group / E;  // power of two, <= 32
    for (int m = lanes_per_group >> 1; m >= 1; m >>= 1) {
        w_min = fminf(w_min, __shfl_xor_sync(0xffffffffu, w_min, m));
        w_max = fmaxf(w_max, __shfl_xor_sync(0xffffffffu, w_max, m));
    }
    const float n_bins = (float)((1 << bits) - 1);
    float scale, bias;
    affine_params(w_min, w_max, n_bins, scale, bias);

    if ((lane % lanes_per_group) == 0) {
        const int g = lane / lanes_per_group;
        scales[g] = from_float<T>(scale);
        biases[g] = from_float<T>(bias);
    }

    // Pack: the lane's E codes occupy E*bits consecutive bits starting at bit
    // lane*E*bits of the row (low bits first).
    const int nbits = E * bits;  // a power of two in [2, 64]
    uint64_t acc = 0;
#pragma unroll
    for (int i = 0; i < E; ++i)
        acc |= (uint64_t)affine_code(v[i], scale, bias, n_bins) << (i * bits);
    if (nbits == 64) {
        dst[lane * 2] = (uint32_t)acc;
        dst[lane * 2 + 1] = (uint32_t)(acc >> 32);
    } else if (nbits == 32) {
        dst[lane] = (uint32_t)acc;
    } else {
        const uint32_t part = (uint32_t)acc;
        const int lpw = 32 / nbits;  // lanes per word
        uint32_t word = part;
        for (int k = 1; k < lpw; ++k) {
            const uint32_t other = __shfl_down_sync(0xffffffffu, part, k);
            word |= other << (k * nbits);
        }
        if ((lane % lpw) == 0) dst[lane / lpw] = word;
    }
}

// One warp per (tensor, b, h, s) row; E elements per lane.
template <typename T, int E>
__global__ void affine_quantize_warp_kernel(QuantAppendArgs ka, QuantAppendArgs va, int64_t k_rows,
                                            int64_t total_rows) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= total_rows) return;
    const bool is_v = row >= k_rows;
    const QuantAppendArgs &a = is_v ? va : ka;
    int64_t r = is_v ? row - k_rows : row;
    const int s = (int)(r % a.S);
    r /= a.S;
    const int h = (int)(r % a.H);
    const int b = (int)(r / a.H);
    const int64_t t = a.pos + s;
    quantize_row_warp<T, E>((const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss, a.s_sd,
                            a.codes + b * a.c_sb + h * a.c_sh + t * a.c_st,
                            (T *)a.scales + b * a.g_sb + h * a.g_sh + t * a.g_st,
                            (T *)a.biases + b * a.g_sb + h * a.g_sh + t * a.g_st, a.group, a.bits, lane);
}

// Codes of VEC values of one group. The correctly rounded quotient (w - bias) / scale lies between
// the products of (w - bias) with the reciprocal scaled by 1 -+ 4e-7. Each product is rounded to an
// integer by a fused multiply-add with 1.5 * 2^23 (one rounding, ties to even, like rint): when both
// ends give the same integer that is rint of the quotient as well; when they differ for any value
// the lane redoes its values with the division itself. So the codes are those of affine_code bit for
// bit. The clamps run on the biased floats (a NaN becomes code 0, as fmaxf(NaN, 0) makes it), and
// the words accumulate the float bit patterns by multiply-add; MAGIC_SUM removes the bias's share.
template <int VEC, int BITS>
__device__ __forceinline__ uint64_t affine_codes_vec(const float (&v)[VEC], float scale, float bias) {
    constexpr float n_bins = (float)((1 << BITS) - 1);
    constexpr float MAGIC = 12582912.f;          // 1.5 * 2^23: x + MAGIC leaves rint(x) in the low mantissa bits
    constexpr uint32_t MAGIC_BITS = 0x4B400000u;
    constexpr int PER_WORD = (VEC * BITS > 32) ? 32 / BITS : VEC;   // values per 32-bit word
    uint32_t magic_sum = 0;
#pragma unroll
    for (int i = 0; i < PER_WORD; ++i) magic_sum += MAGIC_BITS << (i * BITS);
    const float inv = __frcp_rn(scale);
    const float inv_lo = fmaf(inv, -4e-7f, inv), inv_hi = fmaf(inv, 4e-7f, inv);
    uint32_t w[2] = {0u, 0u};
    uint32_t differ = 0;
#pragma unroll
    for (int i = VEC - 1; i >= 0; --i) {
        const float x = __fsub_rn(v[i], bias);
        const float u_lo = __fmaf_rn(x, inv_lo, MAGIC), u_hi = __fmaf_rn(x, inv_hi, MAGIC);
        differ |= __float_as_uint(u_lo) ^ __float_as_uint(u_hi);
        const float u = fminf(fmaxf(u_lo, MAGIC), MAGIC + n_bins);
        w[i / PER_WORD] = (w[i / PER_WORD] << BITS) + __float_as_uint(u);
    }
    w[0] -= magic_sum;
    if (VEC * BITS > 32) w[1] -= magic_sum;
    // (products beyond 2^22 leave the integer grid of the biased floats but are far outside the code
    // range, so the clamps settle them.) A reciprocal below 1e-30 has lost bits to the subnormal
    // range: exact path, like a straddled tie.
    if (differ != 0u || !(fabsf(inv) > 1e-30f) || !(fabsf(inv) < 1e30f)) {
        w[0] = w[1] = 0u;
#pragma unroll
        for (int i = VEC - 1; i >= 0; --i)
            w[i / PER_WORD] = (w[i / PER_WORD] << BITS) | affine_code(v[i], scale, bias, n_bins);
    }
    return (uint64_t)w[0] | ((uint64_t)w[1] << 32);
}

// Contiguous rows, 16 bytes per lane: a row takes LPR = D / VEC lanes (VEC = 8 for 16-bit types, 4 for
// fp32), a warp covers 32 / LPR rows per pass and keeps U passes of loads in flight. Grid: x = chunks
// of consecutive tokens, y = head, z = batch (keys first, then values), so a block works on one
// (tensor, batch, head) and its pointers are uniform. Same parameters and codes as quantize_row_warp
// (min / max are order-free).
template <typename T, int LPR, int BITS, int U>
__device__ __forceinline__ void affine_quantize_vec_body(const QuantAppendArgs &a, int b, int lpg_log2) {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int RPP = 32 / LPR;
    constexpr int NBITS = VEC * BITS;   // code bits per lane: 8, 16, 32 or 64
    constexpr float n_bins = (float)((1 << BITS) - 1);
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPR, l = lane % LPR;
    const int h = blockIdx.y;
    const int s0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (RPP * U) + sub;
    if (s0 - sub >= a.S) return;   // whole warp
    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + l * VEC;
    uint32_t *codes = a.codes + b * a.c_sb + h * a.c_sh + a.pos * a.c_st;
    const int64_t g0 = b * a.g_sb + h * a.g_sh + a.pos * a.g_st;
    T *scales = (T *)a.scales + g0, *biases = (T *)a.biases + g0;

    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int sr = s0 + u * RPP;
        raw[u] = sr < a.S ? *reinterpret_cast<const uint4 *>(src + sr * a.s_ss) : make_uint4(0u, 0u, 0u, 0u);
    }
    const int lpg = 1 << lpg_log2;   // lanes per group
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int sr = s0 + u * RPP;
        float v[VEC];
        const T *e = reinterpret_cast<const T *>(&raw[u]);
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] = to_float<T>(e[i]);
        float w_min = v[0], w_max = v[0];
#pragma unroll
        for (int i = 1; i < VEC; ++i) {
            w_min = fminf(w_min, v[i]);
            w_max = fmaxf(w_max, v[i]);
        }
        for (int m = lpg >> 1; m >= 1; m >>= 1) {
            w_min = fminf(w_min, __shfl_xor_sync(0xffffffffu, w_min, m));
            w_max = fmaxf(w_max, __shfl_xor_sync(0xffffffffu, w_max, m));
        }
        float scale, bias;
        affine_params(w_min, w_max, n_bins, scale, bias);
        const uint64_t acc = affine_codes_vec<VEC, BITS>(v, scale, bias);
        uint32_t word = (uint32_t)acc;
        if (NBITS < 32) {
            constexpr int LPW = NBITS < 32 ? 32 / NBITS : 1;   // lanes per word
#pragma unroll
            for (int k = 1; k < LPW; ++k) word |= __shfl_down_sync(0xffffffffu, (uint32_t)acc, k) << (k * NBITS);
        }
        if (sr < a.S) {
            if ((l & (lpg - 1)) == 0) {
                scales[sr * a.g_st + (l >> lpg_log2)] = from_float<T>(scale);
                biases[sr * a.g_st + (l >> lpg_log2)] = from_float<T>(bias);
            }
            uint32_t *row = codes + sr * a.c_st;
            if (NBITS == 64) {
                *reinterpret_cast<uint2 *>(row + l * 2) = make_uint2((uint32_t)acc, (uint32_t)(acc >> 32));
            } else if (NBITS == 32) {
                row[l] = word;
            } else {
                constexpr int LPW = NBITS < 32 ? 32 / NBITS : 1;
                if ((l % LPW) == 0) row[l / LPW] = word;
            }
        }
    }
}

template <typename T, int LPR, int BITS, int U>
__global__ void __launch_bounds__(256)
affine_quantize_vec_kernel(QuantAppendArgs ka, QuantAppendArgs va, int lpg_log2) {
    dev::pdl_wait();
    dev::pdl_trigger();
    // keys and values share B, H and S; the branch is uniform over the block
    if ((int)blockIdx.z >= ka.B) affine_quantize_vec_body<T, LPR, BITS, U>(va, (int)blockIdx.z - ka.B, lpg_log2);
    else affine_quantize_vec_body<T, LPR, BITS, U>(ka, (int)blockIdx.z, lpg_log2);
}

// The same rows for a list of independent caches (one new token each): row = (sequence, K or V,
// head); every pointer of the table already addresses head 0 at the sequence's append position.
template <typename T, int E>
__global__ void affine_quantize_varlen_kernel(const __grid_constant__ VarlenQuantArgs a) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= a.n * 2 * a.H) return;
    const int i = row / (2 * a.H), rr = row % (2 * a.H);
    const bool is_v = rr >= a.H;
    const int h = rr % a.H;
    const VarlenQuantSeq &q = a.seq[i];
    const T *src = (const T *)(is_v ? q.vsrc : q.ksrc) + (int64_t)h * a.src_sh;
    uint32_t *codes = (is_v ? q.vcodes : q.kcodes) + (int64_t)h * q.c_sh;
    T *scales = (T *)(is_v ? q.vscales : q.kscales) + (int64_t)h * q.g_sh;
    T *biases = (T *)(is_v ? q.vbiases : q.kbiases) + (int64_t)h * q.g_sh;
    quantize_row_warp<T, E>(src, 1, codes, scales, biases, a.group, a.bits, lane);
}

// General shapes: one thread per group.
template <typename T>
__global__ void affine_quantize_group_kernel(QuantAppendArgs ka, QuantAppendArgs va,
                                             int64_t k_groups, int64_t total_groups) {
    dev::pdl_wait();
    dev::pdl_trigger();
    int64_t gidx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gidx >= total_groups) return;
    const bool is_v = gidx >= k_groups;
    const QuantAppendArgs &a = is_v ? va : ka;
    if (is_v) gidx -= k_groups;
    const int gpr = a.D / a.group;
    const int g = (int)(gidx % gpr);
    int64_t r = gidx / gpr;
    const int s = (int)(r % a.S);
    r /= a.S;
    const int h = (int)(r % a.H);
    const int b = (int)(r / a.H);
    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss + (int64_t)g * a.group * a.s_sd;
    float w_min = to_float<T>(src[0]), w_max = w_min;
    for (int i = 1; i < a.group; ++i) {
        const float x = to_float<T>(src[i * a.s_sd]);
        w_min = fminf(w_min, x);
        w_max = fmaxf(w_max, x);
    }
    const float n_bins = (float)((1 << a.bits) - 1);
    float scale, bias;
    affine_params(w_min, w_max, n_bins, scale, bias);
    const int64_t t = a.pos + s;
    const int64_t gi = b * a.g_sb + h * a.g_sh + t * a.g_st + g;
    ((T *)a.scales)[gi] = from_float<T>(scale);
    ((T *)a.biases)[gi] = from_float<T>(bias);
    uint32_t *dst = a.codes + b * a.c_sb + h * a.c_sh + t * a.c_st + (int64_t)g * a.group * a.bits / 32;
    const int per_word = 32 / a.bits;
    for (int w = 0; w < a.group / per_word; ++w) {
        uint32_t word = 0;
        for (int k = 0; k < per_word; ++k)
            word |= affine_code(to_float<T>(src[(int64_t)(w * per_word + k) * a.s_sd]), scale, bias, n_bins)
                    << (k * a.bits);
        dst[w] = word;
    }
}

template <typename T>
__global__ void affine_dequantize_kernel(DequantArgs a, int64_t total) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int d = (int)(i % a.D);
    const int64_t row = i / a.D;
    const uint32_t word = a.codes[row * a.c_srow + (d * a.bits) / 32];
    const uint32_t code = (word >> ((d * a.bits) % 32)) & ((1u << a.bits) - 1u);
    const int g = d / a.group;
    const float sc = to_float<T>(((const T *)a.scales)[row * a.g_srow + g]);
    const float bi = to_float<T>(((const T *)a.biases)[row * a.g_srow + g]);
    // MLX dequantises in the array dtype: scale * q + bias.
    const float val = __fadd_rn(__fmul_rn(sc, (float)code), bi);
    ((T *)a.out)[row * a.o_srow + d] = from_float<T>(val);
}

// The single-token rows of a list of caches of one shape (the layers of a batched step) in one launch:
// z = (layer, K or V, batch).
struct QuantList {
    int32_t tensors;   // 1: keys only, 2: keys and values
    QuantAppendArgs a[KVC_LIST_MAX][2];
};
template <typename T, int LPR, int BITS>
__global__ void __launch_bounds__(256) affine_quantize_list_kernel(const __grid_constant__ QuantList l, int lpg_log2) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const int B = l.a[0][0].B, b = blockIdx.z % B, w = blockIdx.z / B;
    affine_quantize_vec_body<T, LPR, BITS, 1>(l.a[w / l.tensors][w % l.tensors], b, lpg_log2);
}

// 16-byte lanes need contiguous, 16-byte aligned rows
template <typename T> bool quant_vec_ok(const QuantAppendArgs &a) {
    constexpr int VEC = 16 / (int)sizeof(T);
    const int lpr = a.D / VEC;
    if (a.D % VEC != 0 || !(lpr == 8 || lpr == 16 || lpr == 32)) return false;
    if (a.group % VEC != 0 || a.group / VEC > lpr || ((a.group / VEC) & (a.group / VEC - 1))) return false;
    if (a.s_sd != 1 || a.s_sb % VEC || a.s_sh % VEC || a.s_ss % VEC) return false;
    if ((reinterpret_cast<uintptr_t>(a.src) & 15) || (reinterpret_cast<uintptr_t>(a.codes) & 7)) return false;
    return (a.c_sb % 2 == 0) && (a.c_sh % 2 == 0) && (a.c_st % 2 == 0);
}

template <typename T>
bool quantize_list(const QuantAppendArgs *k, const QuantAppendArgs *v, int n, cudaStream_t stream) {
    static thread_local QuantList l;
    const QuantAppendArgs &k0 = k[0];
    l.tensors = v ? 2 : 1;
    for (int i = 0; i < n; ++i)
        for (int w = 0; w < l.tensors; ++w) {
            const QuantAppendArgs &a = w ? v[i] : k[i];
            if (a.B != k0.B || a.H != k0.H || a.S != k0.S || a.D != k0.D || a.group != k0.group || a.bits != k0.bits ||
                a.dtype != k0.dtype || !quant_vec_ok<T>(a))
                return false;
            l.a[i][w] = a;
        }
    const int64_t z = (int64_t)n * l.tensors * k0.B;
    if (k0.H > 65535 || z > 65535) return false;
    constexpr int VEC = 16 / (int)sizeof(T);
    const int lpr = k0.D / VEC, rpp = 32 / lpr;
    int lpg_log2 = 0;
    while ((1 << lpg_log2) < k0.group / VEC) ++lpg_log2;
    const int warps = std::max(1, std::min(8, (k0.S + rpp - 1) / rpp));
    const dim3 grid((unsigned)((k0.S + warps * rpp - 1) / (warps * rpp)), (unsigned)k0.H, (unsigned)z);
#define KVC_QL(LPR)                                                                                                  \
    switch (k0.bits) {                                                                                               \
        case 2: KVC_CUDA(launch_pdl(affine_quantize_list_kernel<T, LPR, 2>, grid, dim3(warps * 32), 0, stream, l, lpg_log2)); break;         \
        case 4: KVC_CUDA(launch_pdl(affine_quantize_list_kernel<T, LPR, 4>, grid, dim3(warps * 32), 0, stream, l, lpg_log2)); break;         \
        default: KVC_CUDA(launch_pdl(affine_quantize_list_kernel<T, LPR, 8>, grid, dim3(warps * 32), 0, stream, l, lpg_log2)); break;        \
    }
    switch (lpr) {
        case 8: KVC_QL(8); break;
        case 16: KVC_QL(16); break;
        default: KVC_QL(32); break;
    }
#undef KVC_QL
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    return true;
}

template <typename T>
void quantize_dispatch(const QuantAppendArgs &k, const QuantAppendArgs &v, bool have_v,
                       cudaStream_t stream) {
    const QuantAppendArgs &vv = have_v ? v : k;
    const int64_t k_rows = (int64_t)k.B * k.H * k.S;
    const int64_t v_rows = have_v ? (int64_t)v.B * v.H * v.S : 0;
    auto warp_ok = [](const QuantAppendArgs &a) {
        if (a.D % 32 != 0) return false;
        const int E = a.D / 32;
        if (!(E == 1 || E == 2 || E == 4 || E == 8)) return false;
        if (a.group % E != 0) return false;
        const int lpg = a.group / E;
        if (lpg < 1 || lpg > 32 || (lpg & (lpg - 1))) return false;
        const int nbits = E * a.bits;
        return (nbits >= 32) ? (nbits % 32 == 0) : (32 % nbits == 0);
    };
    const bool same_shape = !have_v || (k.D == v.D && k.group == v.group && k.bits == v.bits);
    constexpr int VEC = 16 / (int)sizeof(T);
    auto vec_ok = [](const QuantAppendArgs &a) { return quant_vec_ok<T>(a); };
    const bool same_dims = !have_v || (k.B == v.B && k.H == v.H && k.S == v.S);
    if (same_shape && same_dims && vec_ok(k) && (!have_v || vec_ok(v)) && k.H <= 65535 && 2 * (int64_t)k.B <= 65535) {
        const int lpr = k.D / VEC, rpp = 32 / lpr;
        int lpg_log2 = 0;
        while ((1 << lpg_log2) < k.group / VEC) ++lpg_log2;
        const bool deep = (int64_t)k.S >= 8 * rpp * 4;   // a block of 8 warps fills up with 4 passes per warp
        const int rows_per_warp = rpp * (deep ? 4 : 1);
        const int warps = std::max(1, std::min(8, (k.S + rows_per_warp - 1) / rows_per_warp));
        const dim3 grid((unsigned)((k.S + warps * rows_per_warp - 1) / (warps * rows_per_warp)), (unsigned)k.H,
                        (unsigned)(k.B * (have_v ? 2 : 1)));
#define KVC_QVEC(LPR, BITS)                                                                                   \
    do {                                                                                                      \
        if (deep) KVC_CUDA(launch_pdl(affine_quantize_vec_kernel<T, LPR, BITS, 4>, grid, dim3(warps * 32), 0, stream, k, vv, lpg_log2)); \
        else KVC_CUDA(launch_pdl(affine_quantize_vec_kernel<T, LPR, BITS, 1>, grid, dim3(warps * 32), 0, stream, k, vv, lpg_log2));      \
    } while (0)
#define KVC_QVEC_B(LPR)                                            \
    switch (k.bits) {                                              \
        case 2: KVC_QVEC(LPR, 2); break;                           \
        case 4: KVC_QVEC(LPR, 4); break;                           \
        default: KVC_QVEC(LPR, 8); break;                          \
    }
        switch (lpr) {
            case 8: KVC_QVEC_B(8); break;
            case 16: KVC_QVEC_B(16); break;
            default: KVC_QVEC_B(32); break;
        }
#undef KVC_QVEC_B
#undef KVC_QVEC
    } else if (same_shape && warp_ok(k)) {
        const int64_t total = k_rows + v_rows;
        const int warps = 8;
        const unsigned blocks = (unsigned)((total + warps - 1) / warps);
        switch (k.D / 32) {
            case 1: KVC_CUDA(launch_pdl(affine_quantize_warp_kernel<T, 1>, dim3(blocks), dim3(warps * 32), 0, stream, k, vv, k_rows, total)); break;
            case 2: KVC_CUDA(launch_pdl(affine_quantize_warp_kernel<T, 2>, dim3(blocks), dim3(warps * 32), 0, stream, k, vv, k_rows, total)); break;
            case 4: KVC_CUDA(launch_pdl(affine_quantize_warp_kernel<T, 4>, dim3(blocks), dim3(warps * 32), 0, stream, k, vv, k_rows, total)); break;
            case 8: KVC_CUDA(launch_pdl(affine_quantize_warp_kernel<T, 8>, dim3(blocks), dim3(warps * 32), 0, stream, k, vv, k_rows, total)); break;
        }
    } else {
        const int64_t k_groups = k_rows * (k.D / k.group);
        const int64_t v_groups = have_v ? v_rows * (v.D / v.group) : 0;
        const int64_t total = k_groups + v_groups;
        KVC_CUDA(launch_pdl(affine_quantize_group_kernel<T>, dim3((unsigned)((total + 127) / 128)), dim3(128), 0, stream,
            k, vv, k_groups, total));
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

}  // namespace

bool launch_affine_quantize_varlen(const VarlenQuantArgs &a, cudaStream_t stream) {
    if (a.D % 32 != 0 || a.n < 1 || a.n > KVC_VARLEN_MAX) return false;
    const int E = a.D / 32;
    if (!(E == 1 || E == 2 || E == 4 || E == 8) || a.group % E != 0) return false;
    const int lpg = a.group / E;
    if (lpg < 1 || lpg > 32 || (lpg & (lpg - 1))) return false;
    const int nbits = E * a.bits;
    if (!((nbits >= 32) ? (nbits % 32 == 0) : (32 % nbits == 0))) return false;
    const int total = a.n * 2 * a.H, warps = 8;
    const unsigned blocks = (unsigned)((total + warps - 1) / warps);
#define KVC_QV(TT)                                                                                      \
    switch (E) {                                                                                        \
        case 1: KVC_CUDA(launch_pdl(affine_quantize_varlen_kernel<TT, 1>, dim3(blocks), dim3(warps * 32), 0, stream, a)); break;     \
        case 2: KVC_CUDA(launch_pdl(affine_quantize_varlen_kernel<TT, 2>, dim3(blocks), dim3(warps * 32), 0, stream, a)); break;     \
        case 4: KVC_CUDA(launch_pdl(affine_quantize_varlen_kernel<TT, 4>, dim3(blocks), dim3(warps * 32), 0, stream, a)); break;     \
        default: KVC_CUDA(launch_pdl(affine_quantize_varlen_kernel<TT, 8>, dim3(blocks), dim3(warps * 32), 0, stream, a)); break;    \
    }
    if (a.dtype == KVC_BF16) { KVC_QV(__nv_bfloat16) }
    else if (a.dtype == KVC_F16) { KVC_QV(__half) }
    else if (a.dtype == KVC_F32) { KVC_QV(float) }
    else return false;
#undef KVC_QV
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    return true;
}

bool launch_affine_quantize_list(const QuantAppendArgs *k, const QuantAppendArgs *v, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX || (int64_t)k[0].B * k[0].H * k[0].S == 0) return false;
    switch (k[0].dtype) {
        case KVC_F32: return quantize_list<float>(k, v, n, stream);
        case KVC_F16: return quantize_list<__half>(k, v, n, stream);
        case KVC_BF16: return quantize_list<__nv_bfloat16>(k, v, n, stream);
        default: return false;
    }
}

void launch_affine_quantize2(const QuantAppendArgs &k, const QuantAppendArgs *v, cudaStream_t stream) {
    if ((int64_t)k.B * k.H * k.S == 0) return;
    auto check = [](const QuantAppendArgs &a) {
        KVC_REQUIRE(a.bits == 2 || a.bits == 4 || a.bits == 8,
                    "affine quantisation supports 2, 4 or 8 bits");
        KVC_REQUIRE(a.group > 0 && a.D % a.group == 0, "head dim must be a multiple of the group size");
        KVC_REQUIRE((a.group * a.bits) % 32 == 0, "group must fill whole 32-bit words");
    };
    check(k);
    if (v) {
        check(*v);
        KVC_REQUIRE(v->dtype == k.dtype, "keys and values must share a dtype");
    }
    const QuantAppendArgs dummy = k;
    switch (k.dtype) {
        case KVC_F32: quantize_dispatch<float>(k, v ? *v : dummy, v != nullptr, stream); break;
        case KVC_F16: quantize_dispatch<__half>(k, v ? *v : dummy, v != nullptr, stream); break;
        case KVC_BF16: quantize_dispatch<__nv_bfloat16>(k, v ? *v : dummy, v != nullptr, stream); break;
        default: fail(KVC_ERR_INVALID_ARG, "affine quantisation needs a floating dtype");
    }
}

void launch_affine_quantize(const QuantAppendArgs &a, cudaStream_t stream) {
    launch_affine_quantize2(a, nullptr, stream);
}

void launch_affine_dequantize(const DequantArgs &a, cudaStream_t stream) {
    const int64_t total = a.rows * a.D;
    if (total <= 0) return;
    KVC_REQUIRE(a.bits == 2 || a.bits == 4 || a.bits == 8, "affine dequantisation supports 2, 4 or 8 bits");
    const unsigned blocks = (unsigned)((total + 255) / 256);
    switch (a.dtype) {
        case KVC_F32: affine_dequantize_kernel<float><<<blocks, 256, 0, stream>>>(a, total); break;
        case KVC_F16: affine_dequantize_kernel<__half><<<blocks, 256, 0, stream>>>(a, total); break;
        case KVC_BF16: affine_dequantize_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(a, total); break;
        default: fail(KVC_ERR_INVALID_ARG, "affine dequantisation needs a floating dtype");
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

// ---------------------------------------------------------------------
// TurboQuant fused WHT encode
// ---------------------------------------------------------------------
namespace {

template <typename T, int E>
__global__ void turbo_encode_kernel(TurboEncodeArgs ka, TurboEncodeArgs va, int64_t k_rows,
                                    int64_t total_rows, float inv_sqrt_dim) {
    dev::pdl_wait();
    dev::pdl_trigger();
    extern __shared__ uint32_t s_words[];  // [warps][PWmax]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= total_rows) return;  // whole warp exits together
    const bool is_v = row >= k_rows;
    const TurboEncodeArgs &a = is_v ? va : ka;
    int64_t r = is_v ? row - k_rows : row;
    const int s = (int)(r % a.S);
    r /= a.S;
    const int h = (int)(r % a.H);
    const int b = (int)(r / a.H);
    constexpr int D = E * 32;

    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss;
    float v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = to_float<T>(src[(int64_t)(lane * E + i) * a.s_sd]);

    // L2 norm over the fixed reduction tree.
    float sq = __fmul_rn(v[0], v[0]);
#pragma unroll
    for (int i = 1; i < E; ++i) sq = __fadd_rn(sq, __fmul_rn(v[i], v[i]));
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, m));
    const float norm = __fsqrt_rn(sq);
    const float inv_norm = (norm > 1e-8f) ? __fdiv_rn(1.0f, norm) : 0.0f;

    // unit-normalise and flip signs: x * (inv_norm * sign)
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = __fmul_rn(v[i], __fmul_rn(inv_norm, a.signs[lane * E + i]));

    // Walsh-Hadamard butterfly, stage s pairs elements 2^s apart: (a, b) -> (a+b, a-b).
#pragma unroll
    for (int st = 1; st < E; st <<= 1) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
            if ((i & st) == 0) {
                const float lo = v[i], hi = v[i + st];
                v[i] = __fadd_rn(lo, hi);
                v[i + st] = __fsub_rn(lo, hi);
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, v[i], m);
            v[i] = (lane & m) ? __fsub_rn(other, v[i]) : __fadd_rn(other, v[i]);
        }
    }

    // boundary quantise + pack (low bits first, codes may straddle words)
    const int pw = (D * a.bits + 31) / 32;
    uint32_t *words = s_words + warp * ((1024 * 4 + 31) / 32);
    for (int w = lane; w < pw; w += 32) words[w] = 0;
    __syncwarp();
    const int levels_m1 = (1 << a.bits) - 1;
    const uint32_t mask = (uint32_t)levels_m1;
    float recon_sq = 0.f;  // calibrated rows: squared norm of centroid * scale, same reduction tree as the norm
#pragma unroll
    for (int i = 0; i < E; ++i) {
        float rotated = __fmul_rn(v[i], inv_sqrt_dim);
        float cal = 1.f;
        if (a.calib) {
            cal = a.calib[lane * E + i];
            rotated = __fdiv_rn(rotated, cal);
        }
        uint32_t idx = 0;
        for (int bd = 0; bd < levels_m1; ++bd) idx += (rotated > a.boundaries[bd]) ? 1u : 0u;
        idx &= mask;
        if (a.calib) {
            const float cv = __fmul_rn(a.centroids[idx], cal);
            const float sqv = __fmul_rn(cv, cv);
            recon_sq = i == 0 ? sqv : __fadd_rn(recon_sq, sqv);
        }
        const int bit = (lane * E + i) * a.bits;
        const int w = bit >> 5, sh = bit & 31;
        atomicOr(&words[w], idx << sh);
        if (sh + a.bits > 32) atomicOr(&words[w + 1], idx >> (32 - sh));
    }
    float stored = norm;
    if (a.calib) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) recon_sq = __fadd_rn(recon_sq, __shfl_xor_sync(0xffffffffu, recon_sq, m));
        const float recon = __fsqrt_rn(recon_sq);
        if (recon > 1e-8f) stored = __fdiv_rn(norm, recon);
    }
    __syncwarp();
    const int64_t t = a.pos + s;
    uint32_t *dst = a.packed + b * a.p_sb + h * a.p_sh + t * a.p_st;
    for (int w = lane; w < pw; w += 32) dst[w] = words[w];
    if (lane == 0) a.norms[b * a.n_sb + h * a.n_sh + t * a.n_st] = stored;
}

// Dense-rotation encode for head dims that are not powers of two (fusedEncodeSource,
// TurboQuantKernels.swift:103-204): one block per row, thread d owns dimension d. Norm over the fixed tree
// (32 lanes x ceil(D/32) contiguous elements, then the xor butterfly), rotated[d] = sum_j Pi[d][j] * unit[j]
// accumulated left to right with separate multiply and add, boundary count, packing, and the norm
// correction norm / ||centroids[idx]|| over the same tree. With `calib` the rotated value is divided by
// the scale first and the correction uses centroids[idx] * scale (TurboQuantKernels.swift:354-411).
template <typename T>
__global__ void turbo_encode_dense_kernel(TurboEncodeArgs a, int64_t total_rows) {
    asm volatile("griddepcontrol.launch_dependents;");
    extern __shared__ float s_f[];           // [D] unit row, [D] tree scratch, then the packed words
    const int D = a.D;
    float *unit = s_f;
    float *tree = s_f + D;
    uint32_t *words = (uint32_t *)(s_f + 2 * D + 1);   // tree has one slot past the row
    const int d = threadIdx.x;
    const int64_t row = blockIdx.x;
    if (row >= total_rows) return;
    int64_t r = row;
    const int s = (int)(r % a.S);
    r /= a.S;
    const int h = (int)(r % a.H);
    const int b = (int)(r / a.H);
    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss;
    const int E = (D + 31) / 32;
    const float val = d < D ? to_float<T>(src[(int64_t)d * a.s_sd]) : 0.f;

    // sum over the fixed tree of a per-dimension quantity held in `tree`
    auto tree_sum = [&](float mine) -> float {
        if (d < D) tree[d] = mine;
        __syncthreads();
        float lane_sum = 0.f;
        if (d < 32) {
            bool first = true;
            for (int i = 0; i < E; ++i) {
                const int idx = d * E + i;
                const float x = idx < D ? tree[idx] : 0.f;
                lane_sum = first ? x : __fadd_rn(lane_sum, x);
                first = false;
            }
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) lane_sum = __fadd_rn(lane_sum, __shfl_xor_sync(0xffffffffu, lane_sum, m));
            if (d == 0) tree[D] = lane_sum;      // one slot past the row
        }
        __syncthreads();
        const float total = tree[D];
        __syncthreads();
        return total;
    };

    const float norm = __fsqrt_rn(tree_sum(__fmul_rn(val, val)));
    const float inv_norm = (norm > 1e-8f) ? __fdiv_rn(1.0f, norm) : 0.0f;
    if (d < D) unit[d] = __fmul_rn(val, inv_norm);
    const int pw = (D * a.bits + 31) / 32;
    for (int w = d; w < pw; w += blockDim.x) words[w] = 0;
    __syncthreads();
    uint32_t idx = 0;
    float recon = 0.f;
    if (d < D) {
        const float *rot = a.rotation + (int64_t)d * D;
        float acc = 0.f;
        for (int j = 0; j < D; ++j) acc = __fadd_rn(acc, __fmul_rn(rot[j], unit[j]));
        float cal = 1.f;
        if (a.calib) {
            cal = a.calib[d];
            acc = __fdiv_rn(acc, cal);
        }
        const int levels_m1 = (1 << a.bits) - 1;
        for (int bd = 0; bd < levels_m1; ++bd) idx += (acc > a.boundaries[bd]) ? 1u : 0u;
        idx &= (uint32_t)levels_m1;
        const float cv = a.calib ? __fmul_rn(a.centroids[idx], cal) : a.centroids[idx];
        recon = __fmul_rn(cv, cv);
        const int bit = d * a.bits;
        const int w = bit >> 5, sh = bit & 31;
        atomicOr(&words[w], idx << sh);
        if (sh + a.bits > 32) atomicOr(&words[w + 1], idx >> (32 - sh));
    }
    const float recon_norm = __fsqrt_rn(tree_sum(recon));
    const int64_t t = a.pos + s;
    uint32_t *dst = a.packed + b * a.p_sb + h * a.p_sh + t * a.p_st;
    for (int w = d; w < pw; w += blockDim.x) dst[w] = words[w];
    if (d == 0) a.norms[b * a.n_sb + h * a.n_sh + t * a.n_st] = (recon_norm > 1e-8f) ? __fdiv_rn(norm, recon_norm) : norm;
}

// The calibration statistic on the dense path: thread d of a row's block adds its rotated value (computed
// exactly as turbo_encode_dense_kernel computes it) to the fixed-point sums of dimension d.
template <typename T>
__global__ void turbo_calib_stats_dense_kernel(TurboEncodeArgs a, int64_t total_rows, unsigned long long *sums) {
    extern __shared__ float s_f[];           // [D] unit row, [D + 1] tree scratch
    const int D = a.D;
    float *unit = s_f;
    float *tree = s_f + D;
    const int d = threadIdx.x;
    const int64_t row = blockIdx.x;
    if (row >= total_rows) return;
    int64_t r = row;
    const int s = (int)(r % a.S);
    r /= a.S;
    const int h = (int)(r % a.H);
    const int b = (int)(r / a.H);
    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss;
    const int E = (D + 31) / 32;
    const float val = d < D ? to_float<T>(src[(int64_t)d * a.s_sd]) : 0.f;
    if (d < D) tree[d] = __fmul_rn(val, val);
    __syncthreads();
    if (d < 32) {
        float lane_sum = 0.f;
        bool first = true;
        for (int i = 0; i < E; ++i) {
            const int idx = d * E + i;
            const float x = idx < D ? tree[idx] : 0.f;
            lane_sum = first ? x : __fadd_rn(lane_sum, x);
            first = false;
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) lane_sum = __fadd_rn(lane_sum, __shfl_xor_sync(0xffffffffu, lane_sum, m));
        if (d == 0) tree[D] = lane_sum;
    }
    __syncthreads();
    const float norm = __fsqrt_rn(tree[D]);
    const float inv_norm = (norm > 1e-8f) ? __fdiv_rn(1.0f, norm) : 0.0f;
    if (d < D) unit[d] = __fmul_rn(val, inv_norm);
    __syncthreads();
    if (d < D) {
        const float *rot = a.rotation + (int64_t)d * D;
        float acc = 0.f;
        for (int j = 0; j < D; ++j) acc = __fadd_rn(acc, __fmul_rn(rot[j], unit[j]));
        atomicAdd(&sums[d], (unsigned long long)__float2ll_rn(__fmul_rn(acc, 1073741824.0f)));
        atomicAdd(&sums[D + d], (unsigned long long)__float2ll_rn(__fmul_rn(__fmul_rn(acc, acc), 68719476736.0f)));
    }
}

// Fixed-point per-dimension sums of the rotated unit rows (see launch_turbo_calib_stats). One warp per
// row at a time, rows strided over the grid; a block folds its warps in shared memory and adds once
// per dimension to the global sums. The rotated values are computed exactly as turbo_encode_kernel
// computes the ones it quantises.
template <typename T, int E>
__global__ void __launch_bounds__(256)
turbo_calib_stats_kernel(TurboEncodeArgs a, int64_t total_rows, float inv_sqrt_dim, unsigned long long *sums) {
    constexpr int D = E * 32;
    __shared__ unsigned long long s_sum[2 * D];
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) s_sum[i] = 0ull;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    long long acc1[E], acc2[E];
#pragma unroll
    for (int i = 0; i < E; ++i) { acc1[i] = 0; acc2[i] = 0; }
    for (int64_t row = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); row < total_rows; row += (int64_t)gridDim.x * warps) {
        int64_t r = row;
        const int s = (int)(r % a.S);
        r /= a.S;
        const int h = (int)(r % a.H);
        const int b = (int)(r / a.H);
        const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + s * a.s_ss;
        float v[E];
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = to_float<T>(src[(int64_t)(lane * E + i) * a.s_sd]);
        float sq = __fmul_rn(v[0], v[0]);
#pragma unroll
        for (int i = 1; i < E; ++i) sq = __fadd_rn(sq, __fmul_rn(v[i], v[i]));
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, m));
        const float norm = __fsqrt_rn(sq);
        const float inv_norm = (norm > 1e-8f) ? __fdiv_rn(1.0f, norm) : 0.0f;
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = __fmul_rn(v[i], __fmul_rn(inv_norm, a.signs[lane * E + i]));
#pragma unroll
        for (int st = 1; st < E; st <<= 1) {
#pragma unroll
            for (int i = 0; i < E; ++i) {
                if ((i & st) == 0) {
                    const float lo = v[i], hi = v[i + st];
                    v[i] = __fadd_rn(lo, hi);
                    v[i + st] = __fsub_rn(lo, hi);
                }
            }
        }
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const float other = __shfl_xor_sync(0xffffffffu, v[i], m);
                v[i] = (lane & m) ? __fsub_rn(other, v[i]) : __fadd_rn(other, v[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const float rot = __fmul_rn(v[i], inv_sqrt_dim);
            acc1[i] += __float2ll_rn(__fmul_rn(rot, 1073741824.0f));                       // 2^30
            acc2[i] += __float2ll_rn(__fmul_rn(__fmul_rn(rot, rot), 68719476736.0f));      // 2^36
        }
    }
#pragma unroll
    for (int i = 0; i < E; ++i) {
        atomicAdd(&s_sum[lane * E + i], (unsigned long long)acc1[i]);
        atomicAdd(&s_sum[D + lane * E + i], (unsigned long long)acc2[i]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x)
        if (s_sum[i]) atomicAdd(&sums[i], s_sum[i]);
}

// E consecutive elements of a contiguous row in as few loads as their size allows. (Not through the read-only path: a kernel that
// starts under the tail of the one before reads what that one writes, if only after its wait.)
template <typename T, int E>
__device__ __forceinline__ void load_row_elems(const T *p, float (&v)[E]) {
    constexpr int BYTES = E * (int)sizeof(T);
    if constexpr (BYTES % 16 == 0) {
        uint4 raw[BYTES / 16];
#pragma unroll
        for (int i = 0; i < BYTES / 16; ++i) raw[i] = reinterpret_cast<const uint4 *>(p)[i];
        const T *e = reinterpret_cast<const T *>(raw);
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = to_float<T>(e[i]);
    } else if constexpr (BYTES == 8) {
        const uint2 raw = *reinterpret_cast<const uint2 *>(p);
        const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = to_float<T>(e[i]);
    } else if constexpr (BYTES == 4) {
        const uint32_t raw = *reinterpret_cast<const uint32_t *>(p);
        const T *e = reinterpret_cast<const T *>(&raw);
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = to_float<T>(e[i]);
    } else {
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = to_float<T>(p[i]);
    }
}

// The same encode for contiguous rows with E <= 8: vector loads, R rows per warp in flight, the
// boundary count as a binary search over a shared-memory copy when the boundaries ascend (`sorted`),
// the cross-lane butterfly as one fused multiply-add per value (x * (+-1) + other rounds once, like
// the add or subtract it replaces), and the packed words assembled by shuffles. Grid: x = chunks of
// consecutive tokens, y = head, z = batch (keys first, then values): a block works on one (tensor,
// batch, head). Arithmetic and reduction order are those of turbo_encode_kernel, so norms and codes
// are the same bits.
template <typename T, int E, int R>
__device__ __forceinline__ void turbo_encode_vec_body(const TurboEncodeArgs &a, int b, float inv_sqrt_dim, int sorted,
                                                      float *s_bnd) {
    const int lane = threadIdx.x & 31;
    const int bits = a.bits;
    const int levels_m1 = (1 << bits) - 1;
    // unused upper entries hold +inf, so a search of fixed depth 4 serves every bit width
    if (threadIdx.x < 15) s_bnd[threadIdx.x] = threadIdx.x < levels_m1 ? a.boundaries[threadIdx.x] : __int_as_float(0x7f800000);
    __syncthreads();
    const int h = blockIdx.y;
    const int s0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
    if (s0 >= a.S) return;  // whole warp
    const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + lane * E;
    uint32_t *packed = a.packed + b * a.p_sb + h * a.p_sh + a.pos * a.p_st;
    float *norms = a.norms + b * a.n_sb + h * a.n_sh + a.pos * a.n_st;

    float v[R][E];
    float sg[E];
    load_row_elems<float, E>(a.signs + lane * E, sg);
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int i = 0; i < E; ++i) v[r][i] = 0.f;
        if (s0 + r < a.S) load_row_elems<T, E>(src + (s0 + r) * a.s_ss, v[r]);
    }

    // L2 norm over the fixed reduction tree
    float sq[R], norm[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        sq[r] = __fmul_rn(v[r][0], v[r][0]);
#pragma unroll
        for (int i = 1; i < E; ++i) sq[r] = __fadd_rn(sq[r], __fmul_rn(v[r][i], v[r][i]));
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1)
#pragma unroll
        for (int r = 0; r < R; ++r) sq[r] = __fadd_rn(sq[r], __shfl_xor_sync(0xffffffffu, sq[r], m));
#pragma unroll
    for (int r = 0; r < R; ++r) {
        norm[r] = __fsqrt_rn(sq[r]);
        const float inv_norm = (norm[r] > 1e-8f) ? __frcp_rn(norm[r]) : 0.0f;
#pragma unroll
        for (int i = 0; i < E; ++i) v[r][i] = __fmul_rn(v[r][i], __fmul_rn(inv_norm, sg[i]));
        // in-lane butterfly stages
#pragma unroll
        for (int st = 1; st < E; st <<= 1)
#pragma unroll
            for (int i = 0; i < E; ++i)
                if ((i & st) == 0) {
                    const float lo = v[r][i], hi = v[r][i + st];
                    v[r][i] = __fadd_rn(lo, hi);
                    v[r][i + st] = __fsub_rn(lo, hi);
                }
    }
    // cross-lane stages: the upper lane of a pair takes other - own, the lower one other + own
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const float sign = (lane & m) ? -1.f : 1.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int i = 0; i < E; ++i) v[r][i] = __fmaf_rn(v[r][i], sign, __shfl_xor_sync(0xffffffffu, v[r][i], m));
    }

    const int nb = E * bits;               // bits per lane = words per row (<= 32)
#pragma unroll
    for (int r = 0; r < R; ++r) {
        uint32_t chunk = 0;
#pragma unroll
        for (int i = E - 1; i >= 0; --i) {
            const float rotated = __fmul_rn(v[r][i], inv_sqrt_dim);
            uint32_t idx = 0;
            if (sorted) {
#pragma unroll
                for (int step = 8; step >= 1; step >>= 1)
                    if (rotated > s_bnd[idx + step - 1]) idx += step;
            } else {
                for (int bd = 0; bd < levels_m1; ++bd) idx += (rotated > s_bnd[bd]) ? 1u : 0u;
            }
            chunk = (chunk << bits) | idx;
        }
        const bool live = s0 + r < a.S;
        uint32_t *dst = packed + (s0 + r) * a.p_st;
        if (nb == 32) {
            if (live) dst[lane] = chunk;
        } else if ((nb & (nb - 1)) == 0) {
            // 32 / nb lanes per word: fold neighbours in with a shuffle tree
            uint32_t word = chunk;
            for (int span = 1, sh = nb; sh < 32; span <<= 1, sh <<= 1)
                word |= __shfl_down_sync(0xffffffffu, word, span) << sh;
            const int lpw = 32 / nb;
            if (live && (lane & (lpw - 1)) == 0) dst[lane / lpw] = word;
        } else if (nb == 12) {
            // eight lanes hold 96 bits = three words: pairs (24 bits), quads (48 bits), then the octet
            const uint32_t pair = chunk | (__shfl_down_sync(0xffffffffu, chunk, 1) << 12);
            const uint64_t quad = (uint64_t)pair | ((uint64_t)__shfl_down_sync(0xffffffffu, pair, 2) << 24);
            const uint32_t hi_lo = __shfl_down_sync(0xffffffffu, (uint32_t)quad, 4);
            const uint32_t hi_hi = __shfl_down_sync(0xffffffffu, (uint32_t)(quad >> 32), 4);
            const uint64_t upper = (uint64_t)hi_lo | ((uint64_t)hi_hi << 32);   // bits 48..95 of the octet
            if (live && (lane & 7) == 0) {
                uint32_t *w = dst + (lane >> 3) * 3;
                w[0] = (uint32_t)quad;
                w[1] = (uint32_t)(quad >> 32) | (uint32_t)(upper << 16);
                w[2] = (uint32_t)(upper >> 16);
            }
        } else {
            // lane j holds bits [j nb, (j + 1) nb) of the row; lane w gathers word w
            const int j0 = (32 * lane) / nb;
            uint32_t word = 0;
            for (int k = 0; k <= 32 / nb + 1; ++k) {
                const int j = j0 + k;
                const uint32_t c = __shfl_sync(0xffffffffu, chunk, j & 31);
                const int lo = j * nb - 32 * lane;  // where lane j's chunk starts inside this word
                if (j < 32 && lo < 32) word |= lo >= 0 ? c << lo : c >> (-lo);
            }
            if (live && lane < nb) dst[lane] = word;
        }
        if (live && lane == 0) norms[(s0 + r) * a.n_st] = norm[r];
    }
}

template <typename T, int E, int R>
__global__ void __launch_bounds__(256)
turbo_encode_vec_kernel(TurboEncodeArgs ka, TurboEncodeArgs va, float inv_sqrt_dim, int sorted) {
    dev::pdl_wait();
    dev::pdl_trigger();
    __shared__ float s_bnd[16];
    // keys and values share B, H and S; the branch is uniform over the block
    if ((int)blockIdx.z >= ka.B) turbo_encode_vec_body<T, E, R>(va, (int)blockIdx.z - ka.B, inv_sqrt_dim, sorted, s_bnd);
    else turbo_encode_vec_body<T, E, R>(ka, (int)blockIdx.z, inv_sqrt_dim, sorted, s_bnd);
}

// ---------------------------------------------------------------------
// The same encode for many rows: 16 dims per lane, so a warp holds 32 / (D / 16) rows. Issue-bound like the
// one-row-per-warp form above, with a third of its instructions per row: the Walsh-Hadamard stages that pair
// dims less than 16 apart need no shuffle, the shuffles left carry several rows each, a lane's codes fill whole
// words, and a code is found with one table read and one subtraction, whose sign counts the cell's boundary: a monotone
// map (bits of one fused multiply-add) sends the value to one of 256 cells that hold at most one boundary each, so the
// boundaries of lower cells are passed and those of higher cells are not, whatever the rounding of the map. The cells
// span [-1, 1], so a coordinate of a unit vector needs no clamp; other codebooks, calibrated rows and signs that are
// not +-1 clamp. Signs of one turn the sign bits of the packed elements. A block walks neighbouring row groups, so
// that places move by strides, with the next row's loads in flight.
// Sums run over the fixed tree (D / 32 neighbouring dims left to right, then the exchanges 16, 8, 4, 2, 1, of
// which the last ones stay inside a lane), so norms and codes are the bits of turbo_encode_kernel.
// 131072 rows of D 128 bf16, 4 bits (27 instructions an element, 66 % of the issue rate): 22 us; 30 with 64 clamped
// cells, products by signs and a place computed per row. Keys with the calibration statistic (128 registers, two
// blocks an SM): 34 us, 41 before.
// ---------------------------------------------------------------------
constexpr int CELLS = 256;
struct EncodeCells {
    float scale, shift;      // cell = floor(x * scale) + a constant: bits 7 .. 14 of fma(x, scale, shift)
    int32_t clamp;           // 0: the cells span [-1, 1], which no coordinate of a unit vector leaves
};
constexpr float CELL_MAGIC = 98304.f;      // 1.5 * 2^16: a unit in the last place is 2^-7
constexpr float CELL_TOP = CELL_MAGIC + 254.9921875f;
constexpr float SUM_MAGIC = 12582912.f;    // 1.5 * 2^23: a unit in the last place is 1

// The cell of a value (the host and the kernels agree to the bit: one fused multiply-add, exact comparisons).
__host__ __device__ inline int cell_of(const EncodeCells &c, float x) {
    const float u = fminf(fmaxf(fmaf(x, c.scale, c.shift), CELL_MAGIC), CELL_TOP);
#ifdef __CUDA_ARCH__
    const uint32_t bits = __float_as_uint(u);
#else
    uint32_t bits;
    std::memcpy(&bits, &u, sizeof bits);
#endif
    return (int)((bits >> 7) & (CELLS - 1));
}

// No two boundaries in a cell, and none in the first and last one, where values that are no numbers go.
bool cells_hold(const TurboEncodeArgs &a, const EncodeCells &c) {
    int before = 0;
    for (int i = 0; i < (1 << a.bits) - 1; ++i) {
        const int at = cell_of(c, a.boundaries[i]);
        if (at <= before || at >= CELLS - 1) return false;
        before = at;
    }
    return true;
}

// Cell `i` of a codebook's boundaries: the boundary in it (+inf: none) and the number of boundaries below it. The last cell
// holds what is no number, all of whose bits are set, and no number: nothing is passed.
template <int BITS>
__device__ __forceinline__ float2 make_cell(const TurboEncodeArgs &a, const EncodeCells &c, int i) {
    float bound = INFINITY;
    uint32_t below = 0;
#pragma unroll
    for (int j = 0; j < (1 << BITS) - 1; ++j) {
        const int at = cell_of(c, a.boundaries[j]);
        below += at < i ? 1u : 0u;
        if (at == i) bound = a.boundaries[j];
    }
    return make_float2(bound, __uint_as_float(i == CELLS - 1 ? 0u : below));
}

// Cells that need no clamp where the boundaries lie within (-1, 1) and no two share a cell, else cells between the outer boundaries.
bool build_cells(const TurboEncodeArgs &a, EncodeCells *c) {
    const int n = (1 << a.bits) - 1;
    const float lo = a.boundaries[0], hi = a.boundaries[n - 1];
    for (int i = 0; i < n; ++i)
        if (!(fabsf(a.boundaries[i]) < 1e4f) || (i && !(a.boundaries[i - 1] < a.boundaries[i]))) return false;
    c->clamp = 0;
    c->scale = 126.f;
    c->shift = CELL_MAGIC + 128.f;
    if (!a.calib && lo > -1.f && hi < 1.f && cells_hold(a, *c)) return true;
    c->clamp = 1;
    c->scale = n == 1 ? 1.f : 253.f / (hi - lo);
    if (!(c->scale < 1e6f)) return false;
    c->shift = CELL_MAGIC + 1.5f - rintf(lo * c->scale);
    return cells_hold(a, *c);
}

template <int D> __device__ __forceinline__ float tree_sum(float (&p)[16 / (D / 32)]) {
    // p: sums of this lane's runs of D / 32 dims (neighbouring runs of the 32-run tree)
    constexpr int RUNS = 16 / (D / 32);
#pragma unroll
    for (int m = 16; m >= RUNS; m >>= 1)
#pragma unroll
        for (int j = 0; j < RUNS; ++j) p[j] = __fadd_rn(p[j], __shfl_xor_sync(0xffffffffu, p[j], m / RUNS));
#pragma unroll
    for (int m = RUNS / 2; m >= 1; m >>= 1)
#pragma unroll
        for (int j = 0; j < RUNS; ++j)
            if ((j & m) == 0) p[j] = __fadd_rn(p[j], p[j + m]);
    return p[0];
}

// 16 neighbouring elements of a row as they lie in memory, and times their signs. Signs of one turn over the sign bits
// (`flip`: the bits to turn), which is the product to the bit.
template <typename T> struct RawRun {
    static constexpr int WORDS = 16 * sizeof(T) / 4;
    uint32_t w[WORDS];
    __device__ __forceinline__ void load(const T *src) {
#pragma unroll
        for (int i = 0; i < WORDS / 4; ++i) {
            const uint4 x = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint32_t *>(src) + 4 * i);
            w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
        }
    }
    __device__ __forceinline__ void signed_by(const RawRun &flip, float (&v)[16]) const {
#pragma unroll
        for (int i = 0; i < WORDS; ++i) {
            const uint32_t x = w[i] ^ flip.w[i];
            if constexpr (std::is_same<T, float>::value) {
                v[i] = __uint_as_float(x);
            } else if constexpr (std::is_same<T, __half>::value) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&x));
                v[2 * i] = f.x; v[2 * i + 1] = f.y;
            } else {
                v[2 * i] = __uint_as_float(x << 16);
                v[2 * i + 1] = __uint_as_float(x & 0xFFFF0000u);
            }
        }
    }
};

// This lane's dims `v` of a row, signs applied, rotated in place (before 1 / sqrt(D)); the row's norm. SCALED: `scale_by` may
// point at the magnitudes of signs that are not one.
template <int D, bool SCALED>
__device__ __forceinline__ float rotate_wide(int l, const float *scale_by, float (&v)[16]) {
    constexpr int E = D / 32, RUNS = 16 / E, LPR = D / 16;
    using namespace dev;
    uint64_t x[8];                                   // dims 2i and 2i + 1
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = pack_f2(v[2 * i], v[2 * i + 1]);
    float sq[16], p[RUNS];
#pragma unroll
    for (int i = 0; i < 8; ++i) unpack_f2(mul_f2(x[i], x[i]), sq[2 * i], sq[2 * i + 1]);
#pragma unroll
    for (int j = 0; j < RUNS; ++j) {
        p[j] = sq[j * E];
#pragma unroll
        for (int i = 1; i < E; ++i) p[j] = __fadd_rn(p[j], sq[j * E + i]);
    }
    const float norm = __fsqrt_rn(tree_sum<D>(p));
    const float inv_norm = (norm > 1e-8f) ? __frcp_rn(norm) : 0.0f;
    const uint64_t inv2 = pack_f2(inv_norm, inv_norm), minus = pack_f2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint64_t f = inv2;
        if (SCALED && scale_by) f = mul_f2(inv2, pack_f2(fabsf(scale_by[2 * i]), fabsf(scale_by[2 * i + 1])));
        x[i] = mul_f2(x[i], f);
        float lo, hi;
        unpack_f2(x[i], lo, hi);
        x[i] = pack_f2(__fadd_rn(lo, hi), __fsub_rn(lo, hi));
    }
#pragma unroll
    for (int st = 1; st < 8; st <<= 1)               // (dims 2 st apart)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((i & st) == 0) {
                const uint64_t lo = x[i], hi = x[i + st];
                x[i] = add_f2(lo, hi);
                x[i + st] = fma_f2(hi, minus, lo);
            }
#pragma unroll
    for (int m = 1; m < LPR; m <<= 1) {
        const float sign = (l & m) ? -1.f : 1.f;
        const uint64_t sign2 = pack_f2(sign, sign);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float lo, hi;
            unpack_f2(x[i], lo, hi);
            x[i] = fma_f2(x[i], sign2, pack_f2(__shfl_xor_sync(0xffffffffu, lo, m), __shfl_xor_sync(0xffffffffu, hi, m)));
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) unpack_f2(x[i], v[2 * i], v[2 * i + 1]);
    return norm;
}

// Where the rows of one flat row group are: 8 warps x 32 / (D / 16) consecutive tokens of one (batch, head).
template <int D> struct WideRows {
    static constexpr int LPR = D / 16, RPW = 32 / LPR, GROUP = 8 * RPW;
};

// One row: 16 of its dims, its words to `dst`, its norm to `norm_at`. CLAMP: the value's cell is brought into
// the table first. `lane_at`: where this lane's copy of a cell lies in its 128 bytes.
template <typename T, int D, int BITS, bool CAL, bool CLAMP>
__device__ __forceinline__ void turbo_encode_wide_body(const TurboEncodeArgs &a, const EncodeCells &cells, const unsigned char *cells_mem, uint32_t lane_at,
                                                       const RawRun<T> &raw, const RawRun<T> &flip, const float *scale_by, uint32_t *dst, float *norm_at, bool live,
                                                       int l, float inv_sqrt_dim, float (&rot)[16]) {
    constexpr int E = D / 32, RUNS = 16 / E;
    float (&v)[16] = rot;
    raw.signed_by(flip, v);
    const float norm = rotate_wide<D, CLAMP>(l, scale_by, v);
    float place[16];                                 // cell of a value, before it is brought into the table
    {
        using namespace dev;
        const uint64_t dim2 = pack_f2(inv_sqrt_dim, inv_sqrt_dim), scale2 = pack_f2(cells.scale, cells.scale), shift2 = pack_f2(cells.shift, cells.shift);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const uint64_t x = mul_f2(pack_f2(v[i], v[i + 1]), dim2);
            unpack_f2(x, v[i], v[i + 1]);
            if (!CAL) unpack_f2(fma_f2(x, scale2, shift2), place[i], place[i + 1]);
        }
    }
    float stored = norm;
    uint32_t w[2] = {0u, 0u};
    constexpr int PER = BITS > 2 ? 8 : 16;           // codes per word here (3 bits: joined below)
    float p[RUNS];
#pragma unroll
    for (int i = 15; i >= 0; --i) {
        float x = v[i], cal = 1.f;
        if (CAL) {
            cal = a.calib[l * 16 + i];
            x = __fdiv_rn(x, cal);
        }
        float u = CAL ? __fmaf_rn(x, cells.scale, cells.shift) : place[i];
        if (CLAMP) u = fminf(fmaxf(u, CELL_MAGIC), CELL_TOP);
        const float2 e = *reinterpret_cast<const float2 *>(cells_mem + ((__float_as_uint(u) & ((CELLS - 1) << 7)) | lane_at));
        const float bound = e.x;
        const uint32_t below = __float_as_uint(e.y);
        uint32_t &word = w[i / PER];
        if (CAL) {
            const uint32_t idx = below + (x > bound ? 1u : 0u);
            word = (word << BITS) | idx;
            const float cv = __fmul_rn(a.centroids[idx], cal);
            v[i] = __fmul_rn(cv, cv);
        } else {
            // the sign of the difference: set where x is above the boundary (equal: +0; no number, no boundary: clear)
            word = (word << BITS) + below + (__float_as_uint(__fsub_rn(bound, x)) >> 31);
        }
    }
    if (CAL) {
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            p[j] = v[j * E];
#pragma unroll
            for (int i = 1; i < E; ++i) p[j] = __fadd_rn(p[j], v[j * E + i]);
        }
        const float recon = __fsqrt_rn(tree_sum<D>(p));
        if (recon > 1e-8f) stored = __fdiv_rn(norm, recon);
    }
    if constexpr (BITS == 4) {
        if (live) *(uint2 *)dst = make_uint2(w[0], w[1]);
    } else if constexpr (BITS == 2) {
        if (live) *dst = w[0];
    } else if constexpr (BITS == 3) {
        // two lanes hold 96 bits: the even one writes the first two words, the odd one the third
        const uint32_t lo = w[0] | (w[1] << 24), hi = w[1] >> 8, odd_lo = __shfl_down_sync(0xffffffffu, lo, 1);
        if (live) {
            if (l & 1) {
                *dst = (lo >> 16) | (hi << 16);
            } else {
                dst[0] = lo;
                dst[1] = hi | (odd_lo << 16);
            }
        }
    } else {
        const uint32_t other = __shfl_down_sync(0xffffffffu, w[0], 1);
        if (live && !(l & 1)) *dst = w[0] | (other << 16);
    }
    if (live && l == 0) *norm_at = stored;
}
// Words of a row in front of those that lane l writes.
template <int BITS> __device__ __forceinline__ int wide_word(int l) {
    return BITS == 4 ? 2 * l : BITS == 2 ? l : BITS == 3 ? (l >> 1) * 3 + (l & 1) * 2 : l >> 1;
}

// The calibration statistic of the keys, taken from the rotated rows while they are encoded (uncalibrated; when the
// statistic asks for a calibration, which keys without outlier channels do not, they are encoded again). A lane adds
// its 16 dims of every row it meets. The fixed-point integers reach 2^30 and 2^36; conversions run on a slow pipe, so
// each is taken as top * 2^k + rest, both parts rounded by an addition of 1.5 * 2^23 whose low bits are the
// integer (top and rest are exact: a power of two apart and one fused multiply-add; 2^k is even, so a tie of the
// rest rounds like a tie of the whole). The parts are summed modulo 2^32 with the constant left in and taken off at
// the end. The lanes of a dim meet by shuffles and the warps in shared memory without atomics (64-bit shared
// atomics are compare-and-swap loops), then one global add per dim and block.
struct CalibSums {
    uint32_t top[2][16], rest[2][16], rows;
    __device__ __forceinline__ void clear() {
        rows = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) top[0][i] = top[1][i] = rest[0][i] = rest[1][i] = 0u;
    }
    __device__ __forceinline__ void add_row(const float (&rot)[16]) {
        ++rows;
        using namespace dev;
        auto both = [](float x) { return pack_f2(x, x); };
        auto add = [&](int w, int i, uint64_t y, float down, float up) {
            const uint64_t t = fma_f2(y, both(down), both(SUM_MAGIC));
            const uint64_t r = add_f2(fma_f2(add_f2(t, both(-SUM_MAGIC)), both(up), y), both(SUM_MAGIC));
            float t0, t1, r0, r1;
            unpack_f2(t, t0, t1);
            unpack_f2(r, r0, r1);
            top[w][i] += __float_as_uint(t0);
            top[w][i + 1] += __float_as_uint(t1);
            rest[w][i] += __float_as_uint(r0);
            rest[w][i + 1] += __float_as_uint(r1);
        };
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const uint64_t x = pack_f2(rot[i], rot[i + 1]);
            add(0, i, mul_f2(x, both(1073741824.0f)), 6.103515625e-5f, -16384.f);                  // 2^30, parts of 2^14
            add(1, i, mul_f2(mul_f2(x, x), both(68719476736.0f)), 1.52587890625e-5f, -65536.f);    // 2^36, parts of 2^16
        }
    }
};
constexpr int CALIB_ROWS = 1024;      // rows a lane may add up before a part could pass 2^31

// y = keys or values; the row groups of a tensor are dealt to the blocks of x, so a launch is one wave.
template <typename T, int D, int KB, int VB, bool STATS>
__global__ void __launch_bounds__(256, STATS ? 2 : 3)
turbo_encode_wide_kernel(const __grid_constant__ TurboEncodeArgs ka, const __grid_constant__ TurboEncodeArgs va,
                         const __grid_constant__ EncodeCells kc, const __grid_constant__ EncodeCells vc, int groups, int groups_per_plane,
                         float inv_sqrt_dim, unsigned long long *sums) {
    using W = WideRows<D>;
    __shared__ __align__(128) float2 table[CELLS * 16];
    const bool is_v = blockIdx.y != 0;
    const TurboEncodeArgs &a = is_v ? va : ka;
    const int lane = threadIdx.x & 31, l = lane % W::LPR, warp = threadIdx.x >> 5;
    {   // a thread takes a cell; the lanes start at different copies of theirs, so that they meet no bank twice
        static_assert(CELLS == 256, "a thread a cell");
        const float2 c = is_v ? make_cell<VB>(va, vc, threadIdx.x) : make_cell<KB>(ka, kc, threadIdx.x);
        const float4 cc = make_float4(c.x, c.y, c.x, c.y);
#pragma unroll
        for (int j = 0; j < 8; ++j) reinterpret_cast<float4 *>(table)[threadIdx.x * 8 + ((j + lane) & 7)] = cc;
    }
    dev::pdl_wait();      // the cells came from the parameters
    dev::pdl_trigger();
    RawRun<T> flip;
    RawRun<float> signs;
    signs.load(a.signs + l * 16);
    bool unit = true;
#pragma unroll
    for (int i = 0; i < RawRun<T>::WORDS; ++i) flip.w[i] = 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t sg = signs.w[i];
        unit = unit && (sg & 0x7FFFFFFFu) == 0x3F800000u;
        if (sizeof(T) == 4) flip.w[i % RawRun<T>::WORDS] = sg & 0x80000000u;
        else flip.w[i / 2] |= (sg >> 31) << ((i & 1) ? 31 : 15);
    }
    unit = __all_sync(0xffffffffu, unit);
    __syncthreads();
    const unsigned char *cells_mem = reinterpret_cast<const unsigned char *>(table);
    const uint32_t lane_at = (lane & 15) * 8;            // a half warp meets no bank twice
    CalibSums cs;
    if (STATS) cs.clear();
    const bool cal = !is_v && !STATS && ka.calib, clamp = (is_v ? vc.clamp : kc.clamp) || !unit;
    const float *scale_by = unit ? nullptr : a.signs + l * 16;
    // Row groups in runs of neighbours: the place of a group is found once a plane, then moved on by a stride.
    const int share = groups / (int)gridDim.x, extra = groups % (int)gridDim.x, first = blockIdx.x * share + min((int)blockIdx.x, extra);
    int left = share + ((int)blockIdx.x < extra), plane = first / groups_per_plane, in = first % groups_per_plane;
    while (left > 0) {
        const int h = plane % a.H, b = plane / a.H, n = min(left, groups_per_plane - in);
        int s = in * W::GROUP + warp * W::RPW + lane / W::LPR;
        const T *src = (const T *)a.src + b * a.s_sb + h * a.s_sh + (int64_t)s * a.s_ss + l * 16;
        uint32_t *dst = a.packed + b * a.p_sb + h * a.p_sh + (a.pos + s) * a.p_st + (is_v ? wide_word<VB>(l) : wide_word<KB>(l));
        float *norm_at = a.norms + b * a.n_sb + h * a.n_sh + (a.pos + s) * a.n_st;
        const int64_t src_step = W::GROUP * a.s_ss, dst_step = W::GROUP * a.p_st, norm_step = W::GROUP * a.n_st;
        // the row after this one is on its way while this one is encoded (the sums leave no registers for it)
        constexpr bool AHEAD = !STATS && sizeof(T) == 2;
        auto row = [&](const T *at, int t) { return t < a.S ? at : at - (int64_t)(t - (a.S - 1)) * a.s_ss; };
        RawRun<T> raw, next;
        if (AHEAD) next.load(row(src, s));
        for (int k = 0; k < n; ++k, s += W::GROUP, src += src_step, dst += dst_step, norm_at += norm_step) {
            if (s - lane / W::LPR >= a.S) break;      // whole warp
            const bool live = s < a.S;
            if (AHEAD) raw = next;
            else raw.load(row(src, s));
            if (AHEAD && k + 1 < n) next.load(row(src + src_step, s + W::GROUP));
            float rot[16];
#define KVC_EWROW(BITS, CAL, CLAMP, A, C) turbo_encode_wide_body<T, D, BITS, CAL, CLAMP>(A, C, cells_mem, lane_at, raw, flip, scale_by, dst, norm_at, live, l, inv_sqrt_dim, rot)
            if (is_v) {
                if (clamp) KVC_EWROW(VB, false, true, va, vc);
                else KVC_EWROW(VB, false, false, va, vc);
            } else if (cal) KVC_EWROW(KB, true, true, ka, kc);
            else if (clamp) KVC_EWROW(KB, false, true, ka, kc);
            else KVC_EWROW(KB, false, false, ka, kc);
#undef KVC_EWROW
            if (STATS && live) cs.add_row(rot);
        }
        left -= n;
        in = 0;
        ++plane;
    }
    if constexpr (STATS) {
        long long(*part)[D] = (long long(*)[D])table;      // [warps at a time][D]: the cells are no longer read
        constexpr int AT_ONCE = (int)sizeof(table) / (D * 8) < 8 ? (int)sizeof(table) / (D * 8) : 8;
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            long long mine[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                mine[i] = ((long long)(int32_t)(cs.top[w][i] - cs.rows * 0x4B400000u) << (w ? 16 : 14)) + (int32_t)(cs.rest[w][i] - cs.rows * 0x4B400000u);
#pragma unroll
                for (int m = W::LPR; m < 32; m <<= 1) mine[i] += __shfl_xor_sync(0xffffffffu, mine[i], m);
            }
            long long total = 0;
            for (int w0 = 0; w0 < 8; w0 += AT_ONCE) {
                __syncthreads();
                if (warp >= w0 && warp < w0 + AT_ONCE && lane < W::LPR)
#pragma unroll
                    for (int i = 0; i < 16; ++i) part[warp - w0][l * 16 + i] = mine[i];
                __syncthreads();
                if ((int)threadIdx.x < D)
#pragma unroll
                    for (int k = 0; k < AT_ONCE; ++k) total += part[k][threadIdx.x];
            }
            if ((int)threadIdx.x < D && total) atomicAdd(&sums[w * D + threadIdx.x], (unsigned long long)total);
        }
    }
}

// Rows as the wide kernels read them: 16 dims from a 16-byte boundary on, words in pairs.
bool encode_wide_ok(const TurboEncodeArgs &a) {
    if (a.D != 64 && a.D != 128 && a.D != 256) return false;
    const int64_t vec = 16 / (int64_t)dtype_size(a.dtype);
    if (a.s_sd != 1 || a.s_sb % vec || a.s_sh % vec || a.s_ss % vec) return false;
    if ((reinterpret_cast<uintptr_t>(a.src) & 15) || (reinterpret_cast<uintptr_t>(a.signs) & 15)) return false;
    if (a.bits == 4 && ((reinterpret_cast<uintptr_t>(a.packed) & 7) || a.p_sb % 2 || a.p_sh % 2 || a.p_st % 2)) return false;
    return !a.rotation;
}

template <typename T, int D, int KB, int VB, bool STATS>
bool launch_encode_wide(const TurboEncodeArgs &k, const TurboEncodeArgs &v, bool have_v, const EncodeCells &kc, const EncodeCells &vc,
                        unsigned long long *sums, cudaStream_t stream) {
    auto kernel = turbo_encode_wide_kernel<T, D, KB, VB, STATS>;
    static int resident = 0;
    if (!resident) {
        int n = 0;
        KVC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0));
        resident = std::max(1, n);
    }
    const int64_t per_plane = (k.S + WideRows<D>::GROUP - 1) / WideRows<D>::GROUP, groups = per_plane * k.H * k.B;
    if (groups > (int64_t)1 << 30) return false;
    const int64_t slots = std::max<int64_t>(1, (int64_t)sm_count(current_device()) * resident / (have_v ? 2 : 1));
    if (STATS && (groups + slots - 1) / slots > CALIB_ROWS) return false;
    KVC_CUDA(launch_pdl(kernel, dim3((unsigned)std::min(groups, slots), have_v ? 2 : 1), dim3(256), 0, stream, k, v, kc, vc, (int)groups, (int)per_plane, 1.0f / sqrtf((float)D), sums));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    return true;
}

// From 16 rows per head on: below, a warp would hold mostly empty rows and the one-row form has the shorter chain.
// With `sums` (keys alone, uncalibrated) the calibration statistic is added up as well.
template <typename T>
bool encode_wide(const TurboEncodeArgs &k, const TurboEncodeArgs &v, bool have_v, unsigned long long *sums, cudaStream_t stream) {
    if (k.S < 16 || !encode_wide_ok(k) || (have_v && !encode_wide_ok(v))) return false;
    if (have_v && (k.B != v.B || k.H != v.H || k.S != v.S || v.calib)) return false;
    static thread_local EncodeCells kc, vc;
    if (!build_cells(k, &kc) || (have_v && !build_cells(v, &vc))) return false;
#define KVC_EWB(DD, KB, VB)                                                                                          \
    if (k.D == DD && k.bits == KB && (!have_v || v.bits == VB) && !sums)                                             \
        return launch_encode_wide<T, DD, KB, VB, false>(k, v, have_v, kc, vc, nullptr, stream);
#define KVC_EWS(DD, KB)                                                                                              \
    if (k.D == DD && k.bits == KB && sums) return launch_encode_wide<T, DD, KB, KB, true>(k, k, false, kc, kc, sums, stream);
#define KVC_EW(DD) KVC_EWB(DD, 4, 4) KVC_EWB(DD, 3, 3) KVC_EWB(DD, 2, 2) KVC_EWB(DD, 3, 4) KVC_EWB(DD, 4, 2) KVC_EWB(DD, 1, 1) \
    KVC_EWS(DD, 4) KVC_EWS(DD, 3) KVC_EWS(DD, 2) KVC_EWS(DD, 1)
    KVC_EW(64) KVC_EW(128) KVC_EW(256)
#undef KVC_EW
#undef KVC_EWS
#undef KVC_EWB
    return false;
}

// The rows of a list of caches of one shape in one launch: z = (layer, K or V, batch).
struct EncodeList {
    int32_t tensors;
    TurboEncodeArgs a[KVC_LIST_MAX][2];
};
template <typename T, int E>
__global__ void __launch_bounds__(256) turbo_encode_list_kernel(const __grid_constant__ EncodeList l, float inv_sqrt_dim, int sorted) {
    dev::pdl_wait();
    dev::pdl_trigger();
    __shared__ float s_bnd[16];
    const int B = l.a[0][0].B, b = blockIdx.z % B, w = blockIdx.z / B;
    turbo_encode_vec_body<T, E, 1>(l.a[w / l.tensors][w % l.tensors], b, inv_sqrt_dim, sorted, s_bnd);
}

template <int E> bool encode_vec_ok(const TurboEncodeArgs &a) {
    if (a.s_sd != 1 || a.s_sb % E || a.s_sh % E || a.s_ss % E) return false;
    return (reinterpret_cast<uintptr_t>(a.src) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.signs) & 15) == 0;
}

bool boundaries_ascend(const TurboEncodeArgs &a) {
    for (int i = 0; i + 2 < (1 << a.bits); ++i)
        if (!(a.boundaries[i] <= a.boundaries[i + 1])) return false;
    return true;
}

template <typename T, int E>
bool encode_list(const TurboEncodeArgs *k, const TurboEncodeArgs *v, int n, cudaStream_t stream) {
    static thread_local EncodeList l;
    const TurboEncodeArgs &k0 = k[0];
    l.tensors = v ? 2 : 1;
    bool sorted = true;
    for (int i = 0; i < n; ++i)
        for (int w = 0; w < l.tensors; ++w) {
            const TurboEncodeArgs &a = w ? v[i] : k[i];
            if (a.B != k0.B || a.H != k0.H || a.S != k0.S || a.D != k0.D || a.dtype != k0.dtype || a.calib || a.rotation ||
                a.bits < 1 || a.bits > 4 || !encode_vec_ok<E>(a))
                return false;
            sorted = sorted && boundaries_ascend(a);
            l.a[i][w] = a;
        }
    const int64_t z = (int64_t)n * l.tensors * k0.B;
    if (k0.H > 65535 || z > 65535) return false;
    const int vw = std::max(1, std::min(8, k0.S));
    const dim3 grid((unsigned)((k0.S + vw - 1) / vw), (unsigned)k0.H, (unsigned)z);
    KVC_CUDA(launch_pdl(turbo_encode_list_kernel<T, E>, grid, dim3(vw * 32), 0, stream, l, 1.0f / sqrtf((float)k0.D), sorted ? 1 : 0));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    return true;
}

template <typename T>
void turbo_dispatch(const TurboEncodeArgs &k, const TurboEncodeArgs &v, bool have_v, cudaStream_t stream) {
    const int64_t k_rows = (int64_t)k.B * k.H * k.S;
    const int64_t v_rows = have_v ? (int64_t)v.B * v.H * v.S : 0;
    const int64_t total = k_rows + v_rows;
    const int warps = 4;
    const unsigned blocks = (unsigned)((total + warps - 1) / warps);
    const size_t smem = warps * ((1024 * 4 + 31) / 32) * sizeof(uint32_t);
    const float inv_sqrt_dim = 1.0f / sqrtf((float)k.D);
    const int E = k.D / 32;
    auto vec_ok = [&](const TurboEncodeArgs &a) {
        if (a.s_sd != 1 || a.s_sb % E || a.s_sh % E || a.s_ss % E) return false;
        return (reinterpret_cast<uintptr_t>(a.src) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.signs) & 15) == 0;
    };
    auto ascending = [](const TurboEncodeArgs &a) {
        for (int i = 0; i + 2 < (1 << a.bits); ++i)
            if (!(a.boundaries[i] <= a.boundaries[i + 1])) return false;
        return true;
    };
    const bool same_dims = !have_v || (k.B == v.B && k.H == v.H && k.S == v.S);
    if (encode_wide<T>(k, v, have_v, nullptr, stream)) return;
    const bool calibrated = k.calib || (have_v && v.calib);   // few calibrated rows: the generic kernel
    if (!calibrated && E <= 8 && same_dims && vec_ok(k) && (!have_v || vec_ok(v)) && k.H <= 65535 && 2 * (int64_t)k.B <= 65535) {
        const int sorted = ascending(k) && (!have_v || ascending(v)) ? 1 : 0;
        const bool deep = k.S >= 16;
        const int rpw = deep ? 2 : 1;
        const int vw = std::max(1, std::min(8, (k.S + rpw - 1) / rpw));
        const dim3 grid((unsigned)((k.S + vw * rpw - 1) / (vw * rpw)), (unsigned)k.H, (unsigned)(k.B * (have_v ? 2 : 1)));
#define KVC_TV(EE)                                                                                        \
    do {                                                                                                  \
        if (deep) KVC_CUDA(launch_pdl(turbo_encode_vec_kernel<T, EE, 2>, grid, dim3(vw * 32), 0, stream, k, v, inv_sqrt_dim, sorted)); \
        else KVC_CUDA(launch_pdl(turbo_encode_vec_kernel<T, EE, 1>, grid, dim3(vw * 32), 0, stream, k, v, inv_sqrt_dim, sorted));      \
    } while (0)
        switch (E) {
            case 1: KVC_TV(1); break;
            case 2: KVC_TV(2); break;
            case 4: KVC_TV(4); break;
            default: KVC_TV(8); break;
        }
#undef KVC_TV
        KVC_CUDA(cudaGetLastError());
        ++g_launch_count;
        return;
    }
#define KVC_TE(EE)                                                                               \
    KVC_CUDA(launch_pdl(turbo_encode_kernel<T, EE>, dim3(blocks), dim3(warps * 32), smem, stream, k, v, k_rows, total, inv_sqrt_dim))
    switch (k.D / 32) {
        case 1: KVC_TE(1); break;
        case 2: KVC_TE(2); break;
        case 4: KVC_TE(4); break;
        case 8: KVC_TE(8); break;
        case 16: KVC_TE(16); break;
        case 32: KVC_TE(32); break;
        default: fail(KVC_ERR_UNSUPPORTED, "turbo encode: head dim must be a power of two in [32, 1024]");
    }
#undef KVC_TE
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

}  // namespace

static void launch_turbo_encode_dense(const TurboEncodeArgs &a, cudaStream_t stream) {
    const int64_t rows = (int64_t)a.B * a.H * a.S;
    if (rows == 0) return;
    KVC_REQUIRE(a.bits >= 1 && a.bits <= 4, "turbo encode supports 1..4 bits");
    KVC_REQUIRE(a.D >= 2 && a.D <= 1024, "turbo encode (dense rotation) supports head dims up to 1024");
    const int threads = std::max(32, ((a.D + 31) / 32) * 32);
    const size_t smem = (size_t)(2 * a.D + 1) * sizeof(float) + (size_t)((a.D * a.bits + 31) / 32 + 1) * sizeof(uint32_t);
    switch (a.dtype) {
        case KVC_F32: turbo_encode_dense_kernel<float><<<(unsigned)rows, threads, smem, stream>>>(a, rows); break;
        case KVC_F16: turbo_encode_dense_kernel<__half><<<(unsigned)rows, threads, smem, stream>>>(a, rows); break;
        case KVC_BF16: turbo_encode_dense_kernel<__nv_bfloat16><<<(unsigned)rows, threads, smem, stream>>>(a, rows); break;
        default: fail(KVC_ERR_INVALID_ARG, "turbo encode needs a floating dtype");
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_turbo_encode2(const TurboEncodeArgs &k, const TurboEncodeArgs *v, cudaStream_t stream) {
    if ((int64_t)k.B * k.H * k.S == 0) return;
    if (k.rotation || (v && v->rotation)) {
        // dense rotations: one launch per tensor
        KVC_REQUIRE(k.rotation && (!v || v->rotation), "turbo encode: keys and values must both use the dense rotation");
        launch_turbo_encode_dense(k, stream);
        if (v) launch_turbo_encode_dense(*v, stream);
        return;
    }
    KVC_REQUIRE(k.bits >= 1 && k.bits <= 4, "turbo encode supports 1..4 bits");
    KVC_REQUIRE(k.D >= 32 && k.D <= 1024 && (k.D & (k.D - 1)) == 0,
                "turbo encode (Walsh-Hadamard path) needs a power-of-two head dim in [32, 1024]");
    if (v) {
        KVC_REQUIRE(v->D == k.D && v->dtype == k.dtype, "turbo encode: K and V must share dim and dtype");
        KVC_REQUIRE(v->bits >= 1 && v->bits <= 4, "turbo encode supports 1..4 bits");
    }
    const TurboEncodeArgs &vv = v ? *v : k;
    switch (k.dtype) {
        case KVC_F32: turbo_dispatch<float>(k, vv, v != nullptr, stream); break;
        case KVC_F16: turbo_dispatch<__half>(k, vv, v != nullptr, stream); break;
        case KVC_BF16: turbo_dispatch<__nv_bfloat16>(k, vv, v != nullptr, stream); break;
        default: fail(KVC_ERR_INVALID_ARG, "turbo encode needs a floating dtype");
    }
}

bool launch_turbo_encode_list(const TurboEncodeArgs *k, const TurboEncodeArgs *v, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX || (int64_t)k[0].B * k[0].H * k[0].S == 0) return false;
#define KVC_EL(TT)                                                           \
    switch (k[0].D) {                                                        \
        case 64: return encode_list<TT, 2>(k, v, n, stream);                 \
        case 128: return encode_list<TT, 4>(k, v, n, stream);                \
        case 256: return encode_list<TT, 8>(k, v, n, stream);                \
        default: return false;                                               \
    }
    switch (k[0].dtype) {
        case KVC_F16: KVC_EL(__half)
        case KVC_BF16: KVC_EL(__nv_bfloat16)
        default: return false;
    }
#undef KVC_EL
}

void launch_turbo_encode(const TurboEncodeArgs &a, cudaStream_t stream) {
    launch_turbo_encode2(a, nullptr, stream);
}

bool launch_turbo_encode_stats(const TurboEncodeArgs &a, long long *sums, cudaStream_t stream) {
    if ((int64_t)a.B * a.H * a.S == 0 || a.calib || a.rotation || a.bits < 1 || a.bits > 4) return false;
    unsigned long long *o = reinterpret_cast<unsigned long long *>(sums);
    switch (a.dtype) {
        case KVC_F32: return encode_wide<float>(a, a, false, o, stream);
        case KVC_F16: return encode_wide<__half>(a, a, false, o, stream);
        case KVC_BF16: return encode_wide<__nv_bfloat16>(a, a, false, o, stream);
        default: return false;
    }
}

void launch_turbo_calib_stats(const TurboEncodeArgs &a, long long *sums, cudaStream_t stream) {
    const int64_t rows = (int64_t)a.B * a.H * a.S;
    if (rows == 0) return;
    if (a.rotation) {
        const int threads = std::max(32, ((a.D + 31) / 32) * 32);
        const size_t smem = (size_t)(2 * a.D + 1) * sizeof(float);
        unsigned long long *o = reinterpret_cast<unsigned long long *>(sums);
        switch (a.dtype) {
            case KVC_F32: turbo_calib_stats_dense_kernel<float><<<(unsigned)rows, threads, smem, stream>>>(a, rows, o); break;
            case KVC_F16: turbo_calib_stats_dense_kernel<__half><<<(unsigned)rows, threads, smem, stream>>>(a, rows, o); break;
            case KVC_BF16: turbo_calib_stats_dense_kernel<__nv_bfloat16><<<(unsigned)rows, threads, smem, stream>>>(a, rows, o); break;
            default: fail(KVC_ERR_INVALID_ARG, "key calibration needs a floating dtype");
        }
        KVC_CUDA(cudaGetLastError());
        ++g_launch_count;
        return;
    }
    KVC_REQUIRE(a.D >= 32 && a.D <= 1024 && (a.D & (a.D - 1)) == 0,
                "key calibration (Walsh-Hadamard path) needs a power-of-two head dim in [32, 1024]");
    const float inv_sqrt_dim = 1.0f / sqrtf((float)a.D);
    const int warps = 8;
    const unsigned blocks = (unsigned)std::min<int64_t>((rows + warps - 1) / warps, (int64_t)sm_count(current_device()) * 8);
    unsigned long long *out = reinterpret_cast<unsigned long long *>(sums);
#define KVC_CS(TT)                                                                                                \
    switch (a.D / 32) {                                                                                           \
        case 1: turbo_calib_stats_kernel<TT, 1><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
        case 2: turbo_calib_stats_kernel<TT, 2><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
        case 4: turbo_calib_stats_kernel<TT, 4><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
        case 8: turbo_calib_stats_kernel<TT, 8><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
        case 16: turbo_calib_stats_kernel<TT, 16><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
        default: turbo_calib_stats_kernel<TT, 32><<<blocks, warps * 32, 0, stream>>>(a, rows, inv_sqrt_dim, out); break; \
    }
    switch (a.dtype) {
        case KVC_F32: KVC_CS(float) break;
        case KVC_F16: KVC_CS(__half) break;
        case KVC_BF16: KVC_CS(__nv_bfloat16) break;
        default: fail(KVC_ERR_INVALID_ARG, "key calibration needs a floating dtype");
    }
#undef KVC_CS
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

}  // namespace kvc
