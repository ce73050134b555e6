// Cache row movement: linear append, ring scatter and the segment gather the
// rotating cache uses for temporal re-ordering, front trims and logical views.
// All of it is pure data movement (bit-exact by construction) and HBM-bound:
// one thread moves one 16-byte vector, consecutive threads touch consecutive
// vectors of a row, K and V travel in the same launch.
#include "attn_common.cuh"

#include <algorithm>
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

template <typename V>
__global__ void append_kernel(AppendArgs a, int64_t k_units, int64_t total_units,
                              int k_upr, int v_upr /* units per row */) {
    dev::pdl_wait();
    dev::pdl_trigger();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total_units) return;
    const bool is_v = i >= k_units;
    if (is_v) i -= k_units;
    const int upr = is_v ? v_upr : k_upr;
    const int u = (int)(i % upr);
    int64_t row = i / upr;
    const int s = (int)(row % a.S);
    row /= a.S;
    const int h = (int)(row % a.H);
    const int b = (int)(row / a.H);
    constexpr int VB = sizeof(V);
    if (!is_v) {
        const char *src = (const char *)a.k_src +
                          (b * a.ks_sb + h * a.ks_sh + s * a.ks_ss) * (int64_t)a.esize + (int64_t)u * VB;
        char *dst = (char *)a.k_dst +
                    (b * a.kd_sb + h * a.kd_sh + (a.pos + s) * a.kd_st) * (int64_t)a.esize + (int64_t)u * VB;
        *(V *)dst = *(const V *)src;
    } else {
        const char *src = (const char *)a.v_src +
                          (b * a.vs_sb + h * a.vs_sh + s * a.vs_ss) * (int64_t)a.esize + (int64_t)u * VB;
        char *dst = (char *)a.v_dst +
                    (b * a.vd_sb + h * a.vd_sh + (a.pos + s) * a.vd_st) * (int64_t)a.esize + (int64_t)u * VB;
        *(V *)dst = *(const V *)src;
    }
}

// The single-token appends of a list of caches of one shape in one launch: y = cache.
struct AppendList {
    AppendArgs a[KVC_LIST_MAX];
};
__global__ void append_list_kernel(const __grid_constant__ AppendList l, int k_units, int total_units, int k_upr, int v_upr) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const AppendArgs &a = l.a[blockIdx.y];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total_units) return;
    const bool is_v = i >= k_units;
    if (is_v) i -= k_units;
    const int upr = is_v ? v_upr : k_upr, u = i % upr;
    int row = i / upr;
    const int s = row % a.S;
    row /= a.S;
    const int h = row % a.H, b = row / a.H;
    const char *src = is_v ? (const char *)a.v_src + (b * a.vs_sb + h * a.vs_sh + s * a.vs_ss) * (int64_t)a.esize
                           : (const char *)a.k_src + (b * a.ks_sb + h * a.ks_sh + s * a.ks_ss) * (int64_t)a.esize;
    char *dst = is_v ? (char *)a.v_dst + (b * a.vd_sb + h * a.vd_sh + (a.pos + s) * a.vd_st) * (int64_t)a.esize
                     : (char *)a.k_dst + (b * a.kd_sb + h * a.kd_sh + (a.pos + s) * a.kd_st) * (int64_t)a.esize;
    ((uint4 *)dst)[u] = ((const uint4 *)src)[u];
}

// Element-wise fallback for sources whose inner stride is not 1 or whose rows
// are not 16-byte aligned.
template <typename E>
__global__ void append_strided_kernel(AppendArgs a, int64_t k_elems, int64_t total) {
    dev::pdl_wait();
    dev::pdl_trigger();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const bool is_v = i >= k_elems;
    if (is_v) i -= k_elems;
    const int D = is_v ? a.Dv : a.Dk;
    const int d = (int)(i % D);
    int64_t row = i / D;
    const int s = (int)(row % a.S);
    row /= a.S;
    const int h = (int)(row % a.H);
    const int b = (int)(row / a.H);
    if (!is_v) {
        const E *src = (const E *)a.k_src + b * a.ks_sb + h * a.ks_sh + s * a.ks_ss + d * a.ks_sd;
        E *dst = (E *)a.k_dst + b * a.kd_sb + h * a.kd_sh + (a.pos + s) * a.kd_st + d;
        *dst = *src;
    } else {
        const E *src = (const E *)a.v_src + b * a.vs_sb + h * a.vs_sh + s * a.vs_ss + d * a.vs_sd;
        E *dst = (E *)a.v_dst + b * a.vd_sb + h * a.vd_sh + (a.pos + s) * a.vd_st + d;
        *dst = *src;
    }
}

// Rotary positions for queries and keys in one launch (applyRotaryPosition,
// MLXLMCommon/RoPEApplication.swift:58-69; the rotation itself is MLX's published RoPE: pair i of a
// head at position p turns by p * scale * base^(-2i/dims)). One thread per (row, pair); features past
// `dims` are copied. Arithmetic in float32, results rounded to the element type.
// A decode step turns a few KB: what it costs is the launch, the angle's chain and its place in front of the attention.
// So the kernel starts under the tail of the one before it, works out the angles (they need no memory), waits, and
// only then lets the attention kernel start, which may stream the stored rows while this one turns q and k.
template <typename T>
__global__ void rope_kernel(RopeArgs a, int64_t q_items, int64_t total_items) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < total_items;
    if (!live) i = 0;
    const bool is_k = i >= q_items;
    if (is_k) i -= q_items;
    const RopeTensor &t = is_k ? a.k : a.q;
    const int half = a.D / 2;            // items per row: D / 2 (rotated pairs first, then pass-through pairs)
    const int p = (int)(i % half);
    int64_t row = i / half;
    const int l = (int)(row % t.L);
    row /= t.L;
    const int h = (int)(row % t.H);
    const int b = (int)(row / t.H);
    const T *src = (const T *)t.src + b * t.s_sb + h * t.s_sh + l * t.s_sl;
    T *dst = (T *)t.dst + b * t.d_sb + h * t.d_sh + l * t.d_sl;
    const int rp = a.dims / 2;           // rotated pairs
    float sn = 0.f, cs = 1.f;
    if (p < rp) dev::rope_angle(p, a.log2_base_over_half, a.offset + l, a.scale, cs, sn);
    dev::pdl_wait();
    dev::pdl_trigger();
    if (!live) return;
    if (p < rp) {
        const int i0 = a.traditional ? 2 * p : p, i1 = a.traditional ? 2 * p + 1 : p + rp;
        float y0, y1;
        dev::rope_turn(to_float<T>(src[i0]), to_float<T>(src[i1]), cs, sn, y0, y1);
        dst[i0] = from_float<T>(y0);
        dst[i1] = from_float<T>(y1);
    } else {
        // the features past `dims`, two per item
        const int j = a.dims + 2 * (p - rp);
        dst[j] = src[j];
        if (j + 1 < a.D) dst[j + 1] = src[j + 1];
    }
}

// Unit u of destination token j of (b, h).
template <typename V> __device__ __forceinline__ void gather_unit(const GatherArgs &a, int b, int h, int64_t j, int u) {
    // Map destination-relative row j to its source token.
    int64_t src_t = -1;
    int64_t rem = j;
#pragma unroll
    for (int sgi = 0; sgi < 4; ++sgi) {
        if (sgi < a.nseg && src_t < 0) {
            if (rem < a.seg[sgi].count) src_t = a.seg[sgi].src_start + rem;
            else rem -= a.seg[sgi].count;
        }
    }
    if (src_t < 0) return;
    constexpr int VB = sizeof(V);
    const char *src = (const char *)a.src +
                      (b * a.s_sb + h * a.s_sh + src_t * a.s_st) * (int64_t)a.esize + (int64_t)u * VB;
    char *dst = (char *)a.dst +
                (b * a.d_sb + h * a.d_sh + (a.dst_start + j) * a.d_st) * (int64_t)a.esize + (int64_t)u * VB;
    *(V *)dst = *(const V *)src;
}

template <typename V>
__global__ void gather_kernel(GatherArgs a, int64_t total_units, int upr, int64_t rows_per_bh) {
    dev::pdl_wait();
    dev::pdl_trigger();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total_units) return;
    const int u = (int)(i % upr);
    int64_t row = i / upr;
    int64_t j = row % rows_per_bh;
    row /= rows_per_bh;
    gather_unit<V>(a, (int)(row / a.H), (int)(row % a.H), j, u);
}

// The two arrays of a cache in one launch (blockIdx.y), for the rings whose gather is all latency: 3.5 us an array at
// 4 x 1 heads x 512 rows of D 256, a launch each.
__global__ void gather_pair_kernel(const __grid_constant__ GatherArgs k, const __grid_constant__ GatherArgs v, uint32_t total_units,
                                   uint32_t upr, uint32_t rows_per_bh) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total_units) return;
    const uint32_t u = i % upr, row = i / upr, j = row % rows_per_bh, bh = row / rows_per_bh;
    gather_unit<uint4>(blockIdx.y ? v : k, (int)(bh / (uint32_t)k.H), (int)(bh % (uint32_t)k.H), j, (int)u);
}

__global__ void causal_mask_kernel(uint8_t *out, int64_t n, int64_t offset, int64_t window) {
    dev::pdl_wait();
    dev::pdl_trigger();
    // createCausalMask (KVCache.swift:253-275): rows are absolute positions
    // offset..offset+n-1, columns 0..offset+n-1; keep when row >= col and,
    // with a window, row < col + window.
    const int64_t cols = offset + n;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * cols) return;
    const int64_t r = offset + i / cols;
    const int64_t c = i % cols;
    bool keep = r >= c;
    if (window >= 0) keep = keep && (r < c + window);
    out[i] = keep ? 1 : 0;
}

// The same mask per batch entry with prepared lengths: entry b also requires col < lengths[b]
// (createCausalMask's `lengths` argument, KVCache.swift:268-271). out: [batch, 1, n, offset + n].
__global__ void causal_mask_lengths_kernel(uint8_t *out, int64_t n, int64_t offset, int64_t window,
                                           const int32_t *lengths, int64_t total) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const int64_t cols = offset + n;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int64_t b = i / (n * cols), j = i % (n * cols);
    const int64_t r = offset + j / cols;
    const int64_t c = j % cols;
    bool keep = r >= c;
    if (window >= 0) keep = keep && (r < c + window);
    keep = keep && (c < (int64_t)lengths[b]);
    out[i] = keep ? 1 : 0;
}

__global__ void rolled_mask_kernel(uint8_t *out, int64_t size, int64_t window, int64_t shift) {
    dev::pdl_wait();
    dev::pdl_trigger();
    // RotatingKVCache.makeMask single-token branch (KVCache.swift:861-865):
    // mask[i] = i >= size - window, rolled right by `shift`.
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= size) return;
    int64_t srci = ((i - shift) % size + size) % size;
    out[i] = (srci >= size - window) ? 1 : 0;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

namespace {
bool append_vectors(const AppendArgs &a) {
    auto stride_ok = [&](int64_t s) { return (s * a.esize) % 16 == 0; };
    const int64_t kb = (int64_t)a.Dk * a.esize, vb = (int64_t)a.Dv * a.esize;
    return a.ks_sd == 1 && a.vs_sd == 1 && kb % 16 == 0 && vb % 16 == 0 && aligned16(a.k_src) && aligned16(a.v_src) &&
           aligned16(a.k_dst) && aligned16(a.v_dst) && stride_ok(a.ks_sb) && stride_ok(a.ks_sh) && stride_ok(a.ks_ss) &&
           stride_ok(a.vs_sb) && stride_ok(a.vs_sh) && stride_ok(a.vs_ss) && stride_ok(a.kd_sb) && stride_ok(a.kd_sh) &&
           stride_ok(a.kd_st) && stride_ok(a.vd_sb) && stride_ok(a.vd_sh) && stride_ok(a.vd_st);
}
}  // namespace

bool launch_append_list(const AppendArgs *args, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX) return false;
    static thread_local AppendList l;
    const AppendArgs &a0 = args[0];
    const int64_t rows = (int64_t)a0.B * a0.H * a0.S, k_upr = (int64_t)a0.Dk * a0.esize / 16, v_upr = (int64_t)a0.Dv * a0.esize / 16;
    const int64_t total = rows * (k_upr + v_upr);
    if (total <= 0 || total > (int64_t)1 << 30) return false;
    for (int i = 0; i < n; ++i) {
        const AppendArgs &a = args[i];
        if (a.B != a0.B || a.H != a0.H || a.S != a0.S || a.Dk != a0.Dk || a.Dv != a0.Dv || a.esize != a0.esize || !append_vectors(a)) return false;
        l.a[i] = a;
    }
    KVC_CUDA(launch_pdl(append_list_kernel, dim3((unsigned)((total + 255) / 256), (unsigned)n), dim3(256), 0, stream, l, (int)(rows * k_upr), (int)total, (int)k_upr, (int)v_upr));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    return true;
}

void launch_append(const AppendArgs &a, cudaStream_t stream) {
    if (a.B <= 0 || a.H <= 0 || a.S <= 0) return;
    const int64_t rows = (int64_t)a.B * a.H * a.S;
    const int64_t kb = (int64_t)a.Dk * a.esize, vb = (int64_t)a.Dv * a.esize;
    const bool vec = append_vectors(a);
    const int threads = 256;
    if (vec) {
        const int k_upr = (int)(kb / 16), v_upr = (int)(vb / 16);
        const int64_t k_units = rows * k_upr, total = k_units + rows * v_upr;
        const int64_t blocks = (total + threads - 1) / threads;
        KVC_CUDA(launch_pdl(append_kernel<uint4>, dim3((unsigned)blocks), dim3(threads), 0, stream, a, k_units, total, k_upr, v_upr));
    } else {
        const int64_t k_elems = rows * a.Dk, total = k_elems + rows * a.Dv;
        const int64_t blocks = (total + threads - 1) / threads;
        if (a.esize == 2)
            KVC_CUDA(launch_pdl(append_strided_kernel<uint16_t>, dim3((unsigned)blocks), dim3(threads), 0, stream, a, k_elems, total));
        else if (a.esize == 4)
            KVC_CUDA(launch_pdl(append_strided_kernel<uint32_t>, dim3((unsigned)blocks), dim3(threads), 0, stream, a, k_elems, total));
        else
            fail(KVC_ERR_INVALID_ARG, "append: unsupported element size");
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

namespace {
// y = array, x = 16-byte pieces of the tails of its planes; pieces that straddle an end go by half words
__global__ void zero_tails_kernel(const __grid_constant__ ZeroTails z) {
    dev::pdl_wait();
    dev::pdl_trigger();
    const auto &t = z.tail[blockIdx.y];
    const int64_t first = t.from & ~(int64_t)15, per_plane = (t.pitch - first + 15) >> 4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < per_plane * t.planes; i += (int64_t)gridDim.x * blockDim.x) {
        char *plane = t.base + i / per_plane * t.pitch;
        const int64_t at = first + (i % per_plane) * 16;
        if (at >= t.from && at + 16 <= t.pitch && !((uintptr_t)(plane + at) & 15)) {
            *(uint4 *)(plane + at) = make_uint4(0u, 0u, 0u, 0u);
        } else {
            for (int64_t b = max(at, t.from); b < min(at + 16, t.pitch); b += 2) *(uint16_t *)(plane + b) = 0;
        }
    }
}
struct Floats { float v[1024 - 16]; };
__global__ void store_floats_kernel(float *dst, const __grid_constant__ Floats f, int n) {
    dev::pdl_wait();
    dev::pdl_trigger();
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = f.v[i];
}
}  // namespace

void launch_zero_tails(const ZeroTails &z, cudaStream_t stream) {
    if (z.n <= 0) return;
    int64_t most = 0;
    for (int i = 0; i < z.n; ++i) most = std::max<int64_t>(most, (z.tail[i].pitch - z.tail[i].from + 31) / 16 * z.tail[i].planes);
    if (most <= 0) return;
    KVC_CUDA(launch_pdl(zero_tails_kernel, dim3((unsigned)std::min<int64_t>((most + 255) / 256, 1184), (unsigned)z.n), dim3(256), 0, stream, z));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_store_floats(float *dst, const float *src, int n, cudaStream_t stream) {
    constexpr int MOST = sizeof(Floats) / sizeof(float);
    for (int at = 0; at < n; at += MOST) {
        Floats f;
        const int m = std::min(n - at, MOST);
        std::memcpy(f.v, src + at, (size_t)m * sizeof(float));
        KVC_CUDA(launch_pdl(store_floats_kernel, dim3(1), dim3(256), 0, stream, dst + at, f, m));
        KVC_CUDA(cudaGetLastError());
        ++g_launch_count;
    }
}

namespace {
int64_t gather_tokens(const GatherArgs &a) {
    int64_t n = 0;
    for (int i = 0; i < a.nseg; ++i) n += a.seg[i].count;
    return n;
}
// Rows that move 16 bytes at a time.
bool gather_vec(const GatherArgs &a) {
    auto stride_ok = [&](int64_t s) { return (s * a.esize) % 16 == 0; };
    return (int64_t)a.W * a.esize % 16 == 0 && aligned16(a.src) && aligned16(a.dst) && stride_ok(a.s_sb) && stride_ok(a.s_sh) &&
           stride_ok(a.s_st) && stride_ok(a.d_sb) && stride_ok(a.d_sh) && stride_ok(a.d_st);
}
}  // namespace

void launch_gather_pair(const GatherArgs &k, const GatherArgs &v, cudaStream_t stream) {
    const int64_t tokens = gather_tokens(k), upr = (int64_t)k.W * k.esize / 16, total = tokens * k.B * k.H * upr;
    // one shape, and an index of 32 bits: two launches otherwise
    if (tokens <= 0 || tokens != gather_tokens(v) || k.B != v.B || k.H != v.H || k.W != v.W || k.esize != v.esize || k.B <= 0 || k.H <= 0 ||
        total > (int64_t)1 << 30 || !gather_vec(k) || !gather_vec(v)) {
        launch_gather(k, stream);
        launch_gather(v, stream);
        return;
    }
    KVC_CUDA(launch_pdl(gather_pair_kernel, dim3((unsigned)((total + 255) / 256), 2), dim3(256), 0, stream, k, v, (uint32_t)total, (uint32_t)upr, (uint32_t)tokens));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_gather(const GatherArgs &a, cudaStream_t stream) {
    const int64_t rows_per_bh = gather_tokens(a);
    if (rows_per_bh <= 0 || a.B <= 0 || a.H <= 0) return;
    const int64_t rb = (int64_t)a.W * a.esize;
    const bool vec = gather_vec(a);
    const int threads = 256;
    const int64_t rows = (int64_t)a.B * a.H * rows_per_bh;
    if (vec) {
        const int upr = (int)(rb / 16);
        const int64_t total = rows * upr;
        KVC_CUDA(launch_pdl(gather_kernel<uint4>, dim3((unsigned)((total + threads - 1) / threads)), dim3(threads), 0, stream, 
            a, total, upr, rows_per_bh));
    } else if (rb % 4 == 0 && ((uintptr_t)a.src & 3) == 0 && ((uintptr_t)a.dst & 3) == 0 &&
               (a.esize == 4 || (a.s_sb % 2 == 0 && a.s_sh % 2 == 0 && a.s_st % 2 == 0 &&
                                 a.d_sb % 2 == 0 && a.d_sh % 2 == 0 && a.d_st % 2 == 0))) {
        const int upr = (int)(rb / 4);
        const int64_t total = rows * upr;
        KVC_CUDA(launch_pdl(gather_kernel<uint32_t>, dim3((unsigned)((total + threads - 1) / threads)), dim3(threads), 0, stream, 
            a, total, upr, rows_per_bh));
    } else if (a.esize == 2) {
        const int upr = (int)(rb / 2);
        const int64_t total = rows * upr;
        KVC_CUDA(launch_pdl(gather_kernel<uint16_t>, dim3((unsigned)((total + threads - 1) / threads)), dim3(threads), 0, stream, 
            a, total, upr, rows_per_bh));
    } else {
        fail(KVC_ERR_INVALID_ARG, "gather: unsupported row layout");
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_rope(const RopeArgs &a, cudaStream_t s) {
    KVC_REQUIRE(a.dims >= 2 && a.dims % 2 == 0 && a.dims <= a.D && a.D % 2 == 0, "rope: dims must be even and at most the head dim");
    const int half = a.D / 2;
    const int64_t q_items = a.q.src ? (int64_t)a.q.B * a.q.H * a.q.L * half : 0;
    const int64_t k_items = a.k.src ? (int64_t)a.k.B * a.k.H * a.k.L * half : 0;
    const int64_t total = q_items + k_items;
    if (total <= 0) return;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    switch (a.dtype) {
        case KVC_F32: KVC_CUDA(launch_pdl(rope_kernel<float>, dim3(blocks), dim3(256), 0, s, a, q_items, total)); break;
        case KVC_F16: KVC_CUDA(launch_pdl(rope_kernel<__half>, dim3(blocks), dim3(256), 0, s, a, q_items, total)); break;
        case KVC_BF16: KVC_CUDA(launch_pdl(rope_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, s, a, q_items, total)); break;
        default: fail(KVC_ERR_INVALID_ARG, "rope needs a floating dtype");
    }
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
    g_last_chained_launch = g_launch_count;
}

void launch_causal_mask(uint8_t *out, int64_t n, int64_t offset, int64_t window, cudaStream_t s) {
    const int64_t total = n * (offset + n);
    if (total <= 0) return;
    KVC_CUDA(launch_pdl(causal_mask_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, s, out, n, offset, window));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_causal_mask_lengths(uint8_t *out, int64_t n, int64_t offset, int64_t window, const int32_t *lengths,
                                int64_t batch, cudaStream_t s) {
    const int64_t total = batch * n * (offset + n);
    if (total <= 0) return;
    KVC_CUDA(launch_pdl(causal_mask_lengths_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, s, out, n, offset, window, lengths, total));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

void launch_rolled_mask(uint8_t *out, int64_t size, int64_t window, int64_t shift, cudaStream_t s) {
    if (size <= 0) return;
    KVC_CUDA(launch_pdl(rolled_mask_kernel, dim3((unsigned)((size + 255) / 256)), dim3(256), 0, s, out, size, window, shift));
    KVC_CUDA(cudaGetLastError());
    ++g_launch_count;
}

}  // namespace kvc
