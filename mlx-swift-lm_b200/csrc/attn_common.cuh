// Device primitives shared by the TMA-staged attention kernels: mbarrier
// (bounded waits), TMA tile and bulk loads, ldmatrix, fast exp2 and the
// m16n8k16 tensor-core MMA for f16 / bf16 operands.
#pragma once

#include "common.h"

#include <algorithm>
#include <cstdlib>
#include <utility>

#include <cuda.h>

// Measurement aids (switching consumer work off piece by piece to time the producer alone) exist
// only in a build made with -DKVC_MEASURE_AIDS, which the shipped build never sets: without the
// flag the skip bits are the constant 0, the branches on them compile away and no environment
// variable is read.
#ifdef KVC_MEASURE_AIDS
#define KVC_SKIP_BITS(p) ((p).debug_skip)
#else
#define KVC_SKIP_BITS(p) 0
#endif

namespace kvc {

inline int measure_skip_bits() {
#ifdef KVC_MEASURE_AIDS
    static const int bits = [] {
        const char *e = std::getenv("KVC_DECODE_DEBUG_SKIP");
        return e ? std::atoi(e) : 0;
    }();
    return bits;
#else
    return 0;
#endif
}

// KVC_TRACE_DISPATCH=1 makes the chunk paths say on stderr which kernel took a call. Read at each
// use (tests switch it on inside a running process); only chunk launches consult it, never decode.
inline bool trace_dispatch() {
    const char *e = std::getenv("KVC_TRACE_DISPATCH");
    return e && e[0] == '1';
}

// What a chunk on operand pairs takes beside its 16-bit rows: the low halves (k, q: null where the high ones are exact),
// the factors that give scaled operands their size back (per query row; per (batch, KV head); null: 1; values always
// have theirs), and the type of its output.
struct ChunkLow {
    const void *k, *v, *q;
    const float *q_undo, *k_undo, *v_undo;
    int32_t out_dtype;
};

namespace dev {

constexpr uint32_t SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait; returns false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// A consumer warp gives ring entry `bar` back to the copies that fill it. An arrival orders this warp's reads before other
// threads' loads and stores, but not before a bulk or TMA copy (the async proxy): loads whose values are still on their way
// were overtaken by the copy of a later tile (8-bit codes in one group a row, three CTAs an SM: every run gave other outputs,
// off by up to 20 % of a row). So the reads are either fenced off ...
__device__ __forceinline__ void release_fenced(uint64_t *bar, int lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
// ... or the arrival's address is made to need them: `read` joins words that came out of the last loads (those before came back
// before them), `none` is zero and not known to the compiler. A kernel whose later (volatile) shared loads or stores need every
// value that it took from the entry has waited for them already, and arrives as it is.
__device__ __forceinline__ void release_after(uint64_t *bar, int lane, uint32_t read, uint32_t none) {
    __syncwarp();
    if (lane == 0) mbar_arrive((uint64_t *)((unsigned char *)bar + (read & none)));
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y,
                                            int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Programmatic dependent launch: a kernel launched with launch_pdl() may start while the
// kernel before it on the stream is still running; everything it reads from global memory
// must come after pdl_wait(), which returns once that kernel has completed and flushed.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel on the stream (if it was launched with launch_pdl) be scheduled as soon as
// every CTA of this one has issued it or exited. Issued only AFTER pdl_wait(): a kernel that starts
// early then knows that everything up to the kernel before its predecessor has completed.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Bits of 32 mask bytes starting at p (any alignment), the first n of them inside the row.
__device__ __forceinline__ uint32_t mask_bits32(const uint8_t *p, int n) {
    if (n <= 0) return 0;
    n = min(n, 32);
    const uint32_t *w = (const uint32_t *)((uintptr_t)p & ~(uintptr_t)3);
    const int sh = (int)((uintptr_t)p & 3) * 8, words = (n + (sh >> 3) + 3) >> 2;   // only words that hold a byte of the row
    uint32_t bits = 0, cur = *w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t nxt = i + 1 < words ? w[i + 1] : 0u;
        const uint32_t b = __vcmpne4(__funnelshift_r(cur, nxt, sh), 0u) & 0x08040201u;
        bits |= ((b | b >> 8 | b >> 16 | b >> 24) & 15u) << (4 * i);
        cur = nxt;
    }
    return n == 32 ? bits : bits & ((1u << n) - 1u);
}

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 8x8 transpose of b16 elements across the warp: lane (g, c) gives row g, columns 2c, 2c+1
// and receives row g of the transpose.
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

// The 8x8 b16 transpose without `volatile`: every lane of the warp reaches it (callers keep it out of
// divergent branches) and it has no side effect, so the compiler may schedule it among the lookups.
__device__ __forceinline__ uint32_t movmatrix_free(uint32_t x) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

template <typename T> struct MmaType;
template <> struct MmaType<__nv_bfloat16> {
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    }
    static __device__ __forceinline__ void store(void *p, int64_t i, float v) {
        ((__nv_bfloat16 *)p)[i] = __float2bfloat16_rn(v);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t w) {
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
    }
};
template <> struct MmaType<__half> {
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    }
    static __device__ __forceinline__ void store(void *p, int64_t i, float v) {
        ((__half *)p)[i] = __float2half_rn(v);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t w) {
        return __half22float2(*reinterpret_cast<const __half2 *>(&w));
    }
};


// A tile's lines towards L2, where every kernel's writes meet: may run ahead of the wait on the kernel before, whatever that
// one writes.
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap *map, int x, int y, int z, int w) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];"
                 ::"l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(w)
                 : "memory");
}

// Rotary positions: cosine and sine of pair `p` at a position (MLX's published RoPE: p turns by
// position * scale * base^(-2p / dims)). The frequency in double precision, rounded once: at positions in the tens of
// thousands a float32 exp2 would already move the angle by 1e-3.
__device__ __forceinline__ void rope_angle(int p, double log2_base_over_half, int64_t position, float scale, float &cs, float &sn) {
    const float inv_freq = (float)exp2(-(double)p * log2_base_over_half);
    sincosf(__fmul_rn(__fmul_rn((float)position, scale), inv_freq), &sn, &cs);
}
// A pair turned (in float32, one product rounded, one fused).
__device__ __forceinline__ void rope_turn(float x0, float x1, float cs, float sn, float &y0, float &y1) {
    y0 = __fmaf_rn(x0, cs, -__fmul_rn(x1, sn));
    y1 = __fmaf_rn(x0, sn, __fmul_rn(x1, cs));
}

// Untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// ---------------------------------------------------------------------
// End of a work unit: merge the consumer warps of the CTA into one partial,
// publish it, and let the last unit of the (batch, head) merge all splits.
// ---------------------------------------------------------------------
struct UnitOut {
    float *o_part;      // [query row][split][D]
    float2 *ml_part;    // [query row][split] (log2-domain max, sum)
    int *counters;      // one ticket per (batch, head), self-resetting
    void *out;
    int32_t out_dtype;
    int64_t o_sb, o_sh, o_sl;
    const float *o_signs;  // optional: rotate merged rows back (TurboQuant values)
    int32_t splits, Hq, L;
};

__device__ __forceinline__ void store_out(void *p, int32_t dtype, int64_t i, float v) {
    switch (dtype) {
        case KVC_F32: ((float *)p)[i] = v; break;
        case KVC_F16: ((__half *)p)[i] = __float2half_rn(v); break;
        default: ((__nv_bfloat16 *)p)[i] = __float2bfloat16_rn(v); break;
    }
}

// Query row n of a group as head and position: a decode step has one position and needs no division.
__device__ __forceinline__ void split_row(int n, int L, int &head, int &pos) {
    head = n;
    pos = 0;
    if (L != 1) {
        head = n / L;
        pos = n - head * L;
    }
}

// Four neighbouring elements, in one store where they lie on its boundary.
__device__ __forceinline__ void store_out4(void *p, int32_t dtype, int64_t i, float4 v) {
    const uintptr_t at = (uintptr_t)p + (uintptr_t)(i * (dtype == KVC_F32 ? 4 : 2));
    if (at & (dtype == KVC_F32 ? 15 : 7)) {
        store_out(p, dtype, i, v.x);
        store_out(p, dtype, i + 1, v.y);
        store_out(p, dtype, i + 2, v.z);
        store_out(p, dtype, i + 3, v.w);
    } else if (dtype == KVC_F32) {
        *(float4 *)at = v;
    } else if (dtype == KVC_F16) {
        *(uint2 *)at = make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
    } else {
        *(uint2 *)at = make_uint2(pack_bf2(v.x, v.y), pack_bf2(v.z, v.w));
    }
}

// Preconditions: every consumer warp w < NWARPS has written its un-normalised
// rows to red_o[(w*16 + r) * red_stride + d] and (max, sum) to red_ml[(w*16 + r)*2],
// followed by a __syncthreads(). `work` is shared memory that does not overlap
// red_o / red_ml, at least R * max(splits, D) floats; `flag` one int of shared memory.
template <int D, int NWARPS>
__device__ void unit_epilogue(const UnitOut &u, const float *red_o, const float *red_ml, int red_stride,
                              float *work, int *flag, int b, int hk, int rep, int R, int split, int bh) {
    const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
    constexpr int row0 = 0;  // a unit of this epilogue always carries the whole group
    const int64_t qrow0 = ((int64_t)b * u.Hq + hk * rep) * u.L + row0;  // the group's rows are consecutive query rows
    for (int i = tid; i < R * D; i += nthreads) {
        const int r = i / D, d = i % D;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) m = fmaxf(m, red_ml[(w * 16 + r) * 2]);
        float o = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) {
            const float mw = red_ml[(w * 16 + r) * 2];
            const float f = (mw == -INFINITY) ? 0.f : fast_exp2(mw - m);
            o += red_o[(w * 16 + r) * red_stride + d] * f;
            l += red_ml[(w * 16 + r) * 2 + 1] * f;
        }
        const int64_t base = (qrow0 + r) * u.splits + split;
        __stcg(&u.o_part[base * D + d], o);
        if (d == 0) __stcg(&u.ml_part[base], make_float2(m, l));
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int ticket = atomicAdd(&u.counters[bh], 1);
        const int last = (ticket == u.splits - 1) ? 1 : 0;
        if (last) u.counters[bh] = 0;
        *flag = last;
    }
    __syncthreads();
    if (!*flag) return;
    __threadfence();
    // merge weights per (row, split)
    for (int r = warp; r < R; r += nthreads / 32) {
        float m = -INFINITY;
        for (int s = lane; s < u.splits; s += 32) m = fmaxf(m, __ldcg(&u.ml_part[(qrow0 + r) * u.splits + s]).x);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float lsum = 0.f;
        for (int s = lane; s < u.splits; s += 32) {
            const float2 ml = __ldcg(&u.ml_part[(qrow0 + r) * u.splits + s]);
            const float f = (ml.x == -INFINITY || ml.y <= 0.f) ? 0.f : fast_exp2(ml.x - m);
            work[r * u.splits + s] = f;
            lsum += ml.y * f;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
        __syncwarp();
        for (int s = lane; s < u.splits; s += 32) work[r * u.splits + s] *= inv;
    }
    __syncthreads();
    if (!u.o_signs) {
        for (int i = tid; i < R * D; i += nthreads) {
            const int r = i / D, d = i % D;
            float o = 0.f;
            const float *src = u.o_part + ((qrow0 + r) * u.splits) * D + d;
            for (int s = 0; s < u.splits; ++s) o = fmaf(__ldcg(src + (int64_t)s * D), work[r * u.splits + s], o);
            const int hq = hk * rep + (row0 + r) / u.L, lq = (row0 + r) % u.L;
            store_out(u.out, u.out_dtype, b * u.o_sb + hq * u.o_sh + lq * u.o_sl + d, o);
        }
        return;
    }
    // TurboQuant values: the merged rows are in the rotated basis; out = signs * H(o) / sqrt(D).
    float *rows = work + R * u.splits;  // [R][D]
    for (int i = tid; i < R * D; i += nthreads) {
        const int r = i / D, d = i % D;
        float o = 0.f;
        const float *src = u.o_part + ((qrow0 + r) * u.splits) * D + d;
        for (int s = 0; s < u.splits; ++s) o = fmaf(__ldcg(src + (int64_t)s * D), work[r * u.splits + s], o);
        rows[i] = o;
    }
    for (int half = 1; half < D; half <<= 1) {
        __syncthreads();
        for (int pidx = tid; pidx < R * (D / 2); pidx += nthreads) {
            const int r = pidx / (D / 2), j = pidx % (D / 2);
            const int i0 = ((j / half) * 2 * half) + (j % half), i1 = i0 + half;
            const float x = rows[r * D + i0], y = rows[r * D + i1];
            rows[r * D + i0] = x + y;
            rows[r * D + i1] = x - y;
        }
    }
    __syncthreads();
    const float f = rsqrtf((float)D);
    for (int i = tid; i < R * D; i += nthreads) {
        const int r = i / D, d = i % D;
        const int hq = hk * rep + (row0 + r) / u.L, lq = (row0 + r) % u.L;
        store_out(u.out, u.out_dtype, b * u.o_sb + hq * u.o_sh + lq * u.o_sl + d, rows[i] * f * u.o_signs[d]);
    }
}

// ---------------------------------------------------------------------
// Flat tile decomposition shared by the decode kernels. All (batch, head) units have
// `tiles` tiles; CTA c owns the consecutive flat tiles [flat_lo(c), flat_lo(c + 1)) of the
// units * tiles in the launch and walks them as segments (one per unit it touches). The
// partial of a segment goes to slot (c - first CTA of the unit) of the unit's partials.
// ---------------------------------------------------------------------
struct FlatPlan {
    int32_t tiles;     // tiles per unit
    int32_t per, rem;  // CTA c owns per + (c < rem) tiles
    int32_t nslots;    // partial slots per unit
    int32_t red_rows;  // rows of the cross-warp buffers (>= query rows per unit)
};

__device__ __forceinline__ int64_t flat_lo(const FlatPlan &f, int c) { return (int64_t)c * f.per + min(c, f.rem); }

// Flat tile numbers fit 31 bits (the launches check it): a 64-bit division is a call of a few hundred cycles, and several
// stand in front of a segment's first load and behind its last tile.
__device__ __forceinline__ int flat_div(int64_t a, int b) { return (int)((uint32_t)a / (uint32_t)b); }
__device__ __forceinline__ int flat_mod(int64_t a, int b, int quotient) { return (int)((uint32_t)a - (uint32_t)quotient * (uint32_t)b); }
inline bool flat_fits(int64_t tiles) { return tiles <= INT32_MAX; }

__device__ __forceinline__ int flat_cta_of(const FlatPlan &f, int64_t x) {
    const uint32_t big = (uint32_t)f.rem * (uint32_t)(f.per + 1);
    return (uint32_t)x < big ? flat_div(x, f.per + 1) : f.rem + flat_div((uint32_t)x - big, f.per);
}

// The same for units of one length, with the ends of the ranges where they cost least. A range that leaves one unit for the
// next pays for another segment: queries turned and packed, warps folded, a partial, a ticket (v4 kernel, 64 units of nine
// tiles on 148 CTAs: 11 000 .. 17 000 cycles, where a tile takes 2 050). So ranges are multiples of `step` tiles: 1
// where equal ranges are the best, a piece of a unit (its tiles rounded up to whole pieces; a CTA stops at the `real`
// ones) or a whole unit.
struct UnitPlan {
    int32_t tiles;     // tiles per unit, rounded up to whole steps
    int32_t per, rem;  // CTA c owns (per + (c < rem)) * step tiles
    int32_t nslots, red_rows;
    int32_t step, real;
};

__device__ __forceinline__ int64_t flat_lo(const UnitPlan &f, int c) { return ((int64_t)c * f.per + min(c, f.rem)) * f.step; }
__device__ __forceinline__ int flat_cta_of(const UnitPlan &f, int64_t x) {
    const uint32_t xs = f.step == 1 ? (uint32_t)x : (uint32_t)x / (uint32_t)f.step, big = (uint32_t)f.rem * (uint32_t)(f.per + 1);
    return xs < big ? flat_div(xs, f.per + 1) : f.rem + flat_div(xs - big, f.per);
}

// Whether equal ranges would cut a unit into more than 64 partials. Calls of so few units stay with the streaming kernel,
// whose operands are f16 pairs, where a kernel's are single (f16 outputs of one sequence of 5 000 tokens, 28/4 heads,
// err by 2.5 times as much there).
inline bool few_units(int64_t units, int64_t tiles, int64_t slots) {
    const int64_t work = units * tiles, per = work / std::min(slots, work);
    return (tiles + per - 1) / per + 1 > 64;
}

// Plans `units` of `tiles` tiles over at most `slots` CTAs; `segment`: what a segment costs beside its tiles, in tiles.
inline int64_t plan_units(UnitPlan *f, int64_t units, int64_t tiles, int64_t slots, int64_t segment) {
    const int64_t work = units * tiles, n = std::min(slots, work), most = (work + n - 1) / n;
    const bool even = work % n == 0;
    const int64_t touched = even && tiles % most == 0 ? 1 : even && most % tiles == 0 ? most / tiles : (most + tiles - 2) / tiles + 1;
    const int64_t cost = most + segment * touched;
    f->real = (int32_t)tiles;
    f->tiles = (int32_t)tiles;
    f->step = 1;
    f->per = (int32_t)(work / n);
    f->rem = (int32_t)(work % n);
    f->nslots = (int32_t)((tiles + f->per - 1) / f->per + 1);
    if (units <= slots) {
        const int64_t piece = (tiles + slots / units - 1) / (slots / units), pieces = (tiles + piece - 1) / piece;
        if (piece + segment >= cost) return n;
        f->tiles = (int32_t)(pieces * piece);
        f->step = (int32_t)piece;
        f->per = 1;
        f->rem = 0;
        f->nslots = (int32_t)pieces;
        return units * pieces;
    }
    if ((units + slots - 1) / slots * (tiles + segment) >= cost) return n;
    f->step = (int32_t)tiles;
    f->per = (int32_t)(units / slots);
    f->rem = (int32_t)(units % slots);
    f->nslots = 1;
    return slots;
}

// Barrier among the NW consumer warps only (the producer warp never joins it). Every consumer
// warp reaches every one of these whether or not one of its bounded waits has run out.
template <int NW>
__device__ __forceinline__ void consumer_bar() {
    asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
}

// Output rows from the rotated basis: out = signs * H(o) / sqrt(D) for the R rows in `rows` ([R][D]).
// A warp takes a row: lane l holds dims E*l .. E*l + E - 1, the stages that pair dims less
// than E apart stay inside the lane, the other five are lane exchanges. Pairs and operations
// ((a, b) -> (a + b, a - b), lower dim first) are those of the stage-by-stage butterfly.
template <int D, int NW>
__device__ __forceinline__ void rotate_out_rows(const UnitOut &u, const float *rows, int b, int hk, int rep, int R, int row0) {
    static_assert(D % 32 == 0 && D / 32 >= 1 && D / 32 <= 16, "one warp spans a row");
    constexpr int E = D / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float fs = rsqrtf((float)D);
    for (int r = warp; r < R; r += NW) {
        float x[E];
#pragma unroll
        for (int j = 0; j < E; ++j) x[j] = rows[r * D + E * lane + j];
#pragma unroll
        for (int h = 1; h < E; h <<= 1)
#pragma unroll
            for (int i = 0; i < E; ++i)
                if ((i & h) == 0) {
                    const float xa = x[i], ya = x[i + h];
                    x[i] = xa + ya;
                    x[i + h] = xa - ya;
                }
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const bool upper = (lane & m) != 0;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float y = __shfl_xor_sync(0xffffffffu, x[j], m);
                x[j] = upper ? y - x[j] : x[j] + y;
            }
        }
        int hq, lq;
        split_row(row0 + r, u.L, hq, lq);
        hq += hk * rep;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int d = E * lane + j;
            store_out(u.out, u.out_dtype, b * u.o_sb + hq * u.o_sh + lq * u.o_sl + d, x[j] * fs * u.o_signs[d]);
        }
    }
}

// End of a segment, called by all NW consumer warps (tid = 0 .. 32 NW - 1) after each has
// written its un-normalised rows to red_o[(warp * red_rows + r) * red_stride + d] and
// red_ml[(warp * red_rows + r) * 2 + {0, 1}] = (max, sum): merges the warps and, where the segment is the whole unit,
// writes the output rows; else writes the segment's partial, takes a ticket and, in the CTA that completes the unit,
// merges all partials (log-sum-exp) and writes the rows (through signs * H(.) / sqrt(D) when
// o_signs is set; `work` then holds red_rows * D floats, and is not touched otherwise). Lists of short units are mostly
// whole ones, and the divisions behind a segment's place took 64 bits before: 4 layers of 32 sequences of 425 .. 1 761 tokens,
// 64/8 heads, 4 bits: 145 us -> 130.
// NBUF (default NW) is the number of warps that wrote cross-warp buffers: a kernel that has already
// folded its NW warps down to NBUF of them passes the smaller count, all NW warps still take part; `live`: as many
// of these as had tokens (the first ones).
template <int D, int NW, int NBUF = NW, int FLY = 16, typename Plan>
__device__ void segment_epilogue(const UnitOut &u, const Plan &f, const float *red_o, const float *red_ml,
                                 int red_stride, float *work, int *flag, int unit, int b, int hk, int rep, int R,
                                 int64_t x_unit = -1, int unit_tiles = 0, int row0 = 0, int live = NBUF) {
    // row0: the unit covers the query rows row0 .. row0 + R - 1 of its (batch, kv head) group (a group
    // of more rows than one unit carries is cut into several units)
    const int tid = threadIdx.x;
    constexpr int NT = NW * 32;
    consumer_bar<NW>();
    // the unit's flat tile range: uniform units unless the caller passes a var-len range
    if (x_unit < 0) {
        x_unit = (int64_t)unit * f.tiles;
        unit_tiles = f.tiles;
    }
    const int first_cta = flat_cta_of(f, x_unit);
    const int expected = flat_cta_of(f, x_unit + unit_tiles - 1) - first_cta + 1;
    const int slot = (int)blockIdx.x - first_cta;
    const int64_t qrow0 = ((int64_t)b * u.Hq + hk * rep) * u.L + row0;
    // A thread takes four neighbouring dims of a row at a time: the weights of the row are worked out once for them, and
    // where partials are merged, loads of sixteen slots are in flight. (One dim at a time and eight slots, the CTA that
    // merged 17 slots of four rows at D 128 spent 7 us on it, a third of what a decode step of a chat takes in all.)
    constexpr int D4 = D / 4;
    // Four dims of the segment's rows, the warps merged; their row's maximum and sum.
    auto merged = [&](int r, int d, float &m, float &l) {
        m = -INFINITY;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        l = 0.f;
#pragma unroll
        for (int w0 = 0; w0 < NBUF; w0 += 4) {
            if (w0 >= live) break;
#pragma unroll
            for (int w = w0; w < w0 + 4 && w < NBUF; ++w) m = fmaxf(m, red_ml[(w * f.red_rows + r) * 2]);
        }
#pragma unroll
        for (int w0 = 0; w0 < NBUF; w0 += 4) {
            if (w0 >= live) break;
#pragma unroll
            for (int w = w0; w < w0 + 4 && w < NBUF; ++w) {
                const float mw = red_ml[(w * f.red_rows + r) * 2];
                const float fw = (mw == -INFINITY) ? 0.f : fast_exp2(mw - m);
                const float4 x = *(const float4 *)&red_o[(w * f.red_rows + r) * red_stride + d];
                o.x += x.x * fw; o.y += x.y * fw; o.z += x.z * fw; o.w += x.w * fw;
                l += red_ml[(w * f.red_rows + r) * 2 + 1] * fw;
            }
        }
        return o;
    };
    // The finished dims of a row: to the output, or to `work` where they have to be rotated back first.
    auto finish = [&](int r, int d, float4 o, float l) {
        o = l > 0.f ? make_float4(o.x / l, o.y / l, o.z / l, o.w / l) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (u.o_signs) {
            *(float4 *)&work[r * D + d] = o;
        } else {
            int hq, lq;
            split_row(row0 + r, u.L, hq, lq);
            hq += hk * rep;
            store_out4(u.out, u.out_dtype, b * u.o_sb + hq * u.o_sh + lq * u.o_sl + d, o);
        }
    };
    if (expected == 1) {   // the segment is the whole unit: its rows go straight to the output
        for (int i = tid; i < R * D4; i += NT) {
            const int r = i / D4, d = i % D4 * 4;
            float m, l;
            const float4 o = merged(r, d, m, l);
            finish(r, d, o, l);
        }
        consumer_bar<NW>();
        if (u.o_signs) {
            rotate_out_rows<D, NW>(u, work, b, hk, rep, R, row0);
            consumer_bar<NW>();
        }
        return;   // the buffers are free again
    }
    for (int i = tid; i < R * D4; i += NT) {
        const int r = i / D4, d = i % D4 * 4;
        float m, l;
        const float4 o = merged(r, d, m, l);
        const int64_t base = (qrow0 + r) * f.nslots + slot;
        __stcg((float4 *)&u.o_part[base * D + d], o);
        if (d == 0) __stcg(&u.ml_part[base], make_float2(m, l));
    }
    __threadfence();
    consumer_bar<NW>();
    if (tid == 0) {
        const int last = atomicAdd(&u.counters[unit], 1) == expected - 1 ? 1 : 0;
        if (last) u.counters[unit] = 0;
        *flag = last;
    }
    consumer_bar<NW>();
    if (*flag) {
        __threadfence();
        // The (max, sum) pairs and the partial values of FLY slots are loaded together (eight where the kernel has no
        // registers for more), the weights are recomputed per thread; slots are merged eight at a time.
        if (expected <= 4) {
            // Few slots: two of a thread's elements at a time, so that their loads meet.
            for (int i0 = tid; i0 < R * D4; i0 += 2 * NT) {
                float2 ml[2][4];
                float4 ov[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = i0 + e * NT, r = i / D4, d = i % D4 * 4;
                    const int64_t at = (qrow0 + r) * f.nslots;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool in = i < R * D4 && j < expected;
                        ml[e][j] = in ? __ldcg(&u.ml_part[at + j]) : make_float2(-INFINITY, 0.f);
                        ov[e][j] = in ? __ldcg((const float4 *)&u.o_part[(at + j) * D + d]) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = i0 + e * NT;
                    if (i >= R * D4) break;
                    float m = -INFINITY, lsum = 0.f;
                    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < 4; ++j) m = fmaxf(m, (ml[e][j].y > 0.f) ? ml[e][j].x : -INFINITY);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float fw = (ml[e][j].x == -INFINITY || ml[e][j].y <= 0.f) ? 0.f : fast_exp2(ml[e][j].x - m);
                        lsum = fmaf(ml[e][j].y, fw, lsum);
                        o.x = fmaf(ov[e][j].x, fw, o.x); o.y = fmaf(ov[e][j].y, fw, o.y);
                        o.z = fmaf(ov[e][j].z, fw, o.z); o.w = fmaf(ov[e][j].w, fw, o.w);
                    }
                    finish(i / D4, i % D4 * 4, o, lsum);
                }
            }
        } else
        for (int i = tid; i < R * D4; i += NT) {
            const int r = i / D4, d = i % D4 * 4;
            const float2 *mlp = u.ml_part + (qrow0 + r) * f.nslots;
            const float *src = u.o_part + ((qrow0 + r) * f.nslots) * D + d;
            float m = -INFINITY, lsum = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int s0 = 0; s0 < expected; s0 += FLY) {
                float2 ml[FLY];
                float4 ov[FLY];
#pragma unroll
                for (int j = 0; j < FLY; ++j) {
                    const bool in = s0 + j < expected;
                    ml[j] = in ? __ldcg(&mlp[s0 + j]) : make_float2(-INFINITY, 0.f);
                    ov[j] = in ? __ldcg((const float4 *)(src + (int64_t)(s0 + j) * D)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int half = 0; half < FLY; half += 8) {
                    if (s0 + half >= expected) break;
                    float mb = m;
#pragma unroll
                    for (int j = half; j < half + 8; ++j) mb = fmaxf(mb, (ml[j].y > 0.f) ? ml[j].x : -INFINITY);
                    const float keep = (m == -INFINITY) ? 0.f : fast_exp2(m - mb);   // rescale what earlier slots gave
                    o.x *= keep; o.y *= keep; o.z *= keep; o.w *= keep;
                    lsum *= keep;
                    m = mb;
#pragma unroll
                    for (int j = half; j < half + 8; ++j) {
                        const float fw = (ml[j].x == -INFINITY || ml[j].y <= 0.f) ? 0.f : fast_exp2(ml[j].x - m);
                        lsum = fmaf(ml[j].y, fw, lsum);
                        o.x = fmaf(ov[j].x, fw, o.x); o.y = fmaf(ov[j].y, fw, o.y);
                        o.z = fmaf(ov[j].z, fw, o.z); o.w = fmaf(ov[j].w, fw, o.w);
                    }
                }
            }
            finish(r, d, o, lsum);
        }
        if (u.o_signs) {
            consumer_bar<NW>();
            rotate_out_rows<D, NW>(u, work, b, hk, rep, R, row0);
        }
    }
    consumer_bar<NW>();  // buffers and flag are reused by the next segment
}

}  // namespace dev

// Launch with programmatic stream serialization (see dev::pdl_wait). KVC_NO_PDL=1 falls
// back to a plain launch. The small kernels in front of an attention kernel (appends, quantisers, encoders, gathers) are
// launched so too, wait first and release their successors after the wait: a plain launch behind a programmatic one
// started at multiples of 2.05 us behind the one before (steps of an affine or compressed cache took n * 2.05 us a layer),
// a chain of programmatic ones starts at once: 18.5 -> 14.6 us for rotary, append and attention of 64/8 heads over 64 .. 300
// tokens, 8 bits. Kernels that hold TMEM release nobody early: the successor's CTAs could take columns that a CTA
// of theirs has yet to allocate, and wait for it.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args &&...args) {
    static const bool off = [] {
        const char *e = std::getenv("KVC_NO_PDL");
        return e && e[0] == '1';
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = off ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace kvc
