// Pieces shared by the tcgen05 attention kernels: tile constants, matrix / instruction descriptor
// helpers, TMEM loads, and the host-side tensor-map encoding for 128-row x 64-element boxes.
#pragma once
#include <cuda.h>

#include <mutex>

#include "attn_common.cuh"
#include "common.h"
#include "f32x2.cuh"

namespace kvc {
namespace tc {

using namespace dev;

constexpr int TC_ROWS = 128;                 // query rows per CTA = TMEM lanes
constexpr int TC_KEYS = 128;                 // keys per tile
constexpr int TC_BOX = 128 * 128;            // bytes of one 64-element-wide box of 128 rows
constexpr int TC_TILE = 2 * TC_BOX;          // 32 KB: a 128 x 128 16-bit tile (P; Q, K and V at head dim 128)
constexpr uint32_t TC_TMEM_COLS = 512;       // all of the SM

__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    // start address, leading and stride byte offsets in 16-byte units; descriptor version 1 (bit 46);
    // 128-byte swizzle (2 at bits 61..63)
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// The same product with the A operand in TMEM (lane = row; 32-bit column c of the operand = its elements
// 2c and 2c + 1): D[tmem_d] (+)= A[tmem_a] * B[bdesc].
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// Arrives on the barrier once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// The same load without the wait: several can be in flight, tmem_ld_wait() closes them all.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 registers of this thread into 32 columns of its TMEM lane (lane = 32 * (warp % 4) + lane id).
__device__ __forceinline__ void tmem_st32_issue(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
          "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
          "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st16_issue(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <typename T> __device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) { return pack_h2(lo, hi); }
template <> __device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ void tma_load_5d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y, int z, int u, int v) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(u), "r"(v)
        : "memory");
}

// True in one lane of a converged warp. The MMA warp runs its loop with all lanes and picks the lane only around the
// instructions themselves: under a branch on the lane number every descriptor takes the slow way from vector to uniform
// registers (70 ... 100 cycles per product, against the 64 the tensor core needs for it).
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}

// One wait of a whole warp: all its threads carry on, or none does.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}

// After a wait that ran out. Producer lane: the copies into a ring whose next entry is `slot` in its use number `round` have
// arrived (the last use of every entry).
__device__ __forceinline__ void drain_copies(uint64_t *full, uint32_t stages, uint32_t slot, uint32_t round) {
#pragma unroll 1
    for (uint32_t s = 0; s < stages; ++s) {
        const uint32_t uses = round + (s < slot ? 1u : 0u);
        if (uses > 0) (void)mbar_wait(&full[s], (uses - 1) & 1);
    }
}
// The warp that issues products: all of them are done (`bar`: used here alone).
__device__ __forceinline__ void drain_products(uint64_t *bar) {
    if (elect_one()) umma_commit(bar);
    __syncwarp();
    (void)warp_wait(bar, 0);
}

// Keys whose products the tensor core may add up before the sums go on in fp32 instructions. It adds towards zero, and a sum of
// n keys loses 6e-9 n of itself (values of one sign; about half of that for values around zero): 3e-6 of an f16 output, which
// is rounded by 2e-4, and 2.5e-5 of a bf16 one, rounded by eight times that, so that errors against 64 bits grow by 0.01 %.
inline int fold_keys(int32_t dtype) { return dtype == KVC_F16 ? 512 : 4096; }

__device__ __forceinline__ void add4_global(float4 *p, float x, float y, float z, float w) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// The fp32 sums a softmax thread (a row) folds its D columns of O into, in a reference of their own. Behind O in TMEM where
// there is room, otherwise in memory that only this thread touches: [column / 4][128 rows] of float4, added to where they lie
// (no load to wait for) unless the reference has left them far behind.
template <int D, bool IN_TMEM> struct FoldedSums {
    uint32_t o;
    float4 *sums;
    float m = -INFINITY;                 // their reference
    bool any = false;
    __device__ __forceinline__ FoldedSums(uint32_t o_addr, float4 *memory) : o(o_addr), sums(memory) {}
    // 32 columns of O and of the sums, in the reference m_o
    __device__ __forceinline__ void total(int cb, float m_o, float (&x)[32]) {
        tmem_ld32(o + cb * 32, x);
        if (!any) return;
        const float f = m == -INFINITY ? 0.f : fast_exp2(m - m_o);
        if constexpr (IN_TMEM) {
            float s[32];
            tmem_ld32(o + D + cb * 32, s);
#pragma unroll
            for (int k = 0; k < 32; ++k) x[k] = fmaf(s[k], f, x[k]);
        } else
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4) {
            const float4 y = __ldcg(&sums[(cb * 8 + c4) * TC_ROWS]);
            x[c4 * 4 + 0] = fmaf(y.x, f, x[c4 * 4 + 0]);
            x[c4 * 4 + 1] = fmaf(y.y, f, x[c4 * 4 + 1]);
            x[c4 * 4 + 2] = fmaf(y.z, f, x[c4 * 4 + 2]);
            x[c4 * 4 + 3] = fmaf(y.w, f, x[c4 * 4 + 3]);
        }
    }
    // ... all of them to memory of the same layout
    __device__ __forceinline__ void leave(float m_o, float4 *to) {
#pragma unroll 1
        for (int cb = 0; cb < D / 32; ++cb) {
            float x[32];
            total(cb, m_o, x);
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) __stcg(&to[(cb * 8 + c4) * TC_ROWS], make_float4(x[c4 * 4], x[c4 * 4 + 1], x[c4 * 4 + 2], x[c4 * 4 + 3]));
        }
    }
    // A fold: all threads of a warp; O is settled, and the product after it starts from nothing. In memory it is begun here and put()
    // for all columns by the caller, who has work to do it under, unless the reference has moved too far: then it is done at once.
    enum Form { DONE, STORE, ADD };
    __device__ __forceinline__ Form begin(float m_o, float &f) {
        if (IN_TMEM) {
#pragma unroll 1
            for (int cb = 0; cb < D / 32; ++cb) {
                float x[32];
                uint32_t bits[32];
                total(cb, m_o, x);
#pragma unroll
                for (int k = 0; k < 32; ++k) bits[k] = __float_as_uint(x[k]);
                tmem_st32_issue(o + D + cb * 32, bits);
            }
            tmem_st_wait();
            m = m_o;
            any = true;
            return DONE;
        }
        f = 1.f;
        if (any && !__any_sync(0xffffffffu, !(m_o - m <= 64.f))) {
            f = fast_exp2(m_o - m);
            return ADD;
        }
        const bool again = any;
        if (again) leave(m_o, sums);
        m = m_o;
        any = true;
        return again ? DONE : STORE;
    }
    // N columns of O from column 4 * at on
    template <int N> __device__ __forceinline__ void put(Form form, int at, const uint32_t (&x)[N], float f) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const float4 y = make_float4(__uint_as_float(x[4 * i]) * f, __uint_as_float(x[4 * i + 1]) * f, __uint_as_float(x[4 * i + 2]) * f, __uint_as_float(x[4 * i + 3]) * f);
            if (form == ADD) add4_global(&sums[(at + i) * TC_ROWS], y.x, y.y, y.z, y.w);
            else __stcg(&sums[(at + i) * TC_ROWS], y);
        }
    }
    __device__ __forceinline__ void fold(float m_o) {
        float f;
        const Form form = begin(m_o, f);
        if (form == DONE) return;
#pragma unroll 2
        for (int cb = 0; cb < D / 32; ++cb) {
            uint32_t x[32];
            tmem_ld32_issue(o + cb * 32, x);
            tmem_ld_wait();
            put(form, cb * 8, x, f);
        }
    }
};

// 32 output columns of a row as 16-bit values.
template <typename T> __device__ __forceinline__ void store_row32(T *dst, const float *o, float inv) {
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
        uint4 v;
        v.x = pack_pair<T>(o[c8 * 8 + 0] * inv, o[c8 * 8 + 1] * inv);
        v.y = pack_pair<T>(o[c8 * 8 + 2] * inv, o[c8 * 8 + 3] * inv);
        v.z = pack_pair<T>(o[c8 * 8 + 4] * inv, o[c8 * 8 + 5] * inv);
        v.w = pack_pair<T>(o[c8 * 8 + 6] * inv, o[c8 * 8 + 7] * inv);
        *(uint4 *)(dst + c8 * 8) = v;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_tc() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
        if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess) fn = (EncodeTiledFn)ptr;
        else (void)cudaGetLastError();
    });
    return fn;
}

// [B, H, rows, D] view, element strides (inner 1): boxes of box_rows rows x 64 elements, 128-byte swizzle,
// rows beyond `rows` read as zero.
inline bool make_map_tc(CUtensorMap *map, const void *data, int32_t dtype, int D, int64_t rows, int H, int B, int64_t s_row,
                 int64_t s_h, int64_t s_b, int box_rows = 128) {
    EncodeTiledFn fn = encode_tiled_tc();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)H, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)s_row * 2, (cuuint64_t)(H > 1 ? s_h : s_row * rows) * 2,
                                   (cuuint64_t)(B > 1 ? s_b : (H > 1 ? s_h * H : s_row * rows)) * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == KVC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    return fn(map, dt, 4, const_cast<void *>(data), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline bool strides_fit(const void *data, int D, int64_t s_row, int64_t s_h, int64_t s_b, int H, int B) {
    auto ok = [](int64_t st) { return st > 0 && (st * 2) % 16 == 0; };
    if (((uintptr_t)data & 15) != 0 || !ok(s_row) || s_row < D) return false;
    if (H > 1 && !ok(s_h)) return false;
    if (B > 1 && !ok(s_b)) return false;
    return true;
}

// Queries [B, Hq, L, D] as (dim, head of the group, position, KV head, batch): a box is hb heads x lb positions of 64 dims.
inline bool make_query_map(CUtensorMap *map, const AttnArgs &a, int rep, int hb, int lb) {
    EncodeTiledFn fn = encode_tiled_tc();
    if (!fn) return false;
    const int64_t row = a.q_sl * 2, head = a.Hq > 1 ? a.q_sh * 2 : row;
    const cuuint64_t dims[5] = {(cuuint64_t)a.D, (cuuint64_t)rep, (cuuint64_t)a.L, (cuuint64_t)a.Hkv, (cuuint64_t)a.B};
    const cuuint64_t strides[4] = {(cuuint64_t)head, (cuuint64_t)row, (cuuint64_t)(head * rep), (cuuint64_t)(a.B > 1 ? a.q_sb * 2 : head)};
    const cuuint32_t box[5] = {64, (cuuint32_t)hb, (cuuint32_t)lb, 1, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUtensorMapDataType dt = a.q_dtype == KVC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    return fn(map, dt, 5, const_cast<void *>(a.q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Device memory for the length of one call, in stream order (inside a capture: of the graph). Null where there is no room.
struct CallMemory {
    void *ptr = nullptr;
    cudaStream_t stream;
    CallMemory(size_t bytes, cudaStream_t s) : stream(s) {
        if (bytes > 0) ptr = dev_try_alloc(bytes, s);
    }
    ~CallMemory() { dev_free(ptr, stream); }   // nothing for a null pointer
    CallMemory(const CallMemory &) = delete;
    CallMemory &operator=(const CallMemory &) = delete;
};

}  // namespace tc
}  // namespace kvc
