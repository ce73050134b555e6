// Which calls attn_stream_kernel takes, and with which template arguments.
#include "attn_stream.cuh"

#include <cmath>
#include <cstdlib>
#include <mutex>

namespace kvc {

using namespace stream;

int run_stream_bf16_64(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);
int run_stream_bf16_128(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);
int run_stream_bf16_256(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);
int run_stream_f16_64(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);
int run_stream_f16_128(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);
int run_stream_f16_256(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream);

namespace {

__global__ void window_kernel(uint32_t *start) {
    extern __shared__ __align__(1024) unsigned char smem[];
    *start = smem_u32(smem);
}

// Whether dynamic shared memory starts where the kernel's table loads expect it. Asked once per device, on a stream of its
// own (a stream that is being captured cannot be waited for); where it starts elsewhere, or nobody can tell, the calls
// stay with the kernels behind this one. KVC_STREAM=0 says no.
bool window_fits(int device) {
    static std::mutex mu;
    static int known[64] = {0};   // 1: yes, 2: no
    if (device < 0 || device >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (known[device]) return known[device] == 1;
    known[device] = 2;
    const char *e = std::getenv("KVC_STREAM");
    if (e && e[0] == '0') return false;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    KVC_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    cudaStream_t own = nullptr;
    uint32_t *start = nullptr;
    bool asked = cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking) == cudaSuccess && cudaMallocHost(&start, sizeof *start) == cudaSuccess;
    if (asked) {
        *start = 0;
        window_kernel<<<1, 1, 1024, own>>>(start);
        asked = cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(own) == cudaSuccess;
    }
    if (asked && *start == ST_WINDOW) known[device] = 1;
    if (start) (void)cudaFreeHost(start);
    if (own) (void)cudaStreamDestroy(own);
    (void)cudaGetLastError();
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    return known[device] == 1;
}

int source_kind(const KVSource &s, const AttnArgs &a) {
    if (s.kind == SRC_RAW) return s.dtype == a.q_dtype ? SK_RAW : -1;
    if (s.kind == SRC_AFFINE) return s.dtype != a.q_dtype ? -1 : s.bits == 4 ? SK_A4 : s.bits == 8 ? SK_A8 : -1;
    return s.bits == 2 ? SK_T2 : s.bits == 3 ? SK_T3 : s.bits == 4 ? SK_T4 : -1;
}

// Rows contiguous, every (batch, head) slab on a 16-byte boundary.
bool source_streams(const KVSource &s, int D) {
    const int64_t es = s.kind == SRC_RAW ? 2 : 4;
    if ((uintptr_t)s.data & 15 || (s.sb * es) & 15 || (s.sh * es) & 15) return false;
    if (s.kind == SRC_RAW) return s.st == D;
    if (s.st != (int64_t)D * s.bits / 32) return false;
    if (s.kind == SRC_TURBO)
        return s.norms && !((uintptr_t)s.norms & 15) && s.gst == 1 && !((s.gsb * 4) & 15) && !((s.gsh * 4) & 15);
    if (s.group != 32 && s.group != 64 && s.group != 128) return false;
    if (D % s.group || s.gst != D / s.group) return false;
    return !((uintptr_t)s.scales & 15) && !((uintptr_t)s.biases & 15) && !((s.gsb * 2) & 15) && !((s.gsh * 2) & 15);
}

StreamSource stream_source(const KVSource &s) {
    const int64_t es = s.kind == SRC_RAW ? 2 : 4, gs = s.kind == SRC_TURBO ? 4 : 2;
    StreamSource o;
    o.data = s.data;
    o.scales = s.kind == SRC_TURBO ? (const void *)s.norms : s.scales;
    o.biases = s.biases;
    o.sb = s.sb * es; o.sh = s.sh * es; o.gsb = s.gsb * gs; o.gsh = s.gsh * gs;
    return o;
}

bool stream_pick(const AttnArgs &a, StreamPick *out) {
    if (a.q_dtype != KVC_BF16 && a.q_dtype != KVC_F16) return false;
    if (a.D != 64 && a.D != 128 && a.D != 256) return false;
    if (a.mask.mode == KVC_MASK_ARRAY || a.q_rot || a.o_rot) return false;
    if (a.Hkv <= 0 || a.Hq % a.Hkv || a.T < 1 || a.T > (int64_t)1 << 30 || a.L < 1 || a.B < 1) return false;
    const int kk = source_kind(a.k, a), vk = source_kind(a.v, a);
    if (kk < 0 || vk < 0 || (kk == SK_RAW && vk == SK_RAW)) return false;
    if ((kk >= SK_T2) != (a.q_signs != nullptr) || (vk >= SK_T2) != (a.o_signs != nullptr)) return false;
    if (!source_streams(a.k, a.D) || !source_streams(a.v, a.D) || !window_fits(a.device)) return false;
    const int kg = a.k.kind == SRC_AFFINE ? a.k.group : 64, vg = a.v.kind == SRC_AFFINE ? a.v.group : 64;
    out->kk = kk; out->vk = vk;
    out->unit = std::min(kg, vg) == 32 ? 32 : 64;
    return true;
}

void stream_params(const AttnArgs &a, const StreamPick &pk, StreamParams *p) {
    p->q = a.q; p->out = a.out; p->out_dtype = a.q_dtype;
    p->q_sb = a.q_sb; p->q_sh = a.q_sh; p->q_sl = a.q_sl;
    p->o_sb = a.o_sb; p->o_sh = a.o_sh; p->o_sl = a.o_sl;
    p->k = stream_source(a.k); p->v = stream_source(a.v);
    p->q_signs = a.q_signs; p->q_calib = a.q_calib; p->o_signs = a.o_signs;
    // centroids travel times a power of two, so that the low halves of their f16 pairs stay clear of subnormals
    auto scaled = [](const float *cb, int bits, float *out, float *undo) {
        float big = 0.f;
        for (int i = 0; i < (1 << bits); ++i) big = std::max(big, std::fabs(cb[i]));
        int e = 0;
        if (big > 0.f && std::isfinite(big)) std::frexp(big, &e);
        e = std::min(std::max(e, -100), 100);
        for (int i = 0; i < (1 << bits); ++i) out[i] = std::ldexp(cb[i], 3 - e);
        *undo = std::ldexp(1.f, e - 3);
    };
    p->kcb_undo = p->vcb_undo = 1.f;
    if (a.k.kind == SRC_TURBO) scaled(a.k.codebook, a.k.bits, p->kcb, &p->kcb_undo);
    if (a.v.kind == SRC_TURBO) scaled(a.v.codebook, a.v.bits, p->vcb, &p->vcb_undo);
    p->groups_k = a.k.kind == SRC_AFFINE ? a.D / a.k.group : 0;
    p->groups_v = a.v.kind == SRC_AFFINE ? a.D / a.v.group : 0;
    // one table when keys and values share their codebook (the shipped tables depend on dim and bits only)
    const bool k_turbo = pk.kk >= SK_T2, v_turbo = pk.vk >= SK_T2;
    bool shared = k_turbo && v_turbo && pk.kk == pk.vk;
    for (int i = 0; shared && i < (1 << a.k.bits); ++i) shared = a.k.codebook[i] == a.v.codebook[i];
    p->v_table = (k_turbo && v_turbo && !shared && a.v.bits <= a.k.bits) ? (1 << (2 * a.k.bits)) * 256 : 0;   // behind the keys' table, which is no smaller
    p->B = a.B; p->Hq = a.Hq; p->Hkv = a.Hkv; p->L = a.L; p->T = (int32_t)a.T;
    p->causal = a.mask.mode == KVC_MASK_CAUSAL ? 1 : 0;
    p->causal_offset = a.mask.causal_offset;
    p->status = device_status_word(a.device);
    p->scale_log2 = a.scale * 1.4426950408889634f;
}

int run_stream_any(const AttnArgs &a, const StreamPick &pk, const StreamParams &p, StreamList *list, cudaStream_t stream) {
    if (a.q_dtype == KVC_BF16)
        return a.D == 64    ? run_stream_bf16_64(a, pk, p, list, stream)
               : a.D == 128 ? run_stream_bf16_128(a, pk, p, list, stream)
                            : run_stream_bf16_256(a, pk, p, list, stream);
    return a.D == 64    ? run_stream_f16_64(a, pk, p, list, stream)
           : a.D == 128 ? run_stream_f16_128(a, pk, p, list, stream)
                        : run_stream_f16_256(a, pk, p, list, stream);
}

}  // namespace

int launch_attention_stream(const AttnArgs &a, cudaStream_t stream) {
    StreamPick pk;
    if (!stream_pick(a, &pk) || (int64_t)(a.Hq / a.Hkv) * a.L > 64) return 0;
    StreamParams p = {};
    stream_params(a, pk, &p);
    if (!p.status) return 0;
    return run_stream_any(a, pk, p, nullptr, stream);
}

// `n` calls of one shape (lengths, arrays and scales of the codebooks' signs may differ) in one launch.
int launch_attention_stream_list(const AttnArgs *args, int n, cudaStream_t stream) {
    if (n < 1 || n > KVC_LIST_MAX) return 0;
    const AttnArgs &a0 = args[0];
    StreamPick pk;
    if (!stream_pick(a0, &pk) || (int64_t)(a0.Hq / a0.Hkv) * a0.L > 64) return 0;
    StreamParams p = {};
    stream_params(a0, pk, &p);
    if (!p.status) return 0;
    static thread_local StreamList list;
    list.n = n;
    for (int i = 0; i < n; ++i) {
        const AttnArgs &a = args[i];
        StreamPick own;
        if (!stream_pick(a, &own) || own.kk != pk.kk || own.vk != pk.vk || own.unit != pk.unit) return 0;
        if (a.B != a0.B || a.Hq != a0.Hq || a.Hkv != a0.Hkv || a.L != a0.L || a.D != a0.D || a.q_dtype != a0.q_dtype ||
            a.scale != a0.scale || a.mask.mode != a0.mask.mode || a.k.group != a0.k.group || a.v.group != a0.v.group ||
            a.q_sh != a0.q_sh || a.q_sl != a0.q_sl || a.o_sh != a0.o_sh || a.o_sl != a0.o_sl || a.device != a0.device)
            return 0;
        for (int j = 0; j < 16; ++j)
            if (a.k.codebook[j] != a0.k.codebook[j] || a.v.codebook[j] != a0.v.codebook[j]) return 0;
        StreamSeq &sq = list.seq[i];
        sq.q = a.q; sq.out = a.out;
        sq.k = stream_source(a.k); sq.v = stream_source(a.v);
        sq.q_signs = a.q_signs; sq.q_calib = a.q_calib; sq.o_signs = a.o_signs;
        sq.q_sb = a.q_sb; sq.o_sb = a.o_sb;
        sq.T = (int32_t)a.T;
        sq.causal_offset = a.mask.causal_offset;
    }
    return run_stream_any(a0, pk, p, &list, stream);
}

}  // namespace kvc
