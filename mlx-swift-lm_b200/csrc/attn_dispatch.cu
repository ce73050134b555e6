// Chooses the attention kernel for a call: the specialised decode kernels when
// the shape and representation match one, the general kernel otherwise.
#include "common.h"

#include <cstdlib>

namespace kvc {

int launch_attention_general(const AttnArgs &a, cudaStream_t stream);
int launch_attention_decode(const AttnArgs &a, cudaStream_t stream);
int launch_attention_affine(const AttnArgs &a, cudaStream_t stream);
int launch_attention_turbo(const AttnArgs &a, cudaStream_t stream);
int launch_attention_stream(const AttnArgs &a, cudaStream_t stream);
int launch_attention_f32_list(const AttnArgs *args, int n, cudaStream_t stream);
int launch_attention_stream_list(const AttnArgs *args, int n, cudaStream_t stream);
int launch_attention_decode_list(const AttnArgs *args, int n, cudaStream_t stream);
int launch_attention_chunk_packed(const AttnArgs &a, cudaStream_t stream);
int launch_attention_chunk_tc(const AttnArgs &a, cudaStream_t stream);
int launch_attention_chunk_one(const AttnArgs &a, cudaStream_t stream);
int launch_attention_chunk_materialized(const AttnArgs &a, cudaStream_t stream);
int launch_attention_chunk_packed_pairs(const AttnArgs &a, cudaStream_t stream);
int launch_attention_verify_tc_raw(const AttnArgs &a, cudaStream_t stream);

namespace {
// KVC_ATTENTION_PATH=general forces the general kernel (read once per process; used by
// tests that compare the two paths on the device from child processes).
bool force_general() {
    static const bool forced = [] {
        const char *e = std::getenv("KVC_ATTENTION_PATH");
        return e && e[0] == 'g';
    }();
    return forced;
}
}  // namespace

int launch_attention(const AttnArgs &a, cudaStream_t stream) {
    if (!force_general()) {
        int n = launch_attention_chunk_tc(a, stream);   // chunks over raw caches: tcgen05 kernel
        if (n > 0) return n;
        n = launch_attention_chunk_one(a, stream);   // ... under boolean array masks, and at head dim 256
        if (n > 0) return n;
        n = launch_attention_verify_tc_raw(a, stream);   // verify rounds of 17 ... 64 rows per KV head over raw caches
        if (n > 0) return n;
        n = launch_attention_decode(a, stream);
        if (n > 0) return n;
        n = launch_attention_affine(a, stream);
        if (n > 0) return n;
        n = launch_attention_turbo(a, stream);
        if (n > 0) return n;
        n = launch_attention_stream(a, stream);   // up to 64 rows per KV head over every other pair of representations
        if (n > 0) return n;
        n = launch_attention_chunk_materialized(a, stream);   // long chunks over packed caches: rows written out, then tcgen05
        if (n > 0) return n;
        n = launch_attention_chunk_packed(a, stream);
        if (n > 0) return n;
        n = launch_attention_chunk_packed_pairs(a, stream);   // other chunks over packed caches, and those under array masks
        if (n > 0) return n;
        n = launch_attention_f32_list(&a, 1, stream);   // decode and verify over single-precision affine caches
        if (n > 0) return n;
    }
    return launch_attention_general(a, stream);
}

namespace {
// Bytes of K and V one call reads.
double call_bytes(const AttnArgs &a) {
    auto row = [&](const KVSource &s) {
        if (s.kind == SRC_RAW) return (double)a.D * dtype_size(s.dtype);
        if (s.kind == SRC_TURBO) return (double)a.D * s.bits / 8 + 4;
        return (double)a.D * s.bits / 8 + 2.0 * (a.D / s.group) * dtype_size(s.dtype);
    };
    return (double)a.B * a.Hkv * a.T * (row(a.k) + row(a.v));
}
}  // namespace

// One launch costs its ramp, merge and tail once instead of once per call (about 8 us with the launch gap).
// Over packed caches the streaming kernel, which takes lists, reads at about 0.7 of the rate of the kernels
// specialised for head dim 128, so larger calls there stay launches of their own: the line is where the time
// it reads longer, at 4 TB/s, passes the fixed cost it saves.
int launch_attention_list(const AttnArgs *args, int n, cudaStream_t stream) {
    if (force_general() || n < 2) return 0;
    const AttnArgs &a = args[0];
    int made = launch_attention_decode_list(args, n, stream);
    if (made > 0) return made;
    made = launch_attention_f32_list(args, n, stream);
    if (made > 0) return made;
    if ((int64_t)(a.Hq / (a.Hkv > 0 ? a.Hkv : 1)) * a.L > 16) return 0;   // wider verify rounds: the tcgen05 kernel
    const bool specialised = a.D == 128 && ((a.k.kind == SRC_AFFINE && a.v.kind == SRC_AFFINE) || (a.k.kind == SRC_TURBO && a.v.kind == SRC_TURBO));
    if (specialised) {
        double bytes = 0;
        for (int i = 0; i < n; ++i) bytes += call_bytes(args[i]);
        if (0.43 * bytes / 4.0e6 > 8.0 * (n - 1)) return 0;
    }
    return launch_attention_stream_list(args, n, stream);
}

}  // namespace kvc
