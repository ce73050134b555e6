"""The TMA-staged tensor-core decode kernels over packed caches (affine codes,
TurboQuant indices) against the oracle, driven through the cache objects the
way attentionWithCacheUpdate drives them."""
import os
import subprocess
import sys
import tempfile

import numpy as np
import pytest
import torch

from helpers import TOL, bits_equal, max_abs_diff, oracle_f32, seeded, to_oracle, worst_excess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,bits,group,P", [
    (2, 28, 4, 128, 4, 64, 3000),    # Qwen2-7B shape, 4-bit (7 query heads per KV head)
    (2, 32, 8, 128, 8, 64, 1000),
    (1, 32, 8, 64, 8, 64, 1024),     # Llama-3.2-1B shape
    (2, 8, 2, 128, 4, 32, 200),
    (2, 8, 2, 128, 4, 128, 77),
    (1, 64, 8, 128, 8, 128, 129),
    (2, 16, 4, 64, 4, 64, 63),
])
def test_affine_decode_kernel_matches_oracle(kvc, oracle, cuda, dtype, B, Hq, Hkv, D, bits, group, P):
    g, o = kvc.QuantizedKVCache(group, bits), oracle.QuantizedKVCache(group, bits)
    k = seeded((B, Hkv, P, D), 1, dtype, outlier_frac=0.01)
    v = seeded((B, Hkv, P, D), 2, dtype, outlier_frac=0.01)
    g.update_quantized(k.to(cuda), v.to(cuda))
    o.update_quantized(to_oracle(k), to_oracle(v))
    scale = D ** -0.5
    for step in range(3):
        q = seeded((B, Hq, 1, D), 10 + step, dtype)
        k1, v1 = seeded((B, Hkv, 1, D), 20 + step, dtype), seeded((B, Hkv, 1, D), 30 + step, dtype)
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), scale)
        ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, scale)
        # the x20 outlier channels of V make some outputs larger than 1: the stated absolute
        # tolerance on the arithmetic plus one spacing of the 16-bit store (helpers.worst_excess)
        assert worst_excess(out, ref, dtype) <= 0, f"step {step}"
    assert kvc.lib().kvc_device_status() == 0
    for a, b in zip(g.state, o.state):
        assert bits_equal(a, np.ascontiguousarray(b))


def test_affine_small_causal_chunk(kvc, oracle, cuda):
    B, Hq, Hkv, D, L = 2, 4, 2, 128, 6
    g, o = kvc.QuantizedKVCache(64, 4), oracle.QuantizedKVCache(64, 4)
    k, v = seeded((B, Hkv, 500, D), 1, torch.bfloat16), seeded((B, Hkv, 500, D), 2, torch.bfloat16)
    g.update_quantized(k.to(cuda), v.to(cuda))
    o.update_quantized(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, torch.bfloat16)
    k1, v1 = seeded((B, Hkv, L, D), 4, torch.bfloat16), seeded((B, Hkv, L, D), 5, torch.bfloat16)
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), 0.09, "causal")
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, 0.09, "causal")
    assert max_abs_diff(out, ref) <= 2e-2


def test_affine_kernel_with_large_queries_and_scales(kvc, oracle, cuda):
    """Outlier channels x20 in K/V and queries of magnitude ~10: the f16 operand
    path must stay within tolerance."""
    B, Hq, Hkv, D = 1, 8, 2, 128
    g, o = kvc.QuantizedKVCache(64, 4), oracle.QuantizedKVCache(64, 4)
    k = seeded((B, Hkv, 700, D), 1, torch.bfloat16, outlier_frac=0.05)
    v = seeded((B, Hkv, 700, D), 2, torch.bfloat16, outlier_frac=0.05)
    g.update_quantized(k.to(cuda), v.to(cuda))
    o.update_quantized(to_oracle(k), to_oracle(v))
    q = (seeded((B, Hq, 1, D), 3, torch.float32) * 4).to(torch.bfloat16)
    k1, v1 = seeded((B, Hkv, 1, D), 4, torch.bfloat16), seeded((B, Hkv, 1, D), 5, torch.bfloat16)
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5)
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5)
    # outlier channels make outputs larger than 1: stated tolerance plus one spacing of the bf16 store
    assert worst_excess(out, ref, torch.bfloat16) <= 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,P,kb,vb", [
    (1, 64, 8, 3000, 3, 4),     # Llama-3-70B head layout, 3-bit keys / 4-bit values
    (2, 8, 2, 700, 4, 4),
    (2, 8, 2, 130, 4, 2),
    (1, 16, 4, 257, 3, 3),
    (2, 4, 4, 64, 2, 2),
])
def test_turbo_decode_kernel_matches_oracle(kvc, oracle, cuda, dtype, B, Hq, Hkv, P, kb, vb):
    """The lookup-table tensor-core decode kernel over packed TurboQuant rows (D = 128)."""
    D = 128
    kw = dict(bits=max(kb, vb), key_bits=kb, value_bits=vb)
    g = kvc.TurboQuantKVCache(**kw)
    o = oracle.TurboQuantKVCache(**kw)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    g.encode_new_token(k.to(cuda), v.to(cuda))
    o.encode_new_token(to_oracle(k), to_oracle(v))
    scale = D ** -0.5
    n0 = kvc.launch_count(reset=True)
    for step in range(3):
        q = seeded((B, Hq, 1, D), 10 + step, dtype)
        k1, v1 = seeded((B, Hkv, 1, D), 20 + step, dtype), seeded((B, Hkv, 1, D), 30 + step, dtype)
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), scale)
        ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, scale)
        assert max_abs_diff(out, ref) <= TOL[dtype], f"step {step}"
    # one encode launch and ONE attention launch per step: the merge is folded into the kernel
    assert kvc.launch_count(reset=True) <= 6
    assert kvc.lib().kvc_device_status() == 0
    for a, b in zip(g.state, o.state):
        assert bits_equal(a, np.ascontiguousarray(b))


def test_turbo_kernel_small_causal_chunk(kvc, oracle, cuda):
    B, Hq, Hkv, D, L = 2, 4, 2, 128, 4     # 2 query heads per KV head x 4 positions = 8 rows
    kw = dict(bits=4, key_bits=3, value_bits=4)
    g = kvc.TurboQuantKVCache(**kw)
    o = oracle.TurboQuantKVCache(**kw)
    k, v = seeded((B, Hkv, 500, D), 1, torch.bfloat16), seeded((B, Hkv, 500, D), 2, torch.bfloat16)
    g.encode_new_token(k.to(cuda), v.to(cuda))
    o.encode_new_token(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, torch.bfloat16)
    k1, v1 = seeded((B, Hkv, L, D), 4, torch.bfloat16), seeded((B, Hkv, L, D), 5, torch.bfloat16)
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), 0.09, "causal")
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, 0.09, "causal")
    assert max_abs_diff(out, ref) <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,bits,group,P,L", [
    (2, 8, 2, 4, 64, 300, 64),       # prefill chunk over a quantised prefix: 256 rows per KV head
    (1, 28, 4, 4, 64, 2100, 6),      # verify round, Qwen2-7B layout: 7 heads x 6 positions = 42 rows
    (1, 8, 2, 8, 64, 500, 40),       # 8-bit, 160 rows: three row blocks, the last one partial
    (1, 4, 1, 4, 32, 4000, 5),       # group 32; one unit, long prefix: several splits + merge
    (2, 8, 2, 8, 128, 77, 33),       # group 128
    (1, 2, 1, 4, 128, 0, 130),       # chunk into an empty cache
])
def test_affine_chunk_kernel_matches_oracle(kvc, oracle, cuda, dtype, B, Hq, Hkv, bits, group, P, L):
    """Multi-token chunks over the affine cache: dequantise-to-shared-memory tensor-core kernel; the verify round
    of the Qwen2-7B layout (groups of 64, 42 rows per kv head) goes to the tcgen05 verify kernel."""
    D = 128
    g, o = kvc.QuantizedKVCache(group, bits, reserve_tokens=P + L), oracle.QuantizedKVCache(group, bits)
    if P:
        k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
        g.update_quantized(k.to(cuda), v.to(cuda))
        o.update_quantized(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, dtype)
    k1, v1 = seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    kvc.launch_count(reset=True)
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, "causal")
    launches = kvc.launch_count(reset=True)
    if group == 64 and 16 < (Hq // Hkv) * L <= 64:
        assert 3 <= launches <= 4       # quantise-append + the tcgen05 verify kernel behind its query kernel (+ merge)
    else:
        assert launches == 2            # quantise-append + one attention launch
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, "causal")
    assert max_abs_diff(out, ref) <= TOL[dtype]
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,kb,vb,P,L", [
    (1, 64, 8, 3, 4, 2100, 6),       # verify round, Llama-3-70B layout: 8 heads x 6 positions = 48 rows
    (2, 8, 2, 4, 4, 300, 40),        # 160 rows per KV head
    (1, 4, 1, 3, 3, 3000, 5),        # one unit, long prefix: several splits + merge + rotation
    (1, 8, 2, 4, 2, 130, 17),
    (1, 4, 2, 2, 2, 64, 9),
])
def test_turbo_chunk_kernel_matches_oracle(kvc, oracle, cuda, dtype, B, Hq, Hkv, kb, vb, P, L):
    """Verify rounds / chunks over the TurboQuant cache (compressed phase)."""
    D = 128
    kw = dict(bits=max(kb, vb), key_bits=kb, value_bits=vb)
    g = kvc.TurboQuantKVCache(reserve_tokens=P + L, **kw)
    o = oracle.TurboQuantKVCache(**kw)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    g.encode_new_token(k.to(cuda), v.to(cuda))
    o.encode_new_token(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, dtype)
    k1, v1 = seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    kvc.launch_count(reset=True)
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, "causal")
    # encode-append + one attention launch; the tensor-core verify kernel (2- / 3-bit keys, 4-bit values, 9..128
    # rows per kv head) adds the query rotation in front, the output rotation behind and a merge when it splits
    assert kvc.launch_count(reset=True) <= 5
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, "causal")
    assert max_abs_diff(out, ref) <= TOL[dtype]
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("bits", [4, 8])
def test_varlen_decode_over_independent_caches(kvc, oracle, cuda, bits):
    """A ragged decode batch held the reference's way (one cache per sequence): the var-len call
    appends and attends all of them in two launches; per-sequence results equal the oracle's and
    the per-cache calls', and the caches hold identical codes afterwards."""
    Hq, Hkv, D, dtype = 28, 4, 128, torch.bfloat16
    lengths = [37, 64, 1, 300, 2049, 511, 130, 65, 1000, 5]
    n = len(lengths)
    var = [kvc.QuantizedKVCache(64, bits, reserve_tokens=t + 8) for t in lengths]
    one = [kvc.QuantizedKVCache(64, bits, reserve_tokens=t + 8) for t in lengths]
    orc = [oracle.QuantizedKVCache(64, bits) for _ in lengths]
    for i, t in enumerate(lengths):
        k, v = seeded((1, Hkv, t, D), 10 * i, dtype), seeded((1, Hkv, t, D), 10 * i + 1, dtype)
        for c in (var[i], one[i]):
            c.update_quantized(k.to(cuda), v.to(cuda))
        orc[i].update_quantized(to_oracle(k), to_oracle(v))
    scale = D ** -0.5
    for step in range(3):
        q = [seeded((1, Hq, 1, D), 1000 + 100 * step + i, dtype) for i in range(n)]
        k = [seeded((1, Hkv, 1, D), 2000 + 100 * step + i, dtype) for i in range(n)]
        v = [seeded((1, Hkv, 1, D), 3000 + 100 * step + i, dtype) for i in range(n)]
        dq, dk, dv = [t.to(cuda) for t in q], [t.to(cuda) for t in k], [t.to(cuda) for t in v]
        outs = [torch.empty((1, Hq, 1, D), dtype=dtype, device=cuda) for _ in range(n)]
        kvc.launch_count(reset=True)
        kvc.DecodeStep(var, dq, dk, dv, outs, scale).run_varlen()
        assert kvc.launch_count(reset=True) == 2
        for i in range(n):
            ref = oracle.attention_with_cache_update(to_oracle(q[i]), to_oracle(k[i]), to_oracle(v[i]), orc[i], scale)
            assert max_abs_diff(outs[i], ref) <= TOL[dtype], f"step {step} sequence {i}"
            single = one[i].attention(dq[i], dk[i], dv[i], scale)
            assert max_abs_diff(outs[i], to_oracle(single)) <= 1e-2
    assert kvc.lib().kvc_device_status() == 0
    for a, b, o in zip(var, one, orc):
        assert a.offset == b.offset == o.offset
        for x, y in zip(a.state, b.state):
            assert torch.equal(x, y)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,bits,group,P,L,mask", [
    (2, 8, 2, 128, 4, 64, 260, 640, "causal"),     # 80 blocks of 128 rows on a quantised prefix
    (1, 16, 4, 128, 8, 32, 0, 600, "causal"),      # chunk into an empty cache, last block partial
    (5, 16, 2, 128, 2, 128, 1000, 128, "none"),    # 2-bit codes, no mask, ragged last key tile
    (2, 32, 8, 64, 4, 64, 777, 300, "causal"),     # head dim 64
])
def test_affine_prefill_chunk_on_the_tensor_core_kernel(kvc, oracle, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, D, bits,
                                                        group, P, L, mask):
    """Long chunks over the affine cache: the rows are written out once as f16 / bf16 and the
    contraction runs on the tcgen05 kernel."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    g, o = kvc.QuantizedKVCache(group, bits), oracle.QuantizedKVCache(group, bits)
    if P:
        k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
        g.update_quantized(k.to(cuda), v.to(cuda))
        o.update_quantized(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, dtype)
    k1, v1 = seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    capfd.readouterr()
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, mask)
    torch.cuda.synchronize()
    err = capfd.readouterr().err
    assert "chunk_mat" in err and "chunk_tc" in err
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, mask)
    assert max_abs_diff(out, ref) <= TOL[dtype]
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,kb,vb,P,L,mask", [
    (2, 8, 2, 128, 3, 4, 260, 640, "causal"),
    (1, 16, 4, 128, 4, 4, 1, 600, "causal"),
    (5, 16, 2, 128, 2, 2, 1000, 128, "none"),
    (3, 8, 8, 128, 4, 2, 500, 512, "causal"),
    (2, 32, 8, 64, 3, 3, 777, 300, "causal"),      # head dim 64
])
def test_turbo_prefill_chunk_on_the_tensor_core_kernel(kvc, oracle, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, D, kb, vb,
                                                       P, L, mask):
    """Long chunks over the compressed TurboQuant cache: rows written out in the rotated basis,
    queries rotated in, outputs rotated back, contraction on the tcgen05 kernel."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    kw = dict(bits=max(kb, vb), key_bits=kb, value_bits=vb)
    g, o = kvc.TurboQuantKVCache(**kw), oracle.TurboQuantKVCache(**kw)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    g.encode_new_token(k.to(cuda), v.to(cuda))
    o.encode_new_token(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, dtype)
    k1, v1 = seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    capfd.readouterr()
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, mask)
    torch.cuda.synchronize()
    err = capfd.readouterr().err
    assert "chunk_mat" in err and "chunk_tc" in err
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, mask)
    assert max_abs_diff(out, ref) <= TOL[dtype]
    assert kvc.lib().kvc_device_status() == 0


def test_calibrated_turbo_prefill_chunk_on_the_tensor_core_kernel(kvc, oracle, cuda, capfd, monkeypatch):
    """Correlated keys: the cache calibrates at compression, and the chunk's rotated queries carry the
    calibration scale."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    B, Hq, Hkv, D, P, L = 2, 8, 2, 128, 600, 640
    dtype = torch.bfloat16
    kw = dict(bits=4, key_bits=3, value_bits=4)
    g, o = kvc.TurboQuantKVCache(**kw), oracle.TurboQuantKVCache(**kw)
    q = seeded((B, Hq, P, D), 1, dtype)
    from test_gpu_turbo import _correlated_keys
    k, v = _correlated_keys((B, Hkv, P, D), 2, dtype), seeded((B, Hkv, P, D), 3, dtype)
    g.attention(q.to(cuda), k.to(cuda), v.to(cuda), D ** -0.5, "causal")          # raw prefill
    oracle.attention_with_cache_update(to_oracle(q), to_oracle(k), to_oracle(v), o, D ** -0.5, "causal")
    q1, k1, v1 = seeded((B, Hq, 1, D), 4, dtype), _correlated_keys((B, Hkv, 1, D), 5, dtype), seeded((B, Hkv, 1, D), 6, dtype)
    g.attention(q1.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5)                  # compresses and calibrates
    oracle.attention_with_cache_update(to_oracle(q1), to_oracle(k1), to_oracle(v1), o, D ** -0.5)
    assert g.is_compressed and len(g.state) == 5 and len(o.state) == 5
    q2 = seeded((B, Hq, L, D), 7, dtype)
    k2, v2 = _correlated_keys((B, Hkv, L, D), 8, dtype), seeded((B, Hkv, L, D), 9, dtype)
    capfd.readouterr()
    out = g.attention(q2.to(cuda), k2.to(cuda), v2.to(cuda), D ** -0.5, "causal")
    torch.cuda.synchronize()
    assert "chunk_mat" in capfd.readouterr().err
    ref = oracle.attention_with_cache_update(to_oracle(q2), to_oracle(k2), to_oracle(v2), o, D ** -0.5, "causal")
    from helpers import worst_excess
    assert worst_excess(out, ref, dtype) <= 0
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,bits,group,P,L", [
    (2, 28, 4, 4, 64, 1000, 6),      # Qwen2-7B layout, verify round: 42 rows per kv head; tensor-core kernel, split keys
    (1, 32, 4, 8, 64, 517, 5),       # 8-bit codes, 40 rows: tensor-core kernel
    (2, 16, 2, 8, 64, 1300, 6),      # 8-bit codes, 48 rows, bigger
    (2, 8, 1, 4, 128, 2049, 8),      # 64 rows; group 128: units of eight rows on the decode kernel
    (1, 17, 1, 4, 64, 300, 1),       # 17 heads on one kv head, one position, no causal limit to speak of
    (16, 56, 8, 4, 64, 700, 6),      # 128 units: one CTA each, six tiles in a row, no split
    (1, 8, 1, 4, 64, 120, 8),        # 64 rows; the chunk itself crosses the first tile boundary
    (40, 20, 4, 4, 64, 300, 4),      # 160 units of three tiles on fewer SMs: CTAs that walk two or three units
])
def test_affine_verify_rounds(kvc, oracle, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, bits, group, P, L):
    """17 to 64 query rows per kv head over the affine cache. 4- or 8-bit codes in groups of 64: the tcgen05 verify
    kernel (rows decoded once per kv head). Otherwise the group is cut into units of eight rows, each streamed
    through the 8-row decode kernel with its own causal limits (one attention launch)."""
    D = 128
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    g, o = kvc.QuantizedKVCache(group, bits), oracle.QuantizedKVCache(group, bits)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    g.update_quantized(k.to(cuda), v.to(cuda))
    o.update_quantized(to_oracle(k), to_oracle(v))
    mask = "causal" if L > 1 else "none"
    for rnd in range(2):
        q = seeded((B, Hq, L, D), 3 + rnd, dtype)
        k1, v1 = seeded((B, Hkv, L, D), 5 + rnd, dtype), seeded((B, Hkv, L, D), 7 + rnd, dtype)
        kvc.launch_count(reset=True)
        capfd.readouterr()
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, mask)
        torch.cuda.synchronize()
        launches, err = kvc.launch_count(reset=True), capfd.readouterr().err
        if group == 64:
            assert "verify_tc affine" in err
        else:
            assert launches == 2            # quantise-append + one attention launch
        ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, mask)
        assert max_abs_diff(out, ref) <= TOL[dtype], f"round {rnd}"
        assert g.trim(max(L - 1, 0)) == o.trim(max(L - 1, 0))
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("kind", ["turbo_k3v4", "turbo_k4v4", "affine4"])
def test_decode_at_every_context_length_around_the_stage_boundaries(kvc, oracle, cuda, kind):
    """The 15-warp decode kernels stream 240-token stages and cut the last one short at the stored rows
    rounded up to 256: every context length around multiples of 240 and of 256 (and the first tokens of
    an empty cache) against the oracle, in one growing cache."""
    B, Hq, Hkv, D = 1, 8, 1, 128
    dtype = torch.bfloat16
    if kind == "affine4":
        g, o = kvc.QuantizedKVCache(64, 4), oracle.QuantizedKVCache(64, 4)
    else:
        kw = dict(bits=4, key_bits=3 if kind == "turbo_k3v4" else 4, value_bits=4)
        g, o = kvc.TurboQuantKVCache(**kw), oracle.TurboQuantKVCache(**kw)
    scale = D ** -0.5
    check_at = set(range(1, 6)) | {t + d for t in (240, 256, 480, 512, 720, 768, 960, 1024) for d in (-2, -1, 0, 1, 2)}
    T = 0
    for target in sorted(check_at):
        fill = target - 1 - T               # rows to add before the decode step that makes the context `target`
        if fill > 0:
            k, v = seeded((B, Hkv, fill, D), 1000 + target, dtype), seeded((B, Hkv, fill, D), 2000 + target, dtype)
            if kind == "affine4":
                g.update_quantized(k.to(cuda), v.to(cuda))
                o.update_quantized(to_oracle(k), to_oracle(v))
            else:
                g.encode_new_token(k.to(cuda), v.to(cuda))
                o.encode_new_token(to_oracle(k), to_oracle(v))
            T += fill
        q = seeded((B, Hq, 1, D), 3000 + target, dtype)
        k1, v1 = seeded((B, Hkv, 1, D), 4000 + target, dtype), seeded((B, Hkv, 1, D), 5000 + target, dtype)
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), scale)
        ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, scale)
        T += 1
        assert g.offset == o.offset == T == target
        assert max_abs_diff(out, ref) <= TOL[dtype], f"context {target}"
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype,B,Hq,Hkv,kb,vb,P,L,written", [
    (torch.bfloat16, 1, 32, 8, 3, 4, 47, 17, False),      # 64 keys: one tile, decoded in the tile loop
    (torch.bfloat16, 1, 32, 8, 3, 4, 48, 17, True),       # 65
    (torch.float16, 2, 28, 4, 2, 2, 111, 10, True),       # 70 rows of a group
    (torch.float16, 3, 8, 8, 4, 2, 130, 65, True),        # one head a group, 65 positions
    (torch.bfloat16, 1, 64, 8, 3, 3, 1000, 33, True),
])
def test_short_turbo_chunk_with_rows_written_out(kvc, oracle, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, kb, vb, P, L, written):
    """Short chunks over TurboQuant caches: which kernels take them, and the stated 2e-2 plus one spacing of the store."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    D = 128
    g, o = _caches(kvc, oracle, cuda, dtype, dict(key_bits=kb, value_bits=vb), B, Hkv, D, P)
    q, k1, v1 = seeded((B, Hq, L, D), 3, dtype), seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    capfd.readouterr()
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, "causal")
    torch.cuda.synchronize()
    assert ("rows written out" in capfd.readouterr().err) == written
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, "causal")
    assert worst_excess(out, ref, dtype) <= 0
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype,kw,Hq,Hkv,D,P,L", [
    (torch.float16, dict(key_bits=8, value_bits=4), 8, 2, 128, 1, 1),       # a single cached row
    (torch.bfloat16, dict(key_bits=8, value_bits=3), 28, 4, 128, 61, 1),    # 62 rows: the last block is short
    (torch.bfloat16, dict(key_bits=0, value_bits=4), 4, 1, 256, 2050, 1),
    (torch.float16, dict(key_bits=0, value_bits=2), 4, 4, 64, 79, 1),
    (torch.bfloat16, dict(key_bits=3, value_bits=3), 8, 8, 64, 640, 3),     # 48-bit quarters of a row
    (torch.bfloat16, dict(key_bits=4, value_bits=2), 4, 1, 256, 255, 2),    # two tables
    (torch.float16, dict(key_bits=8, value_bits=2), 16, 2, 128, 300, 2),    # 16 rows: two column blocks
    (torch.bfloat16, dict(key_bits=2, value_bits=2), 8, 1, 64, 130, 7),     # 56 rows: four row units
    (torch.bfloat16, dict(key_bits=3, value_bits=4, affine_values=True), 8, 2, 128, 500, 1),
    (torch.float16, dict(bits=4, group=32), 4, 1, 256, 333, 1),
    (torch.bfloat16, dict(bits=8, group=128), 8, 2, 256, 64, 1),
    (torch.bfloat16, dict(bits=8, group=32), 8, 8, 64, 1000, 2),
])
def test_stream_kernel_matches_oracle(kvc, oracle, cuda, dtype, kw, Hq, Hkv, D, P, L):
    """Every family of representations of the warp-streaming kernel, at the edges of its blocks (16 tokens),
    tiles (64) and row units (8 / 16). Bound: the stated 2e-2 on the arithmetic plus one spacing of the store."""
    B = 2
    if "group" in kw:
        make = lambda m: m.QuantizedKVCache(kw["group"], kw["bits"])
    else:
        make = lambda m: m.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw)
    g, o = make(kvc), make(oracle)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    if "group" in kw:
        g.update_quantized(k.to(cuda), v.to(cuda))
        o.update_quantized(to_oracle(k), to_oracle(v))
    else:
        g.encode_new_token(k.to(cuda), v.to(cuda))
        o.encode_new_token(to_oracle(k), to_oracle(v))
    for step in range(2):
        q = seeded((B, Hq, L, D), 10 + step, dtype)
        k1, v1 = seeded((B, Hkv, L, D), 20 + step, dtype), seeded((B, Hkv, L, D), 30 + step, dtype)
        mask = "causal" if L > 1 else "none"
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, mask)
        ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5, mask)
        assert worst_excess(out, ref, dtype) <= 0, f"step {step}"
    for a, b in zip(g.state, o.state):
        assert bits_equal(a, np.ascontiguousarray(b))


@pytest.mark.parametrize("dtype,kw,Hq,Hkv,D,P,L,mask", [
    (torch.bfloat16, None, 4, 1, 256, 511, 129, "window"),        # odd row pitch, 129 rows of a head: three row blocks
    (torch.float16, None, 4, 2, 64, 63, 1, "window"),             # a single row; 64 keys fill one tile
    (torch.bfloat16, None, 8, 8, 128, 100, 37, "heads"),          # a mask per head, one row fully masked
    (torch.bfloat16, None, 4, 1, 128, 70, 20, "additive"),
    (torch.bfloat16, dict(bits=8, group=32), 4, 1, 256, 200, 70, "window"),
    (torch.bfloat16, dict(key_bits=8, value_bits=3), 4, 1, 256, 200, 70, "causal"),
    (torch.bfloat16, dict(key_bits=0, value_bits=4), 8, 2, 128, 130, 40, "causal"),
    (torch.float16, dict(key_bits=0, value_bits=2), 8, 2, 64, 130, 40, "window"),     # keys used in place
    (torch.float16, dict(key_bits=3, value_bits=4), 16, 16, 64, 129, 90, "causal"),
])
def test_masked_and_mixed_chunks_match_oracle(kvc, oracle, cuda, dtype, kw, Hq, Hkv, D, P, L, mask):
    """Chunks under array masks and chunks over the layouts that are decoded to operand pairs. Bound: the stated
    2e-2 on the arithmetic plus one spacing of the store."""
    B, T = 2, P + L
    if kw is None:
        make = lambda m: m.KVCacheSimple()
    elif "group" in kw:
        make = lambda m: m.QuantizedKVCache(kw["group"], kw["bits"])
    else:
        make = lambda m: m.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw)
    g, o = make(kvc), make(oracle)
    fill = "update" if kw is None else "update_quantized" if "group" in kw else "encode_new_token"
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
    getattr(g, fill)(k.to(cuda), v.to(cuda))
    getattr(o, fill)(to_oracle(k), to_oracle(v))
    q = seeded((B, Hq, L, D), 3, dtype)
    k1, v1 = seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
    row, col = torch.arange(P, T)[:, None], torch.arange(T)[None, :]
    m = {"window": (col <= row) & (row - col < 48), "causal": "causal"}.get(mask)
    if mask == "heads":
        m = torch.rand((B, Hq, L, T), generator=torch.Generator().manual_seed(6)) < 0.3
        m[:, :, 5] = False
    elif mask == "additive":
        m = torch.where(col <= row, -0.01 * (row - col).float(), torch.tensor(float("-inf")))
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, m if isinstance(m, str) else m.to(cuda))
    ref = oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, D ** -0.5,
                                             m if isinstance(m, str) else m.numpy())
    assert worst_excess(out, ref, dtype) <= 0
    assert kvc.lib().kvc_device_status() == 0


def _caches(kvc, oracle, cuda, dtype, kw, B, Hkv, D, P, gain=1.0):
    if kw is None:
        make, fill = (lambda m: m.KVCacheSimple()), "update"
    elif "group" in kw:
        make, fill = (lambda m: m.QuantizedKVCache(kw["group"], kw["bits"])), "update_quantized"
    else:
        make, fill = (lambda m: m.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw)), "encode_new_token"
    g, o = make(kvc), make(oracle)
    k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype) * gain
    getattr(g, fill)(k.to(cuda), v.to(cuda))
    getattr(o, fill)(to_oracle(k), to_oracle(v))
    return g, o


@pytest.mark.parametrize("dtype,kw,Hq,lists", [
    *[(torch.float16, dict(bits=b, group=gr), Hq, False) for b, gr in ((8, 128), (8, 64), (8, 32), (4, 64), (4, 128)) for Hq in (8, 16, 24, 32)],
    (torch.bfloat16, dict(bits=8, group=128), 24, False),
    (torch.float16, dict(bits=4, group=64), 80, False),         # ten rows a group
    (torch.float16, dict(bits=8, group=64), 24, True),          # independent sequences
    (torch.float16, dict(bits=4, group=64), 24, True),
    (torch.float16, dict(key_bits=3, value_bits=4), 24, False),
    (torch.float16, dict(key_bits=4, value_bits=2), 24, False),
    (torch.float16, None, 24, False),                            # a raw cache
    (torch.bfloat16, None, 32, False),
])
def test_ring_entries_are_read_before_they_are_filled_again(kvc, oracle, cuda, dtype, kw, Hq, lists):
    """Contexts that walk the rings of packed tiles several times, out of L2, where a copy is back soonest: run after run
    the same bits, and every row within 2^-7 of the oracle's sums (a 16-bit query, weight and store err by up to 2^-11
    each for f16, a bf16 store by 2^-9; sums over 9 000 tokens keep the ratio; a lost tile of 64 tokens is 2^-3.6)."""
    B, Hkv, D, P = 2, 8, 128, 9000
    n = B if lists else 1
    g, o = [], []
    for i in range(n):
        a, b = _caches(kvc, oracle, cuda, dtype, kw, B // n, Hkv, D, P - i)
        g.append(a)
        o.append(b)
    q, k1, v1 = seeded((B, Hq, 1, D), 3, dtype), seeded((B, Hkv, 1, D), 4, dtype), seeded((B, Hkv, 1, D), 5, dtype)
    dq, dk, dv = ([t.to(cuda)[i:i + B // n] for i in range(n)] for t in (q, k1, v1))
    runs = []
    for _ in range(12):
        outs = [torch.empty_like(t) for t in dq]
        if lists:
            kvc.DecodeStep(g, dq, dk, dv, outs, D ** -0.5).run_varlen()
        else:
            outs[0].copy_(g[0].attention(dq[0], dk[0], dv[0], D ** -0.5))
        runs.append(torch.cat(outs).cpu())
        kvc.trim_prompt_cache(g, 1)
    assert all(torch.equal(r, runs[0]) for r in runs[1:])
    for i in range(n):
        at = slice(i * (B // n), (i + 1) * (B // n))
        ref = torch.from_numpy(oracle_f32(oracle.attention_with_cache_update(
            to_oracle(q.float()[at]), to_oracle(k1[at]), to_oracle(v1[at]), o[i], D ** -0.5))).double()
        assert float(((runs[0][at].double() - ref).norm(dim=-1) / ref.norm(dim=-1)).max()) <= 2.0 ** -7
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype,kw,Hq,Hkv,D,P,L,mask", [
    (torch.float16, dict(key_bits=8, value_bits=4), 32, 8, 128, 700, 1, "none"),       # stream kernel: two MMAs a key, three a value
    (torch.float16, dict(key_bits=0, value_bits=3), 8, 4, 256, 700, 1, "none"),
    (torch.float16, dict(key_bits=4, value_bits=4), 16, 8, 64, 700, 2, "causal"),
    (torch.float16, dict(key_bits=8, value_bits=2), 32, 4, 128, 333, 2, "causal"),     # two column blocks
    (torch.float16, dict(bits=4, group=32), 8, 4, 256, 700, 1, "none"),
    (torch.bfloat16, None, 4, 1, 256, 300, 100, "window"),                             # row-split kernel: P as a pair
    (torch.float16, None, 4, 2, 128, 300, 40, "window"),
    (torch.float16, dict(key_bits=8, value_bits=4), 8, 2, 128, 300, 70, "causal"),     # operand pairs
    (torch.float16, dict(key_bits=0, value_bits=4), 8, 2, 64, 300, 70, "causal"),
    (torch.float16, dict(key_bits=3, value_bits=4), 4, 1, 256, 300, 70, "window"),
    (torch.float16, dict(key_bits=4, value_bits=4, affine_values=True), 8, 2, 128, 300, 70, "causal"),
    (torch.float16, dict(bits=8, group=64), 4, 1, 256, 300, 70, "causal"),
])
def test_packed_calls_err_by_the_store_alone(kvc, oracle, cuda, dtype, kw, Hq, Hkv, D, P, L, mask):
    """The arithmetic keeps more than the output type holds. Reference: the oracle's sums for the same codes with an
    unrounded (f32) output. Rounding that to the output type errs by `ideal`; independent arithmetic errors e add in
    quadrature, so 1.05 * ideal allows e up to 0.32 * ideal, 2^-14 of the result for f16. Operands held as one f16
    would err by about 2^-12, as one bf16 by 2^-9."""
    g, o = _caches(kvc, oracle, cuda, dtype, kw, 2, Hkv, D, P)
    T = P + L
    q, k1, v1 = seeded((2, Hq, L, D), 3, dtype), seeded((2, Hkv, L, D), 4, dtype), seeded((2, Hkv, L, D), 5, dtype)
    row, col = torch.arange(P, T)[:, None], torch.arange(T)[None, :]
    m = (col <= row) & (row - col < 100) if mask == "window" else mask
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, m if isinstance(m, str) else m.to(cuda))
    ref = torch.from_numpy(oracle_f32(oracle.attention_with_cache_update(
        to_oracle(q.float()), to_oracle(k1), to_oracle(v1), o, D ** -0.5, m if isinstance(m, str) else m.numpy())))
    ideal = float((ref.to(dtype).double() - ref.double()).norm())
    assert float((out.cpu().double() - ref.double()).norm()) <= 1.05 * ideal


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("kw", [dict(key_bits=0, value_bits=2), dict(key_bits=0, value_bits=3), dict(key_bits=0, value_bits=4),
                                dict(key_bits=3, value_bits=4), dict(key_bits=4, value_bits=2), dict(key_bits=3, value_bits=3, own_codebooks=True),
                                dict(key_bits=2, value_bits=2, own_codebooks=True), dict(key_bits=4, value_bits=4, own_codebooks=True),
                                dict(key_bits=3, value_bits=4, affine_values=True), dict(bits=4, group=32), dict(bits=8, group=32)])
def test_stream_kernel_values_of_every_width(kvc, oracle, cuda, kw, D):
    """A lane's run of a value row is 16 to 128 bits long, 24, 48 and 96 with 3-bit indices; tables lie one behind the other
    where keys and values have their own. One to 33 tokens, fewer and more than eight rows. Bound as above, 1.05 * ideal
    (1.2 where `ideal` is a mean over few roundings); at head dim 128, where kernels with operands of one f16 take the plain
    pairs of representations, the stated 2e-2 and one spacing."""
    dtype, B, Hkv = torch.float16, 2, 2
    kw = dict(kw)
    pairs = D != 128 or kw.get("key_bits") == 0 or "affine_values" in kw
    own = kw.pop("own_codebooks", False)
    for P, L, Hq in ((0, 1, 8), (15, 1, 4), (31, 2, 16)):
        if "group" in kw:
            g, o = kvc.QuantizedKVCache(kw["group"], kw["bits"]), oracle.QuantizedKVCache(kw["group"], kw["bits"])
        else:
            both = dict(bits=max(kw["key_bits"], kw["value_bits"]), **kw)
            g, o = kvc.TurboQuantKVCache(**both), oracle.TurboQuantKVCache(**both)
            if own:
                o._vcb = 1.25 * oracle.codebook(D, kw["value_bits"])
                g.set_codec(key_centroids=oracle.codebook(D, kw["key_bits"]), value_centroids=o._vcb, dim=D)
        if P:
            k, v = seeded((B, Hkv, P, D), 1, dtype), seeded((B, Hkv, P, D), 2, dtype)
            fill = "update_quantized" if "group" in kw else "encode_new_token"
            getattr(g, fill)(k.to(cuda), v.to(cuda))
            getattr(o, fill)(to_oracle(k), to_oracle(v))
        q, k1, v1 = seeded((B, Hq, L, D), 3, dtype), seeded((B, Hkv, L, D), 4, dtype), seeded((B, Hkv, L, D), 5, dtype)
        if not P and "group" not in kw:
            g.encode_new_token(k1.to(cuda), v1.to(cuda))        # compressed from the first row on
            o.encode_new_token(to_oracle(k1), to_oracle(v1))
        mask = "causal" if L > 1 else "none"
        out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), D ** -0.5, mask)
        ref = torch.from_numpy(oracle_f32(oracle.attention_with_cache_update(
            to_oracle(q.float()), to_oracle(k1), to_oracle(v1), o, D ** -0.5, mask)))
        if not pairs:
            assert worst_excess(out, ref.to(dtype).numpy(), dtype) <= 0, (P, L, Hq)
            continue
        ideal = float((ref.to(dtype).double() - ref.double()).norm())
        assert float((out.cpu().double() - ref.double()).norm()) <= (1.05 if P == 31 else 1.2) * ideal, (P, L, Hq)
    assert kvc.lib().kvc_device_status() == 0


def test_calls_without_the_stream_kernel(kvc, cuda):
    """On a device where the stream kernel cannot run (KVC_STREAM=0 stands for one) its calls and lists have other kernels, which differ by
    the operands' rounding: 2^-9 of the result in f16."""
    code = """
import sys, torch, kvcache_b200 as kvc
torch.manual_seed(0)
outs = []
for make in (lambda: kvc.TurboQuantKVCache(bits=8, key_bits=8, value_bits=4), lambda: kvc.TurboQuantKVCache(bits=4, key_bits=0, value_bits=4),
             lambda: kvc.QuantizedKVCache(32, 4)):
    cs = [make(), make()]
    for c in cs:
        k, v = torch.randn(2, 2, 2, 300, 128, dtype=torch.half, device="cuda")
        (c.update_quantized if isinstance(c, kvc.QuantizedKVCache) else c.encode_new_token)(k, v)
    q, k, v = (torch.randn(2, h, 1, 128, dtype=torch.half, device="cuda") for h in (8, 2, 2))
    one = cs[0].attention(q, k, v, 0.09)
    kvc.trim_prompt_cache(cs[:1], 1)
    two = [torch.empty_like(q) for _ in cs]
    kvc.DecodeStep(cs, [q, q], [k, k], [v, v], two, 0.09).run()
    outs += [one, *two]
assert kvc.device_status() == 0
torch.save(torch.stack(outs).cpu(), sys.argv[1])
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    both = []
    for on in "10":
        env = dict(os.environ, PYTHONPATH=os.path.join(root, "mlx-swift-lm_b200", "python"), KVC_STREAM=on)
        with tempfile.NamedTemporaryFile() as out:
            subprocess.run([sys.executable, "-c", code, out.name], check=True, env=env, timeout=300)
            both.append(torch.load(out.name).double())
    assert not torch.equal(*both)
    for x, y in zip(*both):
        assert float((x - y).norm()) <= 2.0 ** -9 * float(y.norm())


@pytest.mark.parametrize("kw,D,L", [(dict(key_bits=8, value_bits=4), 128, 1), (dict(key_bits=4, value_bits=4), 64, 1),
                                    (dict(bits=4, group=64), 256, 1), (dict(key_bits=8, value_bits=4), 128, 70)])
def test_values_and_queries_beyond_the_f16_range(kvc, oracle, cuda, kw, D, L):
    """bf16 values of 1e6 (row norms above 1e7) and queries of 1e5 (scores brought back by the scale): nothing overflows."""
    g, o = _caches(kvc, oracle, cuda, torch.bfloat16, kw, 1, 2, D, 150, gain=1e6)
    q, k1, v1 = seeded((1, 8, L, D), 3, torch.bfloat16) * 1e5, seeded((1, 2, L, D), 4, torch.bfloat16), seeded((1, 2, L, D), 5, torch.bfloat16)
    mask = "causal" if L > 1 else "none"
    out = g.attention(q.to(cuda), k1.to(cuda), v1.to(cuda), 1e-5 * D ** -0.5, mask)
    ref = oracle_f32(oracle.attention_with_cache_update(to_oracle(q), to_oracle(k1), to_oracle(v1), o, 1e-5 * D ** -0.5, mask))
    assert np.linalg.norm(out.float().cpu().numpy() - ref) <= 2.0 ** -8 * np.linalg.norm(ref)    # one spacing of bf16


@pytest.mark.parametrize("dtype,mask_dtype,P", [(torch.bfloat16, torch.float32, 30), (torch.float16, torch.bfloat16, 300),
                                                (torch.bfloat16, torch.bfloat16, 3000)])
def test_row_masked_by_the_lowest_value_is_an_average(kvc, cuda, dtype, mask_dtype, P):
    """A finite mask is added to the scores: a row that holds the type's lowest value everywhere weighs all keys alike."""
    B, Hq, Hkv, D, L = 1, 4, 2, 128, 20
    c = kvc.KVCacheSimple()
    v = seeded((B, Hkv, P + L, D), 2, dtype).to(cuda)
    c.update(seeded((B, Hkv, P, D), 1, dtype).to(cuda), v[:, :, :P])
    m = torch.zeros((L, P + L), dtype=mask_dtype, device=cuda)
    m[3] = torch.finfo(mask_dtype).min
    m[5] = -torch.inf
    out = c.attention(seeded((B, Hq, L, D), 3, dtype).to(cuda), seeded((B, Hkv, L, D), 4, dtype).to(cuda), v[:, :, P:], D ** -0.5, m)
    mean = v.double().mean(2).repeat_interleave(Hq // Hkv, 1)
    assert float((out[:, :, 3].double() - mean).abs().max()) <= 2.0 ** -9     # outputs below 1: half a bf16 spacing
    assert not out[:, :, 5].any() and torch.isfinite(out).all()


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 256), (torch.float16, 256), (torch.bfloat16, 128)])
def test_unmasked_chunk_takes_a_maximum_per_16_tokens(kvc, cuda, dtype, D):
    """P rounds to 16 bits against the running maximum, and tokens that are it are exact: how many tokens share a
    maximum is part of the result's precision. Emulated in 64 bits with 16 and with 32 tokens a step (one tile of 64
    tokens, one split): the kernel's outputs are the first. What is left there is the store's rounding of sums that
    agree to fp32; the two emulations differ by the rounding of P."""
    B, Hq, Hkv, P, L = 4, 4, 1, 34, 30
    k, v, q = (seeded((B, h, n, D), i, dtype) for h, n, i in ((Hkv, P + L, 1), (Hkv, P + L, 2), (Hq, L, 3)))
    out = kvc.scaled_dot_product_attention(q.to(cuda), k.to(cuda), v.to(cuda), D ** -0.5, "causal").cpu()
    s = (q.double() @ k.double().transpose(2, 3)) * D ** -0.5 * 1.4426950408889634
    s = s.masked_fill(torch.arange(P + L)[None, :] > torch.arange(P, P + L)[:, None], -torch.inf)

    def emulate(step):
        m, l, o = torch.full((B, Hq, L, 1), -torch.inf, dtype=torch.float64), 0.0, 0.0
        for t in range(0, P + L, step):
            x = s[..., t:t + step]
            m_new = torch.maximum(m, x.amax(-1, True))
            a, p = torch.exp2(m - m_new), torch.exp2(x - m_new)
            m, l, o = m_new, l * a + p.sum(-1, True), o * a + p.float().to(dtype).double() @ v[:, :, t:t + step].double()
        return o / l
    far = float((emulate(32) - emulate(16)).norm())
    ref = emulate(16)
    store = float((ref.float().to(dtype).double() - ref).norm())
    assert float((out.double() - ref).norm()) <= 1.01 * store          # 32 tokens a step: hypot(store, far)
    assert far > 0.3 * store


def _rows64(oracle, state, kind, D):
    """Keys and values that the arrays of a packed cache stand for, in 64 bits, in the basis of the callers' rows."""
    dev = state[0].device

    def unpack(w, bits):
        return torch.from_numpy(oracle.unpack_low_bit(w.cpu().numpy().view(np.uint32), bits, D).astype(np.int64)).to(dev)

    def affine(codes, scales, biases, bits):
        s, b = (t.double().repeat_interleave(D // scales.shape[-1], -1) for t in (scales, biases))
        return unpack(codes, bits).double() * s + b

    def index(packed, norms, bits, seed):
        h = torch.ones((1, 1), dtype=torch.float64, device=dev)
        while h.shape[0] < D:
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
        book, signs = (torch.from_numpy(a.astype(np.float64)).to(dev) for a in (oracle.codebook(D, bits), oracle.wht_signs(D, seed)))
        return (book[unpack(packed, bits)] @ h) / D ** 0.5 * signs * norms.double().unsqueeze(-1)
    if "group" in kind:
        return affine(*state[:3], kind["bits"]), affine(*state[3:], kind["bits"])
    kb, vb = kind["key_bits"], kind["value_bits"]
    n = {0: 1, 8: 3}.get(kb, 2)
    k = state[0].double() if kb == 0 else affine(*state[:3], 8) if kb == 8 else index(*state[:2], kb, 42)
    return k, affine(*state[n:n + 3], vb) if kind.get("affine_values") else index(*state[n:n + 2], vb, 43)


def _attention64(q, k, v, scale, allowed):
    rep = q.shape[1] // k.shape[1]
    k, v = (t.repeat_interleave(rep, 1) for t in (k, v))
    return torch.softmax((q.double() @ k.transpose(2, 3) * scale).masked_fill(~allowed, -torch.inf), -1) @ v


@pytest.mark.parametrize("kw,Hq,Hkv,D,P,L,gain", [
    (dict(key_bits=4, value_bits=4, affine_values=True), 8, 2, 128, 3000, 100, 4.0),    # operand pairs
    (dict(key_bits=8, value_bits=4), 8, 2, 128, 3000, 100, 4.0),
    (dict(key_bits=0, value_bits=4), 8, 2, 128, 3000, 100, 1.0),
    (dict(bits=4, group=64), 4, 1, 256, 3000, 100, 1.0),
    (dict(key_bits=3, value_bits=4), 4, 1, 256, 3000, 100, 1.0),
    (dict(key_bits=3, value_bits=3), 4, 4, 64, 500, 20, 1.0),
])
@pytest.mark.parametrize("size", [1.0, 2.0 ** -10])
def test_chunks_on_operand_pairs_keep_single_precision(kvc, oracle, cuda, kw, Hq, Hkv, D, P, L, gain, size):
    """f16 callers, one key channel in a hundred 20 times larger, and the same data a thousand times smaller: against
    64-bit sums the outputs err by the store's rounding `ideal` and no more. 1.0005 * ideal leaves the arithmetic 0.03 *
    ideal (errors add in quadrature), 2^-17 of the result, which is what single precision needs for scores near 50;
    products of pairs of bf16 took 1.0034 .. 1.011."""
    make = (lambda: kvc.QuantizedKVCache(kw["group"], kw["bits"])) if "group" in kw else \
        (lambda: kvc.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw))
    c = make()
    g = torch.ones(D)
    g[torch.randperm(D, generator=torch.Generator().manual_seed(3))[:max(1, D // 100)]] = 20.0
    k, v, k1, v1, q = (seeded((2, h, n, D), s) for s, (h, n) in enumerate(((Hkv, P), (Hkv, P), (Hkv, L), (Hkv, L), (Hq, L))))
    k, v, k1, v1, q = (t.half().to(cuda) for t in (k * g * size, v * size, k1 * g * size, v1 * size, q * gain))
    (c.update_quantized if "group" in kw else c.encode_new_token)(k, v)
    out = c.attention(q, k1, v1, D ** -0.5 / size, "causal")
    K, V = _rows64(oracle, c.state, kw, D)
    ref = _attention64(q, K, V, D ** -0.5 / size, torch.arange(P + L, device=cuda) <= torch.arange(P, P + L, device=cuda)[:, None])
    ideal = float((ref.half().double() - ref).norm())
    assert float((out.double() - ref).norm()) <= 1.0005 * ideal


def test_small_probabilities_under_an_array_mask(kvc, cuda):
    """16 000 keys at probabilities around 2^-26 beside one near 1 whose value row is zero: together they are the output.
    f16 probabilities as they are would be zero there."""
    B, H, D, P, L = 1, 2, 128, 16000, 4
    u = seeded((1, 1, 1, D), 1)
    u = u / u.norm()
    k = (seeded((B, H, P + L, D), 2) * 0.02).half()
    k[:, :, 7] = (u * 8.0).half()
    v = (1.0 + 0.1 * seeded((B, H, P + L, D), 3)).half()
    v[:, :, 7] = 0.0
    q = (u * 2.25).expand(B, H, L, D).half().to(cuda)          # score of key 7: 18 nats, 26 powers of two
    k, v = k.to(cuda), v.to(cuda)
    c = kvc.KVCacheSimple()
    c.update(k[:, :, :P], v[:, :, :P])
    m = torch.arange(P + L, device=cuda) <= torch.arange(P, P + L, device=cuda)[:, None]
    out = c.attention(q, k[:, :, P:], v[:, :, P:], 1.0, m)
    ref = _attention64(q, k.double(), v.double(), 1.0, m)
    # outputs around 2^-12, a subnormal of f16 begins at 2^-14: the store rounds to 2^-23 at most
    assert float((out.double() - ref).abs().max()) <= 2.0 ** -23 * 1.01
    assert float(ref.min()) > 2.0 ** -13


@pytest.mark.parametrize("kw,Hq,Hkv,D,L", [
    (dict(key_bits=4, value_bits=4, affine_values=True), 8, 2, 128, 1),
    (dict(key_bits=4, value_bits=4, affine_values=True), 8, 2, 128, 4),     # two column blocks
    (dict(bits=4, group=64), 4, 1, 256, 1),
    (dict(bits=4, group=32), 4, 1, 256, 4),
    (dict(bits=8, group=64), 4, 1, 256, 1),
    (dict(key_bits=8, value_bits=4), 8, 2, 64, 1),
    (dict(key_bits=3, value_bits=4, affine_values=True), 8, 2, 64, 4),
])
def test_stream_kernel_keeps_single_precision_over_affine_codes(kvc, oracle, cuda, kw, Hq, Hkv, D, L):
    """f16 callers over 8 000 keys, where outputs are small beside the values: against 64-bit sums they err by the store's
    rounding `ideal` alone. 1.0003 * ideal leaves the arithmetic 0.025 * ideal; codes that entered the MMA as subnormals
    took 1.0006 .. 1.0011 (4 bits)."""
    P = 8000
    c = kvc.QuantizedKVCache(kw["group"], kw["bits"]) if "group" in kw else \
        kvc.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw)
    g = torch.ones(D)
    g[torch.randperm(D, generator=torch.Generator().manual_seed(3))[:max(1, D // 100)]] = 20.0
    k, v, k1, v1, q = (seeded((4, h, n, D), s) for s, (h, n) in enumerate(((Hkv, P), (Hkv, P), (Hkv, L), (Hkv, L), (Hq, L))))
    k, v, k1, v1, q = (t.half().to(cuda) for t in (k * g, v, k1 * g, v1, q))
    (c.update_quantized if "group" in kw else c.encode_new_token)(k, v)
    out = c.attention(q, k1, v1, D ** -0.5, "causal" if L > 1 else "none")
    K, V = _rows64(oracle, c.state, kw, D)
    ref = _attention64(q, K, V, D ** -0.5, torch.arange(P + L, device=cuda) <= torch.arange(P, P + L, device=cuda)[:, None])
    ideal = float((ref.half().double() - ref).norm())
    assert float((out.double() - ref).norm()) <= 1.0003 * ideal


@pytest.mark.parametrize("bits,group,B,Hq,Hkv,D,P", [
    (4, 64, 4, 16, 8, 128, 1100), (4, 128, 4, 16, 8, 128, 1100), (8, 64, 4, 16, 8, 128, 1100), (8, 128, 8, 32, 8, 128, 300),
    (8, 32, 8, 32, 8, 128, 300), (4, 64, 8, 32, 8, 64, 600), (8, 64, 8, 32, 8, 64, 600),
])
def test_affine_ranges_that_end_where_units_end(kvc, oracle, cuda, bits, group, B, Hq, Hkv, D, P):
    """Units of a few tiles, one or a few whole pieces a CTA. Query, weights and store are f16, `ideal` is what the last of the three
    errs by; a weight's error meets a code's distance from the middle, so that the three are alike: sqrt(3) * ideal, and 15 %
    for how alike they are. (Weights that meet the codes themselves: 2.4 .. 2.9 * ideal.)"""
    c = kvc.QuantizedKVCache(group, bits)
    c.update_quantized(seeded((B, Hkv, P, D), 1, torch.half).to(cuda), seeded((B, Hkv, P, D), 2, torch.half).to(cuda))
    q, k1, v1 = (seeded((B, h, 1, D), s, torch.half).to(cuda) for s, h in ((3, Hq), (4, Hkv), (5, Hkv)))
    out = c.attention(q, k1, v1, D ** -0.5)
    K, V = _rows64(oracle, c.state, dict(bits=bits, group=group), D)
    ref = _attention64(q, K, V, D ** -0.5, torch.ones((1, P + 1), dtype=torch.bool, device=cuda))
    ideal = float((ref.half().double() - ref).norm())
    assert float((out.double() - ref).norm()) <= 2.0 * ideal
    assert kvc.lib().kvc_device_status() == 0


def _packed(kvc, cuda, kw, B, Hkv, D, P, seed=1):
    """A packed f16 cache of P rows."""
    c = kvc.QuantizedKVCache(kw["group"], kw["bits"]) if "group" in kw else kvc.TurboQuantKVCache(bits=max(kw["key_bits"], kw["value_bits"]), **kw)
    k, v = (torch.randn((B, Hkv, P, D), generator=torch.Generator(cuda).manual_seed(seed + i), device=cuda, dtype=torch.half) for i in (0, 100))
    (c.update_quantized if "group" in kw else c.encode_new_token)(k, v)
    return c


def _err_over_ideal(oracle, out, c, q, kw, D, L=1):
    """Distance from 64-bit sums over that of their f16 rounding."""
    K, V = _rows64(oracle, c.state, kw, D)
    T = K.shape[2]
    ref = _attention64(q, K, V, D ** -0.5, torch.arange(T, device=q.device) <= torch.arange(T - L, T, device=q.device)[:, None])
    return float((out.double() - ref).norm() / (ref.half().double() - ref).norm())


@pytest.mark.parametrize("kw,rows,D,B,Hkv,P", [
    # TurboQuant kernels of f16 operands: rotated query, both centroids, weight and store: sqrt(5), and 25 %. Codebooks of two bits have two
    # magnitudes, whose rounding may be the largest there is, 2.4 times the mean one: sqrt(3 + 2 * 2.4^2)
    (dict(key_bits=2, value_bits=2), 4, 128, 16, 8, 300),       # tiles of 64: units of five, three pieces or whole ones
    (dict(key_bits=3, value_bits=3), 4, 128, 4, 8, 1100),
    (dict(key_bits=4, value_bits=2), 4, 128, 48, 8, 130),
    (dict(key_bits=3, value_bits=4), 4, 128, 8, 8, 2047),       # tiles of 240: units of nine in pieces of five
    (dict(key_bits=4, value_bits=4), 4, 128, 32, 8, 300),
    # operand pairs: the store alone, and 5 %
    (dict(key_bits=8, value_bits=4), 4, 128, 8, 8, 300),
    (dict(key_bits=0, value_bits=4), 4, 64, 40, 8, 300),
    (dict(bits=4, group=32), 4, 256, 16, 8, 300),
])
def test_ranges_that_end_where_units_end(kvc, oracle, cuda, kw, rows, D, B, Hkv, P):
    c = _packed(kvc, cuda, kw, B, Hkv, D, P)
    q, k1, v1 = (seeded((B, h, 1, D), s, torch.half).to(cuda) for s, h in ((3, rows * Hkv), (4, Hkv), (5, Hkv)))
    out = c.attention(q, k1, v1, D ** -0.5)
    pairs = "group" in kw or kw["key_bits"] in (0, 8)
    assert _err_over_ideal(oracle, out, c, q, kw, D) <= (1.05 if pairs else 3.9 if kw["key_bits"] == 2 or kw["value_bits"] == 2 else 2.8)
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("kw,n,B,Hkv,D,P,L,dtype", [
    (dict(key_bits=8, value_bits=4), 2, 4, 8, 128, 300, 1, torch.half),      # 64 units of five tiles, rounded up to six
    (dict(key_bits=8, value_bits=4), 4, 16, 8, 128, 300, 1, torch.half),     # whole units
    (dict(key_bits=4, value_bits=4), 3, 2, 8, 64, 300, 2, torch.half),
    (dict(bits=4, group=64), 3, 3, 4, 64, 450, 1, torch.half),
    (dict(bits=8, group=64), 2, 4, 8, 64, 300, 1, torch.float32),
    (dict(bits=4, group=64), 4, 20, 8, 64, 300, 1, torch.float32),
])
def test_lists_whose_units_are_rounded_up(kvc, oracle, cuda, kw, n, B, Hkv, D, P, L, dtype):
    """Layers of one length in one launch, whose ranges end where units end. The bounds of the kernels' own tests."""
    cs = [_packed(kvc, cuda, kw, B, Hkv, D, P, seed=i) for i in range(n)] if dtype == torch.half else []
    for i in range(n - len(cs)):
        cs.append(kvc.QuantizedKVCache(kw["group"], kw["bits"]))
        cs[i].update_quantized(*(seeded((B, Hkv, P, D), 2 * i + j, dtype).to(cuda) for j in (0, 1)))
    qs, ks, vs = ([seeded((B, h, L, D), s + i, dtype).to(cuda) for i in range(n)] for s, h in ((30, 2 * Hkv), (40, Hkv), (50, Hkv)))
    outs = [torch.empty_like(q) for q in qs]
    kvc.launch_count(reset=True)
    kvc.DecodeStep(cs, qs, ks, vs, outs, D ** -0.5, mask="causal" if L > 1 else "none").run()
    assert kvc.launch_count() == (3 if kw.get("key_bits") == 8 else 2)          # the rows (of both representations), the attention
    for c, q, out in zip(cs, qs, outs):
        if dtype == torch.half:
            assert _err_over_ideal(oracle, out, c, q, kw, D, L) <= 1.05
        else:
            K, V = _rows64(oracle, c.state, kw, D)
            ref = _attention64(q, K, V, D ** -0.5, torch.ones((1, P + 1), dtype=torch.bool, device=cuda))
            assert float((out.double() - ref).norm()) <= 2.0 ** -20 * float(ref.norm())
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("kw", [dict(bits=4, group=32), dict(bits=8, group=32), dict(key_bits=4, value_bits=4),
                                dict(key_bits=3, value_bits=4), dict(key_bits=0, value_bits=2), dict(key_bits=8, value_bits=3)])
@pytest.mark.parametrize("rep,L,P", [(1, 17, 2305), (4, 7, 2318), (8, 4, 2367), (3, 11, 2304 + 64), (8, 8, 2400)])
def test_units_of_32_rows(kvc, oracle, cuda, kw, rep, L, P):
    """Verify rounds of 17, 28, 32, 33 and 64 rows a KV head over enough tokens (128 tiles of 64 an SM) for four column blocks a unit;
    the last tile of a unit holds 1 .. 64 tokens of the round and before it."""
    B, Hkv, D = 32, 16, 64
    c = _packed(kvc, cuda, kw, B, Hkv, D, P)
    q, k1, v1 = (seeded((B, h, L, D), s, torch.half).to(cuda) for s, h in ((3, rep * Hkv), (4, Hkv), (5, Hkv)))
    out = c.attention(q, k1, v1, D ** -0.5, "causal")
    assert _err_over_ideal(oracle, out, c, q, kw, D, L) <= 1.05
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype,Hq,Hkv,D,P", [(torch.bfloat16, 8, 1, 128, 20000), (torch.half, 6, 2, 64, 30011), (torch.half, 4, 1, 256, 12000)])
def test_raw_units_of_more_than_64_partials(kvc, cuda, dtype, Hq, Hkv, D, P):
    """One sequence of few heads: every tile of a long context is another CTA's. Weights and store are rounded to the type: two
    errors of `ideal`, and 15 % for how alike they are."""
    c = kvc.KVCacheSimple()
    k, v = (torch.randn((1, Hkv, P, D), generator=torch.Generator(cuda).manual_seed(i), device=cuda).to(dtype) for i in (1, 2))
    c.update(k, v)
    q, k1, v1 = (seeded((1, h, 1, D), s, dtype).to(cuda) for s, h in ((3, Hq), (4, Hkv), (5, Hkv)))
    out = c.attention(q, k1, v1, D ** -0.5)
    K, V = (torch.cat(t, 2).double() for t in ((k, k1), (v, v1)))
    ref = _attention64(q, K, V, D ** -0.5, torch.ones((1, P + 1), dtype=torch.bool, device=cuda))
    ideal = float((ref.to(dtype).double() - ref).norm())
    assert float((out.double() - ref).norm()) <= 1.15 * 2 ** 0.5 * ideal
    assert kvc.lib().kvc_device_status() == 0


def test_chunk_on_operand_pairs_on_a_full_device(kvc, cuda):
    """A chunk whose decoded rows the device has no room for runs on the general kernel instead of failing."""
    code = """
import torch, kvcache_b200 as kvc
torch.manual_seed(0)
c = kvc.QuantizedKVCache(64, 4, reserve_tokens=40960)
for _ in range(10):
    k, v = torch.randn(2, 1, 8, 4000, 256, dtype=torch.half, device="cuda")
    c.update_quantized(k, v)
q, k, v = (torch.randn(1, h, 70, 256, dtype=torch.half, device="cuda") for h in (8, 8, 8))
out = torch.empty_like(q)
torch.cuda.synchronize()
torch.cuda.empty_cache()
hold = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
launches, outs = [], []
for step in range(2):
    kvc.launch_count(reset=True)
    c.attention(q, k, v, 0.0625, "causal", out=out)
    torch.cuda.synchronize()
    launches.append(kvc.launch_count(reset=True))
    outs.append(out.clone())
    c.trim(70)
    del hold
    torch.cuda.empty_cache()
    hold = None
assert launches[0] == 3 and launches[1] == 4, launches
assert float((outs[0].float() - outs[1].float()).abs().max()) < 2e-3
"""
    env = dict(os.environ, PYTHONPATH=os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx-swift-lm_b200", "python"))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)


@pytest.mark.parametrize("B,room,slices", [(2, 250, [1, 2]), (1, 90, [0, 1])])
def test_short_turbo_chunk_on_a_full_device(kvc, cuda, B, room, slices):
    """Rows of 164 MB a sequence that the device has no room for: sequence by sequence, or in the kernel that decodes in its
    tile loop, instead of failing; and all at once when there is room again (`slices`: sequences per slice, 0: not written out)."""
    code = f"""
import torch, kvcache_b200 as kvc
torch.manual_seed(0)
B = {B}
c = kvc.TurboQuantKVCache(bits=4, key_bits=3, value_bits=4, reserve_tokens=40960)
for _ in range(10):
    k, v = torch.randn(2, B, 8, 4000, 128, dtype=torch.half, device="cuda")
    c.encode_new_token(k, v)
q, k, v = (torch.randn(B, h, 17, 128, dtype=torch.half, device="cuda") for h in (32, 8, 8))
out = torch.empty_like(q)
torch.cuda.synchronize()
torch.cuda.empty_cache()
hold = torch.empty(torch.cuda.mem_get_info()[0] - ({room} << 20), dtype=torch.uint8, device="cuda")
outs = []
for step in range(2):
    c.attention(q, k, v, 128 ** -0.5, "causal", out=out)
    torch.cuda.synchronize()
    print("step", file=__import__("sys").stderr, flush=True)
    outs.append(out.cpu().double())
    c.trim(17)
    hold = None
    torch.cuda.empty_cache()
assert c.offset == 40000
assert float((outs[0] - outs[1]).norm()) < 2.0 ** -8 * float(outs[1].norm())
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "mlx-swift-lm_b200", "python"), KVC_TRACE_DISPATCH="1")
    err = subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300, stderr=subprocess.PIPE, text=True).stderr
    for part, n in zip(err.split("step"), slices):
        assert ("rows written out" in part) == (n > 0) and (n == 0 or f"{n} sequences per slice" in part), err


@pytest.mark.parametrize("kw,P,L", [(dict(key_bits=3, value_bits=4), 20000, 17),      # rows from the pool
                                    (dict(key_bits=3, value_bits=4), 300, 17),        # in the arena
                                    (dict(bits=4, group=64), 20000, 512)])
def test_captured_chunk_with_rows_written_out(kvc, cuda, capfd, monkeypatch, kw, P, L):
    """Replays on other inputs give the eager call's bits, wherever the rows lie."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    B, Hq, Hkv, D = 1, 32, 8, 128
    c = _packed(kvc, cuda, kw, B, Hkv, D, P)
    q, k1, v1 = (seeded((B, h, L, D), s, torch.half).to(cuda) for s, h in ((3, Hq), (4, Hkv), (5, Hkv)))
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        c.attention(q, k1, v1, D ** -0.5, "causal", out=out)        # warm: workspaces of this stream
    torch.cuda.synchronize()
    c.trim(L)
    graph = torch.cuda.CUDAGraph()
    capfd.readouterr()
    with torch.cuda.graph(graph, stream=side):
        c.attention(q, k1, v1, D ** -0.5, "causal", out=out)
    assert "rows written out" in capfd.readouterr().err
    for seed in (11, 12):
        q.copy_(seeded(tuple(q.shape), seed, torch.half))
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        c.trim(L)
        assert torch.equal(out, c.attention(q, k1, v1, D ** -0.5, "causal"))
    del graph
    assert kvc.lib().kvc_device_status() == 0


def test_sequences_of_a_call_take_one_kernel(kvc, cuda, capfd, monkeypatch):
    """Rows written out for a chunk are limited to a few GB at a time. Where a last slice of the batch would be too small to be worth it,
    no sequence of the call is treated that way: equal sequences have equal outputs."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    B, Hq, Hkv, D, P, L = 3, 32, 8, 128, 262144, 64
    c = kvc.QuantizedKVCache(64, 4, reserve_tokens=P + L)
    g = torch.Generator(cuda).manual_seed(1)
    rand = lambda h, n: torch.randn((1, h, n, D), generator=g, device=cuda).to(torch.bfloat16).expand(B, h, n, D).contiguous()
    for _ in range(0, P, 32768):
        c.update_quantized(rand(Hkv, 32768), rand(Hkv, 32768))
    capfd.readouterr()
    out = c.attention(rand(Hq, L), rand(Hkv, L), rand(Hkv, L), D ** -0.5, "causal")
    torch.cuda.synchronize()
    assert "rows written out" not in capfd.readouterr().err
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    assert kvc.lib().kvc_device_status() == 0
