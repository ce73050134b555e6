"""The caller's side of the cache path: rotary positions at the cache's ropeOffset ahead of
attentionWithCacheUpdate (MLXLLM/Models/Llama.swift:58-69, MLXLMCommon/RoPEApplication.swift:58-69) and
the cache traffic of a speculative round over a model's layer list (Evaluate.swift:1179-1286,
KVCachePlan.swift:219-300), against the oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from helpers import TOL, bits_equal, max_abs_diff, seeded, to_oracle

pytestmark = pytest.mark.gpu

# one bf16 / f16 spacing at |x| <= 8 (rotated N(0, 1) inputs): the rotation itself is float32 on both sides
ROPE_TOL = {torch.float32: 2e-5, torch.bfloat16: 2 ** -5, torch.float16: 2 ** -8}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,dims,traditional,base,scale", [(128, 128, False, 10000.0, 1.0), (128, 128, True, 500000.0, 1.0),
                                                           (64, 32, False, 10000.0, 0.25), (256, 64, True, 1000000.0, 1.0)])
def test_rope_matches_oracle(kvc, oracle, cuda, dtype, D, dims, traditional, base, scale):
    x = seeded((2, 3, 7, D), 5, dtype)
    for offset in (0, 1, 4096, 131071):
        got = kvc.rope(x.to(cuda), offset, dims, traditional, base, scale)
        want = oracle.rope(to_oracle(x), offset, dims, traditional, base, scale)
        # large positions: float32 angles lose absolute precision on both sides alike (p * f is rounded once);
        # what remains is the sin/cos implementation, a few float32 spacings of the angle
        tol = ROPE_TOL[dtype] + (2e-3 if offset > 100000 else (1e-4 if offset > 1000 else 0.0))
        assert max_abs_diff(got, want) <= tol, (offset, max_abs_diff(got, want))
        if dims < D:
            assert torch.equal(got[..., dims:].cpu(), x[..., dims:])            # pass-through features untouched
    # in place and strided (the [B, L, H, D] storage of a projection output)
    xs = x.to(cuda).transpose(1, 2).contiguous().transpose(1, 2)
    got = kvc.rope(xs, 3, dims, traditional, base, scale, out=xs)
    assert max_abs_diff(got, oracle.rope(to_oracle(x), 3, dims, traditional, base, scale)) <= ROPE_TOL[dtype]


@pytest.mark.parametrize("kind", ["simple", "rotating", "quantized", "turbo", "none"])
def test_attention_block_step_with_rope(kvc, oracle, cuda, kind):
    """Prefill in two chunks, then decode steps: every call rotates q and k at the cache offset before the
    fused update + attention; the cache ends up holding rotated keys (bit-exact where both sides agree on
    the rotated values to the bit is not required: rotated keys are compared at the store tolerance)."""
    B, Hq, Hkv, D = 2, 8, 2, 128
    dtype = torch.bfloat16
    cfg = dict(dims=D, traditional=False, base=500000.0, scale=1.0)
    scale = D ** -0.5
    if kind == "simple":
        g, o = kvc.KVCacheSimple(), oracle.KVCacheSimple()
    elif kind == "rotating":
        g, o = kvc.RotatingKVCache(max_size=96, keep=4), oracle.RotatingKVCache(96, keep=4)
    elif kind == "quantized":
        g, o = kvc.QuantizedKVCache(64, 8), oracle.QuantizedKVCache(64, 8)
    elif kind == "turbo":
        g, o = kvc.TurboQuantKVCache(bits=4), oracle.TurboQuantKVCache(bits=4)
    else:
        g = o = None
    seed = 0
    for S in ((70, 50) + (1,) * 6 if g is not None else (33,)):
        seed += 1
        q, k, v = seeded((B, Hq, S, D), seed, dtype), seeded((B, Hkv, S, D), seed + 50, dtype), seeded((B, Hkv, S, D), seed + 90, dtype)
        if g is not None and S > 1:
            gm, om = g.make_mask(S), o.make_mask(S)
            om_ = om if isinstance(om, str) else om
            gm_ = gm if isinstance(gm, str) else gm
        else:
            gm_, om_ = ("causal", "causal") if S > 1 else ("none", "none")
        out = kvc.attention_rope(q.to(cuda), k.to(cuda), v.to(cuda), g, cfg, scale, gm_)
        ref = oracle.attention_rope(to_oracle(q), to_oracle(k), to_oracle(v), o, cfg, scale, om_)
        # rotated operands may differ by one bf16 spacing between the two sides (float32 sin/cos of the
        # device and of numpy are not the same bits), which moves scores by ~1e-2 at worst
        assert max_abs_diff(out, ref) <= 2 * TOL[dtype], (kind, S)
        if g is not None:
            assert g.offset == o.offset
    if kind == "simple":
        gk, ok_ = g.state[0], o.state[0]
        assert max_abs_diff(gk, np.ascontiguousarray(ok_)) <= 2 ** -5           # rotated keys, one bf16 spacing at |x| < 8


def test_speculative_rounds_over_a_layer_list(kvc, oracle, cuda):
    """A four-layer list (simple, sliding window past its wrap, affine-quantised, TurboQuant): rounds of
    5 draft tokens + 1 through KVCacheStorage-style staged rounds with a scripted number of accepted
    tokens per round; after every commit each layer's state equals the oracle's, where the oracle is
    driven the reference's way (one StagedRound per cache, commit(retaining)). The sliding-window layer is
    also compared with an emitted-only replay (what the cache would hold had only the kept tokens ever
    been written)."""
    B, Hq, Hkv, D, L = 1, 8, 2, 128, 6
    dtype = torch.bfloat16
    scale = D ** -0.5

    def make():
        gs = [kvc.KVCacheSimple(), kvc.RotatingKVCache(max_size=48, keep=0), kvc.QuantizedKVCache(64, 4), kvc.TurboQuantKVCache(bits=4)]
        os_ = [oracle.KVCacheSimple(), oracle.RotatingKVCache(48, keep=0), oracle.QuantizedKVCache(64, 4), oracle.TurboQuantKVCache(bits=4)]
        return gs, os_

    gs, os_ = make()
    replay = oracle.RotatingKVCache(48, keep=0)
    P = 60                                        # prefill past the window: the ring has wrapped
    for i, (g, o) in enumerate(zip(gs, os_)):
        q, k, v = seeded((B, Hq, P, D), 10 + i, dtype), seeded((B, Hkv, P, D), 20 + i, dtype), seeded((B, Hkv, P, D), 30 + i, dtype)
        gm, om = g.make_mask(P, window_size=48 if i == 1 else None), o.make_mask(P, window_size=48 if i == 1 else None)
        g.attention(q.to(cuda), k.to(cuda), v.to(cuda), scale, gm)
        oracle.attention_with_cache_update(to_oracle(q), to_oracle(k), to_oracle(v), o, scale, om)
        if i == 1:
            replay.update(to_oracle(k), to_oracle(v))
    accepted_script = [5, 0, 2, 5, 1, 3]
    for rnd, accepted in enumerate(accepted_script):
        retaining = accepted + 1                  # the accepted drafts plus the token verified before them
        qs = [seeded((B, Hq, L, D), 100 + 10 * rnd + i, dtype) for i in range(4)]
        ks = [seeded((B, Hkv, L, D), 200 + 10 * rnd + i, dtype) for i in range(4)]
        vs = [seeded((B, Hkv, L, D), 300 + 10 * rnd + i, dtype) for i in range(4)]
        outs = [torch.empty((B, Hq, L, D), dtype=dtype, device=cuda) for _ in range(4)]
        rd = kvc.StorageRound(gs, L)
        rd.attention([t.to(cuda) for t in qs], [t.to(cuda) for t in ks], [t.to(cuda) for t in vs], scale, outs, "causal")
        for i, o in enumerate(os_):
            if isinstance(o, (oracle.KVCacheSimple, oracle.RotatingKVCache)):
                ro = oracle.StagedRound(o, L)
                ko, vo = ro.update(to_oracle(ks[i]), to_oracle(vs[i]))
                ref = oracle.sdpa(to_oracle(qs[i]), ko, vo, scale, "causal")
                ro.commit(retaining)
            else:
                # packed caches take the rows through their normal update path and give the rejected ones back
                ref = oracle.attention_with_cache_update(to_oracle(qs[i]), to_oracle(ks[i]), to_oracle(vs[i]), o, scale, "causal")
                if L > retaining:
                    assert o.trim(L - retaining) == L - retaining
            assert max_abs_diff(outs[i], ref) <= TOL[dtype], f"round {rnd}, layer {i}"
        rd.commit(retaining)
        replay.update(to_oracle(ks[1][:, :, :retaining]), to_oracle(vs[1][:, :, :retaining]))
        for i, (g, o) in enumerate(zip(gs, os_)):
            assert g.offset == o.offset, f"round {rnd}, layer {i}"
            for a, b in zip(g.state, o.state):
                assert tuple(a.shape) == tuple(b.shape) and bits_equal(a, np.ascontiguousarray(b)), f"round {rnd}, layer {i}"
            assert list(g.meta_state) == list(o.meta_state)
    # the sliding-window layer holds what an emitted-only history would have left (same logical window)
    tail = min(replay.offset, 47)
    gv = gs[1].logical_view(tail)
    rv = replay.logical_view(tail)
    assert gv is not None and rv is not None
    assert bits_equal(gv[0], np.ascontiguousarray(rv[0])) and bits_equal(gv[1], np.ascontiguousarray(rv[1]))
    assert kvc.device_status() == 0


def test_speculate_rewind_rule(kvc, oracle, cuda):
    """Without staged rounds the main caches give back numDraft - accepted positions and the draft caches
    max(numDraft - accepted - 1, 0) (Evaluate.swift:1262-1264), all or nothing over the list."""
    B, Hkv, D = 1, 2, 64
    caches = [kvc.KVCacheSimple(), kvc.QuantizedKVCache(64, 8)]
    k = seeded((B, Hkv, 20, D), 1, torch.bfloat16).to(cuda)
    caches[0].update(k, k)
    caches[1].update_quantized(k, k)
    assert kvc.speculate_rewind(caches, 5, 2) == 3 and [c.offset for c in caches] == [17, 17]
    assert kvc.speculate_rewind(caches, 5, 5) == 0 and [c.offset for c in caches] == [17, 17]
    assert kvc.speculate_rewind(caches, 5, 2, is_draft=True) == 2 and [c.offset for c in caches] == [15, 15]
    assert kvc.speculate_rewind(caches, 5, 4, is_draft=True) == 0
    ring = kvc.RotatingKVCache(max_size=8)
    kk = seeded((B, Hkv, 12, D), 2, torch.bfloat16).to(cuda)
    ring.update(kk, kk)                                         # wrapped: not trimmable, so the list refuses
    assert kvc.speculate_rewind([caches[0], ring], 5, 1) == 0 and caches[0].offset == 15
    with pytest.raises(kvc.KVCError):
        kvc.speculate_rewind(caches, 3, 4)


@pytest.mark.parametrize("ring,P,D", [(False, 254, 128), (False, 1031, 64), (True, 60, 128), (True, 40, 256)])
def test_chained_rope_steps_are_rope_then_attention(kvc, cuda, ring, P, D):
    """Steps issued back to back, the attention kernel streaming stored rows while the rotary kernel still runs: the
    same bits as turning q and k first and waiting between the calls. Crosses a growth of the buffer and a ring's
    wrap, steps twice in a row over one cache, and gives a step whose input the launch just before it wrote."""
    def caches():
        made = [kvc.RotatingKVCache(max_size=64, keep=0) if ring else kvc.KVCacheSimple() for _ in range(3)]
        for i, c in enumerate(made):
            c.update(seeded((1, 2, P, D), i, torch.bfloat16).to(cuda), seeded((1, 2, P, D), 9 + i, torch.bfloat16).to(cuda))
        return made
    a, b = caches(), caches()
    k, v = ([seeded((1, 2, 1, D), 40 + 10 * j + i, torch.bfloat16).to(cuda) for i in range(6)] for j in (0, 1))
    x = y = seeded((1, 8, 1, D), 30, torch.bfloat16).to(cuda)
    for i in range(6):
        x = kvc.attention_rope(x, k[i], v[i], a[i // 2], {"dims": D, "base": 500000.0}, D ** -0.5) * 2
    for i in range(6):
        c = b[i // 2]
        at = c.offset
        torch.cuda.synchronize()
        y = c.attention(kvc.rope(y, at, D, base=500000.0), kvc.rope(k[i], at, D, base=500000.0), v[i], D ** -0.5)
        torch.cuda.synchronize()
        y = y * 2
    assert torch.equal(x, y)
    for s, t in zip(a, b):
        assert s.offset == t.offset and all(torch.equal(m, n) for m, n in zip(s.state, t.state))


@pytest.mark.parametrize("dtype,Hq,Hkv,D,dims,traditional,rope_scale,B,P,shift,one", [
    (torch.bfloat16, 8, 2, 128, 128, True, 1.0, 2, 70, 0, True),
    (torch.float16, 4, 4, 64, 32, False, 0.5, 3, 70, 0, True),        # half the dims turn
    (torch.bfloat16, 4, 1, 256, 2, True, 1.0, 1, 70, 0, True),        # a single pair
    (torch.bfloat16, 16, 8, 128, 128, False, 1.0, 128, 50, 0, True),  # CTAs of several units: the slots of the query rows come round
    (torch.float16, 8, 4, 256, 256, False, 1.0, 128, 50, 0, True),
    (torch.bfloat16, 16, 1, 256, 2, True, 1.0, 1, 70, 0, False),       # more rows than shared memory holds
    (torch.float16, 20, 1, 128, 128, False, 1.0, 1, 70, 0, False),     # more rows than the decode kernel takes
    (torch.bfloat16, 8, 2, 128, 96, False, 8.0, 2, 70, 4, False),      # queries off a 16-byte boundary: turned into memory of their own
])
def test_rope_inside_the_decode_kernel(kvc, cuda, dtype, Hq, Hkv, D, dims, traditional, rope_scale, B, P, shift, one):
    """One launch that turns its own rows, or the launches it replaces: the bits of turning q and k first."""
    a, b = kvc.KVCacheSimple(), kvc.KVCacheSimple()
    for c in (a, b):
        c.update(seeded((B, Hkv, P, D), 1, dtype).to(cuda), seeded((B, Hkv, P, D), 2, dtype).to(cuda))
    for step in range(3):
        q = torch.empty(B * Hq * D + 8, dtype=dtype, device=cuda)[shift:shift + B * Hq * D].view(B, Hq, 1, D)
        q.copy_(seeded((B, Hq, 1, D), 10 + step, dtype).to(cuda))
        k, v = seeded((B, Hkv, 1, D), 20 + step, dtype).to(cuda), seeded((B, Hkv, 1, D), 30 + step, dtype).to(cuda)
        kept = q.clone(), k.clone()
        kvc.launch_count(reset=True)
        x = kvc.attention_rope(q, k, v, a, {"dims": dims, "base": 10000.0, "traditional": traditional, "scale": rope_scale}, D ** -0.5)
        assert (kvc.launch_count() == 1) == one
        assert torch.equal(q, kept[0]) and torch.equal(k, kept[1])
        rope = lambda t: kvc.rope(t, b.offset, dims, traditional=traditional, base=10000.0, scale=rope_scale)
        y = b.attention(rope(q), rope(k), v, D ** -0.5)
        assert torch.equal(x, y)
    assert a.offset == b.offset and all(torch.equal(m, n) for m, n in zip(a.state, b.state))
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("rope", [False, True])
def test_step_without_memory_leaves_the_cache_as_it_was(ring, rope):
    """A full device refuses a step's buffers (turned rows of 9 MB, or a new stream's partials): the cache does not count a row that
    was never stored, and goes on when there is room again."""
    code = f"""
import torch, kvcache_b200 as kvc
torch.manual_seed(0)
B, Hq, D, P = 1024, 16, 256, 100
make = (lambda: kvc.RotatingKVCache(max_size=100, keep=4)) if {ring} else kvc.KVCacheSimple
a, b = make(), make()
for c in (a, b):
    torch.manual_seed(1)
    for n in (90, 17, 1, 1):
        c.update(*torch.randn(2, B, 1, n, D, dtype=torch.half, device="cuda"))
q = torch.randn(B, Hq, 1, D, dtype=torch.half, device="cuda")
k, v = torch.randn(2, B, 1, 1, D, dtype=torch.half, device="cuda")
out = torch.empty_like(q)
turn = {{"dims": D, "base": 10000.0}}
if {rope}:
    warm = make()
    warm.attention(q, k, v, 0.0625, out=out)        # the partials of this stream are there; the turned rows are not
    step = lambda c: kvc.attention_rope(q, k, v, c, turn, 0.0625, out=out)
    stream = torch.cuda.current_stream()
else:
    step = lambda c: c.attention(q, k, v, 0.0625, out=out)
    stream = torch.cuda.Stream()
torch.cuda.synchronize()
torch.cuda.empty_cache()
before = a.offset, a.meta_state
hold = torch.empty(torch.cuda.mem_get_info()[0] - (5 << 20), dtype=torch.uint8, device="cuda")
with torch.cuda.stream(stream):
    try:
        step(a)
        raise SystemExit("there was memory")
    except kvc.KVCError:
        pass
assert (a.offset, a.meta_state) == before, (a.offset, a.meta_state, before)
del hold
torch.cuda.empty_cache()
step(a)
x = out.clone()
step(b)
assert torch.equal(x, out) and a.offset == b.offset and a.meta_state == b.meta_state
assert all(torch.equal(s, t) for s, t in zip(a.state, b.state))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "mlx-swift-lm_b200", "python"))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)
