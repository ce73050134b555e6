"""The tcgen05 chunk kernel over the ways its work is cut, and under stream capture."""
import numpy as np
import pytest
import torch

from helpers import seeded

pytestmark = pytest.mark.gpu


def _reference(q, k, v, scale, causal):
    """Plain fp32 attention of the same inputs."""
    rep, L, T = q.shape[1] // k.shape[1], q.shape[2], k.shape[2]
    k, v = (x.float().repeat_interleave(rep, 1) for x in (k, v))
    s = (q.float() @ k.transpose(-1, -2)) * scale
    if causal:
        s.masked_fill_(torch.ones(L, T, dtype=torch.bool, device=q.device).triu(T - L + 1), float("-inf"))
    return torch.softmax(s, -1) @ v


def _bound(v, dtype):
    """Probabilities and outputs are each rounded once to `dtype` (2^-9 or 2^-12 of their size), and an output is a mean of
    the values: twice that of the largest one, and as much again for the sums' order and the exponentials."""
    return 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12) * v.abs().max().item()


SHAPES = [
    (1, 7, 1, 128, 10, 90, "causal"),          # 70 rows, 18 positions x 7 heads a row tile: one tile, four references
    (1, 4, 1, 64, 17, 700, "causal"),          # 68 rows, the fewest: one unit in pieces
    (2, 14, 2, 128, 37, 1031, "causal"),       # three row tiles a group: the last unit has one
    (1, 3, 1, 128, 64, 65, "none"),            # one key past the calls that stay on the mma.sync kernel
    (1, 4, 1, 64, 17, 2500, "causal"),         # ... two references a tile
    (1, 130, 1, 64, 64, 129, "causal"),        # more heads than a row tile takes: head by head
    (3, 16, 16, 64, 129, 257, "causal"),       # one position past a tile, one key past a tile
    (1, 8, 2, 128, 1500, 1500, "causal"),      # units of 1 ... 12 key tiles
    (4, 28, 4, 128, 397, 1500, "causal"),      # equal ranges of all units
    (8, 32, 8, 64, 160, 4300, "causal"),       # K and V past the L2 share: rounds of whole units, ranges of the rest
    (8, 16, 8, 128, 640, 129, "none"),         # rounds of whole units alone
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,mask", SHAPES)
def test_chunk_units_and_cuts(kvc, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, D, L, T, mask):
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q = torch.randn((B, Hq, L, D), generator=torch.Generator(cuda).manual_seed(1), device=cuda).to(dtype)
    k, v = (torch.randn((B, Hkv, T, D), generator=torch.Generator(cuda).manual_seed(s), device=cuda).to(dtype) for s in (2, 3))
    ref = _reference(q, k, v, D ** -0.5, mask == "causal")
    by_position = q.transpose(1, 2).contiguous().transpose(1, 2)   # [B, L, H, D] in memory
    for x in (q, by_position):
        out = kvc.scaled_dot_product_attention(x, k, v, D ** -0.5, mask)
        torch.cuda.synchronize()
        assert "chunk_tc" in capfd.readouterr().err
        assert (out.float() - ref).abs().max().item() <= _bound(v, dtype)
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("growing", [False, True])
def test_chunk_scores_that_move_the_reference(kvc, cuda, growing):
    """Scores that rise (or fall) by far more than the exponent range from one key tile to the next."""
    dtype, D, L, T = torch.float16, 128, 100, 1000
    q = torch.ones((1, 8, L, D), device=cuda, dtype=dtype)
    ramp = torch.linspace(-40, 40, T, device=cuda)
    k = (ramp if growing else -ramp)[None, None, :, None].expand(1, 2, T, D).to(dtype).contiguous()
    v = torch.randn((1, 2, T, D), generator=torch.Generator(cuda).manual_seed(3), device=cuda).to(dtype)
    out = kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal")
    assert (out.float() - _reference(q, k, v, D ** -0.5, True)).abs().max().item() <= _bound(v, dtype)


def test_chunk_with_cut_units_can_be_captured(kvc, cuda):
    """The partials of a captured call belong to its graph: replays on other inputs give the eager call's bits."""
    B, Hq, Hkv, D, L, T = 1, 32, 8, 128, 96, 3000
    q, k, v = (seeded((B, h, n, D), s, torch.bfloat16).to(cuda) for h, n, s in ((Hq, L, 1), (Hkv, T, 2), (Hkv, T, 3)))
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal", out=out)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal", out=out)
    for seed in (11, 12):
        q.copy_(seeded(tuple(q.shape), seed, torch.bfloat16))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.view(torch.int16).cpu(), kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal").view(torch.int16).cpu())


def _bias(out, ref):
    """How far the outputs lie from 64-bit ones towards zero (negative) or away from it, of their mean size."""
    return ((out.double() - ref) * ref.sign()).mean().item() / ref.abs().mean().item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,T", [
    (1, 80, 8, 64, 70000),       # equal ranges of all units
    (1, 148, 148, 70, 9000),     # whole units
    (8, 32, 8, 21, 9000),        # pieces of a unit
])
def test_sums_over_long_contexts(kvc, cuda, capfd, monkeypatch, D, B, Hq, Hkv, L, T):
    """f16 sums of one sign: the tensor core adds towards zero and alone loses 6e-9 of them a key, 5e-5 over 9 000; folded into fp32
    sums every 512 or 768 keys they lose 3e-6 or 4.5e-6. The stores' rounding averages out over the outputs (four sigma are allowed)."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q, k, v = (torch.randn((B, h, n, D), generator=torch.Generator(cuda).manual_seed(i), device=cuda) for i, (h, n) in enumerate(((Hq, L), (Hkv, T), (Hkv, T))))
    q, k, v = q.half(), k.half(), (v + 1).half()
    out = kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal")
    torch.cuda.synchronize()
    assert "chunk_tc" in capfd.readouterr().err
    rep, seen = Hq // Hkv, torch.arange(T, device=cuda) <= torch.arange(T - L, T, device=cuda)[:, None]
    ref = torch.stack([torch.stack([torch.softmax((q[b, h].double() @ k[b, h // rep].double().T * D ** -0.5).masked_fill_(~seen, float("-inf")), -1)
                                    @ v[b, h // rep].double() for h in range(Hq)]) for b in range(B)])
    assert abs(_bias(out, ref)) <= 4.5e-6 + 4 * 2.2e-4 * out.numel() ** -0.5
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 2.0 ** -11
    assert kvc.lib().kvc_device_status() == 0
