"""The tcgen05 chunk kernel over the ways its work is cut, and under stream capture."""
import re

import pytest
import torch

from helpers import seeded

pytestmark = pytest.mark.gpu


def _reference(q, k, v, scale, causal, parts):
    """64-bit attention, and what is left of it with the kernel's two roundings: probabilities are stored in 16 bits against the
    largest score of the row so far (one reference a tile of 128 keys) or of every 128 / parts keys, but never more than 2^24
    below the row's, and so are the outputs."""
    rep, (L, D), T = q.shape[1] // k.shape[1], q.shape[2:], k.shape[2]
    exact, kept = (torch.empty(q.shape, dtype=torch.float64, device=q.device) for _ in range(2))
    hidden = torch.ones(L, T, dtype=torch.bool, device=q.device).triu(T - L + 1)
    step = 128 // parts
    for b in range(q.shape[0]):
        for h in range(q.shape[1]):
            s = (q[b, h].double() @ k[b, h // rep].double().T) * scale * 1.4426950408889634
            if causal:
                s.masked_fill_(hidden, float("-inf"))
            vh = v[b, h // rep].double()
            top = s.amax(-1, keepdim=True)
            p = torch.exp2(s - top)
            l = p.sum(-1, keepdim=True)
            exact[b, h] = p @ vh / l
            s = torch.nn.functional.pad(s, (0, -T % step), value=float("-inf")).view(L, -1, step)
            here = s.amax(-1)
            so_far = here.cummax(-1).values
            ref = so_far if parts == 1 else torch.maximum(here, so_far - 24)
            stored = torch.exp2(s - ref[..., None]).to(q.dtype).double()
            p = (stored * torch.exp2(ref - top)[..., None]).view(L, -1)[:, :T]
            kept[b, h] = (p @ vh / l).to(q.dtype).double()
    return exact, kept


def _check(out, exact, kept):
    """Errors against 64 bits are those of the two roundings, as a whole and in the worst row. (The same scores in 32 bits, the
    running maximum of a cut unit and a few roundings that fall the other way move them by some per cent. Outputs lost from one
    unit, or a factor that is off in one of its partials, are ten times the size.)"""
    err, ideal = (out.double() - exact).norm(dim=-1), (kept - exact).norm(dim=-1)
    size = exact.norm(dim=-1)
    assert err.norm() <= 1.1 * ideal.norm()
    assert (err / size).max() <= 1.3 * (ideal / size).max()


# ... and how the kernel takes them: row tiles a unit, references a tile, whether units are cut
SHAPES = [
    (1, 7, 1, 128, 10, 90, "causal", 1, 4, False),         # 70 rows, 18 positions x 7 heads a row tile: one tile, one unit
    (1, 4, 1, 64, 17, 700, "causal", 1, 4, False),         # 68 rows, the fewest
    (2, 14, 2, 128, 37, 1031, "causal", 1, 4, True),       # three row tiles a group, the last one of one position
    (1, 3, 1, 128, 64, 65, "none", 1, 4, False),           # one key past the calls that stay on the mma.sync kernel
    (1, 4, 1, 64, 17, 2500, "causal", 1, 4, True),         # pieces
    (1, 4, 1, 64, 17, 16400, "causal", 1, 2, True),        # two references: equal ranges
    (1, 32, 8, 128, 256, 7680, "causal", 2, 4, True),      # pairs
    (1, 130, 1, 64, 64, 129, "causal", 1, 1, False),       # more heads than a row tile takes: head by head
    (3, 16, 16, 64, 129, 257, "causal", 1, 1, False),      # one position past a tile, one key past a tile
    (1, 8, 2, 128, 1500, 1500, "causal", 1, 1, False),     # units of 1 ... 12 key tiles
    (4, 28, 4, 128, 397, 1500, "causal", 1, 1, False),     # single row tiles in rounds
    (8, 32, 8, 64, 160, 4300, "causal", 2, 1, True),       # K and V past the L2 share: rounds of whole units, ranges of the rest
    (8, 16, 8, 128, 640, 129, "none", 2, 1, False),        # pairs in rounds
]


def _run(kvc, capfd, q, k, v, scale, mask):
    """The outputs, and how the launch took them (as in SHAPES)."""
    out = kvc.scaled_dot_product_attention(q, k, v, scale, mask)
    torch.cuda.synchronize()
    trace = re.search(r"chunk_tc: \d+ units of (\d) .* ranges of (\d+) tiles, (\d+) pieces, (\d) references", capfd.readouterr().err)
    assert trace and kvc.lib().kvc_device_status() == 0
    return out, int(trace[1]), int(trace[4]), int(trace[2]) + int(trace[3]) > 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,mask,wide,parts,cut", SHAPES)
def test_chunk_units_and_cuts(kvc, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, D, L, T, mask, wide, parts, cut):
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q = torch.randn((B, Hq, L, D), generator=torch.Generator(cuda).manual_seed(1), device=cuda).to(dtype)
    k, v = (torch.randn((B, Hkv, T, D), generator=torch.Generator(cuda).manual_seed(s), device=cuda).to(dtype) for s in (2, 3))
    by_position = q.transpose(1, 2).contiguous().transpose(1, 2)   # [B, L, H, D] in memory
    expected = _reference(q, k, v, D ** -0.5, mask == "causal", parts)
    for x in (q, by_position):
        out, *how = _run(kvc, capfd, x, k, v, D ** -0.5, mask)
        assert how == [wide, parts, cut]
        _check(out, *expected)


@pytest.mark.parametrize("growing", [False, True])
@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,wide,parts,cut", [
    (1, 8, 2, 128, 100, 2000, 1, 4, True),
    (1, 8, 2, 64, 100, 400, 1, 4, False),
    (1, 8, 2, 128, 100, 17000, 1, 2, True),
    (1, 32, 8, 128, 400, 1100, 1, 1, False),
    (1, 32, 8, 128, 256, 7680, 2, 4, True),
    (74, 8, 2, 64, 40, 17000, 2, 2, False),
    (4, 32, 8, 128, 130, 9000, 2, 1, True),
    (8, 32, 8, 128, 128, 1000, 2, 1, False),
])
def test_chunk_scores_that_move_the_reference(kvc, cuda, capfd, monkeypatch, growing, B, Hq, Hkv, D, L, T, wide, parts, cut):
    """Scores that rise and fall by more than the span between a part and the row from one key tile to the next."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    dtype = torch.float16
    q = torch.ones((B, Hq, L, D), device=cuda, dtype=dtype)
    # up and down by 650 in the exponent every 700 keys, the peaks a little higher or lower each time
    wave = (2 * ((torch.arange(T, device=cuda) / 700) % 2 - 1).abs() - 1) * torch.linspace(30, 40, T, device=cuda) * (128 / D) ** 0.5
    k = (wave if growing else wave.flip(0))[None, None, :, None].expand(B, Hkv, T, D).to(dtype).contiguous()
    v = torch.randn((B, Hkv, T, D), generator=torch.Generator(cuda).manual_seed(3), device=cuda).to(dtype)
    out, *how = _run(kvc, capfd, q, k, v, D ** -0.5, "causal")
    assert how == [wide, parts, cut]
    some = [0, B - 1] if B > 8 else range(B)
    _check(out[some], *_reference(q[some], k[some], v[some], D ** -0.5, True, parts))


@pytest.mark.parametrize("dtype,B,L,T,cut", [
    (torch.bfloat16, 1, 96, 3000, True),      # partials of cut units
    (torch.float16, 8, 128, 2000, False),     # sums that are folded into memory
])
def test_chunk_with_memory_of_its_own_can_be_captured(kvc, cuda, capfd, monkeypatch, dtype, B, L, T, cut):
    """The memory of a captured call belongs to its graph: replays on other inputs give the eager call's bits."""
    Hq, Hkv, D = 32, 8, 128
    q, k, v = (seeded((B, h, n, D), s, dtype).to(cuda) for h, n, s in ((Hq, L, 1), (Hkv, T, 2), (Hkv, T, 3)))
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    assert _run(kvc, capfd, q, k, v, D ** -0.5, "causal")[-1] == cut
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal", out=out)
    for seed in (11, 12):
        q.copy_(seeded(tuple(q.shape), seed, dtype))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, "causal"))


def _bias(out, ref):
    """How far the outputs lie from 64-bit ones towards zero (negative) or away from it, of their mean size."""
    return ((out.double() - ref) * ref.sign()).mean().item() / ref.abs().mean().item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,T", [
    (1, 80, 8, 64, 70000),       # pairs, equal ranges of all units
    (1, 148, 148, 70, 9000),     # single row tiles, whole units
    (8, 32, 8, 21, 9000),        # ... in ranges
    (8, 32, 8, 512, 3000),       # pairs in rounds
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
