"""The tcgen05 chunk kernel that keeps P as pairs: boolean array masks, and head dim 256."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(cuda, dtype, B, Hq, Hkv, D, L, T, seed=1):
    def rand(i, *shape):
        return torch.randn(shape, generator=torch.Generator(cuda).manual_seed(seed + i), device=cuda).to(dtype)
    return rand(0, B, Hq, L, D), rand(1, B, Hkv, T, D), rand(2, B, Hkv, T, D)


def _check(kvc, capfd, q, k, v, mask, seen):
    """Against plain fp32 attention; P is exact to 2^-16 (pairs), so what is left is the store: half a spacing of the output,
    and 2^-14 of the largest value for P, the exponentials and sums in another order."""
    dtype, rep, scale = q.dtype, q.shape[1] // k.shape[1], q.shape[-1] ** -0.5
    kr, vr = (x.float().repeat_interleave(rep, 1) for x in (k, v))
    s = ((q.float() @ kr.transpose(-1, -2)) * scale).masked_fill(~seen, float("-inf"))
    ref = torch.nan_to_num(torch.softmax(s, -1), nan=0.0) @ vr
    out = kvc.scaled_dot_product_attention(q, k, v, scale, mask)
    torch.cuda.synchronize()
    assert "chunk_one" in capfd.readouterr().err
    store = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert ((out.float() - ref).abs() <= store * ref.abs() + 2.0 ** -14 * v.abs().max()).all()
    assert not out[~seen.expand_as(s).any(-1)].any()
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,window", [
    (4, 4, 1, 256, 512, 1023, 512),     # sliding window, its tiles shared among pieces
    (1, 16, 16, 64, 70, 300, 100),      # one head a row tile; two CTAs an SM
    (2, 28, 4, 128, 37, 65, 30),        # one key past the calls of the mma.sync kernel; 126 rows a row tile
    (1, 8, 1, 256, 20, 4097, 64),       # most tiles unseen: pieces with nothing to do
    (9, 32, 8, 128, 129, 200, 128),     # more row tiles than places: no pieces
])
def test_window_masks(kvc, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, D, L, T, window):
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q, k, v = _case(cuda, dtype, B, Hq, Hkv, D, L, T)
    i, j = torch.arange(T - L, T, device=cuda)[:, None], torch.arange(T, device=cuda)[None]
    seen = (j <= i) & (j > i - window)
    _check(kvc, capfd, q, k, v, seen, seen)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("form", ["heads", "batch", "odd rows"])
def test_masks_of_any_form(kvc, cuda, capfd, monkeypatch, D, form):
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    B, Hq, Hkv, L, T = 2, 6, 2, 75, 333
    q, k, v = _case(cuda, torch.bfloat16, B, Hq, Hkv, D, L, T)
    shape = {"heads": (1, Hq, L, T + 3), "batch": (B, 1, L, T + 3), "odd rows": (L, T + 3)}[form]
    m = torch.rand(shape, generator=torch.Generator(cuda).manual_seed(7), device=cuda) < 0.3
    m[..., 5, :] = False                      # a position that sees nothing
    m[..., 64:192] = False                    # tiles that nobody sees
    m = m[..., 3:]                            # rows that begin anywhere
    _check(kvc, capfd, q, k, v, m, m)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,L,T,mask", [
    (1, 4, 1, 512, 2048, "causal"), (3, 8, 8, 66, 127, "none"), (1, 2, 1, 129, 129, "causal"), (2, 4, 1, 17, 3000, "causal"),
])
def test_head_dim_256(kvc, cuda, capfd, monkeypatch, dtype, B, Hq, Hkv, L, T, mask):
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q, k, v = _case(cuda, dtype, B, Hq, Hkv, 256, L, T)
    seen = torch.ones(L, T, dtype=torch.bool, device=cuda)
    if mask == "causal":
        seen = seen.tril(T - L)
    _check(kvc, capfd, q, k, v, mask, seen)
    _check(kvc, capfd, q.transpose(1, 2).contiguous().transpose(1, 2), k, v, mask, seen)


@pytest.mark.parametrize("D,mask", [(64, "array"), (128, "array"), (256, "array"), (256, "causal")])
@pytest.mark.parametrize("B,Hq,Hkv,L,T", [
    (1, 4, 1, 64, 70000),        # pieces
    (1, 160, 160, 70, 9000),     # whole units
])
def test_sums_over_long_contexts(kvc, cuda, capfd, monkeypatch, D, mask, B, Hq, Hkv, L, T):
    """f16 sums of one sign: the tensor core adds towards zero and alone loses 6e-9 of them a key, 5e-5 over 9 000; folded into fp32
    sums every 512 keys they lose 3e-6. The stores' rounding averages out over the outputs (four sigma are allowed)."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q, k, v = _case(cuda, torch.float32, B, Hq, Hkv, D, L, T)
    q, k, v = q.half(), k.half(), (v + 1).half()
    seen = torch.arange(T, device=cuda) <= torch.arange(T - L, T, device=cuda)[:, None]
    out = kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, seen if mask == "array" else mask)
    torch.cuda.synchronize()
    assert "chunk_one" in capfd.readouterr().err
    ref = torch.stack([torch.softmax((q[0, h].double() @ k[0, h * Hkv // Hq].double().T * D ** -0.5).masked_fill_(~seen, float("-inf")), -1)
                       @ v[0, h * Hkv // Hq].double() for h in range(Hq)])
    assert abs(((out[0].double() - ref) * ref.sign()).mean().item()) <= (3e-6 + 4 * 2.2e-4 * out.numel() ** -0.5) * ref.abs().mean().item()
    assert ((out[0].double() - ref).norm() / ref.norm()).item() <= 2.0 ** -11
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,array", [(1, 4, 1, 256, 40, 3000, False), (1, 4, 1, 256, 40, 3000, True), (1, 8, 2, 128, 70, 2000, True)])
def test_cut_units_can_be_captured(kvc, cuda, capfd, monkeypatch, B, Hq, Hkv, D, L, T, array):
    """The partials of a captured call belong to its graph: replays on other inputs give the eager call's bits."""
    monkeypatch.setenv("KVC_TRACE_DISPATCH", "1")
    q, k, v = _case(cuda, torch.bfloat16, B, Hq, Hkv, D, L, T)
    mask = torch.arange(T, device=cuda) <= torch.arange(T - L, T, device=cuda)[:, None] if array else "causal"
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, mask, out=out)
    assert int(re.search(r"chunk_one: .* (\d+) pieces", capfd.readouterr().err)[1]) > 1
    for seed in (11, 12):
        q.copy_(_case(cuda, torch.bfloat16, B, Hq, Hkv, D, L, T, seed)[0])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, kvc.scaled_dot_product_attention(q, k, v, D ** -0.5, mask))
    assert kvc.lib().kvc_device_status() == 0
