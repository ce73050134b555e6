"""Scales of zero and below: hidden keys stay hidden whatever the factor of the scores (scale 0: a plain mean of the visible
values; negative: the least similar key weighs most)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _error(out, q, k, v, scale, seen):
    """Relative 2-norm of what is left against 64-bit attention."""
    rep = q.shape[1] // k.shape[1]
    k, v = (x.double().repeat_interleave(rep, 1) for x in (k, v))
    s = (q.double() @ k.transpose(-1, -2) * scale).masked_fill(~seen, float("-inf"))
    ref = torch.softmax(s, -1) @ v
    return ((out.double() - ref).norm() / ref.norm()).item()


def _seen(cuda, mask, L, T):
    i, j = torch.arange(T - L, T, device=cuda)[:, None], torch.arange(T, device=cuda)[None]
    return {"none": j >= 0, "causal": j <= i, "window": (j <= i) & (j > i - 100)}[mask].expand(L, T)


# P and the outputs are each rounded to 16 bits: 2^-9 of a value (bf16) or 2^-12 at most, both far from lined up over a row
BOUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scale", [0.0, -0.1, 0.1])
@pytest.mark.parametrize("B,Hq,Hkv,D,L,T,mask", [
    (1, 8, 2, 128, 20, 333, "causal"),     # few row blocks
    (4, 32, 8, 64, 300, 333, "causal"),    # many
    (4, 32, 8, 128, 64, 333, "none"),      # a last key tile that is not full
    (1, 8, 2, 64, 40, 333, "window"),
    (2, 8, 2, 128, 300, 333, "window"),
    (1, 4, 1, 256, 20, 333, "window"),
    (1, 4, 1, 256, 70, 333, "causal"),
    (2, 32, 8, 128, 6, 333, "causal"),     # verify rounds
    (1, 4, 1, 128, 6, 333, "none"),
])
def test_chunks(kvc, cuda, dtype, scale, B, Hq, Hkv, D, L, T, mask):
    q, k, v = (torch.randn((B, h, n, D), generator=torch.Generator(cuda).manual_seed(i), device=cuda).to(dtype)
               for i, (h, n) in enumerate(((Hq, L), (Hkv, T), (Hkv, T))))
    seen = _seen(cuda, mask, L, T)
    out = kvc.scaled_dot_product_attention(q, k, v, scale, seen if mask == "window" else mask)
    assert _error(out, q, k, v, scale, seen) <= BOUND[dtype]
    assert kvc.lib().kvc_device_status() == 0


@pytest.mark.parametrize("make", ["affine", "turbo"])
@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("L", [6, 64, 300])
def test_packed_caches(kvc, cuda, make, scale, L):
    """Verify rounds and prompt chunks. 8-bit codes: half a step of a group's range in the values, and as
    much again for the keys; 4-bit centroids err by a tenth of a value, averaged over the keys like the values themselves."""
    B, Hq, Hkv, D, P = 4, 32, 8, 128, 269
    c = kvc.QuantizedKVCache(64, 8) if make == "affine" else kvc.TurboQuantKVCache(bits=4, key_bits=4, value_bits=4)
    x = [torch.randn((B, h, n, D), generator=torch.Generator(cuda).manual_seed(i), device=cuda).to(torch.bfloat16)
         for i, (h, n) in enumerate(((Hkv, P), (Hkv, P), (Hq, L), (Hkv, L), (Hkv, L)))]
    (c.update_quantized if make == "affine" else c.encode_new_token)(x[0], x[1])
    out = c.attention(x[2], x[3], x[4], scale, "causal")
    k, v = torch.cat([x[0], x[3]], 2), torch.cat([x[1], x[4]], 2)
    assert _error(out, x[2], k, v, scale, _seen(cuda, "causal", L, P + L)) <= (0.02 if make == "affine" else 0.2)
    assert kvc.lib().kvc_device_status() == 0
