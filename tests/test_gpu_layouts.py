"""Calls in the layouts, mask forms and sizes callers have, on the kernels the dispatch picks and on the general one."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = 160

CODE = """
import random, sys
import torch, kvcache_b200 as kvc
dev = torch.device("cuda")

def rows(rng, g, B, H, L, D, dt):
    R = lambda *s: torch.randn(*s, generator=g, dtype=torch.float32, device=dev).to(dt)
    how = rng.choice(["plain", "tokens first", "padded rows", "slice", "one batch for all"])
    if how == "tokens first": return R(B, L, H, D).transpose(1, 2)
    if how == "padded rows": return R(B, H, L, D + 8)[..., :D]
    if how == "slice": return R(B, H + 1, L + 2, D)[:, 1:, 1:L + 1]
    return R(1, H, L, D).expand(B, H, L, D) if how == "one batch for all" else R(B, H, L, D)

def mask(rng, g, B, Hq, L, T):
    kind = rng.choice(["none", "causal", "bool", "pitch", "broadcast", "heads", "columns first", "f32", "f16"])
    if kind in ("none", "causal"): return kind
    row, col = torch.arange(T - L, T, device=dev)[:, None], torch.arange(T, device=dev)[None]
    keep = (col <= row) & (torch.rand(L, T, generator=g, device=dev) < 0.7) | (col == 0)
    if L > 3: keep[2] = False
    if kind == "pitch":
        w = torch.zeros(L, T + 5, dtype=torch.bool, device=dev)
        w[:, 3:T + 3] = keep
        return w[:, 3:T + 3]
    if kind == "broadcast": return keep[None, None].expand(B, Hq, L, T)
    if kind == "heads": return keep[None, None] & (torch.rand(B, Hq, L, T, generator=g, device=dev) < 0.8)
    if kind == "columns first": return keep.T.contiguous().T
    add = torch.where(keep, torch.randn(L, T, generator=g, device=dev), torch.tensor(-torch.inf, device=dev))
    return {"bool": keep, "f32": add, "f16": add.half()}[kind]

found = []
for i in range(int(sys.argv[1])):
    rng, g = random.Random(i), torch.Generator(device=dev).manual_seed(i)
    D, Hkv, B = rng.choice([64, 128, 256]), rng.choice([1, 2, 4]), rng.randint(1, 3)
    Hq, P = Hkv * rng.choice([1, 2, 4, 7]), rng.choice([1, 16, 63, 65, 200, 513, 1000])
    kind = rng.choice(["raw", "affine", "index", "index"])
    dt = rng.choice([torch.bfloat16, torch.float16] + ([torch.float32] if kind != "index" else []))
    if kind == "raw":
        c = kvc.KVCacheSimple()
    elif kind == "affine":
        c = kvc.QuantizedKVCache(rng.choice([32, 64]), rng.choice([2, 4, 8]))
    else:
        kb, vb = rng.choice([(0, 4), (8, 4), (8, 2), (4, 4), (3, 3), (3, 4), (0, 2), (4, 2)])
        c = kvc.TurboQuantKVCache(bits=4, key_bits=kb, value_bits=vb, affine_values=vb == 4 and rng.random() < 0.3)
    fill = {"raw": getattr(c, "update", None), "affine": getattr(c, "update_quantized", None), "index": getattr(c, "encode_new_token", None)}[kind]
    fill(rows(rng, g, B, Hkv, P, D, dt), rows(rng, g, B, Hkv, P, D, dt))
    for L in (1, rng.choice([2, 9, 17, 40, 100])):
        q, k, v = rows(rng, g, B, Hq, L, D, dt), rows(rng, g, B, Hkv, L, D, dt), rows(rng, g, B, Hkv, L, D, dt)
        out = torch.empty(B, L, Hq, D, dtype=dt, device=dev).transpose(1, 2) if rng.random() < 0.3 else None
        found.append(c.attention(q, k, v, D ** -0.5, mask(rng, g, B, Hq, L, c.offset + L), out=out).cpu())
assert kvc.device_status() == 0
torch.save(found, sys.argv[2])
"""


def test_layouts_masks_and_sizes_agree_with_the_general_kernel(tmp_path):
    """Bounds on the relative 2-norm: one spacing of bf16 (2^-8), two of f16 (2^-9: probabilities of 16 bits and two
    stores), 2e-5 for f32 (the order of up to 1 100 terms); rows a mask leaves empty are zero in both."""
    files = []
    for path in ("", "general"):
        files.append(str(tmp_path / (path or "default")))
        env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "mlx-swift-lm_b200", "python"), KVC_ATTENTION_PATH=path)
        subprocess.run([sys.executable, "-c", CODE, str(CASES), files[-1]], check=True, env=env, timeout=600)
    mine, general = (torch.load(f) for f in files)
    assert len(mine) == len(general) == 2 * CASES
    bound = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -9, torch.float32: 2e-5}
    for i, (a, b) in enumerate(zip(mine, general)):
        assert torch.isfinite(a).all()
        assert float((a.double() - b.double()).norm()) <= bound[a.dtype] * float(b.double().norm()), i
