"""The Python binding where no kernel runs: what its calls raise, and what importing it needs."""
import os
import subprocess
import sys

import pytest
import torch

PY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx-swift-lm_b200", "python")


def test_calls_without_a_device_fail_by_the_library_status(kvc):
    if kvc.device_available():
        pytest.skip("a device is there")
    q, k = torch.zeros(1, 4, 1, 64, dtype=torch.half), torch.zeros(1, 2, 1, 64, dtype=torch.half)
    c = kvc.KVCacheSimple()
    for call in (lambda: c.attention(q, k, k, 0.1), lambda: kvc.scaled_dot_product_attention(q, k, k, 0.1),
                 lambda: kvc.attention_rope(q, k, k, c, {"dims": 64}, 0.1), lambda: c.update(k, k)):
        with pytest.raises(kvc.KVCError):
            call()


def test_tensors_the_library_cannot_describe(kvc):
    c, k = kvc.KVCacheSimple(), torch.zeros(1, 2, 1, 64, dtype=torch.half)
    with pytest.raises(IndexError):
        c.attention(torch.zeros(1, 1, 1, 1, 1, 1), k, k, 0.1)
    with pytest.raises(KeyError):
        c.attention(k.double(), k, k, 0.1)


def test_import_needs_neither_torch_nor_the_binding_module():
    """The C ABI is there for hosts that bring their own tensors; what takes torch tensors asks for torch then."""
    code = """
import sys
sys.modules["torch"] = None
sys.modules["kvcache_b200._binding"] = None
import kvcache_b200 as kvc
assert "sm_100a" in kvc.version() and kvc.lib().kvc_launch_count(0) == 0
c = kvc.KVCacheSimple()
assert c.offset == 0 and c.meta_state == [""]
try:
    kvc.scaled_dot_product_attention(None, None, None, 1.0)
    raise SystemExit("torch was not asked for")
except ImportError:
    pass
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=120, env=dict(os.environ, PYTHONPATH=PY))
