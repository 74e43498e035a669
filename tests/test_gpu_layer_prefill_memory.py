"""The layer's prefill as one native call needs no more device memory at its peak than the stages called from Python."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi

pytestmark = pytest.mark.gpu


def test_native_call_peaks_no_higher(monkeypatch):
    torch.manual_seed(0)
    layer = gdn2.GatedDeltaNet2(gdn2.GatedDeltaNet2Config(hidden_size=1024, num_heads=16, num_kv_heads=8, head_dim_k=128, head_dim_v=128))
    layer = layer.to("cuda", torch.bfloat16).eval()
    x = torch.randn(8, 2000, 1024, device="cuda", dtype=torch.bfloat16)      # normalised outputs of 65 MB
    cache = layer.prefill(x)[1]

    def peak():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        layer.prefill(x, gdn2.GDN2Cache(cache.recurrent_state, cache.conv_state))
        torch.cuda.synchronize()
        return torch.cuda.max_memory_allocated() - before

    native = peak()
    monkeypatch.setattr(_cabi.kernels(), "host", None)
    assert native <= peak() + (16 << 20)                   # the allocator rounds large blocks up
