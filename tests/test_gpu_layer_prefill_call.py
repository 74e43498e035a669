"""The layer's prefill as one native call against the stages called from Python: the same kernels with the same arguments, so the
same bits; prompts shorter than a chunk (the recurrent state is updated in place), of whole chunks, and ragged."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.float16, 128), (torch.float32, 64)])
@pytest.mark.parametrize("S", [1, 5, 40, 64, 150])
def test_native_equals_general(monkeypatch, S, dtype, D):
    torch.manual_seed(S)
    layer = gdn2.GatedDeltaNet2(gdn2.GatedDeltaNet2Config(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim_k=D, head_dim_v=D))
    layer = layer.to(DEV, dtype).eval()
    x = torch.randn(2, S, 256, device=DEV, dtype=dtype)
    state = 0.05 * torch.randn(2, 4, D, D, device=DEV)
    conv = torch.randn(2, 8 * D, 3, device=DEV, dtype=dtype)
    K = _cabi.kernels()

    def call():
        before = K.launches
        out0, fresh = layer.prefill(x)
        cache = gdn2.GDN2Cache(state.clone(), conv.clone())
        mine = cache.recurrent_state
        out, cache = layer.prefill(x, cache)
        assert (cache.recurrent_state is mine) == (S < 64)
        return out0, fresh.recurrent_state, fresh.conv_state, out, cache.recurrent_state, cache.conv_state, K.launches - before

    native = call()
    with monkeypatch.context() as m:
        m.setattr(K, "host", None)
        general = call()
    K.check_device_status()
    assert all(torch.equal(a, b) for a, b in zip(native[:6], general[:6])) and native[6] == general[6]
    wide = torch.cat([x, x], 2)[..., :256]                 # not dense: the general path
    assert torch.equal(layer.prefill(wide)[0], native[0])
