"""One token through the layer in three kernels (``gdn2_layer_step``) against the stages called one by one, at the edges of its
range: one and two groups of eight tokens and what fills neither, reductions of one and of an odd number of 64-step groups, more
heads than the output kernel keeps weights in registers for, shared key heads, no convolution bias."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(hidden, H, HK, dtype, bias):
    torch.manual_seed(hidden + H)
    layer = gdn2.GatedDeltaNet2(gdn2.GatedDeltaNet2Config(hidden_size=hidden, num_heads=H, num_kv_heads=HK, head_dim_k=128, head_dim_v=128))
    if not bias:
        for c in (layer.q_conv, layer.k_conv, layer.v_conv):
            c.conv.bias = None
    return layer.to(DEV, dtype).eval()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,hidden,H,HK,bias", [(1, 64, 1, 1, True), (2, 192, 4, 2, False), (8, 256, 2, 2, True), (9, 320, 3, 1, True),
                                                (16, 1024, 18, 9, True)])
def test_step_equals_its_stages(monkeypatch, B, hidden, H, HK, bias, dtype):
    layer = _layer(hidden, H, HK, dtype, bias)
    K = _cabi.kernels()
    assert K.lib.gdn2_layer_step_workspace_bytes(B, hidden, H, HK, 128, 128, 4, _cabi.dtype_code(dtype)) > 0
    gen = torch.Generator().manual_seed(5)
    s0 = (0.02 * torch.randn(B, H, 128, 128, generator=gen)).to(DEV)
    c0 = torch.randn(B, (2 * HK + H) * 128, 3, generator=gen).to(DEV, dtype)
    xs = torch.randn(3, B, hidden, generator=gen).to(DEV, dtype)

    def steps():
        cache, outs = gdn2.GDN2Cache(s0.clone(), c0.clone()), []
        for x in xs:
            y, cache = layer.step(x, cache)
            outs.append(y)
        return torch.stack(outs), cache

    got, cache = steps()
    with monkeypatch.context() as m:                       # without the host extension: the same kernels, the same bits
        m.setattr(K, "host", None)
        again, cache_again = steps()
        m.setattr(K, "layer_step", lambda *a: None)        # and the stages one by one
        want, cache_want = steps()
    K.check_device_status()
    assert torch.equal(got, again) and torch.equal(cache.recurrent_state, cache_again.recurrent_state)
    assert torch.equal(cache.conv_state, cache_again.conv_state)
    # The products are summed in another order, so a projection may round to the neighbouring 16-bit value: one unit in the
    # last place (2^-8 in bf16, 2^-11 in f16) of single entries, which the following stages pass on as such. The bounds leave
    # a factor of four.
    ulp = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    assert orc.rel_max_err(got.float().cpu(), want.float().cpu()) < 8 * ulp
    assert orc.rel_fro_err(got.float().cpu(), want.float().cpu()) < 4 * ulp
    assert orc.rel_fro_err(cache.recurrent_state.cpu(), cache_want.recurrent_state.cpu()) < 4 * ulp
    assert orc.rel_max_err(cache.conv_state.float().cpu(), cache_want.conv_state.float().cpu()) < 2 * ulp


def test_more_sequences_than_the_kernels_take_go_stage_by_stage():
    layer = _layer(256, 2, 2, torch.bfloat16, True)
    K = _cabi.kernels()
    assert K.lib.gdn2_layer_step_workspace_bytes(17, 256, 2, 2, 128, 128, 4, _cabi.dtype_code(torch.bfloat16)) == 0
    x = torch.randn(17, 256, generator=torch.Generator().manual_seed(1)).to(DEV, torch.bfloat16)
    y, cache = layer.step(x, layer.init_cache(17))
    z, _ = layer.step(x[:1], layer.init_cache(1))
    assert orc.rel_max_err(y[:1].float().cpu(), z.float().cpu()) < 2.0**-5
    with pytest.raises((TypeError, ValueError, RuntimeError)):
        layer.step(x.float(), cache)
