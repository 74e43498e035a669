"""The native host path against the general one: the same kernels with the same arguments, so the same bits; and calls that
are not plain (strided, converted, wrong shapes) still go through the general path or raise what it raises."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _both(monkeypatch, call):
    """The results of ``call()`` with and without the host extension."""
    native = call()
    with monkeypatch.context() as m:
        m.setattr(_cabi.kernels(), "host", None)
        general = call()
    return native, general


def _inputs(B, S, H, HK, D, dtype, seed=0):
    q, k, _, g, b, _ = orc.make_inputs(B, S, HK, D, D, seed=seed)
    _, _, v, _, _, w = orc.make_inputs(B, S, H, D, D, seed=seed + 1)
    return [t.to(DEV, dtype) for t in (q, k, v)] + [g.to(DEV)] + [t.to(DEV, dtype) for t in (b, w)]


@pytest.mark.parametrize("n,H,HK,D,dtype", [(1, 4, 2, 128, torch.bfloat16), (5, 2, 2, 128, torch.float16), (3, 2, 1, 64, torch.float32)])
def test_decode(monkeypatch, n, H, HK, D, dtype):
    ins = _inputs(2, n, H, HK, D, dtype)
    s0 = torch.randn(2, H, D, D, device=DEV)

    def call():
        s = s0.clone()
        o = gdn2.gdn2_decode(*ins, s)
        if n == 1:
            s2 = s0.clone()
            assert torch.equal(gdn2.gdn2_decode_step(*(t[:, 0].contiguous() for t in ins), s2, D**-0.5), o[:, 0]) and torch.equal(s, s2)
        # strided tokens, a scale of its own, double-precision decay: not plain
        wide = [torch.cat([t, t], 1)[:, :n] for t in ins]
        s3 = s0.clone()
        o3 = gdn2.gdn2_decode(*wide[:3], wide[3].double(), *wide[4:], s3, scale=D**-0.5)
        assert torch.equal(o, o3) and torch.equal(s, s3)
        return o, s

    (o, s), (o2, s2) = _both(monkeypatch, call)
    assert torch.equal(o, o2) and torch.equal(s, s2)
    for bad in (s0[:1], s0.double(), s0.transpose(2, 3)):
        with pytest.raises(ValueError):
            gdn2.gdn2_decode(*ins, bad)
    with pytest.raises(ValueError):
        gdn2.gdn2_decode(ins[0], ins[1][:, :, :, :32], *ins[2:], s0.clone())
    with pytest.raises(TypeError):
        gdn2.gdn2_decode(ins[0].double(), *ins[1:], s0.clone())


@pytest.mark.parametrize("S", [20, 64, 150])
@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (64, torch.float32)])
def test_prefill_and_attention(monkeypatch, S, D, dtype):
    ins = _inputs(1, S, 2, 1, D, dtype)
    s0 = torch.randn(1, 2, D, D, device=DEV).mul_(0.1)

    def call():
        return (*gdn2.gdn2_prefill(*ins), *gdn2.gdn2_prefill(*ins, s0.clone()), *gdn2.gdn2_prefill(*ins, s0.double()),
                *gdn2.gdn2_attention(*ins, initial_state=s0, output_final_state=True), gdn2.gdn2_attention(*ins)[0])

    native, general = _both(monkeypatch, call)
    assert all(torch.equal(a, b) for a, b in zip(native, general))
    with pytest.raises(ValueError):
        gdn2.gdn2_prefill(*ins, s0[:, :1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_layer_step(monkeypatch, dtype):
    torch.manual_seed(0)
    cfg = gdn2.GatedDeltaNet2Config(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim_k=128, head_dim_v=128)
    layer = gdn2.GatedDeltaNet2(cfg).to(DEV, dtype).eval()
    x = torch.randn(2, 70, 256, device=DEV, dtype=dtype)

    def call():
        out, cache = layer.prefill(x[:, :66])
        outs = [out]
        for t in range(66, 68):
            y, cache = layer.step(x[:, t], cache)
            outs.append(y)
        y, cache = layer.decode(x[:, 68:70], cache)
        return (*outs, y, cache.recurrent_state, cache.conv_state)

    native, general = _both(monkeypatch, call)
    assert all(torch.equal(a, b) for a, b in zip(native, general))
    with torch.no_grad():                                # a parameter changes: the fused tables follow
        layer.q_proj.weight.mul_(2.0)
        layer.o_proj.weight = torch.nn.Parameter(layer.o_proj.weight * 3.0)
    native, general = _both(monkeypatch, call)
    assert all(torch.equal(a, b) for a, b in zip(native, general))
    seen = []
    handle = layer.o_proj.register_forward_hook(lambda *a: seen.append(1))
    call()
    handle.remove()
    assert len(seen) == 4                                # hooks on the output projection still run, in every call


@pytest.mark.parametrize("D,launched", [(128, 3), (64, 4)])
def test_launches_are_counted(monkeypatch, D, launched):
    """The benchmark's accounting, by either path: the general front of the layer is two kernels."""
    cfg = gdn2.GatedDeltaNet2Config(hidden_size=256, num_heads=2, head_dim_k=D)
    layer = gdn2.GatedDeltaNet2(cfg).to(DEV, torch.bfloat16)
    x = torch.randn(2, 256, device=DEV, dtype=torch.bfloat16)
    K = _cabi.kernels()

    def call():
        cache, before = layer.init_cache(2), K.launches
        layer.step(x, cache)
        return K.launches - before

    assert _both(monkeypatch, call) == (launched, launched)
