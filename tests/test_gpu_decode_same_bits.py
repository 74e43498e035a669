"""A sequence's result has the same bits however many others are decoded with it: the kernel is chosen by the number of tokens alone."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(B, n, H, HK, dtype, seed):
    gen = torch.Generator(DEV).manual_seed(seed)

    def normal(heads):
        return torch.randn(B, n, heads, 128, generator=gen, device=DEV)

    q, k = (torch.nn.functional.normalize(normal(HK), dim=-1).to(dtype) for _ in "qk")
    v, w = normal(H).to(dtype), torch.sigmoid(normal(H)).to(dtype)
    g, b = torch.nn.functional.logsigmoid(normal(HK)) / 16, torch.sigmoid(normal(HK)).to(dtype)
    return (q, k, v, g, b, w), 0.1 * torch.randn(B, H, 128, 128, generator=gen, device=DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("call", [gdn2.gdn2_decode, gdn2.gdn2_prefill])
@pytest.mark.parametrize("n", [1, 4, 8, 9, 16, 37, 63])
def test_a_sequence_alone_equals_the_same_in_a_batch(n, call, dtype):
    B, H, HK = 48, 4, 2                                    # 192 tiles, more than the GPU has SMs; alone 4
    ins, s0 = _inputs(B, n, H, HK, dtype, n)
    s = s0.clone()
    o = call(*ins, s)
    for i in (0, 29, B - 1):
        s1 = s0[i:i + 1].clone()
        o1 = call(*(t[i:i + 1] for t in ins), s1)
        if call is gdn2.gdn2_prefill:
            assert torch.equal(o[0][i:i + 1], o1[0])
        else:
            assert torch.equal(o[i:i + 1], o1)
        assert torch.equal(s[i:i + 1], s1)
    _cabi.kernels().check_device_status()


def test_a_prompt_alone_equals_the_same_in_a_batch_and_packed():
    B, H, HK, S = 24, 4, 2, 64 * 3 + 13                    # short enough for no scan to be cut
    ins, s0 = _inputs(B, S, H, HK, torch.bfloat16, 5)
    o, s = gdn2.gdn2_prefill(*ins, s0)
    packed = [t.reshape(1, B * S, *t.shape[2:]) for t in ins]
    op, sp = gdn2.gdn2_attention(*packed, initial_state=s0, output_final_state=True, cu_seqlens=list(range(0, B * S + 1, S)))
    _cabi.kernels().check_device_status()
    assert torch.equal(op.view_as(o), o) and torch.equal(sp, s)
    for i in (0, B - 1):
        o1, s1 = gdn2.gdn2_prefill(*(t[i:i + 1] for t in ins), s0[i:i + 1])
        assert torch.equal(o1, o[i:i + 1]) and torch.equal(s1, s[i:i + 1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("call", [gdn2.gdn2_decode, gdn2.gdn2_prefill])
@pytest.mark.parametrize("n", [2, 3])
def test_two_and_three_tokens_equal_single_steps(n, call, dtype):
    """Also where they are more tiles than the GPU has SMs: they are swept token by token like a single one."""
    B, H, HK = 24, 16, 8
    ins, s0 = _inputs(B, n, H, HK, dtype, n)
    s, single = s0.clone(), s0.clone()
    res = call(*ins, s)
    o = res if call is gdn2.gdn2_decode else res[0]
    want = torch.cat([gdn2.gdn2_decode(*(t[:, i:i + 1].contiguous() for t in ins), single) for i in range(n)], 1)
    _cabi.kernels().check_device_status()
    assert torch.equal(o, want) and torch.equal(s, single)
