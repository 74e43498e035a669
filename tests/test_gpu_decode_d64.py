"""Decode at DK = DV = 64: the register-tile kernel, and the generic one that a state without 16-byte alignment keeps.

Tolerance: float32 sums of 64 terms per token in another order than the oracle's; the bound of the decode tests at
D = 128 (2e-5 of the largest value over up to 23 tokens) covers them with room. 16-bit outputs round once, to 2^-8 of a value
of a few at most: 2e-2."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 2, 8, 9, 17])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("aligned", [True, False])
def test_decode_d64(n, dtype, aligned):
    B, H, HK, D = 2, 6, 3, 64
    q, k, _, g, b, _ = orc.make_inputs(B, n, HK, D, D, seed=n, gate="softplus", decay_scale=4.0)
    _, _, v, _, _, w = orc.make_inputs(B, n, H, D, D, seed=n + 1, gate="softplus")
    q, k, v, b, w = (t.to(dtype) for t in (q, k, v, b, w))
    s0 = golden_state(B, H, D, D, n, 0.3)
    room = torch.zeros(s0.numel() + 4, device=DEV)
    state = room[0 if aligned else 1:][:s0.numel()].view(s0.shape)
    state.copy_(s0)
    o = gdn2.gdn2_decode(*(t.to(DEV) for t in (q, k, v, g, b, w)), state)
    ex = [t.float().repeat_interleave(H // HK, dim=2) for t in (q, k, g, b)]
    s_ref = s0.clone()
    o_ref = orc.decode(ex[0], ex[1], v.float(), ex[2], ex[3], w.float(), s_ref)
    assert orc.rel_max_err(state.cpu(), s_ref) < 2e-5
    if dtype == torch.float32:
        assert orc.rel_max_err(o.cpu(), o_ref) < 2e-5
    else:
        assert orc.max_abs_err(o.float().cpu(), o_ref) < 2e-2
