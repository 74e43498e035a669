"""The chunk-local stage's factorisation by sub-blocks of 16 tokens and its exact redo, on both sides of the line between them: a chunk
goes by sub-blocks while no 8 tokens decay by 2^96 in any channel, else to the exact kernel. One channel over the line is enough, and
chunks of one launch take different ways. The gates around -4 a token, 2^96 in 16 tokens, are well inside."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,HK", [(2, 2), (4, 2)])
@pytest.mark.parametrize("gate", [-3.9, -4.1, -4.3, -8.1, -8.4, -12.0])      # 2^96 lies at 66.5: -8.3 a token over 8
@pytest.mark.parametrize("where", ["all", "one_channel", "second_chunk", "half_block"])
def test_decays_around_the_lines(gate, where, H, HK):
    B, S, D = 1, 192, 128
    q, k, _, g, b, _ = orc.make_inputs(B, S, HK, D, D, seed=7)
    _, _, v, _, _, w = orc.make_inputs(B, S, H, D, D, seed=8)
    if where == "all":
        g = torch.full_like(g, gate)
    elif where == "one_channel":
        g[..., 77] = gate
    elif where == "second_chunk":
        g[:, 64:128] = gate
    else:                                                  # sixteen tokens that are the second half of a block of 32
        g[:, 80:96, :, ::2] = gate
    low = [t.bfloat16() for t in (q, k, v)] + [g] + [t.bfloat16() for t in (b, w)]
    s0 = golden_state(B, H, D, D, 3, 0.3)
    o, s = gdn2.gdn2_prefill(*(t.to(DEV) for t in low), s0.to(DEV))
    _cabi.kernels().check_device_status()
    rep = [t.repeat_interleave(H // HK, 2) if t.shape[2] == HK else t for t in low]
    o_ref, s_ref = orc.recurrence(*rep, initial_state=s0, dtype=torch.float64)
    assert torch.isfinite(o).all() and torch.isfinite(s).all()
    # the erase and query operands are bf16 (3e-3 of the outputs' norm), the states carry eleven bits (1e-3)
    assert orc.rel_fro_err(o.cpu(), o_ref) < 1e-2 and orc.rel_fro_err(s.cpu(), s_ref) < 2e-3
