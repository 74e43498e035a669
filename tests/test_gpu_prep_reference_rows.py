"""The chunk-local stage scales the rows of every sub-block of 16 tokens by their decay to its row 8. On that row the factors are 1
and the bf16 operands are the inputs themselves, so the diagonal entries of the pair matrix there carry one rounding, the record's own."""

from __future__ import annotations

import pytest
import torch

from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.ws_records import decode_tc_workspace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decay_scale", [0.05, 1.0, 4.0])
def test_reference_rows_are_not_rounded(decay_scale):
    B, S, H, D = 1, 256, 2, 128
    q, k, v, g, b, w = orc.make_inputs(B, S, H, D, D, seed=5, decay_scale=decay_scale)
    dev = [t.bfloat16().to("cuda") for t in (q, k, v)] + [g.to("cuda")] + [t.bfloat16().to("cuda") for t in (b, w)]
    K = _cabi.kernels()
    ws, path = K.chunk_prep(*dev, D**-0.5, path="tcgen05")
    rec = decode_tc_workspace(ws, K.workspace_layout(B, S, H, D, D, torch.bfloat16, path), B, S, H)
    assert int(rec["flags"].sum()) == 0
    rows = torch.tensor([8, 24, 40, 56])
    got = rec["Aqk"][..., rows, rows].double()                              # [B, H, chunks, 4]
    exact = (q.bfloat16().double() * k.bfloat16().double()).sum(-1) * D**-0.5
    exact = exact.reshape(B, S // 64, 64, H).permute(0, 3, 1, 2)[..., rows]
    # half a unit of the fp16 record, and fp32 sums of 128 products of at most 1 in all, times the scale
    assert ((got - exact).abs() <= 2.0**-11 * exact.abs() + 128 * 2.0**-24 * D**-0.5).all()
