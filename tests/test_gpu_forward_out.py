"""``chunk_gdn2_fwd`` into a caller's output: the stages composed in Python, the ragged tail on a second stream beside the
correction pass where the scan is cut. The kernels are those of the one-call form, so the results are the same bits."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,S,H", [
    (1, 64 * 40 + 13, 2),         # cut scan, tail on the second stream
    (1, 64 * 40, 2),              # ... without a tail
    (2, 64 * 3 + 5, 40),          # one walk per head, tail after it
    (1, 63, 2),                   # a tail alone
])
def test_output_tensor_of_the_caller(B, S, H):
    D = 128
    ins = [t.to(DEV) for t in orc.make_inputs(B, S, H, D, D, seed=S, dtype=torch.bfloat16)]
    ref = gdn2.chunk_gdn2_fwd(*ins, D**-0.5, output_final_state=True)
    wide = torch.full((B, S + 9, H, D), 7.0, device=DEV, dtype=torch.bfloat16)
    o, s = gdn2.chunk_gdn2_fwd(*ins, D**-0.5, output_final_state=True, out=wide[:, :S])
    _cabi.kernels().check_device_status()
    assert torch.equal(o, ref[0]) and torch.equal(s, ref[1])
    assert (wide[:, S:] == 7.0).all()
    o_ref, s_ref = orc.recurrence(*(t.cpu() for t in ins))
    assert orc.rel_fro_err(o.cpu(), o_ref) < 1e-2 and orc.rel_fro_err(s.cpu(), s_ref) < 1e-2
