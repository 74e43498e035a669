"""The exact family's scan in tiles of four rows by four columns over quarters of the reduction: value tiles of 8, 16 and 32 columns,
head sizes that are no multiple of the 32 rows of a warp or of the 16 steps of a quarter round, one, two, three and odd numbers of
chunks, and a ragged tail."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,H,DK,DV", [(1, 2, 64, 64), (5, 8, 64, 64), (1, 2, 128, 128), (10, 4, 128, 128), (1, 3, 128, 20), (2, 2, 32, 72),
                                       (1, 2, 8, 4), (2, 3, 40, 12), (1, 1, 96, 36), (16, 8, 24, 40)])
@pytest.mark.parametrize("S", [64, 128, 192 + 5, 5 * 64 + 63])
def test_attention_f32(B, H, DK, DV, S):
    ins = orc.make_inputs(B, S, H, DK, DV, seed=S + DK)
    s0 = golden_state(B, H, DK, DV, 3, 0.3)
    o, s = gdn2.gdn2_attention(*(t.to(DEV) for t in ins), initial_state=s0.to(DEV), output_final_state=True)
    _cabi.kernels().check_device_status()
    o_ref, s_ref = orc.recurrence(*ins, initial_state=s0, dtype=torch.float64)
    # float32 sums and a substitution over 64 rows: a few 1e-7 of the norm (measured 3e-7 on the timed case)
    assert orc.rel_fro_err(o.cpu(), o_ref) < 2e-6 and orc.rel_fro_err(s.cpu(), s_ref) < 2e-6
