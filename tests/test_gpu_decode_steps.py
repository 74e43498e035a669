"""The blocked decode's steps of 4, 6 and 8 tokens: every number of tokens around them, full and padded last steps, with more (sequence,
head) tiles than the GPU has SMs, so that a block walks two or three of them; and the token-by-token sweeps of 2 and 3 there."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,HK", [(24, 16, 8), (50, 3, 1)])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 9, 12, 13, 18, 37])
def test_steps(n, B, H, HK, dtype):
    D = 128
    q, k, _, g, b, _ = orc.make_inputs(B, n, HK, D, D, seed=n)
    _, _, v, _, _, w = orc.make_inputs(B, n, H, D, D, seed=n + 1)
    q, k, v, b, w = (t.to(dtype) for t in (q, k, v, b, w))
    s0 = golden_state(B, H, D, D, n, 0.3)
    state = s0.to(DEV)
    # tokens of a longer row: the batch stride is not n
    wide = [torch.cat([t, t], 1).to(DEV)[:, :n] for t in (q, k, v, g, b, w)]
    o = gdn2.gdn2_decode(*wide, state)
    _cabi.kernels().check_device_status()
    rep = [t.double().repeat_interleave(H // HK, 2) for t in (q, k, g, b)]
    o_ref, s_ref = orc.recurrence(rep[0], rep[1], v.double(), rep[2], rep[3], w.double(), initial_state=s0.double(), dtype=torch.float64)
    # float32 sums of some hundred terms; the outputs rounded to the storage type
    tol = {torch.float32: 1e-6, torch.bfloat16: 3e-3, torch.float16: 4e-4}[dtype]
    assert orc.rel_fro_err(o.cpu().double(), o_ref) < tol
    assert orc.rel_fro_err(state.cpu().double(), s_ref) < 1e-6
