"""Decode with gates that wipe a channel, among ordinary ones: the blocked form, which takes up to eight tokens at a time, keeps what
the token-by-token recurrence keeps. Both sides sum a few hundred float32 terms, 2e-7 of the outputs' norm; 1e-6 leaves room for
the order. (With differences of prefix sums a gate of -1e6 costs 1e-2 and -inf gives NaN.)"""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("gate", [-20.0, -100.0, -1e4, -1e6, -1e30, float("-inf")])
@pytest.mark.parametrize("n,D", [(1, 128), (3, 128), (4, 128), (8, 128), (21, 128), (8, 64), (9, 48)])
def test_strong_gates(n, D, gate):
    B, H = 2, 2
    q, k, v, g, b, w = orc.make_inputs(B, n, H, D, D, seed=n)
    g[0, 1::5] = gate
    g[1, 2::3, :, ::3] = gate
    g[:, 3::4, :, 1::2] = gate
    s0 = golden_state(B, H, D, D, n, 0.3)
    state = s0.to(DEV)
    o = gdn2.gdn2_decode(*(t.to(DEV) for t in (q, k, v, g, b, w)), state)
    _cabi.kernels().check_device_status()
    o_ref, s_ref = orc.recurrence(q, k, v, g, b, w, initial_state=s0, dtype=torch.float64)
    assert orc.rel_fro_err(o.cpu(), o_ref) < 1e-6 and orc.rel_fro_err(state.cpu(), s_ref) < 1e-6


@pytest.mark.parametrize("gate", [-20.0, -1e6, float("-inf")])
@pytest.mark.parametrize("n", [2, 3, 4, 6, 12, 16, 21])
def test_strong_gates_in_every_step_size(n, gate):
    """Steps of 4, 6 and 8 tokens, one and several of them, and the sweeps of two and three; more tiles than the GPU has SMs, so
    that the tables of the next tile are built while this one is worked on."""
    B, H, HK, D = 54, 3, 1, 128
    q, k, _, g, b, _ = orc.make_inputs(B, n, HK, D, D, seed=n)
    _, _, v, _, _, w = orc.make_inputs(B, n, H, D, D, seed=n + 1)
    g[::2, 1::5] = gate
    g[1::2, 0::3, :, ::3] = gate
    g[:, 3::4, :, 1::2] = gate
    s0 = golden_state(B, H, D, D, n, 0.3)
    state = s0.to(DEV)
    o = gdn2.gdn2_decode(*(t.to(DEV) for t in (q, k, v, g, b, w)), state)
    _cabi.kernels().check_device_status()
    q, k, g, b = (t.repeat_interleave(H, 2) for t in (q, k, g, b))
    o_ref, s_ref = orc.recurrence(q, k, v, g, b, w, initial_state=s0, dtype=torch.float64)
    assert orc.rel_fro_err(o.cpu(), o_ref) < 1e-6 and orc.rel_fro_err(state.cpu(), s_ref) < 1e-6


@pytest.mark.parametrize("gate", [-1e6, float("-inf")])
def test_tail_of_a_tensor_core_prefill(gate):
    """bf16: chunks with such gates are redone exactly, the tail is decoded."""
    B, S, H, D = 1, 64 * 3 + 21, 2, 128
    q, k, v, g, b, w = orc.make_inputs(B, S, H, D, D, seed=4)
    g[:, 5::17] = gate
    g[:, 64 * 3 + 2::6, :, ::2] = gate
    low = [t.bfloat16() for t in (q, k, v)] + [g] + [t.bfloat16() for t in (b, w)]
    o, s = gdn2.gdn2_prefill(*(t.to(DEV) for t in low))
    _cabi.kernels().check_device_status()
    o_ref, s_ref = orc.recurrence(*low, dtype=torch.float64)
    assert orc.rel_fro_err(o.cpu(), o_ref) < 1e-2 and orc.rel_fro_err(s.cpu(), s_ref) < 1e-3
