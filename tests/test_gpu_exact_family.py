"""The exact (CUDA-core) chunkwise family at the edges of its tiles: head sizes around the eight-lane channel split and
the value tiles of the scan, ragged tails taken as one more chunk, shared key heads, fast decay and every tile width.

Tolerance: both sides are float32 sums of at most a few hundred terms in different orders, so they differ by some
sqrt(256) * 2^-24 = 1e-6 of the largest value; the bound of the reference's own float32 tests, 2e-5, covers that."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,S,H,HK,DK,DV,decay", [
    (2, 65, 3, 3, 64, 64, 1.0),        # a tail of one token
    (1, 191, 2, 1, 8, 4, 1.0),         # the smallest head, shared key head, a tail of 63
    (1, 64 * 5 + 37, 4, 2, 24, 100, 1.0),    # channel and value counts that no tile divides
    (1, 130, 2, 2, 128, 36, 40.0),     # two channels per thread, fast decay
    (2, 200, 10, 10, 64, 128, 8.0),    # 16 value columns per block
    (3, 100, 37, 37, 16, 96, 1.0),     # 32 value columns per block
])
def test_ragged_lengths_float32(B, S, H, HK, DK, DV, decay):
    q, k, _, g, b, _ = orc.make_inputs(B, S, HK, DK, DV, seed=S, gate="softplus", decay_scale=decay)
    _, _, v, _, _, w = orc.make_inputs(B, S, H, DK, DV, seed=S + 1, gate="softplus")
    s0 = golden_state(B, H, DK, DV, S, 0.3)
    o, s = gdn2.gdn2_attention(*(t.to(DEV) for t in (q, k, v, g, b, w)), initial_state=s0.to(DEV), output_final_state=True)
    _cabi.kernels().check_device_status()
    ex = [t.repeat_interleave(H // HK, dim=2) for t in (q, k, g, b)]
    s_ref = s0.clone()
    o_ref = orc.decode(ex[0], ex[1], v, ex[2], ex[3], w, s_ref)
    assert torch.isfinite(o).all()
    assert orc.rel_max_err(o.cpu(), o_ref) < 2e-5
    assert orc.rel_max_err(s.cpu(), s_ref) < 2e-5


def test_workspace_for_whole_chunks_keeps_the_decoded_tail():
    """A caller that sized the workspace for the whole chunks only gets the tail decoded, with the same results."""
    K = _cabi.kernels()
    B, S, H, D = 1, 150, 2, 64
    ins = [t.to(DEV) for t in orc.make_inputs(B, S, H, D, D, seed=3)]
    code = _cabi.dtype_code(torch.float32)
    res = []
    for nbytes in (K.lib.gdn2_prefill_workspace_bytes(B, 128, H, H, D, D, code, _cabi.PATH_SIMT),
                   K.lib.gdn2_prefill_ragged_workspace_bytes(B, S, H, H, D, D, code, _cabi.PATH_SIMT)):
        ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        o, s = torch.empty_like(ins[2]), torch.empty(B, H, D, D, device=DEV)
        rc = K.lib.gdn2_prefill_ragged(*(t.data_ptr() for t in ins), None, o.data_ptr(), s.data_ptr(), ws.data_ptr(), nbytes,
                                       B, S, H, H, D, D, S, S, D**-0.5, code, _cabi.PATH_SIMT, None,
                                       torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        res.append((o.cpu(), s.cpu()))
    assert orc.rel_max_err(res[0][0], res[1][0]) < 2e-5 and orc.rel_max_err(res[0][1], res[1][1]) < 2e-5


@pytest.mark.parametrize("gate", [None, -20.0, -100.0, -1e4, -1e6, -1e30, float("-inf")])
@pytest.mark.parametrize("form", ["tail", "packed", "whole"])
def test_strong_gates_keep_the_ones_after_them(gate, form):
    """A gate that wipes a channel must not cost the later, ordinary ones any digits: the recurrence forms every decay by
    itself. Against it in 64 bits the float32 outputs are sums of a few hundred rounded terms, 1.6e-7 of their norm when
    evaluated token by token; 1e-6 leaves room for another order and is below what prefix sums lose from -100 on (5e-6)."""
    D, H = 64, 2
    lengths = {"tail": [64 + 40], "packed": [40, 3, 64, 41], "whole": [128]}[form]
    T = sum(lengths)
    q, k, v, g, b, w = orc.make_inputs(1, T, H, D, D, seed=5)
    if gate is not None:                                    # whole tokens, single channels, neighbours inside a group of four
        g[:, 9::31] = gate
        g[:, 10::37, :, ::3] = gate
        g[:, 17::29, :, 1::2] = gate
    s0 = golden_state(len(lengths), H, D, D, 1, 0.3)
    dev = [t.to(DEV) for t in (q, k, v, g, b, w)]
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    o, s = gdn2.gdn2_attention(*dev, initial_state=s0.to(DEV), output_final_state=True,
                               **({"cu_seqlens": cu} if form == "packed" else {}))
    _cabi.kernels().check_device_status()
    for i, n in enumerate(lengths):
        part = [t[:, cu[i]:cu[i + 1]] for t in (q, k, v, g, b, w)]
        o_ref, s_ref = orc.recurrence(*part, initial_state=s0[i:i + 1], dtype=torch.float64)
        assert orc.rel_fro_err(o[:, cu[i]:cu[i + 1]].cpu(), o_ref) < 1e-6
        assert orc.rel_fro_err(s[i:i + 1].cpu(), s_ref) < 1e-6
