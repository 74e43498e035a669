"""Packed sequences in one launch per stage against the same sequences evaluated one call each: sequences shorter than a
chunk, empty ones, more than one table of them, shared key heads, both kernel families, strided inputs and scans that are
cut into segments.

Tolerance: the kernels are the same, so a sequence whose scan is cut alike gives the same bits; where the cut differs,
or a tail is decoded by another kernel, float32 sums are taken in another order (2e-5 of the largest value in float32)
and a bf16 output may round the other way (one step of 2^-8 of a value of a few, against the 2e-2 bound of the bf16
tests); states stay within that bound's 1e-3."""

from __future__ import annotations

import pytest
import torch

import gdn2_tilelang_b200 as gdn2
from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENGTHS = {
    "short": [5, 1, 63, 0, 17, 3],                 # no whole chunk anywhere
    "mixed": [64 * 9 + 5, 0, 64, 130, 1, 64 * 3],
    "long": [64 * 70 + 9, 64 * 2, 64 * 41],        # scans cut into segments
    "many": [(i * 37) % 150 for i in range(131)],  # more than one table holds
}


@pytest.mark.parametrize("name", sorted(LENGTHS))
@pytest.mark.parametrize("H,HK,DK,DV,dtype", [
    (2, 2, 128, 128, torch.bfloat16), (4, 2, 128, 128, torch.bfloat16), (2, 1, 64, 64, torch.float32),
    (3, 3, 32, 40, torch.float16), (2, 2, 128, 128, torch.float16)])
@pytest.mark.parametrize("with_state", [False, True])
def test_packed_equals_one_call_per_sequence(name, H, HK, DK, DV, dtype, with_state):
    lens = LENGTHS[name]
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    T = offs[-1]
    q, k, _, g, b, _ = orc.make_inputs(1, T, HK, DK, DV, seed=T)
    _, _, v, _, _, w = orc.make_inputs(1, T, H, DK, DV, seed=T + 1)
    q, k, v, b, w = (t.to(DEV, dtype) for t in (q, k, v, b, w))
    g = g.to(DEV)
    s0 = torch.randn(len(lens), H, DK, DV, generator=torch.Generator().manual_seed(1)).mul_(0.1).to(DEV) if with_state else None
    o, s = gdn2.gdn2_attention(q, k, v, g, b, w, initial_state=s0, output_final_state=True, cu_seqlens=offs)
    _cabi.kernels().check_device_status()
    # the same from strided tensors and a tensor of offsets, without the final state
    wide = torch.cat([q, q], -1)[..., :DK]
    o2, none = gdn2.gdn2_attention(wide, k, v, g, b, w, initial_state=s0, cu_seqlens=torch.tensor(offs))
    assert none is None and torch.equal(o, o2)
    for i, (lo, hi) in enumerate(zip(offs, offs[1:])):
        one = s0[i:i + 1] if with_state else None
        if hi == lo:
            assert torch.equal(s[i], s0[i]) if with_state else not s[i].any()
            continue
        if name == "many" and i % 10:
            continue
        o1, s1 = gdn2.gdn2_attention(*(t[:, lo:hi].contiguous() for t in (q, k, v, g, b, w)), initial_state=one,
                                     output_final_state=True)
        if dtype == torch.float32:
            assert orc.rel_max_err(o[:, lo:hi].cpu(), o1.cpu()) < 2e-5 and orc.rel_max_err(s[i:i + 1].cpu(), s1.cpu()) < 2e-5
        else:
            assert orc.max_abs_err(o[:, lo:hi].float().cpu(), o1.float().cpu()) < 2e-2, i
            assert orc.rel_fro_err(s[i:i + 1].cpu(), s1.cpu()) < 1e-3, i
    _cabi.kernels().check_device_status()


@pytest.mark.parametrize("H,D,DV,dtype,lens", [
    (64, 128, 128, torch.bfloat16, [64 * 70 + 9, 64 * 61, 0, 130, 64 * 2]),     # the second sequence opens a new group
    (128, 8, 4, torch.float32, [64 * 30 + 1, 64 * 34, 70, 5]),                  # the third does
    (70, 8, 4, torch.float32, [10, 64 * 118, 3]),                               # a sequence beyond the bound by itself
])
def test_groups_that_share_a_workspace(H, D, DV, dtype, lens):
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    gen = torch.Generator(device=DEV).manual_seed(3)
    q, k = (torch.nn.functional.normalize(torch.randn(1, offs[-1], H, D, generator=gen, device=DEV), dim=-1).to(dtype) for _ in "qk")
    v, w = (torch.randn(1, offs[-1], H, DV, generator=gen, device=DEV).to(dtype) for _ in "vw")
    g = torch.nn.functional.logsigmoid(torch.randn(1, offs[-1], H, D, generator=gen, device=DEV)) / 16
    b = torch.sigmoid(torch.randn(1, offs[-1], H, D, generator=gen, device=DEV)).to(dtype)
    w = torch.sigmoid(w)
    s0 = torch.randn(len(lens), H, D, DV, generator=gen, device=DEV) * 0.1
    o, s = gdn2.gdn2_attention(q, k, v, g, b, w, initial_state=s0, output_final_state=True, cu_seqlens=offs)
    _cabi.kernels().check_device_status()
    for i, (lo, hi) in enumerate(zip(offs, offs[1:])):
        if hi == lo:
            assert torch.equal(s[i], s0[i])
            continue
        o1, s1 = gdn2.gdn2_attention(*(t[:, lo:hi] for t in (q, k, v, g, b, w)), initial_state=s0[i:i + 1], output_final_state=True)
        tol = 2e-5 if dtype == torch.float32 else 1e-2
        assert orc.rel_fro_err(o[:, lo:hi].cpu(), o1.cpu()) < tol and orc.rel_fro_err(s[i:i + 1].cpu(), s1.cpu()) < min(tol, 1e-3)
    _cabi.kernels().check_device_status()
