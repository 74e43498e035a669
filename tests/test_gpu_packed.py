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
from tests.conftest import note
from tests.test_gpu_kernels import O_ABS_BF16, STATE_FRO, _guarded, _guards_intact

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


def _decays(g, offs, kind):
    """The inputs' ordinary decay made fast, absent or slow; "mixed" gives every sequence another one."""
    scale = {"fast": 30.0 * 16, "none": 0.0, "slow": 1 / 64, "usual": 1.0}
    g = g.clone()
    for i, (lo, hi) in enumerate(zip(offs, offs[1:])):
        g[:, lo:hi] *= scale[("fast", "none", "usual", "slow")[i % 4] if kind == "mixed" else kind]
    return g


@pytest.mark.parametrize("kind", ["mixed", "fast", "none", "slow"])
@pytest.mark.parametrize("H,HK,D,DV,dtype", [(4, 2, 128, 128, torch.bfloat16), (2, 1, 64, 40, torch.float32), (2, 2, 128, 128, torch.float16)])
def test_packed_against_the_oracle(H, HK, D, DV, dtype, kind):
    """Sequences whose scans are cut, with decays that flag chunks for the exact redo (fast: some chunks of the tensor-core
    family, in some sequences only), that let a segment's transition matrix vanish at once, and that keep it to the end.
    Bounds of the unpacked kernels' tests; without forgetting the cut's hand-over rounds to 4e-3 of the state, as in the
    test of the unpacked cut."""
    lens = [64 * 70 + 9, 64 * 41, 40, 64 * 24 + 63]
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    q, k, _, g, b, _ = orc.make_inputs(1, offs[-1], HK, D, D, seed=11)
    _, _, v, _, _, w = orc.make_inputs(1, offs[-1], H, D, DV, seed=12)
    g = _decays(g, offs, kind)
    q, k, v, b, w = (t.to(dtype) for t in (q, k, v, b, w))
    s0 = torch.randn(len(lens), H, D, DV, generator=torch.Generator().manual_seed(1)) * 0.1
    K = _cabi.kernels()
    if dtype == torch.bfloat16:
        cu = (_cabi.ctypes.c_int64 * len(offs))(*offs)
        assert K.lib.gdn2_packed_launches(cu, len(lens), H, HK, D, DV, _cabi.GDN2_BF16, 0) == 6      # the scan is cut
    o, s = gdn2.gdn2_attention(*(t.to(DEV) for t in (q, k, v, g, b, w)), initial_state=s0.to(DEV), output_final_state=True,
                               cu_seqlens=offs)
    K.check_device_status()
    o, s = o.cpu(), s.cpu()
    ex = [t.repeat_interleave(H // HK, dim=2) for t in (q, k, g, b)]
    for i, (lo, hi) in enumerate(zip(offs, offs[1:])):
        part = [t[:, lo:hi].double() for t in (ex[0], ex[1], v, ex[2], ex[3], w)]
        o_ref, s_ref = orc.recurrence(*part, initial_state=s0[i:i + 1], dtype=torch.float64)
        eo, es = orc.rel_fro_err(o[:, lo:hi], o_ref), orc.rel_fro_err(s[i:i + 1], s_ref)
        note("packed_against_the_oracle", dtype=str(dtype), kind=kind, seq=i, o=eo, s=es)
        if dtype == torch.float32:
            assert orc.rel_max_err(o[:, lo:hi], o_ref) < 2e-5 and orc.rel_max_err(s[i:i + 1], s_ref) < 2e-5, i
        elif dtype == torch.float16:
            assert orc.max_abs_err(o[:, lo:hi], o_ref) < O_ABS_BF16 / 8 and orc.rel_max_err(s[i:i + 1], s_ref) < 2e-5, i
        else:
            assert orc.max_abs_err(o[:, lo:hi], o_ref) < O_ABS_BF16 and es < (STATE_FRO if kind == "fast" else 4e-3), i


@pytest.mark.parametrize("lens,H,HK,D,dtype", [
    ([64 * 70 + 9, 0, 64 * 41, 5], 2, 1, 128, torch.bfloat16),      # a cut scan's segment records
    ([7, 64, 1], 3, 3, 128, torch.bfloat16),
    ([64 * 3 + 1, 63, 0, 70], 2, 1, 24, torch.float32),
    ([64 * 2 + 40], 2, 2, 64, torch.float16),
])
def test_packed_calls_stay_inside_their_buffers(lens, H, HK, D, dtype):
    """Guard bytes around a workspace of exactly the size asked for, the outputs and the states; and, in the exact family,
    around those of the unpacked call that takes its tail as one more chunk."""
    K = _cabi.kernels()
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    T, N, code = offs[-1], len(lens), _cabi.dtype_code(dtype)
    q, k, _, g, b, _ = orc.make_inputs(1, T, HK, D, D, seed=T)
    _, _, v, _, _, w = orc.make_inputs(1, T, H, D, D, seed=T + 1)
    ins = [t.to(DEV, dtype) for t in (q, k, v)] + [g.to(DEV)] + [t.to(DEV, dtype) for t in (b, w)]
    cu = (_cabi.ctypes.c_int64 * (N + 1))(*offs)
    st = torch.cuda.current_stream().cuda_stream
    nbytes = K.lib.gdn2_packed_workspace_bytes(cu, N, H, HK, D, D, code, 0)
    bufs = [_guarded((nbytes,), torch.uint8), _guarded((1, T, H, D), dtype), _guarded((N, H, D, D), torch.float32)]
    rc = K.lib.gdn2_packed_forward(*(t.data_ptr() for t in ins), cu, N, None, bufs[1][1].data_ptr(), bufs[2][1].data_ptr(),
                                   bufs[0][1].data_ptr(), nbytes, H, HK, D, D, D**-0.5, code, 0, st)
    assert rc == 0
    assert K.lib.gdn2_packed_forward(*(t.data_ptr() for t in ins), cu, N, None, bufs[1][1].data_ptr(), bufs[2][1].data_ptr(),
                                     bufs[0][1].data_ptr(), nbytes - 1024, H, HK, D, D, D**-0.5, code, 0, st) == -5
    torch.cuda.synchronize()
    assert all(_guards_intact(buf, gd) for buf, _, gd in bufs)
    assert torch.isfinite(bufs[1][1].float()).all() and torch.isfinite(bufs[2][1]).all()
    if dtype != torch.bfloat16 and T >= 64:
        nbytes = K.lib.gdn2_prefill_ragged_workspace_bytes(1, T, H, HK, D, D, code, 0)
        bufs = [_guarded((nbytes,), torch.uint8), _guarded((1, T, H, D), dtype), _guarded((1, H, D, D), torch.float32)]
        rc = K.lib.gdn2_prefill_ragged(*(t.data_ptr() for t in ins), None, bufs[1][1].data_ptr(), bufs[2][1].data_ptr(),
                                       bufs[0][1].data_ptr(), nbytes, 1, T, H, HK, D, D, T, T, D**-0.5, code, 0, None, st)
        torch.cuda.synchronize()
        assert rc == 0 and all(_guards_intact(buf, gd) for buf, _, gd in bufs)
    K.check_device_status()
