"""The states entering every chunk from a scan that is cut into segments, against the one-block walk of the same problem.

Tolerances are those of the cut scan's own test: the two forms differ by the rounding of the state hand-over, and without
decay nothing forgets it (1e-3 and 4e-3 of the states' norm, outputs within the 2e-2 of the bf16 tests)."""

from __future__ import annotations

import pytest
import torch

from gdn2_tilelang_b200 import _cabi
from oracle import gdn2_oracle as orc
from tests.conftest import golden_state, note

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,H,HK,NC,decay", [(1, 2, 1, 40, 1.0), (2, 16, 16, 64, 1.0), (2, 16, 16, 64, 0.0), (1, 1, 1, 130, 1 / 64)])
def test_chunk_states_of_a_cut_scan(B, H, HK, NC, decay):
    K = _cabi.kernels()
    S, D = 64 * NC, 128
    q, k, _, g, b, _ = orc.make_inputs(B, S, HK, D, D, seed=NC)
    _, _, v, _, _, w = orc.make_inputs(B, S, H, D, D, seed=NC + 1)
    dev = [t.bfloat16().to(DEV) for t in (q, k, v)] + [(g * decay).to(DEV)] + [t.bfloat16().to(DEV) for t in (b, w)]
    s0 = golden_state(B, H, D, D, NC, 0.1).to(DEV)
    assert K.scan_segments(B, S, H, D, D, torch.bfloat16, _cabi.PATH_TCGEN05) > 1
    o, s, h = K.chunk_forward(*dev, D**-0.5, s0, want_chunk_states=True, path="tcgen05")
    o1, s1, h1 = K.chunk_forward(*dev, D**-0.5, s0, want_chunk_states=True, path="tcgen05_serial")
    K.check_device_status()
    tol = 1e-3 if decay == 1.0 else 4e-3
    assert torch.equal(h[:, 0], s0)
    assert orc.max_abs_err(o.float(), o1.float()) < 2e-2
    assert orc.rel_fro_err(s, s1) < tol
    for n in range(NC):                                   # chunk by chunk: one stale record must not hide in the norm of all
        assert orc.rel_fro_err(h[:, n], h1[:, n]) < tol, n


@pytest.mark.parametrize("decay", [16.0, 1.0, 1 / 8, 1 / 64, 0.0])
def test_chunk_states_against_the_recurrence(decay):
    """Both forms against 64-bit arithmetic: the cut may not cost precision. The operands of the products are 16-bit, so
    either form is off by 6e-4 of the states' norm with the usual decay and by 1.7e-3 where nothing is forgotten; a cut's
    errors are other ones, not larger ones."""
    K = _cabi.kernels()
    B, H, NC, D = 1, 2, 40, 128
    S = 64 * NC
    q, k, v, g, b, w = orc.make_inputs(B, S, H, D, D, seed=NC)
    low = [t.bfloat16() for t in (q, k, v)] + [g * decay] + [t.bfloat16() for t in (b, w)]
    s0 = golden_state(B, H, D, D, NC, 0.1)
    state, h_ref = s0, []
    for n in range(NC):
        h_ref.append(state)
        _, state = orc.recurrence(*(t[:, 64 * n:64 * n + 64] for t in low), initial_state=state, dtype=torch.float64)
    h_ref = torch.stack(h_ref, 1)
    dev = [t.to(DEV) for t in low]
    assert K.scan_segments(B, S, H, D, D, torch.bfloat16, _cabi.PATH_TCGEN05) > 1
    err = {}
    for path in ("tcgen05", "tcgen05_serial"):
        _, s, h = K.chunk_forward(*dev, D**-0.5, s0.to(DEV), want_chunk_states=True, path=path)
        K.check_device_status()
        err[path] = [orc.rel_fro_err(h.cpu(), h_ref), max(orc.rel_fro_err(h[:, n].cpu(), h_ref[:, n]) for n in range(NC)),
                     orc.rel_fro_err(s.cpu(), state)]
    note("chunk_states_against_the_recurrence", decay=decay, cut=str(err["tcgen05"]), walk=str(err["tcgen05_serial"]))
    tol = 1e-3 if decay >= 1.0 else 4e-3
    assert max(err["tcgen05"]) < tol and max(err["tcgen05_serial"]) < tol
    assert all(c < 1.2 * w1 + 1e-6 for c, w1 in zip(err["tcgen05"], err["tcgen05_serial"]))
