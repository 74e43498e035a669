"""``GatedDeltaNet2.step`` called with gradients enabled leaves no graph behind: the weight tables that the layer keeps can be copied
with it, and whatever ``decode`` a program has put in place of the layer's own runs without gradients, as it does through ``decode``."""

from __future__ import annotations

import copy

import pytest
import torch

from gdn2_tilelang_b200 import _cabi, attention
from gdn2_tilelang_b200.config import GatedDeltaNet2Config
from tests.fake_kernels import OracleKernels


class Replaced(attention.GatedDeltaNet2):
    def decode(self, hidden_states, cache):
        self.grad_mode = torch.is_grad_enabled()
        return self.o_proj.weight.sum() * hidden_states, cache


@pytest.fixture
def kernels(monkeypatch):
    K = OracleKernels()
    K.layer_step = lambda *args: None                        # offered the call with the layer's tables, declines
    monkeypatch.setattr(_cabi, "_kernels", K)
    return K


def _layer(cls=attention.GatedDeltaNet2):
    torch.manual_seed(0)
    return cls(GatedDeltaNet2Config(hidden_size=32, num_heads=2, head_dim_k=16))


@pytest.mark.parametrize("change", [False, True])
def test_the_kept_tables_have_no_graph(kernels, change):
    net = _layer()
    x = torch.randn(2, 32)
    if change:                                               # built without gradients once, then again by a step
        net.decode(x.unsqueeze(1), net.init_cache(2))
        with torch.no_grad():
            net.q_proj.weight.mul_(1.5)
    y, _ = net.step(x, net.init_cache(2))
    w_cat, _, conv_w, conv_b = net._fused
    assert not any(t.requires_grad for t in (y, w_cat, conv_w, conv_b))
    assert torch.equal(w_cat[: net.q_proj.weight.shape[0]], net.q_proj.weight)
    other = copy.deepcopy(net)
    torch.testing.assert_close(other.step(x, other.init_cache(2))[0], y)


def test_a_replaced_decode_runs_without_gradients(kernels):
    net = _layer(Replaced)
    y, _ = net.step(torch.randn(2, 32, requires_grad=True), net.init_cache(2))
    assert not net.grad_mode and not y.requires_grad
    net = _layer()
    net.decode = lambda x, cache: (net.o_proj(torch.zeros(2, 1, 32)) + x, cache)
    y, _ = net.step(torch.randn(2, 32, requires_grad=True), net.init_cache(2))
    assert not y.requires_grad
