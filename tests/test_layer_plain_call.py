"""The layer's one-call decode steps aside for a layer that a program has customised: what ran when the output projection was
called as a module, or a stage as a method, still runs."""

from __future__ import annotations

import types

import pytest
import torch
from torch import nn

from gdn2_tilelang_b200 import _cabi, attention
from gdn2_tilelang_b200.config import GatedDeltaNet2Config
from tests.fake_kernels import OracleKernels


class Host:
    def __init__(self):
        self.calls = 0

    def parameter_key(self, params):
        return b""

    def decode(self, *args):
        return None

    def layer_decode(self, *args):
        self.calls += 1                                      # (None: not a plain call after all)


@pytest.fixture
def layer(monkeypatch):
    K = OracleKernels()
    K.host = Host()
    monkeypatch.setattr(_cabi, "_kernels", K)
    torch.manual_seed(0)
    net = attention.GatedDeltaNet2(GatedDeltaNet2Config(hidden_size=32, num_heads=2, head_dim_k=16))
    return net, K.host


def _instance_forward(net):
    inner = net.o_proj.forward
    net.o_proj.forward = types.MethodType(lambda self, x: inner(x) * 2, net.o_proj)
    return lambda: None


def _instance_stage(net):
    inner = net._project_out
    net._project_out = lambda normed: inner(normed) * 2
    return lambda: None


def _hook(net):
    return net.o_proj.register_forward_hook(lambda m, i, o: o * 2).remove


def _pre_hook(net):
    return net.o_proj.register_forward_pre_hook(lambda m, i: (i[0] * 2,)).remove


def _global_hook(net):
    return nn.modules.module.register_module_forward_hook(lambda m, i, o: o * 2 if m is net.o_proj else None).remove


def _global_pre_hook(net):
    return nn.modules.module.register_module_forward_pre_hook(lambda m, i: (i[0] * 2,) if m is net.o_proj else None).remove


@pytest.mark.parametrize("customise", [_instance_forward, _instance_stage, _hook, _pre_hook, _global_hook, _global_pre_hook])
def test_a_customised_output_projection_runs(layer, customise):
    net, host = layer
    x = torch.randn(2, 1, 32)
    plain = net.decode(x, net.init_cache(2))[0]
    assert host.calls == 1                                   # the plain layer is offered to the native call
    undo = customise(net)
    try:
        out = net.decode(x, net.init_cache(2))[0]
    finally:
        undo()
    assert host.calls == 1
    torch.testing.assert_close(out, 2 * plain)


def test_parameters_replaced_by_tensors(layer):
    """A program that computes a decay parameter and sets the tensor in the parameter's place takes the general path."""
    net, host = layer
    x = torch.randn(2, 1, 32)
    plain = net.decode(x, net.init_cache(2))[0]
    for name in ("A_log", "dt_bias"):
        value = getattr(net, name).detach().clone()
        delattr(net, name)
        setattr(net, name, value)
        for call in (net.decode, net.prefill):
            torch.testing.assert_close(call(x, net.init_cache(2))[0], plain)
        torch.testing.assert_close(net.step(x[:, 0], net.init_cache(2))[0], plain[:, 0])
    assert host.calls == 1
