"""The host extension is optional: where it cannot be built or loaded the package works through the general path."""

from __future__ import annotations

import subprocess
import sys

import pytest
import torch

from gdn2_tilelang_b200 import _cabi, build

NAME = "gdn2_tilelang_b200._gdn2_host"


@pytest.fixture(autouse=True)
def not_loaded(monkeypatch):
    monkeypatch.delitem(sys.modules, NAME, raising=False)


def test_it_loads():
    host = _cabi.load_host()
    assert host is not None and callable(host.decode) and _cabi.load_host() is host


def test_no_compiler(monkeypatch, tmp_path):
    def no_compiler(*args, **kw):
        raise FileNotFoundError("g++")

    monkeypatch.setattr(build, "host_lib", lambda: tmp_path / "_gdn2_host.none.so")
    monkeypatch.setattr(subprocess, "run", no_compiler)
    with pytest.warns(UserWarning, match="host extension"):
        K = _cabi.NativeKernels()
    assert K.host is None and K.lib.gdn2_abi_version() == 3
    monkeypatch.setattr(build, "_stale", lambda target, deps: target.name.startswith("_gdn2_host"))
    with pytest.warns(UserWarning, match="host extension"):
        assert build.build() == build.LIB                    # the kernels do not need it


def test_an_object_that_does_not_load(monkeypatch, tmp_path):
    bad = tmp_path / "_gdn2_host.bad.so"
    bad.write_bytes(b"built for something else")
    monkeypatch.setattr(build, "host_lib", lambda: bad)
    with pytest.warns(UserWarning, match="host extension"):
        assert _cabi.NativeKernels().host is None


def test_another_torch_is_another_object(monkeypatch):
    mine = build.host_lib()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert build.host_lib() != mine
