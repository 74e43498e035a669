"""Every bounded wait of the kernels has its result looked at, and whole-warp code waits as a warp.

A wait that ran out must lead out of the code that depends on it: tensor memory that a product may still be writing is not
read, and lanes that leave a wait by different exits do not go straight on to warp-collective instructions."""

from __future__ import annotations

import pathlib
import re

import pytest

SOURCES = sorted((pathlib.Path(__file__).resolve().parents[1] / "gdn2_tilelang_b200" / "csrc").glob("*.cu*"))
WAIT = re.compile(r"\b(?:tc::)?(mbar_wait(?:_warp|_limit|_relaxed)?)\s*\(")


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_wait_is_ignored(path):
    code = _code(path)
    for m in WAIT.finditer(code):
        before = code[:m.start()].rstrip()
        line = code.count("\n", 0, m.start()) + 1
        # a call that is a statement of its own follows a separator, a closing parenthesis of an if / for, or an else
        dropped = before.endswith((";", "{", "}", ":")) or before.endswith("else")
        if before.endswith(")"):
            depth, i = 0, len(before) - 1
            while i >= 0:
                depth += {")": 1, "(": -1}.get(before[i], 0)
                if depth == 0:
                    break
                i -= 1
            dropped = re.search(r"\b(if|for|while)\s*$", before[:i]) is not None
        assert not dropped, f"{path.name}:{line}: the result of {m.group(1)} is ignored"


@pytest.mark.parametrize("name", ["scan_tc.cu", "prep_tc.cu", "scan_simt.cu"])
def test_warps_wait_together(name):
    """Per-lane waits are left to the one copying thread of the tensor-core scan."""
    code = _code(next(p for p in SOURCES if p.name == name))
    lanes = [m for m in WAIT.finditer(code) if m.group(1) == "mbar_wait"]
    copying = code.find("if (lane == 0) {\n      auto load_wq"), code.find("} else if (wid == 8)")
    assert all(copying[0] < m.start() < copying[1] for m in lanes)
