"""Kernels that are launched as programmatic dependents wait for the kernel before them as the first thing they do."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "crosslayer_coding_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu"))


def _kernels(text):
    """``{name: first statement}`` of the ``__global__`` functions."""
    found = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        body = text[text.index("{", i) + 1:]
        found[m[1]] = body[: body.index(";") + 1].strip()
    return found


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_chained_kernels_wait_first(path):
    text = path.read_text()
    assert "<<<" not in text, "launch through launch_chained or launch_alone"
    kernels = _kernels(text)
    assert len(kernels) == len(re.findall(r"^.*__global__", text, flags=re.M)) - len(re.findall(r"^\s*//.*__global__", text, flags=re.M))
    chained = set(re.findall(r"launch_chained\((\w+)", text))
    alone = set(re.findall(r"launch_alone\((\w+)", text))
    for name in chained:
        assert kernels[name] == "if (chain_wait()) return;", name
    # a kernel that may run early is never taken for one that may not, and the other way round
    assert not chained & alone
    for name, first in kernels.items():
        assert (first == "if (chain_wait()) return;") == (name in chained), name
