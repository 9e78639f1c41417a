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


def _bodies(text):
    """``{name: body}`` of the ``__global__`` functions, without comments."""
    text = re.sub(r"//[^\n]*", "", text)
    found = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        start = i = text.index("{", i) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        found[m[1]] = text[start: i - 1]
    return found


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_kernels_that_wait_for_another_rank_hold_their_successors(path):
    """A chained kernel releases the next one as its second statement, except with several ranks when it polls a peer's flag: CTAs that came early would
    hold the SMs until the peer arrives."""
    for name, body in _bodies(path.read_text()).items():
        head = [s.strip() for s in body.split(";")[:2]]
        releases = body.count("chain_release()")
        polls = re.search(r"exchange_gather\(|exchange_sum\(|ld_acquire_sys", body) is not None
        if head[0] != "if (chain_wait()) return":
            assert releases == 0, name
        elif not polls:
            assert releases == 1 and head[1] == "chain_release()", name
        else:
            assert releases == 0 or (releases == 1 and re.fullmatch(r"if \((p\.)?ex\.world <= 1\) chain_release\(\)", head[1])), name


def test_the_kernels_that_poll_are_known():
    polling = {n for p in SOURCES for n, b in _bodies(p.read_text()).items() if re.search(r"exchange_gather\(|exchange_sum\(|ld_acquire_sys", b)}
    assert polling == {"peer_barrier_kernel", "find_bin_kernel", "refine_kernel", "step_control_kernel"}
    # the wait alone does not release anything
    wait = (CSRC / "common.cuh").read_text().split("bool chain_wait()")[1].split("\n}")[0]
    assert "griddepcontrol.wait" in wait and "launch_dependents" not in wait


def test_rules_on_resident_ctas_ask_the_device():
    """What is launched early, and which decodes are taken in slices, depends on the SMs of the device at hand, not on those of one product."""
    common, decode = ((CSRC / n).read_text() for n in ("common.cuh", "decode.cu"))
    assert "kChainedCtasPerSm * device_sms()" in common and "kSliceCtasPerSm * device_sms()" in decode
    rules = common.split("inline cudaError_t launch_chained")[1].split("\n}")[0] + decode.split("static bool takes_slices")[1].split("\n}")[0]
    assert not re.search(r"\b(148|592|1184)\b", rules)
