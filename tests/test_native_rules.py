"""Host-side rules of the native library, which need no GPU: sizes at which a call takes another form or is refused."""
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def ext():
    from crosslayer_coding_b200.ops import ext as ext_mod

    return ext_mod.load()  # built here where it is missing


@pytest.mark.parametrize("k", [0, -1, -(1 << 40), 64])
def test_scratch_of_the_token_topk_for_any_count(ext, k):
    """A count that is not positive is left to the refusal that follows; in a child process, which a failure would end."""
    code = ("from crosslayer_coding_b200.ops import ext\nm = ext.load()\n"
            f"print([m.token_topk_scratch(6, 2048, F, {k}) for F in (8192, 32768)])")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    small, large = eval(r.stdout.strip().splitlines()[-1])
    assert small == 0 and (large > 0) == (k > 0)


# both sides of every line: elements, columns (fewest and most), count; and counts of list words and maxima by what the scratch holds
@pytest.mark.parametrize("L,B,F,k,room", [(6, 1365, 32768, 64, 0), (6, 1366, 32768, 64, 1024), (4, 4096, 32760, 24, 0), (4, 4096, 32768, 24, 1024), (8, 2048, 32768, 24, 1024),
                                          (8, 2048, 32776, 24, 0), (4, 4096, 32768, 64, 1024), (4, 4096, 32768, 65, 0), (8, 2048, 32768, 64, 1024), (8, 2048, 32768, 65, 2048),
                                          (8, 2048, 32768, 128, 2048), (8, 2048, 32768, 129, 0), (1, 65600, 4096, 1, 0), (1, 1 << 22, 256, 1, 0)])
def test_sizes_of_the_four_pass_token_topk(ext, L, B, F, k, room):
    got = ext.token_topk_scratch(L, B, F, k)
    maxima = -(-(-(-(L * F // 8) // 256) * 32) // 256) * 256  # one group of eight columns in eight, in whole blocks
    assert got == (B * (8 * room + 4 * maxima + 8) if room else 0)
    assert got <= B * L * F * 2 // 8  # an eighth of the matrix at most


def _waits():
    """(file, line, openers of the blocks around it) of every plain bounded wait on an mbarrier outside its helpers."""
    for path in sorted((ROOT / "crosslayer_coding_b200" / "csrc").glob("*.cu")):
        src = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"\bmbar_wait\(", src):
            line = src[src.rfind("\n", 0, m.start()) + 1: src.find("\n", m.start())].strip()
            around, depth = [], 0
            for i in range(m.start() - 1, -1, -1):
                if src[i] == "}":
                    depth += 1
                elif src[i] == "{" and depth:
                    depth -= 1
                elif src[i] == "{":
                    around.append(src[max(src.rfind(c, 0, i) for c in ";{}") + 1: i].strip())
            yield path.name, line, around


def test_bounded_waits_do_not_split_a_warp():
    """A lane that gives up at a bounded wait must not leave the others of its warp at a shuffle: a plain wait belongs to one thread, which
    goes on alone or shares the verdict; a whole warp waits through ``mbar_wait_warp`` or, its first lane for all, ``mbar_wait_leader``."""
    one_thread = re.compile(r"\b(lane|tid|etid) == \w+")
    waits = list(_waits())
    assert len(waits) > 10
    split = [(name, line) for name, line, around in waits if not one_thread.search(line) and not any(one_thread.search(a) for a in around)]
    assert not split, split


def test_a_verdict_that_one_lane_brings_home_is_ordered():
    """What one lane saw at an mbarrier is not seen by the others through a shuffle alone: a lane's own verdict for its warp comes from
    ``mbar_wait_leader``, which puts a ``__syncwarp`` behind it; a thread's for a whole CTA role through shared memory and a barrier."""
    alone = [(name, line) for name, line, around in _waits() if re.search(r"\blane == 0\) \w+ = mbar_wait", line)]
    assert not alone, alone
    helper = (ROOT / "crosslayer_coding_b200" / "csrc" / "common.cuh").read_text().split("bool mbar_wait_leader(")[1].split("\n}")[0]
    assert helper.index("mbar_wait(") < helper.index("__shfl_sync") < helper.index("__syncwarp")
