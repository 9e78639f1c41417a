"""Host-side rules of the native library, which need no GPU: sizes at which a call takes another form or is refused."""
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
