"""The index-checking build (-DCLT_DEBUG_BOUNDS): a training step runs clean under it, and an entry whose feature index lies
outside the decoder is reported through the status word while its access is skipped (the regular build trusts its lists)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r'''
import sys, torch
sys.path.insert(0, %r)
from crosslayer_coding_b200 import CLTConfig, CrossLayerTranscoder, TrainingConfig
from crosslayer_coding_b200.ops import ext
from crosslayer_coding_b200.training.fused_engine import FusedBatchTopKEngine, EngineStatusError
e = ext.load()
assert e.__name__.endswith("_dbg"), e.__name__
dev = torch.device("cuda:0")
torch.manual_seed(0)
L, B, d, F = 3, 128, 64, 256
cfg = CLTConfig(num_features=F, num_layers=L, d_model=d, activation_fn="batchtopk", batchtopk_k=6, clt_dtype="bfloat16")
model = CrossLayerTranscoder(cfg, device=dev)
tc = TrainingConfig(learning_rate=1e-3, training_steps=10, activation_path="unused", precision="bf16", sparsity_lambda=0.01, preactivation_coef=0.0)
eng = FusedBatchTopKEngine(model, tc, B)
X = torch.randn(L, B, d, device=dev).bfloat16()
Y = torch.randn(L, B, d, device=dev).bfloat16()
for step in range(3):
    out = eng.train_step(X, Y, step, 1e-3, sparsity_lambda=0.01)
torch.cuda.synchronize()
eng.check_status()                       # no index complaint on a regular step
# an entry that names feature F (one past the last): the debug build reports it and leaves the row untouched
eng.encode_select(X)
torch.cuda.synchronize()
eng.tcsr_col[0] = (1 << 24) | F
eng.decode_loss(Y)
torch.cuda.synchronize()
try:
    eng.check_status()
    print("NO-REPORT")
except EngineStatusError as exc:
    print("REPORTED", exc)
'''


def test_debug_build_runs_clean_and_reports_a_bad_entry():
    env = dict(os.environ, CLT_DEBUG_BOUNDS="1")
    res = subprocess.run([sys.executable, "-c", SCRIPT % REPO], env=env, capture_output=True, text=True, timeout=900)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-3000:]
    assert "REPORTED" in res.stdout and "index out of range" in res.stdout and "value 256" in res.stdout, res.stdout[-1000:]


LISTS = r"""
import sys, torch
sys.path.insert(0, %r)
from crosslayer_coding_b200.ops import ext
e = ext.load()
assert e.__name__.endswith("_dbg"), e.__name__
dev, I32 = torch.device("cuda:0"), torch.int32
L, F, B = 2, 24, 40
hyper = [1e-3, 0.9, 0.999, 1e-8, 0.01, 0.5, 0.5, 1.0, 0.7, 0.0, 1.0]
n = torch.full((L * F,), 7)
off = torch.zeros(L * F + 1, dtype=I32, device=dev)
off[1:] = n.cumsum(0).to(I32).to(dev)
total = int(off[-1])

def call(what, tying, d, dtype, bad, with_status=True):
    g = torch.Generator(device=dev).manual_seed(d)
    tok = torch.randint(0, B, (total,), device=dev, generator=g, dtype=I32)
    val = torch.randn(total, device=dev, generator=g)
    if bad is not None:
        tok[bad] = B
    rows = [L - s if tying == 0 else 1 for s in range(L)]
    w = [torch.randn(F, r, d, device=dev, generator=g).to(dtype) for r in rows]
    m, v = ([torch.zeros(F, r, d, device=dev) for r in rows] for _ in range(2))
    # the row behind the last layer's, which the bad token names, is there
    seeds = torch.randn(L * B + 1, d, device=dev, generator=g).bfloat16()[: L * B].view(L, B, d)
    ctl = torch.zeros(16, device=dev)
    ctl[1] = ctl[6] = 1.0
    status = torch.zeros(4, dtype=I32, device=dev)
    norm = what.startswith("norm")
    if what.endswith("decoder"):
        e.decoder_rows_adam(w, m, v, L, B, d, F, tying, off, tok, val, seeds, torch.zeros(total, device=dev), None, None, None, None, None, hyper, status,
                            None, None, ctl, norm)
    else:
        enc, z = torch.randn(L, F, d, device=dev, generator=g).to(dtype), lambda: torch.zeros(L, F, d, device=dev)
        b = torch.zeros(L, F, device=dev)
        e.encoder_rows_adam(enc, z(), z(), b.to(dtype), b.clone(), b.clone(), off, tok, val, seeds, None, None, hyper, status, None, None, None, ctl, norm)
    torch.cuda.synchronize()
    return status.tolist()

b16, f32 = torch.bfloat16, torch.float32
CASES = [("norm decoder", 0, 264, b16), ("norm decoder", 0, 1032, f32), ("norm encoder", 0, 264, b16), ("norm decoder", 1, 264, b16), ("decoder", 0, 264, b16),
         ("decoder", 0, 520, b16), ("decoder", 0, 520, f32), ("decoder", 2, 264, b16), ("decoder", 2, 520, b16), ("decoder", 1, 264, b16), ("encoder", 0, 264, b16),
         ("encoder", 0, 520, b16), ("decoder", 0, 2056, b16), ("encoder", 0, 2056, b16)]
for case in CASES:
    assert call(*case, None) == [0, 0, 0, 0], case
    for at in (0, 5):  # among the first four entries of a list, which several forms hold ahead, and behind them
        got = call(*case, (L * F - 1) * 7 + at)
        assert got[0] == 5 and 200 < got[2] < 300 and got[3] == B, (case, at, got)
print("ALL-REPORTED")
"""


def test_debug_build_checks_the_tokens_of_every_row_update():
    """The norm pre-pass, the row pipeline with its entries beyond the staged ones, a warp per row, the general sweeps."""
    env = dict(os.environ, CLT_DEBUG_BOUNDS="1")
    res = subprocess.run([sys.executable, "-c", LISTS % REPO], env=env, capture_output=True, text=True, timeout=900)
    assert res.returncode == 0 and "ALL-REPORTED" in res.stdout, res.stdout[-2000:] + res.stderr[-3000:]
