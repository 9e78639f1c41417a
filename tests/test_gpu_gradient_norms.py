"""The norm pre-pass of gradient clipping against fp64: row lengths around the vectors of a warp, lists around the entries held in registers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HYPER = [1e-3, 0.9, 0.999, 1e-8, 0.01, 0.5, 0.5, 1.0, 0.7, 0.0]  # the ninth is the gradient scale
SC_INV_SCALE, SC_GRAD_NORM_SQ, SC_CLIP = 1, 5, 6


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from crosslayer_coding_b200.ops import ext as e

    return e.load()


def _lists(g, L, F, B, dev):
    """CSR lists of 0 to 45 entries per feature: none, up to the four in registers, up to the 32 beyond them, more."""
    n = torch.randint(0, 9, (L * F,), device=dev, generator=g)
    n[:: 7] = 0
    n[:: 11] = torch.randint(30, 46, (n[:: 11].numel(),), device=dev, generator=g)
    off = torch.zeros(L * F + 1, dtype=torch.int32, device=dev)
    off[1:] = n.cumsum(0).int()
    total = int(off[-1])
    tok = torch.randint(0, B, (total,), device=dev, generator=g, dtype=torch.int32)
    val = torch.randn(total, device=dev, generator=g)
    return off, tok, val, torch.repeat_interleave(torch.arange(L * F, device=dev), n)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("L,F,B,d", [(1, 40, 33, 8), (3, 64, 100, 256), (2, 48, 64, 264), (3, 72, 50, 520), (2, 40, 64, 776), (2, 40, 40, 1032), (1, 24, 16, 2048)])
def test_decoder_and_encoder_norms(ext, dtype, extra, L, F, B, d):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(F + d)
    t16 = torch.float16 if dtype == torch.float16 else torch.bfloat16
    off, tok, val, owner = _lists(g, L, F, B, dev)
    gs = torch.randn(L, B, d, device=dev, generator=g).to(t16)
    rows = [L - s for s in range(L)]
    w = [torch.randn(F, r, d, device=dev, generator=g).to(dtype) for r in rows]
    mom = [[torch.zeros(F, r, d, device=dev) for r in rows] for _ in range(2)]
    pen = torch.randn(L * F, device=dev, generator=g) if extra else None
    idx = torch.where(torch.arange(L * F, device=dev) % 5 == 0, torch.arange(L * F, device=dev), -1).int() if extra else None
    xrows = torch.randn(L * F, d, device=dev, generator=g) if extra else None
    ctl = torch.zeros(16, device=dev)
    ctl[SC_INV_SCALE], ctl[SC_CLIP] = 0.25, 1.0
    grad_a = torch.zeros(len(val), device=dev)
    kept = [t.clone() for t in w]
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    ext.decoder_rows_adam(w, mom[0], mom[1], L, B, d, F, 0, off, tok, val, gs, grad_a, pen, None, None, None, None, HYPER, status, idx, xrows, ctl, True)
    layer, feat, scale = owner // F, owner % F, 0.7 * 0.25
    eps = 2.0 ** -24
    norm, dots, size = 0.0, torch.zeros(len(val), device=dev, dtype=torch.float64), torch.zeros(len(val), device=dev, dtype=torch.float64)
    for s in range(L):
        at = layer == s
        t, a, f = tok[at].long(), val[at].double(), feat[at]
        for r in range(rows[s]):
            seed, wr = gs[s + r].double()[t], w[s][:, r].double()
            grad = torch.zeros(F, d, device=dev, dtype=torch.float64).index_add_(0, f, a[:, None] * seed) * scale
            if extra:
                grad += pen.view(L, F)[s].double()[:, None] * wr * (torch.bincount(f, minlength=F) + (idx.view(L, F)[s] >= 0) > 0)[:, None]
                if r == 0:
                    grad += torch.where((idx.view(L, F)[s] >= 0)[:, None], xrows.view(L, F, d)[s].double(), 0.0)
            norm += float(grad.square().sum())
            dots[at] += (seed * wr[f]).sum(1) * scale
            size[at] += (seed * wr[f]).abs().sum(1) * scale
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and all(torch.equal(a, b) for a, b in zip(w, kept)) and not mom[0][0].any()
    # fp32 sums: R d products per dL/da; a row's gradient of up to 45 entries, then L F d squares
    assert ((grad_a.double() - dots).abs() <= (L * d + 8) * eps * size + 1e-30).all()
    assert abs(float(ctl[SC_GRAD_NORM_SQ]) - norm) <= (2 * 64 + 2048) * eps * norm

    # encoder: rows of the layer inputs, biases
    enc, mv = torch.randn(L, F, d, device=dev, generator=g).to(dtype), torch.zeros(L, F, d, device=dev)
    bias = torch.zeros(L, F, device=dev, dtype=dtype)
    ctl[SC_GRAD_NORM_SQ] = 0
    ext.encoder_rows_adam(enc, mv, mv.clone(), bias, torch.zeros(L, F, device=dev), torch.zeros(L, F, device=dev), off, tok, val, gs, None, None, HYPER,
                          status, idx, xrows, None, ctl, True)
    grad = torch.zeros(L * F, d, device=dev, dtype=torch.float64).index_add_(0, owner, val.double()[:, None] * gs.double()[layer, tok.long()]) * 0.7
    if extra:
        grad += torch.where((idx >= 0)[:, None], xrows.double(), 0.0)
    gb = torch.zeros(L * F, device=dev, dtype=torch.float64).index_add_(0, owner, val.double()) * 0.7
    norm = float(grad.square().sum() + gb.square().sum())
    assert abs(float(ctl[SC_GRAD_NORM_SQ]) - norm) <= (2 * 64 + 2048) * eps * norm


# weights that are not finite make the norm so, without a sparsity penalty too (the update forms 0 x w as well), wherever the row is touched at all: the step
# is then skipped
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [8, 264, 1032])
@pytest.mark.parametrize("touched", ["extra row", "entry", "none"])
def test_decoder_norm_of_weights_that_are_not_finite(ext, dtype, d, touched):
    dev = torch.device("cuda:0")
    L, F, B = 2, 16, 20
    g = torch.Generator(device=dev).manual_seed(d)
    w = [torch.randn(F, L - s, d, device=dev, generator=g).to(dtype) for s in range(L)]
    w[1][5, 0, d - 1] = float("inf")
    n = torch.ones(L * F, dtype=torch.int64)
    n[F + 5] = 1 if touched == "entry" else 0
    off = torch.zeros(L * F + 1, dtype=torch.int32, device=dev)
    off[1:] = n.cumsum(0).int().to(dev)
    total = int(off[-1])
    tok, val = torch.zeros(total, dtype=torch.int32, device=dev), torch.ones(total, device=dev)
    gs = torch.randn(L, B, d, device=dev, generator=g).bfloat16()
    idx = torch.full((L * F,), -1, dtype=torch.int32, device=dev)
    if touched == "extra row":
        idx[F + 5] = 0
    ctl = torch.zeros(16, device=dev)
    ctl[SC_INV_SCALE] = ctl[SC_CLIP] = 1.0
    zero = [torch.zeros(F, L - s, d, device=dev) for s in range(L)]
    ext.decoder_rows_adam(w, zero, zero, L, B, d, F, 0, off, tok, val, gs, torch.zeros(total, device=dev), None, None, None, None, None, HYPER,
                          torch.zeros(4, dtype=torch.int32, device=dev), idx, torch.ones(1, d, device=dev), ctl, True)
    assert bool(torch.isnan(ctl[SC_GRAD_NORM_SQ])) == (touched != "none")
    assert touched != "none" or float(ctl[SC_GRAD_NORM_SQ]) > 0
