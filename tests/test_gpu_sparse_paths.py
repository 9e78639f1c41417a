"""Kernels of the sparse step at the sizes where their dispatch changes, each against a plain PyTorch restatement."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
I32, F32 = torch.int32, torch.float32


@pytest.fixture(scope="module")
def ext():
    from crosslayer_coding_b200.ops import ext as ext_mod

    return ext_mod.load()


def _dev():
    return torch.device("cuda:0")


def _csr(ext, tok, col, val, B, ncols, pitch, sort=3):
    """Both CSR views of an entry list, as the engine builds them."""
    dev, n = tok.device, tok.numel()
    ctl = torch.zeros(16, dtype=torch.int64, device=dev)
    ctl[3] = n
    z = lambda k, dt=I32: torch.zeros(max(k, 1), dtype=dt, device=dev)  # noqa: E731
    r = dict(tok_off=z(B + 1), feat_off=z(ncols + 1), tcsr_col=z(n), tcsr_val=z(n, F32), fcsr_tok=z(n), fcsr_val=z(n, F32))
    ext.build_csr(tok, col, val, ctl, B, ncols, z(B), z(ncols), r["tok_off"], r["feat_off"], z(B), z(ncols), r["tcsr_col"], r["tcsr_val"],
                  r["fcsr_tok"], r["fcsr_val"], None, sort, pitch)
    return r


def _entries(g, L, B, F, n, dev):
    """n distinct (token, layer, feature) entries in random order; every third value negative, a few exactly zero."""
    flat = torch.randperm(B * L * F, generator=g)[:n]
    val = torch.randn(n, generator=g)
    val[::17] = 0.0
    return (flat // (L * F)).to(I32).to(dev), (flat % (L * F)).to(I32).to(dev), val.to(dev)


def _dense_decode(L, B, d, F, tying, tok, col, val, W, off, sc, rows_limit=0):
    """``[L, B, d]`` in 64 bits: the sums over the entries, without biases."""
    acts = torch.zeros(L, B, F, device=tok.device, dtype=torch.float64)
    acts[(col // F).long(), tok.long(), (col % F).long()] = val.double()
    want = torch.zeros(L, B, d, device=tok.device, dtype=torch.float64)
    for t in range(L):
        for s in range(t + 1):
            if rows_limit and t - s >= rows_limit:
                continue
            a = acts[s]
            if off is not None:
                a = torch.where(a != 0, (a + off[t].double()) * sc[t].double(), a)
            w = W[s][:, t - s] if tying == 0 else W[s if tying == 1 else t][:, 0]
            want[t] += a @ w.double()
    return want


def _check_decode(ext, L, B, d, tying, affine, dtype=torch.bfloat16, addend=False, rows_limit=0, F=24, entries=None, expected=0, equal=False):
    dev = _dev()
    g = torch.Generator().manual_seed(L * 1000 + B + d)
    tok, col, val = (entries or _entries)(g, L, B, F, min(B * L * F, 7 * B), dev)
    rows = [L - s if tying == 0 else 1 for s in range(L)]
    W = [(torch.randn(F, r, d, generator=g) / 4).to(dtype).to(dev) for r in rows]
    off = torch.randn(L, F, generator=g).to(dev) if affine else None
    sc = torch.randn(L, F, generator=g).to(dev) if affine else None
    bias = torch.randn(L, d, generator=g).to(dev)
    add = torch.randn(L, B, d, generator=g).to(dev) if addend else None
    y = torch.randn(L, B, d, generator=g).to(dtype).to(dev)
    sigma = (0.5 + torch.rand(L, d, generator=g)).to(dev)
    want = _dense_decode(L, B, d, F, tying, tok, col, val, W, off, sc, rows_limit) + bias.double()[:, None, :]
    if addend:
        want += add.double()
    status = torch.zeros(4, dtype=I32, device=dev)
    for sort in (3, 0):  # the order of a token's entries changes only the order of the sums
        c = _csr(ext, tok, col, val, B, L * F, F, sort)

        def decode(mode, partial=None, bias=None, addend=None, target=None, sigma=None, gs=None, yhat=None, sq=None, peers=(), rows_per_rank=0, rank=0):
            ext.sparse_decode(W, L, B, d, F, tying, c["tok_off"], c["tcsr_col"], c["tcsr_val"], off, sc, partial, bias, addend, target, sigma, gs, yhat, sq, mode,
                              list(peers), rows_per_rank, rank, status, None, rows_limit, expected, equal)

        yhat = torch.full((L, B, d), float("nan"), device=dev)
        gs = torch.empty(L, B, d, device=dev, dtype=dtype)
        sq = torch.zeros(L, device=dev, dtype=torch.float64)
        decode(1, bias=bias, addend=add, target=y, sigma=sigma, gs=gs, yhat=yhat, sq=sq)
        # fp32 sums of at most a few dozen products: 2^-24 each on terms of the size of the result
        scale = want.abs().max()
        assert (yhat.double() - want).abs().max() < 1e-5 * scale
        r = (want - y.double()) * sigma.double()[:, None]
        assert torch.allclose(sq, r.square().sum((1, 2)), rtol=1e-5)
        # bf16 keeps 8 bits (fp16 has 11): half a unit in the last place of the value, plus the fp32 error of the sum
        assert ((gs.double() - r * sigma.double()[:, None]).abs() <= 2 ** -8 * (r * sigma.double()[:, None]).abs() + 1e-4).all()
        # the reconstruction alone
        plain = torch.full((L, B, d), float("nan"), device=dev)
        decode(1, bias=bias, addend=add, yhat=plain)
        assert torch.equal(plain, yhat) if sort == 3 else (plain.double() - want).abs().max() < 1e-5 * scale
        # partial sums only (the tensor-parallel form before the exchange)
        sums = want - bias.double()[:, None] - (add.double() if addend else 0)
        part = torch.full((L, B, d), float("nan"), device=dev)
        decode(0, partial=part)
        assert (part.double() - sums).abs().max() < 1e-5 * scale
        # the same sums pushed to the owners of the tokens, three of them with the last block not full: each holds an area [ranks, L,
        # rows, d] per sending rank; here all areas lie in this GPU's memory (the kernel only stores, no rank waits for another)
        world, rank = 3, 1
        rows_per_rank = (B + world - 1) // world
        areas = torch.full((world, world, L, rows_per_rank, d), float("nan"), device=dev)
        decode(2, peers=[areas[o].data_ptr() for o in range(world)], rows_per_rank=rows_per_rank, rank=rank)
        pushed = torch.cat([areas[o, rank] for o in range(world)], dim=1)
        assert torch.equal(pushed[:, :B], part) if sort == 3 else (pushed[:, :B].double() - sums).abs().max() < 1e-5 * scale
        assert bool(pushed[:, B:].isnan().all()) and bool(areas[:, [0, 2]].isnan().all())
    assert int(status[0]) == 0


# d: one to four 16-byte vectors per lane, partly filled ones, two column chunks; B: the split walk (few (token, target) warps), the
# walk, the walk of two rows per step (2048 tokens and three or four vectors) and (per source) the running sum, each with a last
# CTA that is not full
@pytest.mark.parametrize("tying,affine", [(0, False), (1, False), (1, True), (2, False), (2, True)])
@pytest.mark.parametrize("L,B,d", [(2, 3, 8), (3, 5, 264), (12, 2, 768), (2, 3, 1024), (3, 4, 2048), (4, 1030, 256), (4, 1030, 512), (5, 1027, 520), (2, 2055, 768),
                                   (2, 2051, 1024), (3, 1500, 1024), (2, 2051, 1032), (3, 700, 2048), (2, 2050, 2048)])
def test_gather_decode_matches_dense(ext, L, B, d, tying, affine):
    _check_decode(ext, L, B, d, tying, affine)


# the half-precision build, the skip connection's addend, a limit on the target rows (which keeps per-source decoders off the
# running sum), more layers than any other test has
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,d", [(3, 5, 264), (4, 1100, 512), (2, 2055, 768), (20, 70, 264), (32, 1030, 64)])
@pytest.mark.parametrize("opts", [dict(dtype=torch.float16), dict(addend=True), dict(rows_limit=1), dict(rows_limit=2, dtype=torch.float16, addend=True)])
def test_gather_decode_options(ext, L, B, d, tying, opts):
    _check_decode(ext, L, B, d, tying, False, **opts)


def _uneven_entries(g, L, B, F, n, dev):
    """Lists of very different length: every 64th token has up to 600 entries, most have a few, every fifth none."""
    tok, flat = [], []
    for b in range(B):
        k = 0 if b % 5 == 4 else (600 if b % 64 == 0 else (130 if b % 64 == 1 else b % 4))
        pick = torch.randperm(L * F, generator=g)[:k]
        tok.append(torch.full((pick.numel(),), b))
        flat.append(pick)
    tok, flat = torch.cat(tok), torch.cat(flat)
    mix = torch.randperm(tok.numel(), generator=g)
    return tok[mix].to(I32).to(dev), flat[mix].to(I32).to(dev), torch.randn(tok.numel(), generator=g).to(dev)


# lists of several batches per warp next to empty ones, on both sides of every line of the dispatch: eight warps per token, four, two tokens
# of narrow rows per CTA, two rows per step with the tokens by length (also with two column chunks), the running sum with and without
# that order
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,d", [(3, 70, 264), (3, 70, 1032), (4, 1030, 136), (13, 1900, 136), (4, 1030, 512), (14, 2049, 520), (4, 4097, 512), (7, 2050, 1800)])
def test_gather_decode_of_uneven_lists(ext, L, B, d, tying):
    _check_decode(ext, L, B, d, tying, False, F=72, entries=_uneven_entries)


# two warps per token, which callers with a small k ask for (and get for many (token, target) pairs): the sums do not depend on how
# true the expectation is
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,d", [(13, 1303, 512), (13, 1303, 520), (9, 1001, 1800), (3, 70, 520)])
@pytest.mark.parametrize("expected,equal", [(20, False), (20, True), (60, True)])
def test_gather_decode_with_an_expected_length(ext, L, B, d, tying, expected, equal):
    _check_decode(ext, L, B, d, tying, tying != 0, F=72, entries=_uneven_entries, expected=expected, equal=equal)


# lists of one length of 128 and more entries: one warp or four per token on either side of the lines, without the order by length
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,d", [(13, 1303, 520), (9, 1303, 520), (7, 2050, 1800), (3, 600, 1032), (13, 1303, 512), (4, 4100, 200)])
@pytest.mark.parametrize("expected", [127, 200, 300])
def test_gather_decode_of_equal_long_lists(ext, tying, L, B, d, expected):
    _check_decode(ext, L, B, d, tying, False, F=72, entries=_uneven_entries, expected=expected, equal=True)


# slices of 256 columns per CTA where all of them are on the chip at once, at most 592: on both sides of the line, the last slice with one vector,
# half and whole, next to short expected lists, which keep whole rows
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,d", [(2, 98, 520), (2, 99, 520), (4, 37, 1024), (4, 38, 1024), (12, 16, 768), (3, 2, 776), (1, 197, 640)])
@pytest.mark.parametrize("opts", [dict(), dict(expected=20), dict(expected=200, equal=True, dtype=torch.float16), dict(addend=True, rows_limit=2)])
def test_gather_decode_of_few_tokens(ext, tying, L, B, d, opts):
    _check_decode(ext, L, B, d, tying, tying != 0 and opts.get("rows_limit") is None, F=300, entries=_uneven_entries, **opts)


@pytest.mark.parametrize("d", [520, 768, 1024])
def test_decode_in_slices_equals_whole_rows(ext, d):
    """An element's sum takes the same entries in the same order in both forms: few tokens (slices) give the bits that they give among many."""
    dev = _dev()
    g = torch.Generator().manual_seed(d)
    L, F, few, many = 3, 400, 16, 512
    tok, col, val = _uneven_entries(g, L, many, F, 0, dev)
    W = [(torch.randn(F, L - s, d, generator=g) / 4).to(torch.bfloat16).to(dev) for s in range(L)]
    out = []
    for B in (few, many):
        keep = tok < B
        c = _csr(ext, tok[keep].contiguous(), col[keep].contiguous(), val[keep].contiguous(), B, L * F, F)
        part = torch.full((L, B, d), float("nan"), device=dev)
        ext.sparse_decode(W, L, B, d, F, 0, c["tok_off"], c["tcsr_col"], c["tcsr_val"], None, None, part, None, None, None, None, None, None, None, 0, [], 0, 0,
                          torch.zeros(4, dtype=I32, device=dev), None, 0, 0, False)
        out.append(part[:, :few])
    assert torch.equal(*out)


@pytest.mark.parametrize("L,B,d", [(3, 1303, 200), (3, 1303, 512)])
def test_gather_decode_of_equal_short_lists_in_narrow_rows(ext, L, B, d):
    _check_decode(ext, L, B, d, 0, False, F=72, entries=_uneven_entries, expected=20, equal=True)


# the running sum over lists of unknown length: on both sides of the line between four and two warps per token, one and two column chunks
@pytest.mark.parametrize("B,d", [(8191, 200), (8192, 200), (4095, 520), (4096, 520)])
def test_running_decode_of_many_tokens(ext, B, d):
    _check_decode(ext, 2, B, d, 1, False, F=72, entries=_uneven_entries)


# the running sum with one and with two warps per token
@pytest.mark.parametrize("d", [200, 520])
@pytest.mark.parametrize("expected,equal", [(20, False), (40, False), (100, True)])
def test_running_decode_with_an_expected_length(ext, d, expected, equal):
    _check_decode(ext, 5, 1303, d, 1, False, F=72, entries=_uneven_entries, expected=expected, equal=equal)


def test_decode_refuses_loss_outputs_without_a_target(ext):
    """Without a target neither the gradient seed nor the error sums are written: a call that hands them in is an error."""
    dev = _dev()
    L, B, d, F = 2, 3, 64, 24
    g = torch.Generator().manual_seed(0)
    c = _csr(ext, *_entries(g, L, B, F, 20, dev), B, L * F, F)
    W = [torch.randn(F, L - s, d, generator=g).bfloat16().to(dev) for s in range(L)]
    bias, yhat = torch.zeros(L, d, device=dev), torch.empty(L, B, d, device=dev)
    gs, sq = torch.empty(L, B, d, device=dev, dtype=torch.bfloat16), torch.zeros(L, device=dev, dtype=torch.float64)
    target = torch.zeros(L, B, d, device=dev, dtype=torch.bfloat16)

    def call(target, gs, yhat, sq):
        ext.sparse_decode(W, L, B, d, F, 0, c["tok_off"], c["tcsr_col"], c["tcsr_val"], None, None, None, bias, None, target, None, gs, yhat, sq, 1, [], 0, 0,
                          torch.zeros(4, dtype=I32, device=dev))

    for bad in ((None, gs, yhat, sq), (None, gs, yhat, None), (None, None, yhat, sq), (None, None, None, None), (target, None, yhat, sq), (target, gs, yhat, None)):
        with pytest.raises(RuntimeError, match="mode 1"):
            call(*bad)
    call(None, None, yhat, None)
    call(target, gs, None, sq)


# long segments in shared memory, ranges beyond it, one feature per CTA, tokens beyond the token sort's buffer
@pytest.mark.parametrize("B,L,F,n", [(40, 2, 300, 900), (3000, 1, 8, 20000), (5000, 1, 2, 9000), (9000, 1, 3, 27000), (2, 2, 4000, 9000), (700, 3, 512, 200000)])
def test_csr_segments_are_sorted(ext, B, L, F, n):
    dev = _dev()
    g = torch.Generator().manual_seed(n)
    tok, col, val = _entries(g, L, B, F, n, dev)
    c = _csr(ext, tok, col, val, B, L * F, F)
    order = torch.argsort(col.long() * B + tok.long())
    assert torch.equal(c["fcsr_tok"], tok[order]) and torch.equal(c["fcsr_val"], val[order])
    order = torch.argsort(tok.long() * (L * F) + col.long())
    packed = ((col // F) << 24) | (col % F)
    assert torch.equal(c["tcsr_col"], packed[order].to(I32)) and torch.equal(c["tcsr_val"], val[order])
    assert torch.equal(c["feat_off"].cpu(), torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(col.cpu().long(), minlength=L * F).cumsum(0)]).to(I32))
    assert torch.equal(c["tok_off"].cpu(), torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(tok.cpu().long(), minlength=B).cumsum(0)]).to(I32))


# ranks over the list and buckets by layer (few and many tokens), one to eight entries per thread, a bucket that is too long, the network
# beyond, one and several tiles of the scan
@pytest.mark.parametrize("B,L,F,n", [(1, 2, 4000, 250), (3, 4, 1000, 1530), (2, 4, 1000, 1600), (2, 12, 1000, 3800), (2, 2, 4000, 1700), (2, 3, 2000, 4500),
                                     (5000, 3, 64, 40000), (700, 32, 16, 90000), (1100, 8, 64, 200000), (1100, 8, 80, 450000), (1100, 5, 300, 900000)])
def test_token_view_alone(ext, B, L, F, n):
    """The token-major view without the feature-major one: equal to that of the full build, entries outside the problem left out."""
    dev = _dev()
    g = torch.Generator().manual_seed(n)
    tok, col, val = _entries(g, L, B, F, n, dev)
    c = _csr(ext, tok, col, val, B, L * F, F)
    stray = torch.tensor([-1, B, 0, 0], dtype=I32, device=dev), torch.tensor([0, 0, -1, L * F], dtype=I32, device=dev), torch.ones(4, device=dev)
    tok2, col2, val2 = (torch.cat([a, b]) for a, b in zip((tok, col, val), stray))
    ctl = torch.zeros(16, dtype=torch.int64, device=dev)
    ctl[3] = n + 4
    z = lambda k, dt=I32: torch.zeros(k, dtype=dt, device=dev)  # noqa: E731
    off, tc, tv, per_layer = z(B + 1), z(n + 4), z(n + 4, F32), z(L)
    ext.build_token_csr(tok2, col2, val2, ctl, B, L * F, z(B), off, z(B), tc, tv, per_layer, F)
    assert torch.equal(off, c["tok_off"]) and torch.equal(tc[:n], c["tcsr_col"]) and torch.equal(tv[:n], c["tcsr_val"])
    assert torch.equal(per_layer.long(), torch.bincount((col // F).long(), minlength=L))


# the same number of entries in every layer: one layer (ranks, then the network), too few layers for the buckets, buckets that all start at a multiple of 32
# words, the longest buckets of every number of entries per thread, the last of the 128 layers a key can number
@pytest.mark.parametrize("B,L,per_layer", [(800, 1, 200), (800, 1, 256), (800, 1, 300), (800, 2, 300), (800, 2, 64), (800, 2, 128), (800, 2, 256), (40, 4, 256), (40, 8, 256), (800, 8, 32),
                                           (800, 16, 64), (40, 20, 100), (40, 128, 15), (800, 128, 3)])
def test_token_segments_of_even_layers(ext, B, L, per_layer):
    dev = _dev()
    F = 320
    g = torch.Generator().manual_seed(B + L + per_layer)
    f = torch.stack([torch.randperm(F, generator=g)[:per_layer] for _ in range(B * L)])  # distinct features of a (token, layer)
    row = torch.arange(B * L).repeat_interleave(per_layer)
    tok, col = row // L, (row % L) * F + f.reshape(-1)
    mix = torch.randperm(tok.numel(), generator=g)
    tok, col, val = tok[mix].to(I32).to(dev), col[mix].to(I32).to(dev), torch.randn(tok.numel(), generator=g).to(dev)
    c = _csr(ext, tok, col, val, B, L * F, F)
    order = torch.argsort(tok.long() * L * F + col.long())
    assert torch.equal(c["tcsr_col"], ((col[order] // F) << 24) | (col[order] % F)) and torch.equal(c["tcsr_val"], val[order])


@pytest.mark.parametrize("fn", ["batchtopk", "topk", "jumprelu"])
def test_views_after_a_reconstruction(ext, fn):
    """``reconstruct`` builds the token-major view; the feature-major one and the counts per layer are those of the same selection, and a
    batch that lies in one tensor gives what separate tensors give."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    sf = SparseForward(_serving_model(fn, "none", dev), 200)
    x = torch.randn(3, 200, 64, device=dev).bfloat16()
    sf.encode(x)
    names = ("tok_off", "tcsr_col", "tcsr_val", "feat_off", "fcsr_tok", "fcsr_val")
    want, n, l0 = {k: getattr(sf, k).clone() for k in names}, sf.num_entries(), sf.l0_per_layer()
    sf.encode(torch.randn(3, 200, 64, device=dev).bfloat16())
    a = sf.forward_dict({l: x[l] for l in range(3)})
    assert torch.equal(sf.l0_per_layer(), l0)
    for k in names:  # beyond the entries of this selection the arrays hold what earlier ones left
        assert torch.equal(getattr(sf, k)[: n if "csr" in k else None], want[k][: n if "csr" in k else None]), k
    assert torch.equal(sf.l0_per_layer(), l0)
    y = x.clone()
    for other in ({l: x[l].clone() for l in range(3)}, {l: x[l].float() for l in range(3)}, {0: x[0], 1: x[1], 2: y[2]}):
        b = sf.forward_dict(other)
        assert all(torch.equal(a[l], b[l]) for l in range(3))
    swapped = sf.forward_dict({0: x[1], 1: x[0], 2: x[2]})
    assert not torch.equal(swapped[0], a[0])
    sf.check_status()


FEATURE_VIEW = ("feat_off", "feat_cnt", "feat_cursor", "fcsr_tok", "fcsr_val")


def _views(sf):
    """Copies of both views and the counts per layer; the arrays as long as the entry list end where its entries do."""
    n = sf.num_entries()
    return [getattr(sf, k)[: n if "csr" in k else None].clone() for k in ("tok_off", "tcsr_col", "tcsr_val") + FEATURE_VIEW] + [sf.l0_per_layer()]


def _encoded(model, B, x):
    """The views of a selection by ``encode`` on an object of its own."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    sf = SparseForward(model, B)
    sf.encode(x)
    return _views(sf)


def test_expected_length_of_threshold_lists(ext):
    """What the caller expects of the lists changes the order of the sums and nothing else; a small room says as much."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    B = 6000  # enough (token, target) pairs for two warps per token
    model = _serving_model("jumprelu", "none", dev)
    with torch.no_grad():
        model.log_threshold.fill_(0.9)
    x = _batches(1, dev, B)[0]
    y = torch.randn(3, B, 64, device=dev).bfloat16()
    runs = {}
    for name, kw in (("open", {}), ("short", dict(expected_active_per_token=3)), ("none", dict(expected_active_per_token=0)), ("long", dict(expected_active_per_token=500)),
                     ("room", dict(max_active_per_token=60))):
        sf = SparseForward(model, B, **kw)
        runs[name] = (sf.reconstruct(x, y), sf.sq_err.clone(), sf.expected_entries)
        sf.check_status()
    assert [r[2] for r in runs.values()] == [0, 3, 1, 500, 60]
    scale = runs["open"][0].abs().max()
    for yhat, sq, _ in runs.values():
        assert (yhat - runs["open"][0]).abs().max() < 1e-5 * scale and torch.allclose(sq, runs["open"][1], rtol=1e-5)


def _batches(n, dev, B=200, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed)
    return [torch.randn(3, B, 64, device=dev, generator=g).bfloat16() for _ in range(n)]


@pytest.mark.parametrize("fn", ["batchtopk", "topk", "jumprelu"])
@pytest.mark.parametrize("taken", ["at the start", "after a call"])
def test_held_feature_arrays_follow_the_calls(ext, fn, taken):
    """The feature-major arrays are buffers: whoever holds one has the last selection in it, whichever call made it."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model(fn, "none", dev)
    sf = SparseForward(model, 200)
    x = _batches(3, dev)
    if taken == "after a call":
        sf.reconstruct(x[2])
    held = {k: getattr(sf, k) for k in FEATURE_VIEW}
    for b in x:
        sf.reconstruct(b)
        want, n = _encoded(model, 200, b), sf.num_entries()
        for k, w in zip(FEATURE_VIEW, want[3:]):
            assert torch.equal(held[k][: n if "csr" in k else None], w), k
        assert all(torch.equal(a, b) for a, b in zip(_views(sf), want))


@pytest.mark.parametrize("fn", ["batchtopk", "topk", "jumprelu"])
@pytest.mark.parametrize("read_before", [False, True])
def test_feature_view_after_graph_replays(ext, fn, read_before):
    """Replays of a recorded ``reconstruct``: the views and the counts per layer are those of the replay, before and after the first read
    and next to eager calls."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model(fn, "none", dev)
    sf = SparseForward(model, 200)
    x = _batches(4, dev)
    inp = x[0].clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        sf.reconstruct(inp)  # warm-up
    torch.cuda.current_stream().wait_stream(side)
    if read_before:
        sf.feat_off
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sf.reconstruct(inp)
    l0 = []
    for step, b in enumerate(x[1:] + x[:2]):
        if step == 2:
            sf.reconstruct(x[0])  # an eager call in between
            assert all(torch.equal(a, w) for a, w in zip(_views(sf), _encoded(model, 200, x[0])))
        inp.copy_(b)
        graph.replay()
        l0.append(sf.l0_per_layer())
        if step != 0:  # the first replay passes without a read of the feature-major view
            assert all(torch.equal(a, w) for a, w in zip(_views(sf), _encoded(model, 200, b)))
        assert torch.equal(l0[-1], _encoded(model, 200, b)[-1])
    sf.check_status()


def test_feature_view_read_inside_a_recording_and_on_another_stream(ext):
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model("batchtopk", "none", dev)
    x = _batches(2, dev, seed=1)
    want = [_encoded(model, 200, b) for b in x]
    sf = SparseForward(model, 200)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(20):
            sf.reconstruct(x[1])
        sf.reconstruct(x[0])
    off = sf.feat_off  # taken on the current stream while the calls run on the other one
    side.synchronize()
    assert torch.equal(off, want[0][3])
    # a recording that only reads, behind an eager call that left the view out: each replay reads the list of its moment
    sf = SparseForward(model, 200)
    sf.reconstruct(x[0])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        copy = sf.feat_off.clone()
    graph.replay()
    assert torch.equal(copy, want[0][3])
    sf.reconstruct(x[1])
    graph.replay()
    assert torch.equal(copy, want[1][3])


def test_equal_keys_in_a_token_segment_are_all_kept(ext):
    """A caller's list may name one column twice for a token: both entries stay."""
    dev = _dev()
    tok = torch.zeros(40, dtype=I32, device=dev)
    col = torch.tensor([7] * 20 + list(range(20)), dtype=I32, device=dev)
    val = torch.arange(40, device=dev).float()
    c = _csr(ext, tok, col, val, 1, 64, 64)
    assert torch.equal(c["tcsr_col"].long(), torch.sort(col.long()).values)
    assert torch.equal(torch.sort(c["tcsr_val"]).values, val)


def _check_token_topk(ext, x, mean, rstd, k, F, dev):
    L, B, Fl = x.shape
    status = torch.zeros(4, dtype=I32, device=dev)
    ctl = torch.zeros(16, dtype=torch.int64, device=dev)
    tok, col = torch.zeros(B * k, dtype=I32, device=dev), torch.zeros(B * k, dtype=I32, device=dev)
    val = torch.zeros(B * k, device=dev)
    ext.token_topk_select(x, mean, rstd, Fl, k, ctl, tok, col, val, status, F)
    torch.cuda.synchronize(dev)
    assert int(status[0]) == 0 and int(ctl[3]) == B * k
    assert torch.equal(tok.view(B, k), torch.arange(B, device=dev, dtype=I32)[:, None].expand(B, k))
    assert torch.equal(x.float()[(col // Fl).long(), tok.long(), (col % Fl).long()], val)
    z = ((x.float() - mean[:, None]) * rstd[:, None])[:, :, :F].permute(1, 0, 2).reshape(B, L * F)
    order = torch.sort(z, dim=1, descending=True, stable=True).indices[:, :k]
    want = torch.sort((order // F) * Fl + order % F, dim=1).values.to(I32)
    assert torch.equal(torch.sort(col.view(B, k), dim=1).values, want)


# one, two and four tokens per CTA with a last CTA that is not full; k up to the radix rounds; padding columns
@pytest.mark.parametrize("L,B,Fl,F,k", [(3, 5, 4096, 4096, 64), (2, 601, 2056, 2050, 24), (4, 1779, 520, 520, 7), (4, 1401, 520, 520, 7), (2, 33, 1032, 1030, 513), (1, 9, 64, 64, 64),
                                        (2, 40, 16384, 16384, 300)])
def test_token_topk(ext, L, B, Fl, F, k):
    dev = _dev()
    torch.manual_seed(k)
    x = torch.randn(L, B, Fl, device=dev).bfloat16()
    if B == 33:
        x[0, :, 100:400] = 1.5  # equal columns after standardisation: ties at and around the cut of the radix rounds
    mean, rstd = torch.empty(L, Fl, device=dev), torch.empty(L, Fl, device=dev)
    ext.colstats(x, mean, rstd)
    if B == 40:
        x[1, 3] = 30.0  # a token with half of its keys far above the other half: the bound from the sample rises with them
        ext.colstats(x, mean, rstd)
    _check_token_topk(ext, x, mean, rstd, k, F, dev)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B", [6, 602, 1401, 1781])
def test_token_topk_hands_overflowing_lists_to_the_radix_rounds(ext, B, dtype):
    """The bound on a token's k-th key comes from every eighth block of 2048 columns here.  Large values in the blocks between stay
    above it, more of them than the list holds: those tokens are marked for the radix kernel, which takes them and their
    neighbours in a group of four."""
    dev = _dev()
    L, F, k = 2, 65536 if B == 6 else 16384, 16
    g = torch.Generator().manual_seed(B)
    x = torch.randn(L, B, F, generator=g).to(dtype).to(dev)
    step = min(8, L * F // 8 // 2048)  # as the launcher picks it for k = 16: list of 2048, 1024 maxima
    assert step > 1
    block = torch.arange(L * F, device=dev).view(L, F) // 2048
    unsampled = (block % step != 0) & (block < 4)
    assert int(unsampled.sum()) > 2048
    for t in {1, B // 2 + 1, B - 1}:
        x[:, t][unsampled] = (10 + 2 * torch.rand(int(unsampled.sum()), generator=g)).to(dtype).to(dev)  # with ties: 16-bit values
        assert float(x[:, t][~unsampled].max()) < 10
    _check_token_topk(ext, x, torch.zeros(L, F, device=dev), torch.ones(L, F, device=dev), k, F, dev)


@pytest.mark.parametrize("B,k", [(5, 64), (700, 24), (1400, 7)])
def test_token_topk_list_takes_ties_by_the_lowest_index(ext, B, k):
    """Keys with a spacing of a half: dozens of columns share the key at the cut, and the list kernel keeps the first of them."""
    dev = _dev()
    L, F = 2, 16384
    g = torch.Generator().manual_seed(k)
    x = ((2 * torch.randn(L, B, F, generator=g)).round() / 2).bfloat16().to(dev)
    z = x.float().permute(1, 0, 2).reshape(B, L * F)
    cut = torch.topk(z, k, dim=1).values[:, -1:]
    assert bool(((z >= cut).sum(1) > k).any()) and int((z >= cut - 0.5).sum(1).max()) < 2048  # ties, and a list that holds them
    _check_token_topk(ext, x, torch.zeros(L, F, device=dev), torch.ones(L, F, device=dev), k, F, dev)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_token_topk_on_two_devices_of_one_process(ext):
    for i in (0, 1):
        dev = torch.device("cuda", i)
        x = torch.randn(2, 1401, 512, device=dev).bfloat16()
        mean, rstd = torch.empty(2, 512, device=dev), torch.empty(2, 512, device=dev)
        ext.colstats(x, mean, rstd)
        _check_token_topk(ext, x, mean, rstd, 8, 512, dev)


# the four-pass form of large matrices: shard padding, columns and tokens that do not fill a tile, the smallest and the largest number of columns, k on both
# sides of the two list sizes and at its largest; and large matrices that keep the other forms (too few columns, too large a k, too many columns)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,B,Fl,F,k,passes", [(4, 2050, 32768, 32761, 64, True), (16, 1100, 16376, 16370, 24, True), (8, 1030, 32768, 32765, 65, True), (8, 1031, 32768, 32760, 100, True),
                                               (8, 1029, 32768, 32761, 128, True), (3, 4400, 20488, 20481, 24, False), (8, 1030, 32768, 32760, 200, False),
                                               (8, 1029, 32776, 32776, 512, False)])
def test_token_topk_of_large_matrices(ext, L, B, Fl, F, k, passes, dtype):
    dev = _dev()
    assert B * L * Fl >= 1 << 28 and (ext.token_topk_scratch(L, B, Fl, k) > 0) == passes
    g = torch.Generator(device=dev).manual_seed(k)
    x = (torch.randn(L, B, Fl, generator=g, device=dev) * 0.7 + 0.3 * torch.randn(L, 1, Fl, generator=g, device=dev)).to(dtype)
    mean = torch.stack([x[l].float().mean(0) for l in range(L)])
    rstd = torch.stack([1.0 / (x[l].float().std(0) + 1e-6) for l in range(L)])
    _check_token_topk(ext, x, mean, rstd, k, F, dev)


def test_token_topk_of_large_matrices_with_values_that_are_not_finite(ext):
    """A column with a NaN has NaN statistics and sorts above everything in every row, and infinities sort by their sign: as in the form for
    small matrices, which the same rows are put through a few at a time."""
    dev = _dev()
    L, B, F, k = 4, 2048, 33000, 40
    assert ext.token_topk_scratch(L, B, F, k) > 0  # the four passes; 256 rows at a time take the other form
    g = torch.Generator(device=dev).manual_seed(3)
    x = torch.randn(L, B, F, generator=g, device=dev).bfloat16()
    x[0, 7, 100] = float("nan")
    x[1, 9, 200] = float("inf")
    x[1, 5, 300] = float("-inf")
    x[:, 11] = 1000.0  # a row far above the others: its whole list reaches the bound
    x[:, 12, :8192] = 50.0
    mean, rstd = x.float().mean(1), 1.0 / (x.float().std(1) + 1e-6)
    rstd[1, 400] = 0.0

    def select(rows):
        xs = x[:, rows].contiguous()
        n = xs.shape[1]
        tok, col = torch.zeros(n * k, dtype=I32, device=dev), torch.zeros(n * k, dtype=I32, device=dev)
        val, status = torch.zeros(n * k, device=dev), torch.zeros(4, dtype=I32, device=dev)
        ext.token_topk_select(xs, mean, rstd, F, k, torch.zeros(16, dtype=torch.int64, device=dev), tok, col, val, status, F)
        return torch.sort(col.view(n, k), dim=1).values, int(status[0])

    want = [select(slice(b, b + 256)) for b in range(0, B, 256)]
    got = select(slice(0, B))
    assert torch.equal(got[0], torch.cat([w[0] for w in want])) and got[1] == max(w[1] for w in want)


def test_launches_are_counted(ext):
    """What a caller adds to its count of kernels: the per-token selection by its three forms, the decode with and without the order by length."""
    dev = _dev()
    z = lambda n, dt=I32: torch.zeros(n, dtype=dt, device=dev)  # noqa: E731
    for (L, B, F, k), kernels in (((2, 40, 64, 8), 2), ((2, 40, 1024, 600), 1), ((4, 2050, 32768, 8), 5)):
        x = torch.randn(L, B, F, device=dev).bfloat16()
        got = ext.token_topk_select(x, z((L, F), F32), torch.ones(L, F, device=dev), F, k, z(16, torch.int64), z(B * k), z(B * k), z(B * k, F32), z(4), F)
        assert got == kernels
    for B, expected, equal, kernels in ((40, 0, False, 1), (10000, 0, False, 2), (10000, 20, False, 1), (10000, 200, False, 2), (10000, 200, True, 1)):
        L, d = 3, 520
        got = ext.sparse_decode([z((8, L - s, d), torch.bfloat16) for s in range(L)], L, B, d, 8, 0, z(B + 1), z(8), z(8, F32), None, None, None, z((L, d), F32), None, None, None,
                                None, z((L, B, d), F32), None, 1, [], 0, 0, z(4), None, 0, expected, equal)
        assert got == kernels


@pytest.mark.parametrize("L,B,F", [(2, 40, 64), (6, 2048, 8192), (6, 2048, 32768)])  # the last one is large enough for the four passes
@pytest.mark.parametrize("k", [0, -1, -(1 << 40)])
def test_token_topk_refuses_a_count_that_is_not_positive(ext, L, B, F, k):
    dev = _dev()
    x = torch.zeros(L, B, F, dtype=torch.bfloat16, device=dev)
    z = lambda n, dt=I32: torch.zeros(n, dtype=dt, device=dev)  # noqa: E731
    with pytest.raises(RuntimeError):
        ext.token_topk_select(x, z((L, F), F32), z((L, F), F32), F, k, z(16, torch.int64), z(B), z(B), z(B, F32), z(4), F)


def _serving_model(fn, tying, dev, L=3, d=64, F=512):
    from crosslayer_coding_b200 import CLTConfig, CrossLayerTranscoder

    torch.manual_seed(0)
    cfg = CLTConfig(num_features=F, num_layers=L, d_model=d, activation_fn=fn, batchtopk_k=9, topk_k=9, jumprelu_threshold=0.1, clt_dtype="bfloat16",
                    decoder_tying=tying)
    model = CrossLayerTranscoder(cfg, device=dev)
    with torch.no_grad():
        for w in model.dec_weight:
            w.uniform_(-0.1, 0.1)
        model.dec_bias.uniform_(-0.5, 0.5)
        model.enc_weight.uniform_(-0.02, 0.02)
    return model


@pytest.mark.parametrize("fn,tying", [("batchtopk", "none"), ("topk", "per_source"), ("jumprelu", "per_target"), ("relu", "none")])
def test_sparse_forward_with_and_without_targets(ext, fn, tying):
    """Without targets only the reconstruction is written; the loss sums of an earlier call with targets survive `encode`; changed
    parameters (biases, thresholds) are seen by the next call."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model(fn, tying, dev)
    B = 200
    sf = SparseForward(model, B)
    x = torch.randn(3, B, 64, device=dev).bfloat16()
    y = torch.randn(3, B, 64, device=dev).bfloat16()
    a = sf.reconstruct(x, y)
    sq = sf.sq_err.clone()
    assert torch.allclose(sq, (a.double() - y.double()).square().sum((1, 2)), rtol=1e-5)
    sf.encode(x)
    assert torch.equal(sf.sq_err, sq)
    b = sf.forward_dict({l: x[l] for l in range(3)})
    for l in range(3):
        assert torch.equal(a[l], b[l])
    with torch.no_grad():
        model.dec_bias.add_(0.25)
    shift = {"none": torch.arange(1, 4), "per_source": torch.arange(1, 4), "per_target": torch.ones(3)}[tying].to(dev).float() * 0.25
    c = sf.reconstruct(x)
    assert torch.allclose(c, a + shift[:, None, None], atol=2e-2)
    if fn == "jumprelu":
        n = sf.num_entries()
        with torch.no_grad():
            model.log_threshold.add_(0.5)
        sf.encode(x)
        assert sf.num_entries() < n
    sf.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32, torch.float64])
@pytest.mark.parametrize("strided", [False, True])
def test_decoder_bias_of_any_type_and_stride(ext, dtype, strided):
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model("jumprelu", "none", dev)
    bias = model.dec_bias.data.to(dtype)
    if strided:
        bias = torch.stack([bias, bias + 1], dim=2)[:, :, 0]
    model.dec_bias.data = bias
    sf = SparseForward(model, 200)
    x = torch.randn(3, 200, 64, device=dev).bfloat16()
    got = sf.reconstruct(x)
    model.dec_bias.data = torch.zeros_like(bias).contiguous().float()
    want = sf.reconstruct(x) + (sf.bias_sel.double() @ bias.double()).float()[:, None]
    assert torch.allclose(got, want, rtol=0, atol=1e-5)  # fp32 sums of a few terms of about one
    sf.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32, torch.float64])
def test_thresholds_are_computed_in_32_bits(ext, dtype):
    """``model.bfloat16()`` turns ``log_threshold`` into a 16-bit parameter; the threshold is its exponential in fp32 all the same."""
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model("jumprelu", "none", dev)
    with torch.no_grad():
        # a fifth to four times the spread of the pre-activations; the exponentials of 16-bit values lie between 16-bit values
        model.log_threshold.data = (3.0 * torch.rand(3, 512, device=dev) - 4.0).to(dtype)
    sf = SparseForward(model, 200)
    x = torch.randn(3, 200, 64, device=dev).bfloat16()
    sf.encode(x)
    sf.check_status()
    theta = model.log_threshold.data.double().exp()
    assert ((sf.theta.double() / theta - 1).abs() <= 2.0 ** -22).all()  # fp32: 2^-24, and the error bound of expf (2 ulp)
    want = torch.where(sf.preact.float() >= model.log_threshold.data.float().exp()[:, None, :], sf.preact.float(), torch.zeros((), device=dev))
    assert torch.equal(sf.activations_dense(), want)


@pytest.mark.parametrize("fn", ["batchtopk", "topk"])
def test_threshold_statistics_match_the_dense_form(ext, fn):
    from crosslayer_coding_b200.models import theta
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model(fn, "none", dev)
    sf = SparseForward(model, 150)
    dense, sparse = theta._new_stats(model), theta._new_stats(model)
    for i in range(3):
        x = torch.randn(3, 150, 64, device=dev).bfloat16()
        theta.accumulate_theta_batch(model, {l: x[l] for l in range(3)}, dense)
        theta.accumulate_theta_batch_sparse(sf, x, sparse)
    sf.check_status()
    assert torch.equal(sparse["batches"], dense["batches"])
    # 16-bit pre-activations of two GEMMs: single elements differ by one rounding (2^-8 relative), a selection by few entries
    for n in ("mean", "std"):
        assert torch.allclose(sparse[n], dense[n], atol=2e-3, rtol=2e-3), n
    assert float((sparse["cnt_min"] != dense["cnt_min"]).float().mean()) < 0.02
    same = sparse["cnt_min"] == dense["cnt_min"]
    assert float(((sparse["sum_min"] - dense["sum_min"]).abs()[same] > 0.05).float().mean()) < 0.02


def test_threshold_statistics_of_any_type_and_stride(ext):
    """The sums may be 64-bit, a view of a wider table, or narrower than the shard: every form gets what the fp32 planes get."""
    from crosslayer_coding_b200.models import theta
    from crosslayer_coding_b200.models.sparse_forward import SparseForward

    dev = _dev()
    model = _serving_model("batchtopk", "none", dev)
    sf = SparseForward(model, 150)
    x = torch.randn(3, 150, 64, device=dev).bfloat16()
    want = theta._new_stats(model)
    theta.accumulate_theta_batch_sparse(sf, x, want)
    names = ("sum_min", "cnt_min", "mean", "std")
    double = {n: t.double() for n, t in theta._new_stats(model).items()}
    table = torch.zeros(4, 3, 1024, device=dev)
    views = {n: table[i][:, 256:768] for i, n in enumerate(names)} | {"batches": torch.zeros(6, device=dev)[::2]}
    narrow = {n: torch.zeros(3, 200, device=dev, dtype=torch.float64) for n in names} | {"batches": torch.zeros((), device=dev)}
    for stats, width in ((double, 512), (views, 512), (narrow, 200)):
        theta.accumulate_theta_batch_sparse(sf, x, stats)
        for n in names:
            assert torch.equal(stats[n].float(), want[n][:, :width]), n
        assert bool((stats["batches"] == 1).all())
    assert float(table[:, :, :256].abs().sum() + table[:, :, 768:].abs().sum()) == 0.0
    sf.check_status()


HYPER = [1e-3, 0.9, 0.999, 1e-8, 0.01, 1 - 0.9 ** 3, 1 - 0.999 ** 3, 1.0, 0.5, 0.0, 1.0]


def _row_update(ext, L, B, d, tying, counts, rows_of=None, dtype=torch.bfloat16, ctl=False, extra=False, seed=0):
    """One call of the decoder sweep against 64 bits: moments, weights, norms and dL/da.  ``counts``: entries per feature (the same
    in every layer); ``rows_of``: target rows per feature of a tensor; ``ctl``: loss scale and clip coefficient; ``extra``: compact
    extra gradients of every third feature's first row; ``seed``: stochastic rounding of the weights."""
    dev = _dev()
    g = torch.Generator().manual_seed(d + tying)
    F = len(counts)
    ent = [(l * F + f, t) for l in range(L) for f, c in enumerate(counts) for t in torch.randperm(B, generator=g)[:c].tolist()]
    col = torch.tensor([e[0] for e in ent], dtype=I32, device=dev)
    tok = torch.tensor([e[1] for e in ent], dtype=I32, device=dev)
    val = torch.randn(len(ent), generator=g).to(dev)
    c = _csr(ext, tok, col, val, B, L * F, F)
    rows = [(rows_of or (lambda s: L - s if tying == 0 else 1))(s) for s in range(L)]
    W = [(torch.randn(F, r, d, generator=g) / 8).to(dtype).to(dev) for r in rows]
    M = [(torch.randn(F, r, d, generator=g) * 0.01).to(dev) for r in rows]
    V = [(torch.rand(F, r, d, generator=g) * 1e-3 + 1e-4).to(dev) for r in rows]
    gs = torch.randn(L, B, d, generator=g).to(dtype).to(dev)
    pen = (torch.rand(L * F, generator=g) * 0.01).to(dev)
    acts = torch.zeros(L, B, F, device=dev, dtype=torch.float64)
    acts[(col // F).long(), tok.long(), (col % F).long()] = val.double()
    control, inv_scale, clip = None, 1.0, 1.0
    if ctl:
        inv_scale, clip = 0.25, 0.625
        control = torch.zeros(16, device=dev)
        control[1], control[2], control[6] = inv_scale, 4.0, clip
    gsc, (lr, b1, b2, eps, wd, bc1, bc2) = HYPER[8] * inv_scale, HYPER[:7]
    xi = xr = None
    if extra:
        n_extra = (L * F + 2) // 3
        xi = torch.full((L * F,), -1, dtype=I32)
        xi[::3] = torch.arange(n_extra, dtype=I32)
        xr = torch.randn(n_extra, d, generator=g).to(dev)
        xi = xi.to(dev)
    want, norm2 = [], []
    dlda = torch.zeros(L, B, F, device=dev, dtype=torch.float64)
    for i in range(L):
        grad = torch.zeros(F, rows[i], d, device=dev, dtype=torch.float64)
        for r in range(rows[i]):
            t = i + r if tying == 0 else i
            for s in ([i] if tying == 0 else range(i + 1)):
                grad[:, r] += gsc * acts[s].t() @ gs[t].double()
                dlda[s] += gsc * gs[t].double() @ W[i][:, r].double().t()
        pc = pen.view(L, F).double()
        grad += (pc[i] if tying == 0 else pc[: i + 1].sum(0))[:, None, None] * W[i].double()
        if extra:
            has = xi[i * F: (i + 1) * F] >= 0
            grad[has, 0] += xr[xi[i * F: (i + 1) * F][has].long()].double()
        grad *= clip
        m = b1 * M[i].double() + (1 - b1) * grad
        v = b2 * V[i].double() + (1 - b2) * grad.square()
        w = W[i].double() * (1 - lr * wd) - lr / bc1 * m / ((v / bc2).sqrt() + eps)
        want.append((w, m, v))
    grad_a = torch.zeros(len(ent), device=dev)
    n2 = torch.zeros(L * F, device=dev)
    status = torch.zeros(4, dtype=I32, device=dev)
    hyper = HYPER[:9] + [float(seed)] + HYPER[10:]
    ext.decoder_rows_adam(W, M, V, L, B, d, F, tying, c["feat_off"], c["fcsr_tok"], c["fcsr_val"], gs, grad_a, pen, n2, None, None, None, hyper, status, xi,
                          xr, control, False, None, None)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    ulp = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11  # half a unit in the last place; all of it when rounded stochastically
    for i in range(L):
        w, m, v = want[i]
        # m, v: fp32 sums of up to 90 * L products of unit size, 2^-24 each (1 - beta is itself rounded to 2^-24 of one, a relative
        # 6e-5 of 0.001); w: one rounding to 16 bits (below 2^-14 fp16 has a fixed spacing of 2^-24)
        assert (M[i].double() - m).abs().max() < 4e-6 * m.abs().max() and (V[i].double() - v).abs().max() < 1e-4 * v.abs().max()
        assert ((W[i].double() - w).abs() <= (2 if seed else 1) * ulp * w.abs() + 1e-7).all()
        # norms of the updated rows, of the stored weights in the per-target layout, before they are rounded in the other: fp32 sums of up to 64
        # squares per thread and a tree over the threads and rows (below 100 additions in a row, 2^-24 each), and in the second case
        # weights that are themselves fp32 results of a few operations
        size = (W[i].double() if tying == 2 else w).square().sum((1, 2))
        assert ((n2.view(L, F)[i].double() - size).abs() <= 1e-5 * size).all()
    order = torch.argsort(col.long() * B + tok.long())
    got_l, got_f, got_t = (col[order] // F).long(), (col[order] % F).long(), tok[order].long()
    assert (grad_a.double() - dlda[got_l, got_t, got_f]).abs().max() < 1e-5 * dlda.abs().max()


COUNTS = [0, 1, 3, 4, 5, 7, 8, 9, 35, 36, 37, 60, 0, 2]


# entry counts around the four staged slots, the batches of four and the 32 a warp fetches at once; d with idle lanes, with four
# and with eight elements per thread
@pytest.mark.parametrize("tying", [0, 2])
@pytest.mark.parametrize("L,B,d", [(3, 90, 64), (2, 90, 520), (4, 70, 768), (2, 60, 1536)])
def test_decoder_row_update(ext, L, B, d, tying):
    _row_update(ext, L, B, d, tying, COUNTS)


# per-target tied rows on both sides of the width at which they change to the row pipeline; more rows than resident CTAs, so that
# every CTA has several, of several tensors (600 and 148 features per tensor: a grid that divides the number of features), features
# with many entries among them
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,d,F", [(3, 256, 600), (5, 264, 600), (12, 512, 148), (2, 1032, 800)])
def test_per_target_rows_dealt_over_the_grid(ext, L, d, F, dtype):
    counts = [0] * F
    for i, n in enumerate([90, 1, 0, 33, 4] * 4):
        counts[(i * 37) % F] = n
    _row_update(ext, L, 90, d, 2, counts, dtype=dtype)


# the forms of the row pipeline with 64 registers (one row per feature up to 512 wide, several rows with short lists up to 640), with
# 80 (1288 to 1408 wide) and without batches (one row of more than 1024), next to the widths and lists that keep batches of four
@pytest.mark.parametrize("opts", [dict(), dict(seed=99), dict(dtype=torch.float16)])
@pytest.mark.parametrize("single,d,short", [(True, 392, False), (True, 512, False), (True, 520, False), (False, 520, True), (False, 640, True), (False, 520, False),
                                            (True, 1032, False), (True, 1400, False), (False, 1400, False), (True, 2048, False)])
def test_decoder_row_update_register_forms(ext, single, d, short, opts):
    _row_update(ext, 3, 90, d, 0, COUNTS + [0] * 100 if short else COUNTS, rows_of=(lambda s: 1) if single else None, **opts)


# one warp per row: every number of 128-element blocks with full and partly filled lanes, more rows than three times the resident
# warps (a stage is refilled), one and several rows per feature, rows of all tensors of a per-target layout
@pytest.mark.parametrize("tying,single", [(0, False), (0, True), (2, True)])
@pytest.mark.parametrize("d", [8, 128, 136, 256, 264, 392, 512])
@pytest.mark.parametrize("opts", [dict(), dict(ctl=True, extra=True, dtype=torch.float16), dict(seed=7)])
def test_decoder_row_update_one_warp_per_row(ext, tying, single, d, opts):
    counts = COUNTS + [1, 0, 2] * (900 if d <= 136 else 700)
    _row_update(ext, 3, 90, d, tying, counts, rows_of=(lambda s: 1) if single else None, **opts)


# rows of more than 256 elements: as many of the resident CTAs as the lists need, from almost empty ones to more than need all of them
@pytest.mark.parametrize("tying,single", [(0, False), (0, True), (2, True)])
@pytest.mark.parametrize("d", [264, 384, 512])
@pytest.mark.parametrize("more", [[0, 0, 0], [2, 1, 2], [7, 5, 9]])
def test_decoder_row_update_by_the_length_of_the_lists(ext, tying, single, d, more):
    _row_update(ext, 2, 90, d, tying, COUNTS + more * 700, rows_of=(lambda s: 1) if single else None)


# what the engine adds to the sweep: loss scale and clip coefficient from the control block, compact extra rows, stochastic rounding
@pytest.mark.parametrize("tying,d", [(0, 264), (2, 200), (2, 264), (2, 1032)])
@pytest.mark.parametrize("opts", [dict(ctl=True), dict(extra=True), dict(seed=1234), dict(ctl=True, extra=True, dtype=torch.float16)])
def test_decoder_row_update_options(ext, tying, d, opts):
    _row_update(ext, 3, 90, d, tying, COUNTS, **opts)


def test_affine_gradients_without_affine_terms(ext):
    """The gradients of the offsets and scales of per-target tied rows are formed whenever their accumulators are given, also while the
    terms themselves are left out (offset 0, scale 1)."""
    dev = _dev()
    L, B, d, F = 3, 40, 520, 16
    g = torch.Generator().manual_seed(5)
    tok, col, val = _entries(g, L, B, F, 200, dev)
    c = _csr(ext, tok, col, val, B, L * F, F)
    W = [(torch.randn(F, 1, d, generator=g) / 8).bfloat16().to(dev) for _ in range(L)]
    M, V = ([torch.zeros(F, 1, d, device=dev) for _ in range(L)] for _ in range(2))
    gs = torch.randn(L, B, d, generator=g).bfloat16().to(dev)
    acts = torch.zeros(L, B, F, device=dev, dtype=torch.float64)
    acts[(col // F).long(), tok.long(), (col % F).long()] = val.double()
    want_off, want_sc = (torch.zeros(L, F, device=dev, dtype=torch.float64) for _ in range(2))
    for t in range(L):
        dots = HYPER[8] * gs[t].double() @ W[t][:, 0].double().t()
        want_off[t] = ((acts[: t + 1] != 0) * dots).sum((0, 1))
        want_sc[t] = (acts[: t + 1] * dots).sum((0, 1))
    d_off, d_sc = torch.zeros(L, F, device=dev), torch.zeros(L, F, device=dev)
    status = torch.zeros(4, dtype=I32, device=dev)
    ext.decoder_rows_adam(W, M, V, L, B, d, F, 2, c["feat_off"], c["fcsr_tok"], c["fcsr_val"], gs, torch.zeros(tok.numel(), device=dev), None, None, None, None,
                          None, HYPER, status, None, None, None, False, d_off, d_sc)
    assert int(status[0]) == 0
    # fp32 sums of some ten thousand products: 2^-24 times the square root of their number, on terms of the size of the result
    assert (d_off.double() - want_off).abs().max() < 1e-5 * want_off.abs().max()
    assert (d_sc.double() - want_sc).abs().max() < 1e-5 * want_sc.abs().max()


def test_refused_sizes_raise(ext):
    """Sizes that an entry point refuses on the host (nothing is launched) come back as an exception with the code, not as the end of
    the process."""
    dev = _dev()
    L, B, F = 2, 4, 8
    off, idx, val = torch.zeros(L * F + 1, dtype=I32, device=dev), torch.zeros(1, dtype=I32, device=dev), torch.zeros(1, device=dev)
    status = torch.zeros(4, dtype=I32, device=dev)

    def rows(d):
        W = [torch.zeros(F, 1, d, device=dev, dtype=torch.bfloat16) for _ in range(L)]
        M, V = ([torch.zeros(F, 1, d, device=dev) for _ in range(L)] for _ in range(2))
        gs = torch.zeros(L, B, d, device=dev, dtype=torch.bfloat16)
        ext.decoder_rows_adam(W, M, V, L, B, d, F, 0, off, idx, val, gs, None, None, None, None, None, None, HYPER, status, None, None, None, False, None, None)

    def decode(d):
        W = [torch.zeros(F, L - s, d, device=dev, dtype=torch.bfloat16) for s in range(L)]
        ext.sparse_decode(W, L, B, d, F, 0, torch.zeros(B + 1, dtype=I32, device=dev), idx, val, None, None, torch.zeros(L, B, d, device=dev), None, None, None,
                          None, None, None, None, 0, [], 0, 0, status)

    for call, d in ((rows, 12), (decode, 12), (decode, 2056)):
        with pytest.raises(RuntimeError, match="failed with code -1"):
            call(d)
    rows(16)
    decode(16)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
