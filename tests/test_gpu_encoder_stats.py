"""Encoder GEMM with the batch statistics in its epilogue: the outputs of the GEMM without them, the statistics of the separate pass, bit
for bit where its additions have a fixed order (rows in at most two chunks)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from crosslayer_coding_b200.ops import ext as e

    return e.load()


def _row_chunks(L, B, F):
    """Chunks of rows that the separate pass splits its sums into; with more than two, its additions have no fixed order."""
    z = 1
    while -(-F // 256) * L * z < 592 and z < 16 and B // (2 * z) >= 128:
        z *= 2
    return z


# below 256 tokens one CTA per tile; whole strips in one round and in several; strips that are left over; a last tile of 1, 9, 44, 232, 256 tokens;
# the end of a chunk of rows inside a tile (2 x 264 and 300 rows); a last strip of 8, 72, 136 features; K below and beyond one ring of stages
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize(
    "L,M,N,K",
    [(2, 200, 264, 64), (2, 256, 256, 64), (1, 257, 72, 8), (1, 300, 520, 136), (3, 528, 1032, 520), (9, 1000, 8200, 128), (75, 265, 2048, 64),
     (6, 1536, 16384, 64), (3, 2100, 32768, 72)],
)
def test_encoder_gemm_stats(ext, dtype, L, M, N, K):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(L + M + N + K)
    x = torch.randn(L, M, K, device=dev, generator=g).to(dtype)
    w = (torch.randn(L, N, K, device=dev, generator=g) / math.sqrt(K)).to(dtype)
    b = (3 * torch.randn(L, N, device=dev, generator=g)).to(dtype)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    nan = float("nan")
    plain, out = (torch.full((L, M, N), nan, device=dev, dtype=dtype) for _ in range(2))
    mean, rstd, mean_p, rstd_p = (torch.full((L, N), nan, device=dev) for _ in range(4))
    assert ext.encoder_gemm_stats(x, w, b, out, mean, rstd, status) >= 1
    ext.encoder_gemm(x, w, b, plain, status, None)
    ext.colstats(plain, mean_p, rstd_p)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    assert torch.equal(out.view(torch.int16), plain.view(torch.int16))
    if _row_chunks(L, M, N) <= 2:
        assert torch.equal(mean, mean_p) and torch.equal(rstd, rstd_p)
    # fp32 sums of M values (the shift keeps them at the size of the spread): M + 16 roundings of 2^-24 of sums below M times the largest value
    of = out.double()
    spread = (of - of[:, :1]).abs().amax(1)
    eps = (M + 16) * 2.0 ** -24
    assert ((mean.double() - of.mean(1)).abs() <= eps * spread + 2.0 ** -23 * of.mean(1).abs()).all()
    var = of.var(1)
    got = (1 / rstd.double() - 1e-6).square()
    assert ((got - var).abs() <= 4 * eps * spread.square() + 2.0 ** -20 * var + 1e-12).all()


def test_encoder_gemm_stats_refuses_other_shapes(ext):
    dev = torch.device("cuda:0")
    x, w = torch.zeros(1, 256, 64, device=dev).bfloat16(), torch.zeros(1, 256, 64, device=dev).bfloat16()
    out, st = torch.zeros(1, 256, 256, device=dev).bfloat16(), torch.zeros(4, dtype=torch.int32, device=dev)
    m = torch.zeros(1, 256, device=dev)
    with pytest.raises(RuntimeError, match="mean/rstd"):
        ext.encoder_gemm_stats(x, w, None, out, m, torch.zeros(1, 128, device=dev), st)
    with pytest.raises(RuntimeError, match="dtype"):
        ext.encoder_gemm_stats(x, w, None, out, m.double(), m, st)


# few strips with many rows, whose tiles would go one after the other on a part of the chip while the rest of it stood idle: no strip is taken whole.  A full
# round of strips and a few more: the few are not.  Rounds that are nearly full: all of them are.
@pytest.mark.parametrize("L,M,N,K,way", [(2, 4100, 2056, 72, "none"), (1, 8192, 2048, 64, "none"), (79, 4100, 256, 8, "full rounds"), (297, 3000, 256, 8, "full rounds"), (3, 4096, 5120, 64, "all")])
def test_encoder_gemm_stats_of_few_strips(ext, L, M, N, K, way):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(M + N)
    x = torch.randn(L, M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(L, N, K, device=dev, generator=g) / math.sqrt(K)).bfloat16()
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    plain, out = (torch.full((L, M, N), float("nan"), device=dev, dtype=torch.bfloat16) for _ in range(2))
    mean, rstd = (torch.full((L, N), float("nan"), device=dev) for _ in range(2))
    kernels = ext.encoder_gemm_stats(x, w, None, out, mean, rstd, status)
    ext.encoder_gemm(x, w, None, plain, status, None)
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and kernels == (1 if way == "all" else 3)  # the pass over the others: sums of row chunks, conversion
    assert torch.equal(out.view(torch.int16), plain.view(torch.int16))
    if _row_chunks(L, M, N) <= 2:
        mean_p, rstd_p = torch.empty_like(mean), torch.empty_like(rstd)
        ext.colstats(plain, mean_p, rstd_p)
        assert torch.equal(mean, mean_p) and torch.equal(rstd, rstd_p)
    of = out.double()
    spread = (of - of[:, :1]).abs().amax(1)
    eps = (M + 16) * 2.0 ** -24  # as above
    assert ((mean.double() - of.mean(1)).abs() <= eps * spread + 2.0 ** -23 * of.mean(1).abs()).all()
    var = of.var(1)
    assert (((1 / rstd.double() - 1e-6).square() - var).abs() <= 4 * eps * spread.square() + 2.0 ** -20 * var + 1e-12).all()


# the GEMM by CTA pairs with and without sums against 64 bits, with tiles of all 256 tokens, and the sums per block of 128 rows of both GEMMs
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,M,N,K", [(1, 4096, 1024, 768), (2, 300, 520, 136), (2, 1025, 264, 520), (3, 200, 136, 72), (1, 128, 8, 8)])
def test_encoder_gemm_forms_against_64_bits(ext, dtype, L, M, N, K):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x = torch.randn(L, M, K, device=dev, generator=g).to(dtype)
    w = (torch.randn(L, N, K, device=dev, generator=g) / math.sqrt(K)).to(dtype)
    b = torch.randn(L, N, device=dev, generator=g).to(dtype)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    want = torch.einsum("lmk,lnk->lmn", x.double(), w.double()) + b.double()[:, None]
    size = torch.einsum("lmk,lnk->lmn", x.double().abs(), w.double().abs()) + b.double().abs()[:, None]
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    mean, rstd = (torch.full((L, N), float("nan"), device=dev) for _ in range(2))
    sums = torch.full((L, (M + 127) // 128, N, 2), float("nan"), device=dev)
    calls = [lambda o: ext.encoder_gemm(x, w, b, o, status, None), lambda o: ext.encoder_gemm_stats(x, w, b, o, mean, rstd, status),
             lambda o: ext.encoder_gemm(x, w, b, o, status, sums)]
    for call in calls:
        out = torch.full((L, M, N), float("nan"), device=dev, dtype=dtype)
        call(out)
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        # an fp32 sum of K products and the bias, then one rounding to 16 bits (fp16: at least 2^-25 apart)
        assert ((out.double() - want).abs() <= 1.01 * half_ulp * want.abs() + (K + 2) * 2.0 ** -23 * size + 2.0 ** -25).all()
    of = torch.nn.functional.pad(out.double(), (0, 0, 0, -M % 128)).view(L, -1, 128, N)
    for got, terms in ((sums[..., 0], of), (sums[..., 1], of.square())):
        assert ((got.double() - terms.sum(2)).abs() <= 130 * 2.0 ** -24 * terms.abs().sum(2)).all()  # 128 additions in fp32


# pairs without sums take more tiles than there are CTAs: many layers of few tiles, whose last one ends in its first or second half of features, in a store of 64, in the
# first or second half of tokens, in a chunk of 64; the same matrices with few layers go one CTA per tile
@pytest.mark.parametrize("L", [80, 3])
@pytest.mark.parametrize("M,N", [(256, 8), (257, 136), (300, 200), (520, 328), (400, 72)])
@pytest.mark.parametrize("K", [8, 72, 520])
def test_encoder_gemm_of_many_small_layers(ext, L, M, N, K):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x = torch.randn(L, M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(L, N, K, device=dev, generator=g) / math.sqrt(K)).bfloat16()
    b = torch.randn(L, N, device=dev, generator=g).bfloat16()
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    out = torch.full((L, M, N), float("nan"), device=dev, dtype=torch.bfloat16)
    ext.encoder_gemm(x, w, b, out, status, None)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    want = torch.einsum("lmk,lnk->lmn", x.double(), w.double()) + b.double()[:, None]
    size = torch.einsum("lmk,lnk->lmn", x.double().abs(), w.double().abs()) + b.double().abs()[:, None]
    assert ((out.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + (K + 2) * 2.0 ** -23 * size).all()  # fp32 sums, one rounding to bf16
