"""Threshold-gradient GEMM by CTA pairs: tile edges and decoder layouts against a dense fp64 restatement."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from crosslayer_coding_b200.ops import ext as e

    return e.load()


# one CTA per tile (1 and 3 times 128 rows) and pairs: a second CTA with 2 rows, with none (640), a last tile of one row; the last feature tile with 8
# columns and with one CTA's half empty; more tiles than pairs
@pytest.mark.parametrize("tying", [0, 1, 2])
@pytest.mark.parametrize("L,B,F,d", [(2, 100, 264, 72), (2, 130, 256, 64), (3, 384, 136, 64), (2, 640, 520, 136), (1, 257, 8, 8), (4, 1025, 6152, 64)])
def test_theta_grad_gemm_tiles(ext, tying, L, B, F, d):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(B + F + d + tying)
    gs = (torch.randn(L, B, d, device=dev, generator=g) * 0.1).bfloat16()
    rows = [L - s if tying == 0 else 1 for s in range(L)]
    ws = [(torch.randn(F, r, d, device=dev, generator=g) * 0.2).bfloat16() for r in rows]
    x = (torch.randn(L, B, F, device=dev, generator=g) * 0.6).bfloat16()
    theta = torch.rand(L, F, device=dev, generator=g) * 0.5 + 0.05
    S1, S2 = torch.zeros(L, F, device=dev), torch.zeros(L, F, device=dev)
    status = torch.zeros(4, dtype=torch.int32, device=dev)
    cum = gs.double().flip(0).cumsum(0).flip(0).bfloat16().contiguous()
    ext.theta_grad_gemm(gs, ws, x, theta, 1.0, S1, S2, status, tying, cum if tying == 1 else None)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    for s in range(L):
        if tying == 1:
            G, size = cum[s].double() @ ws[s][:, 0].double().t(), cum[s].double().abs() @ ws[s][:, 0].double().abs().t()
        else:
            G = size = 0
            for t in range(s, L):
                w = (ws[s][:, t - s] if tying == 0 else ws[t][:, 0]).double()
                G, size = G + gs[t].double() @ w.t(), size + gs[t].double().abs() @ w.abs().t()
        wx = x[s].double() * ((x[s].float() - theta[s]).abs() <= 0.5)
        # fp32 sums of (L - s) d products and of B rows: 2^-24 for each of their roundings, on the sum of the sizes
        eps = (L * d + B + 8) * 2.0 ** -24
        assert ((S2[s].double() - wx.sum(0)).abs() <= eps * wx.abs().sum(0) + 1e-30).all()
        assert ((S1[s].double() - (wx * G).sum(0)).abs() <= eps * (wx.abs() * size).sum(0) + 1e-30).all()
