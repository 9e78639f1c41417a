"""Global top-k that keeps about one element in 130: the tracked range fits its queue, so that no full-range pass runs, and the selection is exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,B,F,k", [(4, 1500, 2048, 62), (3, 33, 4104, 90), (2, 260, 24, 1)])
def test_dense_selection_stays_in_the_tracked_range(L, B, F, k):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from crosslayer_coding_b200.ops import ext as e
    from crosslayer_coding_b200.training.fused_engine import histogram_range

    ext, dev, i32, f32 = e.load(), torch.device("cuda:0"), torch.int32, torch.float32
    g = torch.Generator(device=dev).manual_seed(B + k)
    k_total = k * B
    key_lo, shift = histogram_range(k_total, B * L * F)
    assert key_lo != 0
    sel = torch.tensor([key_lo, shift], dtype=torch.int64, device=dev)
    pool = torch.empty(4, min(B * L * F, 10 * k_total + (1 << 16)), dtype=i32, device=dev)
    for call in range(3):
        x = (torch.randn(L, B, F, device=dev, generator=g) * (0.5 + torch.rand(L, 1, F, device=dev, generator=g))).bfloat16()
        mean, rstd = torch.empty(L, F, device=dev), torch.empty(L, F, device=dev)
        ext.colstats(x, mean, rstd)
        hist, ctl, status = torch.zeros(2 * 8192 + 32, dtype=i32, device=dev), torch.zeros(16, dtype=torch.int64, device=dev), torch.zeros(4, dtype=i32, device=dev)
        ent = [torch.empty(k_total, dtype=t, device=dev) for t in (i32, i32, f32)]
        cand = [torch.empty(1 << 20, dtype=t, device=dev) for t in (i32, i32, i32, f32)]
        ext.batchtopk_select(x, mean, rstd, F, F, 0, F, k_total, key_lo, shift, hist, ctl, *ent, *cand, status, 1, 0, [], [], 0, 0, sel, pool)
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and int(ctl[3]) == k_total
        assert call == 0 or int(ctl[10]) == 0  # no full-range pass once the range has been found
        z = ((x.float() - mean[:, None]) * rstd[:, None]).permute(1, 0, 2).reshape(-1)  # token-major: the lowest flat index wins a tie
        want = torch.zeros(B * L * F, dtype=torch.bool, device=dev)
        want[torch.sort(z, descending=True, stable=True).indices[:k_total]] = True
        got = torch.zeros_like(want)
        got[ent[0].long() * L * F + ent[1].long()] = True
        assert torch.equal(got, want)


# more densely, up to the one in seven that a tracked range still takes: full tiles of 2048 columns in 16 and 8 rows per CTA; a few columns, whose tiles hold
# all pieces with many rows; more tokens than a grid has rows of CTAs with 32 each, and the same without a tracked range
@pytest.mark.parametrize("L,B,F,k", [(2, 700, 2048, 60), (2, 700, 2048, 136), (3, 300, 4104, 1000), (2, 519, 2048, 512), (2, 1000, 72, 10), (1, 2100000, 8, 1),
                                     (1, 2100000, 8, 2), (3, 300, 2056, 1300)])
def test_denser_selections_stay_in_the_tracked_range(L, B, F, k):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from crosslayer_coding_b200.ops import ext as e
    from crosslayer_coding_b200.training.fused_engine import histogram_range

    ext, dev, i32, f32 = e.load(), torch.device("cuda:0"), torch.int32, torch.float32
    g = torch.Generator(device=dev).manual_seed(B + k)
    k_total = k * B
    key_lo, shift = histogram_range(k_total, B * L * F)
    sel = torch.tensor([key_lo, shift], dtype=torch.int64, device=dev) if key_lo else None
    pool = torch.empty(4, min(B * L * F, 10 * k_total + (1 << 16)), dtype=i32, device=dev) if key_lo else None
    for call in range(3):
        x = (torch.randn(L, B, F, device=dev, generator=g) * (0.5 + torch.rand(L, 1, F, device=dev, generator=g))).bfloat16()
        mean, rstd = torch.empty(L, F, device=dev), torch.empty(L, F, device=dev)
        ext.colstats(x, mean, rstd)
        hist, ctl, status = torch.zeros(2 * 8192 + 32, dtype=i32, device=dev), torch.zeros(16, dtype=torch.int64, device=dev), torch.zeros(4, dtype=i32, device=dev)
        ent = [torch.empty(k_total, dtype=t, device=dev) for t in (i32, i32, f32)]
        cand = [torch.empty(1 << 20, dtype=t, device=dev) for t in (i32, i32, i32, f32)]
        ext.batchtopk_select(x, mean, rstd, F, F, 0, F, k_total, key_lo, shift, hist, ctl, *ent, *cand, status, 1, 0, [], [], 0, 0, sel, pool)
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and int(ctl[3]) == k_total
        assert call == 0 or not key_lo or int(ctl[10]) == 0
        z = ((x.float() - mean[:, None]) * rstd[:, None]).permute(1, 0, 2).reshape(-1)  # token-major: the lowest flat index wins a tie
        want = torch.zeros(B * L * F, dtype=torch.bool, device=dev)
        want[torch.sort(z, descending=True, stable=True).indices[:k_total]] = True
        got = torch.zeros_like(want)
        got[ent[0].long() * L * F + ent[1].long()] = True
        assert torch.equal(got, want)
