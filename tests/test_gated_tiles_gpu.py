"""The gated product of more than 64 rows in every width of tile: rows, features and K at the edges of tiles, rows that leave whole
warps without one, no more tiles than SMs and more, both gated forms, and the rule that chooses."""
import pytest
import torch

DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


def gated(f, F, glu):
    limit, alpha, shift = glu or (0.0, 1.0, 0.0)
    g, u = f[:, :F], f[:, F:]
    if limit:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(alpha * g) * (u + shift)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [64, 128, 256, 2])
@pytest.mark.parametrize("m", [65, 96, 127, 128, 129, 161, 300])
@pytest.mark.parametrize("F,k", [(32, 64), (100, 200), (129, 520), (4800, 72)])
def test_gated_tiles(tile, m, F, k):
    gen = torch.Generator().manual_seed(m * 7 + F)
    a = torch.randn(m, k, generator=gen).bfloat16()
    w = (2.0 * torch.randn(2 * F, k, generator=gen) * k ** -0.5).bfloat16()
    f = a.double() @ w.double().t()
    for glu in (None, (2.0, 1.702, 1.0)):
        want = gated(f, F, glu)
        for dt, rel in ((torch.float32, 2e-5), (torch.bfloat16, 2.0 ** -8)):
            base = torch.full((m + 1, F + 8 - F % 8), float("nan"), dtype=dt, device=DEV)
            out = base[:m, :F]
            args = (a.to(DEV), w.to(DEV), out, ops().EPI_SWIGLU)
            if tile == 2:
                ops().gemm_tc2(*args, up_row_offset=F, glu=glu)
            else:
                ops().gemm_tc(*args, up_row_offset=F, glu=glu, tile=tile)
            ops().check_device_errors()
            # a rounding of the result, and float32 sums of k products of size about 2 (a gate of size about 2 times an up row)
            assert bool(((out.cpu().double() - want).abs() <= want.abs() * rel + 40 * k * 2.0 ** -24).all())
            assert bool(base[m].isnan().all()) and bool(base[:, F:].isnan().all())


@pytest.mark.gpu
@pytest.mark.parametrize("tile,m,F,k", [(64, 900, 4800, 520), (128, 900, 4800, 520), (64, 333, 6400, 1024), (128, 2048, 3072, 1024),
                                        (256, 2048, 3072, 1024)])
def test_three_tiles_a_cta_and_more(tile, m, F, k):
    """Both accumulators and every stage of the ring are used again: at least three tiles a CTA, more blocks of K than stages, and
    in the last row of tiles warps without a row."""
    a = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).bfloat16()
    w = (2.0 * torch.randn(2 * F, k, generator=torch.Generator().manual_seed(F)) * k ** -0.5).bfloat16()
    ctas = ops().sm_count(torch.device(DEV)) * (1 if tile == 256 else 2)
    assert -(-m // 128) * -(-F // (tile // 2)) > 2 * ctas and k > 8 * 64
    want = gated(a.double() @ w.double().t(), F, None)
    for dt, rel in ((torch.float32, 2e-5), (torch.bfloat16, 2.0 ** -8)):
        base = torch.full((m + 1, F + 8), float("nan"), dtype=dt, device=DEV)
        ops().gemm_tc(a.to(DEV), w.to(DEV), base[:m, :F], ops().EPI_SWIGLU, up_row_offset=F, tile=tile)
        ops().check_device_errors()
        # as above
        assert bool(((base[:m, :F].cpu().double() - want).abs() <= want.abs() * rel + 40 * k * 2.0 ** -24).all())
        assert bool(base[m].isnan().all()) and bool(base[:, F:].isnan().all())


def test_the_rule():
    tile = ops()._gated_tile
    assert [tile(m, 3072, 1024) for m in (65, 128, 384, 385, 512, 4096)] == [64, 64, 64, 128, 128, 128]
    assert [tile(m, 12288, 4096) for m in (65, 128, 129, 256, 257, 384, 512)] == [128, 128, 2, 2, 256, 256, 2]
    assert tile(77, 25600, 5120) in (256, 2) and tile(300, 6144, 2048) == 128
