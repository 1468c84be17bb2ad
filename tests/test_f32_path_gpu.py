"""The kernels of the float32 path at the sizes where they can go wrong: edges of tiles and classes, few and many rows,
operands that are not aligned, every mask."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


def ops():
    from rllm_b200.csrc import ops as o
    return o


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16, 17, 64, 65, 129])
@pytest.mark.parametrize("n,k", [(1, 1), (33, 7), (64, 256), (70, 260), (257, 513), (1030, 1024)])
def test_products(m, n, k):
    """Every output within the bound of its order of summation (a chain of ceil(k / 256) * 8 terms, then one of 32), the
    same bits whatever the other rows and the alignment of the operands."""
    a, w, base = rnd(m, k, seed=1), rnd(n, k, seed=2), rnd(m, n, seed=3)
    exact, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = (-(-k // 256) * 8 + 33) * U * size + 1e-30
    out = torch.full((m, n), float("nan"), device=DEV)
    ops().gemm_plain(a.to(DEV), w.to(DEV), out)
    assert bool(((out.cpu().double() - exact).abs() <= bound).all())
    acc = base.to(DEV)
    ops().gemm_plain(a.to(DEV), w.to(DEV), acc, accumulate=True)
    assert torch.equal(acc.cpu(), out.cpu() + base)
    # one column and one row further in wider matrices: another alignment, the same sums
    aw, ww = torch.full((m + 1, k + 3), 7.0), torch.full((n + 1, k + 5), 7.0)
    aw[1:, 1:k + 1], ww[1:, 1:k + 1] = a, w
    other = torch.full((m, n + 3), float("nan"), device=DEV)
    ops().gemm_plain(aw.to(DEV)[1:, 1:k + 1], ww.to(DEV)[1:, 1:k + 1], other[:, 1:n + 1])
    assert torch.equal(other[:, 1:n + 1], out) and bool(other[:, 0].isnan().all()) and bool(other[:, n + 1:].isnan().all())
    for r in {0, m // 2, m - 1}:
        alone = torch.empty(1, n, device=DEV)
        ops().gemm_plain(a[r:r + 1].to(DEV), w.to(DEV), alone)
        assert torch.equal(alone[0], out[r])


@pytest.mark.parametrize("T", [1, 6, 40])
def test_products_per_head(T):
    H, m, k = 3, 50, 68
    a, w = rnd(T, H, k, seed=4), rnd(H, m, k, seed=5)
    out = torch.empty(T, H, m, device=DEV)
    ops().head_linear(a.to(DEV), w.to(DEV), out)
    exact = torch.einsum("thk,hmk->thm", a.double(), w.double())
    size = torch.einsum("thk,hmk->thm", a.double().abs(), w.double().abs())
    assert bool(((out.cpu().double() - exact).abs() <= 41 * U * size).all())
