"""float32 products whose k makes the odd cases of the order of summation: less than a run, runs of one class each (k up to 256),
an odd number of runs a class, and the row counts at which another tile is taken."""
import pytest
import torch

from test_f32_path_gpu import DEV, U, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [3, 8, 16, 20, 32, 33, 40, 64, 136, 256, 264, 777, 1030])
@pytest.mark.parametrize("n", [5, 300, 9600])
def test_small_k(n, k):
    """The bound of the order (a chain of ceil(k / 256) * 8 terms, then one of 32), and the same bits for a row alone, among 16 (the
    streaming kernel), among 17 to 64 and among more."""
    a, w = rnd(150, k, seed=1), rnd(n, k, seed=2)
    exact, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = (-(-k // 256) * 8 + 33) * U * size + 1e-30
    got = {}
    for m in (1, 16, 17, 64, 65, 150):
        out = torch.full((m, n), float("nan"), device=DEV)
        ops().gemm_plain(a[:m].to(DEV), w.to(DEV), out)
        got[m] = out.cpu()
        assert bool(((got[m].double() - exact[:m]).abs() <= bound[:m]).all()), m
    for m in (1, 16, 17, 64, 65):
        assert torch.equal(got[m], got[150][:m]), m
