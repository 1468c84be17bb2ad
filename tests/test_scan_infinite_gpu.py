"""An infinite input of the selective scan gives infinities, not NaN, also where the number of states does not fill its lanes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N", [1, 5, 16, 30, 64, 70])
@pytest.mark.parametrize("tokens", [1, 3, 20])
def test_infinite_input(N, tokens):
    from rllm_b200.csrc import ops as o
    inner, taps = 40, 4
    g = torch.Generator().manual_seed(N)
    rnd = lambda *s: torch.rand(*s, generator=g) + 0.1                                   # noqa: E731
    x, xz, low, dtr = rnd(tokens, inner), rnd(tokens, 2 * inner), rnd(tokens, 2 * N), rnd(tokens, inner)
    x[tokens // 2, 7] = float("inf")
    b, A, D = rnd(inner), -rnd(inner, N), rnd(inner)
    state = torch.zeros(1, inner * (N + taps), device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                       # noqa: E731
    for one in ([False, True] if tokens == 1 else [False]):
        out = torch.empty(tokens, inner, device=DEV)
        st = state.clone()
        o.selective_scan(x.to(DEV), xz.to(DEV), low.to(DEV), 0, N, dtr.to(DEV), b.to(DEV), A.to(DEV), D.to(DEV), st, inner * N,
                         i32([0, tokens]), i32([0]), out, 1, inner, N, taps, one_token=one)
        out = out.cpu()
        assert bool(out[tokens // 2:, 7].isinf().all()) and bool((out[tokens // 2:, 7] > 0).all())
        out[:, 7] = 0
        assert bool(out.isfinite().all())
        kept = st[0, :inner * N].view(inner, N).cpu()
        assert bool(kept[7].isinf().all())
