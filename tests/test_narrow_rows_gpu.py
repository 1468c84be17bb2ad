"""The row-wise helpers that take four columns a thread, over rows narrower than a block (several rows a block), as wide, and
wider, with row counts that do not fill the last block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ACT = {None: lambda x: x, "silu": lambda x: x * torch.sigmoid(x), "relu2": lambda x: x.clamp(min=0) ** 2, "sigmoid": torch.sigmoid,
       "tanh": torch.tanh, "softplus": torch.nn.functional.softplus}


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


@pytest.mark.parametrize("cols", [4, 12, 64, 128, 508, 1020, 1024, 1028, 4100])
@pytest.mark.parametrize("n", [1, 3, 65, 257])
def test_rows(n, cols):
    """Bound: an activation and five roundings of float32 (2^-24 each, the activations within 4 units), terms of size up to 40."""
    from rllm_b200.csrc import ops as o
    a, b, s, f = rnd(n, cols, seed=1), rnd(cols, seed=2), rnd(n, seed=3), rnd(n, cols, seed=4)
    gate = rnd(n, cols // 4, seed=5)
    for act, fn in ACT.items():
        out = torch.full((n + 1, cols), float("nan"), device=DEV)
        o.rows_act(a.to(DEV), out[:n], act=act, bias=b.to(DEV), mul=f.to(DEV), mul_act="sigmoid", factor=0.5, row_scale=s.to(DEV))
        want = 0.5 * fn(a.double() * s.double()[:, None] + b.double()) * torch.sigmoid(f.double())
        bound = 16 * 2.0 ** -24 * want.abs() + 2.0 ** -21 * (1 + a.abs() * s.abs()[:, None] + b.abs()) ** 2
        assert bool(((out[:n].cpu().double() - want).abs() <= bound).all()), act
        assert bool(out[n].isnan().all())
    out = torch.empty(n, cols, dtype=torch.bfloat16, device=DEV)
    o.rows_act(a.bfloat16().to(DEV), out, mul=gate.to(DEV), mul_act="tanh", mul_group=4)
    want = a.bfloat16().double() * torch.tanh(gate.double()).repeat_interleave(4, 1)
    assert bool(((out.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
    x, y, e = rnd(n, cols, seed=6), rnd(n, cols, seed=7), rnd(n, cols, seed=8)
    out = torch.full((n + 1, 2 * cols), float("nan"), device=DEV)
    o.cat2_cast(x.to(DEV), y.to(DEV), out[:n], delta=e.to(DEV), delta_scale=0.25)
    assert float((out[:n, :cols].cpu() - (x + 0.25 * e)).abs().max()) < 1e-6
    assert torch.equal(out[:n, cols:].cpu(), y) and bool(out[n].isnan().all())
