"""Row-wise helpers: the kernels that take four columns a thread against the ones that take any shape (same arithmetic: the
same bits, but for the norm's sums, which are added in another order)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


def wide(t, pad):
    """The same values with `pad` columns more to the row (another stride; an odd one takes the plain kernel)."""
    w = torch.full((t.shape[0], t.shape[1] + pad), 9.0, dtype=t.dtype)
    w[:, :t.shape[1]] = t
    return w.to(DEV)[:, :t.shape[1]]


@pytest.mark.parametrize("n,cols", [(1, 4), (3, 1024), (130, 1028), (2, 4096)])
@pytest.mark.parametrize("src,dst", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("group", [0, 1, 4])
def test_rows_act(n, cols, src, dst, group):
    a, bias = rnd(n, cols, seed=1).to(src), rnd(cols, seed=2).to(DEV)
    mul = rnd(n, cols // group, seed=3) if group else None
    outs = []
    for pad in (4, 3):
        out = torch.zeros(n, cols, dtype=dst, device=DEV)
        kw = dict(mul=wide(mul, pad), mul_act="sigmoid") if group else {}
        if group > 1:
            kw["mul_group"] = group
        ops().rows_act(wide(a, pad), out, act="silu", bias=bias, **kw)
        outs.append(out)
    assert torch.equal(*outs)


@pytest.mark.parametrize("n,d", [(1, 4), (3, 1024), (129, 1028)])
def test_axpby_cat2(n, d):
    o = ops()
    x, y, e = (rnd(n, d, seed=s).to(DEV) for s in (1, 2, 3))
    off = lambda t: torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(n, d)             # noqa: E731  (not on 16 bytes)
    outs = [o.axpby(0.7, f(x), -0.3, f(y), torch.empty(n, d, device=DEV)) for f in (lambda t: t, off)]
    assert torch.equal(*outs)
    for dt in (torch.float32, torch.bfloat16):
        for delta in (None, e, e.bfloat16()):
            outs = []
            for f in (lambda t: t, off):
                out = torch.empty(n, 2 * d, dtype=dt, device=DEV)
                o.cat2_cast(f(x), f(y), out, *(() if delta is None else (delta, 0.5)))
                outs.append(out)
            assert torch.equal(*outs)
            want = torch.cat([x if delta is None else x + 0.5 * delta.float(), y], 1)
            assert float((outs[0].float() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("n", [1, 5, 130])
@pytest.mark.parametrize("H,G,dk,dv", [(4, 1, 64, 64), (32, 8, 128, 128), (3, 3, 20, 36)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_qkv_rownorm_store(n, H, G, dk, dv, dt):
    """Aligned rows against rows of an odd stride; the two kernels add the squares in different orders, at most (H dk) / 4
    terms each: the normed values agree to 2^-24 times that, and to one rounding of the stored type."""
    bs, pages = 16, -(-n // 16) + 1
    wq, wk, wv = H * dk, G * dk, G * dv
    qkv, bias = rnd(n, wq + wk + wv, seed=1), rnd(wq + wk + wv, seed=2).to(DEV)
    qw, kw = rnd(wq, seed=3).to(DEV), rnd(wk, seed=4).to(DEV)
    slots = torch.randperm(pages * bs, generator=torch.Generator().manual_seed(5))[:n].int()
    slots[0] = -1 if n > 1 else slots[0]
    outs = []
    for pad in (4, 3):
        q = torch.zeros(n, wq, dtype=dt, device=DEV)
        kc, vc = torch.zeros(pages, G, bs, dk, dtype=dt, device=DEV), torch.zeros(pages, G, bs, dv, dtype=dt, device=DEV)
        ops().qkv_rownorm_store(wide(qkv, pad), bias, qw, kw, slots.to(DEV), q, kc, vc, H, G, dk, dv, bs, 1e-6)
        outs.append((q, kc, vc))
    eps = 2.0 ** -24 * (8 + wq / 4) + (2.0 ** -8 if dt == torch.bfloat16 else 0.0)
    for a, b in zip(*outs):
        assert bool(((a.double() - b.double()).abs() <= eps * b.double().abs()).all())
    assert torch.equal(outs[0][2], outs[1][2])
