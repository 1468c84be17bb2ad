"""The norms of whole rows that keep a row in registers: every number of columns a thread holds, the longest rows, delta and rows
of either alignment, rows of which several groups of warps add their sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


def close(got, want, bits):
    """A few roundings of float32 on the way, the sum of squares in any order (its relative error is halved by the root), and
    one rounding to `bits` bits at the end."""
    bound = (want.abs() * (2.0 ** -bits + 24 * 2.0 ** -24) + 1e-30)
    assert bool(((got.cpu().double() - want).abs() <= bound).all())


@pytest.mark.parametrize("n", [1, 130])
@pytest.mark.parametrize("d", [4, 8, 32, 252, 1024, 1028, 2048, 4092, 4096, 4100, 8192, 8196, 12288])
@pytest.mark.parametrize("low", [torch.float32, torch.bfloat16])
def test_norm_rows(n, d, low):
    a, x, w = rnd(n, d, seed=1), rnd(n, d, seed=2), rnd(d, seed=3)
    unit = a.double() / torch.sqrt((a.double() ** 2).mean(1, keepdim=True) + 1e-6) * w.double()
    xs, out = x.to(DEV), torch.full((n, d + 4), float("nan"), dtype=low, device=DEV)
    ops().norm_rows(a.to(DEV), w.to(DEV), 1e-6, x=xs, add=True, low=out[:, :d])
    total = x.double() + unit
    assert bool(((xs.cpu().double() - total).abs() <= (x.double().abs() + unit.abs()) * 24 * 2.0 ** -24 + 1e-30).all())
    close(out[:, :d], xs.cpu().double(), 8 if low is torch.bfloat16 else 24)
    assert bool(out[:, d:].isnan().all())
    alone = torch.empty(n, d, dtype=low, device=DEV)
    ops().norm_rows(a.to(DEV), None, 1e-6, low=alone)
    close(alone, a.double() / torch.sqrt((a.double() ** 2).mean(1, keepdim=True) + 1e-6), 8 if low is torch.bfloat16 else 24)
    own = a.to(DEV)
    ops().norm_rows(own, w.to(DEV), 1e-6, x=own)                      # the rows are the stream itself
    close(own, unit, 24)


@pytest.mark.parametrize("n,d", [(1, 4), (8, 252), (127, 1024), (8, 2048), (130, 2048), (1, 4096), (130, 4096), (127, 8192), (130, 8192),
                                 (1, 8196), (130, 12288)])
def test_a_row_is_joined_in_one_rounding(n, d):
    """Bit for bit, in every form that reads four columns at a time: v * (rs * w) + x with one rounding behind the product rs * w.
    The rows are whole numbers, so that their sum of squares is exact in any order; the sum in 64 bits of a 48-bit product is
    rounded twice, which matters in one of 2^29 cases."""
    a = torch.randint(-6, 7, (n, d), generator=torch.Generator().manual_seed(7)).float()
    a[:, 0] = 3.0
    x, w = rnd(n, d, seed=8), rnd(d, seed=9)
    xs, low = x.to(DEV), torch.empty(n, d, dtype=torch.bfloat16, device=DEV)
    ops().norm_rows(a.to(DEV), w.to(DEV), 1e-6, x=xs, add=True, low=low)
    rs = 1.0 / torch.sqrt((a.double() ** 2).sum(1, keepdim=True).float() / torch.tensor(float(d)) + torch.tensor(1e-6))
    want = (a.double() * (rs * w).double() + x.double()).float()
    assert torch.equal(xs.cpu(), want) and torch.equal(low.cpu(), want.bfloat16())


@pytest.mark.parametrize("n", [1, 9, 130])
@pytest.mark.parametrize("d", [4, 1024, 1028, 2052, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("dt,shift", [(torch.float32, 0), (torch.float32, 1), (torch.bfloat16, 0), (torch.bfloat16, 1)])
def test_add_rms_norm(n, d, dt, shift):
    """shift: the sublayer's output starts one entry behind an aligned address."""
    x, delta, w = rnd(n, d, seed=4), rnd(n, d, seed=5).to(dt), rnd(d, seed=6)
    base = torch.zeros(n * d + 1, dtype=dt, device=DEV)
    moved = base[shift:shift + n * d].view(n, d)
    moved.copy_(delta)
    total = x.double() + 0.5 * delta.double()
    unit = total / torch.sqrt((total ** 2).mean(1, keepdim=True) + 1e-5) * w.double()
    for out_dt, bits in ((torch.float32, 24), (torch.bfloat16, 8)):
        xs, out = x.to(DEV), torch.empty(n, d, dtype=out_dt, device=DEV)
        ops().add_rms_norm(xs, moved, w.to(DEV), out, 1e-5, delta_scale=0.5)
        size = x.double().abs() + 0.5 * delta.double().abs()
        assert bool(((xs.cpu().double() - total).abs() <= size * 2.0 ** -23 + 1e-30).all())
        exact = xs.cpu().double()
        close(out, exact / torch.sqrt((exact ** 2).mean(1, keepdim=True) + 1e-5) * w.double(), bits)
    rows = torch.tensor([n - 1, 0], dtype=torch.int32, device=DEV)
    kept, out = x.to(DEV), torch.empty(2, d, device=DEV)
    ops().add_rms_norm(kept, moved, w.to(DEV), out, 1e-5, rows=rows, write_x=False, delta_scale=0.5)
    assert torch.equal(kept.cpu(), x)
    assert bool(((out.cpu().double() - unit[[n - 1, 0]]).abs() <= (unit[[n - 1, 0]].abs() + 1) * 1e-5).all())


def odd_rows(n, d):
    """Rows with an infinity, with a NaN, with a square beyond float32, and ordinary ones; their weights."""
    a = rnd(n, d, seed=10)
    a[0, d // 2], a[1, d - 1], a[2, 0] = float("inf"), float("nan"), 3e20
    return a, rnd(d, seed=11)


def formula(a, w, eps=1e-6):
    return a * (1.0 / torch.sqrt((a * a).sum(1, keepdim=True) / a.shape[1] + eps)) * w


def alike(got, want, bits):
    """NaN where the formula has it (an infinity times 0 too), 0 beside an infinity or a square beyond the range."""
    got = got.cpu().double()
    assert torch.equal(got.isnan(), want.isnan())
    ok = ~want.isnan()
    assert bool(((got - want.double()).abs() <= want.double().abs() * (2.0 ** -bits + 64 * 2.0 ** -24) + 1e-30)[ok].all())


@pytest.mark.parametrize("n", [4, 130])
@pytest.mark.parametrize("d", [64, 1024, 4096, 8192])
def test_infinities_and_nans_stay_in_their_rows(n, d):
    """float32's own rules: the sum of squares of an ordinary row is short of 64 roundings of its value by far (any order)."""
    a, w = odd_rows(n, d)
    want = formula(a, w)
    for low, bits in ((torch.float32, 24), (torch.bfloat16, 8)):
        out = torch.empty(n, d, dtype=low, device=DEV)
        ops().norm_rows(a.to(DEV), w.to(DEV), 1e-6, low=out)
        alike(out, want, bits)
        ops().add_rms_norm(a.to(DEV), None, w.to(DEV), out, 1e-6)
        alike(out, want, bits)
    stream = torch.zeros(n, d, device=DEV)
    ops().norm_rows(a.to(DEV), w.to(DEV), 1e-6, x=stream, add=True)
    alike(stream, want, 24)
    # the same columns as the query row of a projection; keys and values are ordinary
    G, dk, bs = 1, 64, 8
    H = d // dk
    other = rnd(n, 2 * dk, seed=12)
    q = torch.empty(n, d, device=DEV)
    kc, vc = (torch.zeros(n // bs + 1, G, bs, dk, device=DEV) for _ in range(2))
    ops().qkv_rownorm_store(torch.cat([a, other], 1).to(DEV), None, w.to(DEV), w[:dk].contiguous().to(DEV),
                            torch.arange(n, dtype=torch.int32, device=DEV), q, kc, vc, H, G, dk, dk, bs, 1e-6)
    alike(q, want, 24)
    alike(kc.view(-1, dk)[:n], formula(other[:, :dk], w[:dk]), 24)
    assert torch.equal(vc.view(-1, dk)[:n].cpu(), other[:, dk:])


@pytest.mark.parametrize("n", [1, 130])
@pytest.mark.parametrize("d", [1024, 2052, 4096, 8192])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_a_delta_that_begins_anywhere(n, d, dt, shift):
    """The same kernel, and so the same bits, as at an aligned address."""
    x, delta, w = rnd(n, d, seed=13).to(DEV), rnd(n, d, seed=14).to(dt).to(DEV), rnd(d, seed=15).to(DEV)
    moved = torch.zeros(n * d + 4, dtype=dt, device=DEV)[shift:shift + n * d].view(n, d)
    moved.copy_(delta)
    got = []
    for t in (delta, moved):
        xs, out = x.clone(), torch.empty(n, d, device=DEV)
        ops().add_rms_norm(xs, t, w, out, 1e-5, delta_scale=0.5)
        got.append((xs, out))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("n", [1, 130])
@pytest.mark.parametrize("H,G,dk", [(8, 2, 64), (32, 8, 128)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_projection_weights_that_begin_anywhere(n, H, G, dk, dt, which):
    """Bias, query norm or key norm one entry behind an aligned address: the same bits as with all of them aligned."""
    wq, wk, bs = H * dk, G * dk, 8
    rows = rnd(n, wq + 2 * wk, seed=16).to(DEV)
    weights = [rnd(k, seed=17 + i).to(DEV) for i, k in enumerate((wq + 2 * wk, wq, wk))]
    moved = list(weights)
    moved[which] = torch.cat([torch.zeros(1, device=DEV), weights[which]])[1:]
    slots = torch.arange(n, dtype=torch.int32, device=DEV)
    got = []
    for bias, qn, kn in (weights, moved):
        q = torch.empty(n, wq, dtype=dt, device=DEV)
        kc, vc = (torch.zeros(n // bs + 1, G, bs, dk, dtype=dt, device=DEV) for _ in range(2))
        ops().qkv_rownorm_store(rows, bias, qn, kn, slots, q, kc, vc, H, G, dk, dk, bs, 1e-5)
        got.append((q, kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*got))
