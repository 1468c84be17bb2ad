"""The recurrent kernels of decode steps against the general ones (the same sums: the same bits), and the kernels that take
four columns a thread against those that take any shape."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def layout(q_lens):
    cu = [0]
    for q in q_lens:
        cu.append(cu[-1] + q)
    return i32(cu), i32([r for r, q in enumerate(q_lens) for _ in range(q)]), i32([len(q_lens) + 1 - r for r in range(len(q_lens))])


@pytest.mark.parametrize("H,D", [(3, 32), (5, 20), (2, 64), (3, 100), (1, 256)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_wkv_one_token(H, D, dt):
    o = ops()
    R, width = 5, 48
    cu, _, slots = layout([1] * R)
    r, k, v, w, g = ((0.5 * rnd(R, H * D, seed=s)).to(DEV) for s in range(5))
    w0, u, nw = (rnd(H * D, seed=s).to(DEV) for s in (6, 7, 8))
    h = rnd(R, width, seed=9).to(dt).to(DEV)
    off = o.wkv_state_floats(H, D)
    state = rnd(R + 2, off + width, seed=10).to(DEV)
    got = []
    for one in (False, True):
        st, out = state.clone(), torch.empty(R, H * D, dtype=dt, device=DEV)
        o.wkv(r, k, v, w, g, w0, u, nw, 1e-6, st, off, h, cu, slots, out, R, H, D, one_token=one)
        got.append((out, st))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool(got[0][0].float().isfinite().all()) and not torch.equal(got[1][1], state)


@pytest.mark.parametrize("inner,N,taps", [(64, 16, 4), (40, 5, 3), (33, 70, 2), (100, 256, 1)])
def test_scan_one_token(inner, N, taps):
    o = ops()
    R = 4
    cu, _, slots = layout([1] * R)
    x, xz, low, dtr = rnd(R, inner, seed=1).to(DEV), rnd(R, 2 * inner, seed=2).to(DEV), rnd(R, 3 + 2 * N, seed=3).to(DEV), rnd(R, inner, seed=4).to(DEV)
    b, A, D = rnd(inner, seed=5).to(DEV), -rnd(inner, N, seed=6).abs().to(DEV), rnd(inner, seed=7).to(DEV)
    state = rnd(R + 2, inner * (N + taps), seed=8).to(DEV)
    got = []
    for one in (False, True):
        st, out = state.clone(), torch.empty(R, inner, device=DEV)
        o.selective_scan(x, xz, low, 3, 3 + N, dtr, b, A, D, st, inner * N, cu, slots, out, R, inner, N, taps, one_token=one)
        got.append((out, st))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and not torch.equal(got[1][1], state)


@pytest.mark.parametrize("q_lens", [[1], [1, 1, 1], [2, 1, 3, 40, 4], [700, 1, 90]])
@pytest.mark.parametrize("cols", [4, 516, 8192])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_rows_of_four(q_lens, cols, dt):
    """Requests that begin anywhere in a thread's run of tokens.  (An odd row stride, or a base off 16 bytes, takes the plain
    kernels; a rounding of the stored type or of float32 apart, since the compiler may fuse differently.)"""
    o = ops()
    n, (cu, seq, slots) = sum(q_lens), layout(q_lens)
    wide = rnd(n, 2 * cols + 3, seed=1).to(DEV)
    w, b, state = rnd(cols, 4, seed=2).to(DEV), rnd(cols, seed=3).to(DEV), rnd(len(q_lens) + 2, 5 * cols, seed=4).to(DEV)
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -22
    got = []
    for xz in (wide[:, :2 * cols].contiguous(), wide[:, :2 * cols]):
        out = torch.empty(n, cols, dtype=dt, device=DEV)
        o.conv_silu(xz, w, b, state, cols, seq, cu, slots, out, cols)
        got.append(out.double())
    assert float((got[0] - got[1]).abs().max()) <= 2 * eps * float(got[1].abs().max())
    h, mu = rnd(n, cols, seed=5).to(dt).to(DEV), rnd(5, cols, seed=6).sigmoid()
    off = torch.cat([torch.zeros(1), mu.reshape(-1)]).to(DEV)[1:].view(5, cols)
    got = []
    for m in (mu.to(DEV), off):
        out = torch.empty(5, n, cols, dtype=dt, device=DEV)
        o.token_shift(h, m, state, 4 * cols, seq, cu, slots, out)
        got.append(out.double())
    assert float((got[0] - got[1]).abs().max()) <= 2 * eps * float(got[1].abs().max())
