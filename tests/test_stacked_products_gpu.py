"""Products of one shape on inputs of their own in one launch: shares that begin, end and pass over at the end of a matrix, one row to
sixteen, and what goes to the single products instead."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


@pytest.mark.parametrize("m", [1, 3, 8, 9, 16, 17])
@pytest.mark.parametrize("G,n,k", [(4, 4096, 2112), (2, 3000, 4096), (5, 4104, 2048), (3, 8192, 1024), (4, 256, 512), (2, 4096, 2050)])
def test_linear_stack(m, G, n, k):
    if k % 8:
        m = min(m, 3)
    x, w = rnd(G, m, k, seed=1).bfloat16(), (rnd(G, n, k, seed=2) * k ** -0.5).bfloat16()
    base = torch.full((G + 1, m, n), float("nan"), device=DEV)
    out = ops().linear_stack(x.to(DEV), w.to(DEV), base[:G])
    ops().check_device_errors()
    f = x.double() @ w.double().transpose(1, 2)
    size = x.double().abs() @ w.double().abs().transpose(1, 2)
    assert bool(((out.cpu().double() - f).abs() <= k * 2.0 ** -24 * size).all())
    assert bool(base[G].isnan().all())


@pytest.mark.parametrize("grid", [8, 9, 12, 17, 31, 32])
@pytest.mark.parametrize("m", [2, 11])
def test_where_the_shares_pass_over(grid, m):
    """32 granules in four matrices: shares of four granules and fewer, cut in every place."""
    import ctypes
    o, G, n, k = ops(), 4, 64, 256
    x, w = rnd(G, m, k, seed=3).bfloat16().to(DEV), rnd(G, n, k, seed=4).bfloat16().to(DEV)
    out = torch.full((G, m, n), float("nan"), device=DEV)
    c = ctypes.c_int
    st = o._lib("stream").rllm_gemv_stream_stack(o._ptr(w), o._ptr(x), o._ptr(out), c(m), c(n), c(k), c(G), c(grid), c(3),
                                                 o._ptr(o.error_word(DEV)), o._stream())
    assert st == 0
    o.check_device_errors()
    want = x.cpu().double() @ w.cpu().double().transpose(1, 2)
    size = x.cpu().double().abs() @ w.cpu().double().abs().transpose(1, 2)
    assert bool(((out.cpu().double() - want).abs() <= k * 2.0 ** -24 * size).all())
    assert o._lib("stream").rllm_gemv_stream_stack(o._ptr(w), o._ptr(x), o._ptr(out), c(m), c(n), c(k), c(G), c(3), c(3),
                                                   o._ptr(o.error_word(DEV)), o._stream()) != 0      # a share longer than a matrix
