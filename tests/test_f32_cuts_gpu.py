"""float32 attention gives a token the same bits however its prompt is cut into portions, and treats infinite scores and values as
the plain kernel does."""
import pytest
import torch

from test_f32_path_gpu import DEV, Step, attend64, ops, rnd

pytestmark = pytest.mark.gpu


def paged(x, bs):
    """[L, K, hd] -> pages [n, K, bs, hd] in order."""
    L, K, hd = x.shape
    n = -(-L // bs)
    return torch.cat([x, torch.zeros(n * bs - L, K, hd)]).view(n, bs, K, hd).transpose(1, 2).contiguous().to(DEV)


def run(q, k, v, start, H, K, hd, bs, fn="paged_attention", **mask):
    """Attention of the tokens start.. of one request whose queries are q."""
    n, L = q.shape[0], start + q.shape[0]
    step = Step([L], [n])
    out = torch.full((n, H * hd), float("nan"), device=DEV)
    table = torch.arange(-(-k.shape[0] // bs), dtype=torch.int32, device=DEV)[None]
    args = (q.reshape(n, -1).to(DEV), paged(k, bs), paged(v, bs), out)
    m = (hd ** -0.5, mask.get("window", 0), mask.get("keep", 0), None, mask.get("chunk", 0), mask.get("cap", 0.0),
         mask.get("sink"), mask.get("slopes"))
    if fn == "paged_attention":
        ops().paged_attention(*args, step, table, H, K, hd, bs, *m)
    else:
        ops().paged_attention_generic(*args, step.positions, step.seq_ids, table, H, K, hd, bs, *m)
    ops().check_device_errors()
    return out


@pytest.mark.parametrize("hd,H,K", [(128, 4, 2), (128, 8, 2), (128, 2, 2), (64, 3, 1), (64, 2, 2), (64, 10, 2), (128, 40, 1)])
@pytest.mark.parametrize("form", ["all", "window", "kept", "chunk", "extras"])
def test_cuts(hd, H, K, form):
    """One portion of 70 tokens behind 600, and the same tokens in portions of 1 to 40: equal bits."""
    start, n, bs = 600, 70, 16
    dev = lambda x: x.to(DEV)                                                            # noqa: E731
    mask = {"all": {}, "window": dict(window=100), "kept": dict(window=100, keep=37), "chunk": dict(chunk=144),
            "extras": dict(cap=5.0, sink=dev(rnd(H, seed=9)), slopes=dev(rnd(H, seed=10).abs() * 0.05))}[form]
    q, k, v = rnd(n, H, hd, seed=1), rnd(start + n, K, hd, seed=2), rnd(start + n, K, hd, seed=3)
    whole = run(q, k, v, start, H, K, hd, bs, **mask)
    at = 0
    for size in (1, 2, 8, 9, 10, 40):
        part = run(q[at:at + size], k, v, start + at, H, K, hd, bs, **mask)
        assert torch.equal(part, whole[at:at + size]), (form, at, size)
        at += size
    assert at == n


@pytest.mark.parametrize("n", [1, 9, 40])
def test_scores_of_minus_infinity(n):
    """Some keys score -inf for every query (a query entry of one sign against a key entry of -inf): beside finite scores they
    weigh nothing, wherever they lie; 32 of them in a row are one chunk of the kernels."""
    H, K, hd, bs, L = 2, 1, 64, 16, 100
    q, k, v = rnd(n, H, hd, seed=1), rnd(L, K, hd, seed=2), rnd(L, K, hd, seed=3)
    q[..., 0] = q[..., 0].abs() + 0.5
    k[0:64, :, 0] = float("-inf")
    got = run(q, k, v, L - n, H, K, hd, bs)
    plain = run(q, k, v, L - n, H, K, hd, bs, fn="generic")
    rows = plain.isfinite().all(1)
    assert bool(rows.any())
    want = attend64(q, [k[64:]], [v[64:]], [(0, p - 64) for p in range(L - n, L)], hd ** -0.5, 0, 0, 0, 0.0, None, None) if n < 36 else None
    assert bool(got[rows].isfinite().all())
    assert float((got[rows] - plain[rows]).abs().max()) < 1e-5
    if want is not None:
        assert float((got.cpu().double() - want).abs().max()) < 1e-5


@pytest.mark.parametrize("n", [1, 9, 40])
def test_an_infinite_value_whose_weight_underflows(n):
    """A key that is seen with a weight of exactly zero and an infinite value: not a number, as in the plain kernel."""
    H, K, hd, bs, L = 2, 2, 128, 16, 64
    q, k, v = rnd(n, H, hd, seed=1), rnd(L, K, hd, seed=2), rnd(L, K, hd, seed=3)
    q[..., 0] = 40.0
    k[:, :, 0] = 0.0
    k[5, :, 0] = -1000.0
    v[5] = float("inf")
    got, plain = run(q, k, v, L - n, H, K, hd, bs), run(q, k, v, L - n, H, K, hd, bs, fn="generic")
    assert torch.equal(got.isnan(), plain.isnan()) and bool(plain.isnan().any())
