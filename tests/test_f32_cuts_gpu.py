"""float32 attention gives a token the same bits however its prompt is cut into portions."""
import pytest
import torch

from test_f32_path_gpu import DEV, Step, ops, rnd

pytestmark = pytest.mark.gpu


def paged(x, bs):
    """[L, K, hd] -> pages [n, K, bs, hd] in order."""
    L, K, hd = x.shape
    n = -(-L // bs)
    return torch.cat([x, torch.zeros(n * bs - L, K, hd)]).view(n, bs, K, hd).transpose(1, 2).contiguous().to(DEV)


def run(q, k, v, start, H, K, hd, bs, **mask):
    """Attention of the tokens start.. of one request whose queries are q."""
    n, L = q.shape[0], start + q.shape[0]
    step = Step([L], [n])
    out = torch.full((n, H * hd), float("nan"), device=DEV)
    table = torch.arange(-(-k.shape[0] // bs), dtype=torch.int32, device=DEV)[None]
    args = (q.reshape(n, -1).to(DEV), paged(k, bs), paged(v, bs), out)
    m = (hd ** -0.5, mask.get("window", 0), mask.get("keep", 0), None, mask.get("chunk", 0), mask.get("cap", 0.0),
         mask.get("sink"), mask.get("slopes"))
    ops().paged_attention(*args, step, table, H, K, hd, bs, *m)
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
