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


class Step:
    """The fields of a step that attention reads, for requests of `lens` keys of which the last `q_lens` are the step's."""

    def __init__(self, lens, q_lens):
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                  # noqa: E731
        self.q_lens, self.n_tokens, self.n_requests, self.plans = list(q_lens), sum(q_lens), len(lens), {}
        cu = [0]
        for k in q_lens:
            cu.append(cu[-1] + k)
        self.where = [(r, p) for r, (L, k) in enumerate(zip(lens, q_lens)) for p in range(L - k, L)]
        self.cu_q, self.positions = i32(cu), i32([p for _, p in self.where])
        self.seq_ids = i32([r for r, _ in self.where])


def attend64(q, k, v, where, scale, window, keep, chunk, cap, sink, slopes):
    """Row by row in 64 bits; k and v per request [L, K, hd]."""
    n, H, hd = q.shape
    out = torch.empty(n, H, hd, dtype=torch.float64)
    for i, (r, pos) in enumerate(where):
        p = torch.arange(pos + 1)
        see = torch.ones(pos + 1, dtype=torch.bool)
        if window:
            see &= (pos - p < window) | (p < keep)
        if chunk:
            see &= (p >= pos - pos % chunk) | ((p < keep) if window else False)
        p = p[see]
        kk, vv = (x[r][p].double().repeat_interleave(H // x[r].shape[1], 1) for x in (k, v))
        s = torch.einsum("hd,phd->hp", q[i].double(), kk) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes.double()[:, None] * (pos - p).double()
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None]], 1)
        w = torch.softmax(s, 1)[:, :len(p)]
        out[i] = torch.einsum("hp,phd->hd", w, vv)
    return out.reshape(n, H * hd)


@pytest.mark.parametrize("hd,H,K,bs", [(128, 16, 8, 32), (64, 3, 1, 16), (128, 5, 1, 8), (64, 2, 2, 7), (128, 40, 1, 32)])
@pytest.mark.parametrize("form", ["all", "window", "kept", "chunk", "extras"])
def test_attention(hd, H, K, bs, form):
    """Few tokens and portions in one step, at the edges of chunks (32 keys, 16 warps) and tiles.  Whatever no row sees
    holds NaN.  Bound: scores of size |q||k| / sqrt(hd) < 16 rounded hd + 2 times, as a factor of their exponential, and
    sums of at most 700 terms taken in chains of at most 32 + 22: 3e-5 of the largest value."""
    lens = [1, 33, 32, 600, 513, 65, 300, 700, 9]
    q_lens = [1, 1, 8, 1, 2, 65, 40, 9, 9]
    window, keep, chunk, cap, sink, slopes = 0, 0, 0, 0.0, None, None
    if form in ("window", "kept"):
        window, keep = 50, (37 if form == "kept" else 0)
    if form == "chunk":
        chunk = 48
    if form == "extras":
        cap, sink, slopes = 5.0, rnd(H, seed=9), rnd(H, seed=10).abs() * 0.05
    step = Step(lens, q_lens)
    q = rnd(step.n_tokens, H, hd, seed=6)
    width = -(-max(lens) // bs)
    pages = sum(-(-L // bs) for L in lens) + 2
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(7)).tolist()
    kc, vc = (torch.full((pages, K, bs, hd), float("nan")) for _ in range(2))
    table = torch.zeros(len(lens), width, dtype=torch.int32)
    ks, vs = [], []
    for r, (L, ql) in enumerate(zip(lens, q_lens)):
        k, v = rnd(L, K, hd, seed=20 + r), rnd(L, K, hd, seed=50 + r)
        ks.append(k), vs.append(v)
        first = L - ql
        lo = max(0, first + 1 - window) if window else first - first % chunk if chunk else 0
        for p in range(L):
            page = table[r, p // bs] = perm.pop() if p % bs == 0 else table[r, p // bs]
            if p >= lo or p < keep:
                kc[page, :, p % bs], vc[page, :, p % bs] = k[p], v[p]
    scale = hd ** -0.5
    want = attend64(q, ks, vs, step.where, scale, window, keep, chunk, cap, sink, slopes)
    dev = lambda x: None if x is None else x.to(DEV)                                     # noqa: E731
    out = torch.full((step.n_tokens, H * hd), float("nan"), device=DEV)
    args = (dev(kc), dev(vc))
    o = ops()
    o.paged_attention(dev(q.view(-1, H * hd)), *args, out, step, dev(table), H, K, hd, bs, scale, window, keep, None, chunk, cap,
                      dev(sink), dev(slopes))
    o.check_device_errors()
    assert float((out.cpu().double() - want).abs().max()) < 3e-5 * float(want.abs().max())
    # no further off than the plain kernel, which sums in chunks of 128 keys (up to what two orders of summation differ by)
    plain = torch.empty_like(out)
    o.paged_attention_generic(dev(q.view(-1, H * hd)), *args, plain, step.positions, step.seq_ids, dev(table), H, K, hd, bs, scale,
                              window, keep, None, chunk, cap, dev(sink), dev(slopes))
    off = [float((x.cpu().double() - want).norm()) for x in (out, plain)]
    assert off[0] <= 1.1 * off[1]
    # each request alone: the same bits
    at = 0
    for r, (L, ql) in enumerate(zip(lens, q_lens)):
        one = torch.empty(ql, H * hd, device=DEV)
        o.paged_attention(dev(q[at:at + ql].reshape(ql, -1)), *args, one, Step([L], [ql]), dev(table[r:r + 1]), H, K, hd, bs, scale,
                          window, keep, None, chunk, cap, dev(sink), dev(slopes))
        assert torch.equal(one, out[at:at + ql])
        at += ql


def test_attention_ignores_what_a_row_does_not_see():
    """An infinite value of a later token of the portion reaches only the rows that see it."""
    H, K, hd, bs, L = 2, 1, 64, 16, 40
    step = Step([L], [L])
    q, k, v = rnd(L, H * hd, seed=1), rnd(L, K, hd, seed=2), rnd(L, K, hd, seed=3)
    v[25] = float("inf")
    pad = lambda x: torch.cat([x, torch.zeros(8, K, hd)]).view(3, bs, K, hd).transpose(1, 2).contiguous().to(DEV)   # noqa: E731
    out = torch.empty(L, H * hd, device=DEV)
    ops().paged_attention(q.to(DEV), pad(k), pad(v), out, step, torch.arange(3, dtype=torch.int32, device=DEV)[None], H, K, hd, bs,
                          hd ** -0.5)
    assert bool(out[:25].isfinite().all()) and not bool(out[25:].isfinite().any())
