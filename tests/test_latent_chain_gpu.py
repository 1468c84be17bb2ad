"""Merging the splits of attention through latents and storing its rotated parts, where their loops end: one split and more than are in
flight at once, splits without keys, values narrower and wider than a block's columns, latents longer than the threads hold."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from rllm_b200.csrc import ops as o
    return o


@pytest.mark.parametrize("L", [1, 33, 130, 700, 2500])
@pytest.mark.parametrize("H,rank,rot", [(1, 64, 64), (32, 512, 64), (40, 512, 0), (8, 128, 64)])
def test_latent_decode(L, H, rank, rot):
    """Two tokens of one context of L keys and of one of 5 keys: the longer one decides the number of splits."""
    o, W, bs = ops(), rank + rot, 32
    g = torch.Generator().manual_seed(L + H)
    lens = [L, 5]
    rows = [torch.randn(n, W, generator=g).bfloat16() for n in lens]
    q = torch.randn(2, H * W, generator=g).bfloat16()
    if not o.latent_decode_ok(q.to(DEV), W, rank):
        pytest.skip("not a size of this kernel")
    blocks = [-(-n // bs) for n in lens]
    cache = torch.full((sum(blocks), 1, bs, W), float("nan")).bfloat16()
    table = torch.zeros(2, max(blocks), dtype=torch.int32)
    at = 0
    for r, x in enumerate(rows):
        table[r, :blocks[r]] = torch.arange(at, at + blocks[r])
        flat = torch.zeros(blocks[r] * bs, W).bfloat16()
        flat[:lens[r]] = x
        cache[at:at + blocks[r], 0] = flat.view(blocks[r], bs, W)
        at += blocks[r]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                       # noqa: E731
    out = torch.empty(2, H * rank, dtype=torch.bfloat16, device=DEV)
    scale = W ** -0.5
    span = 128 if L <= 128 else -(-L // 128) * 128
    o.latent_decode_attention(q.to(DEV), cache.to(DEV), out, i32([n - 1 for n in lens]), i32([0, 1]), table.to(DEV), H, W, rank, bs,
                              scale, 0.0, span)
    o.check_device_errors()
    for r, x in enumerate(rows):
        k = x.double()
        p = torch.softmax(q[r].double().view(H, W) @ k.t() * scale, -1)
        want = (p @ k[:, :rank]).reshape(-1)
        # probabilities and the result in bfloat16: 2^-8 of sums of |p v|, twice
        size = (p @ k[:, :rank].abs()).reshape(-1)
        assert bool(((out[r].cpu().double() - want).abs() <= 2.0 ** -7 * size + 1e-6).all()), r


@pytest.mark.parametrize("H,rank,r", [(1, 64, 2), (5, 250, 64), (32, 512, 64), (128, 1100, 32), (16, 1024, 64)])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_latent_rope_store(H, rank, r, pairs, dt):
    o, n, dq, bs = ops(), 3, 16, 4
    g = torch.Generator().manual_seed(rank + r)
    q, kv, w = torch.randn(n, H * (dq + r), generator=g), torch.randn(n, rank + r, generator=g), torch.randn(rank, generator=g)
    ang = torch.rand(n, r // 2, generator=g) * 6.0
    cs = torch.stack([torch.cos(ang), torch.sin(ang)], -1).contiguous()
    slots = torch.tensor([6, -1, 1], dtype=torch.int32)
    W = rank + r
    q_att, cache = torch.full((n, H * W), 7.0, dtype=dt), torch.full((2, 1, bs, W), 7.0, dtype=dt)
    got_q, got_c = q_att.to(DEV), cache.to(DEV)
    o.latent_rope_store(q.to(DEV), kv.to(DEV), w.to(DEV), cs.to(DEV), 1.5, slots.to(DEV), got_q, got_c, H, dq, r, rank, bs, 1e-6,
                        pairs=pairs)
    o.check_device_errors()

    def rotate(x, c):                                                                    # x [..., r], c [r / 2, 2]
        co, si = c[..., 0].double() * 1.5, c[..., 1].double() * 1.5
        out = torch.empty_like(x, dtype=torch.float64)
        u, v = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., :r // 2], x[..., r // 2:])
        a, b = u.double() * co - v.double() * si, v.double() * co + u.double() * si
        if pairs:
            out[..., 0::2], out[..., 1::2] = a, b
        else:
            out[..., :r // 2], out[..., r // 2:] = a, b
        return out

    eps = 2.0 ** -8 if dt is torch.bfloat16 else 2.0 ** -20
    for t in range(n):
        head = got_q[t].cpu().view(H, W)
        assert bool((head[:, :rank] == 7.0).all())
        want = rotate(q[t].view(H, dq + r)[:, dq:], cs[t])
        assert bool(((head[:, rank:].double() - want).abs() <= eps * (want.abs() + 4.0)).all())
        if slots[t] < 0:
            continue
        row = got_c.cpu().view(-1, W)[slots[t]].double()
        lat = kv[t, :rank].double()
        want = lat / torch.sqrt((lat ** 2).mean() + 1e-6) * w.double()
        assert bool(((row[:rank] - want).abs() <= eps * want.abs() + 1e-5 * want.abs()).all())
        want = rotate(kv[t, rank:], cs[t])
        assert bool(((row[rank:] - want).abs() <= eps * (want.abs() + 4.0)).all())
    rest = [s for s in range(2 * bs) if s not in (6, 1)]
    assert bool((got_c.cpu().view(-1, W)[rest] == 7.0).all())


@pytest.mark.parametrize("n_splits", [6143, 6144, 8192])
def test_the_longest_contexts(n_splits):
    """As many splits as the kernels take.  The context's logical pages go round eight pages of the cache, so that a key counts as
    often as its page; beside it a token that sees only the first few keys of as many splits."""
    o, W, bs = ops(), 64, 64
    L = n_splits * o.LATENT_SPLIT_KEYS
    g = torch.Generator().manual_seed(n_splits)
    cache = torch.randn(8, 1, bs, W, generator=g).bfloat16()
    q = torch.randn(2, W, generator=g).bfloat16()
    table = (torch.arange(L // bs, dtype=torch.int32) % 8).repeat(2, 1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                       # noqa: E731
    out = torch.full((2, W), float("nan"), dtype=torch.bfloat16, device=DEV)
    o.latent_decode_attention(q.to(DEV), cache.to(DEV), out, i32([L - 1, 4]), i32([0, 1]), table.to(DEV), 1, W, W, bs, W ** -0.5,
                              0.0, L)
    o.check_device_errors()
    keys = cache.double().view(-1, W)
    for r, k in enumerate((keys, keys[:5])):
        times = torch.ones(len(k), dtype=torch.float64)
        if r == 0:
            pages = torch.bincount(table[0].long(), minlength=8).double()
            times = pages.repeat_interleave(bs)
        s = q[r].double() @ k.t() * W ** -0.5
        e = times * torch.exp(s - s.max())
        want, size = (e @ k) / e.sum(), (e @ k.abs()) / e.sum()
        # probabilities and the result in bfloat16: 2^-8 of sums of |p v|, twice; a million keys' sums in float32
        assert bool(((out[r].cpu().double() - want).abs() <= (2.0 ** -7 + 2e-4) * size + 1e-6).all()), r


def test_more_pairs_a_token_than_a_grid_has_blocks():
    """65,534 blocks of 256 pairs and some more: the blocks go round."""
    o, H, dq, r, rank = ops(), (1 << 18) + 77, 1, 130, 2
    assert H * (r // 2) > 65534 * 256
    g = torch.Generator(device=DEV).manual_seed(3)
    q = torch.randn(1, H * (dq + r), generator=g, device=DEV)
    kv = torch.randn(1, rank + r, generator=g, device=DEV)
    ang = torch.rand(1, r // 2, generator=g, device=DEV) * 6.0
    q_att = torch.full((1, H * (rank + r)), 7.0, device=DEV)
    cache = torch.zeros(1, 1, 4, rank + r, device=DEV)
    o.latent_rope_store(q, kv, torch.ones(rank, device=DEV), torch.stack([torch.cos(ang), torch.sin(ang)], -1).contiguous(), 1.0,
                        torch.zeros(1, dtype=torch.int32, device=DEV), q_att, cache, H, dq, r, rank, 4, 1e-6)
    o.check_device_errors()
    u, w = q.view(H, dq + r)[:, dq:].split(r // 2, 1)
    c, s = torch.cos(ang), torch.sin(ang)
    want = torch.cat([u * c - w * s, w * c + u * s], 1)
    got = q_att.view(H, rank + r)
    assert bool((got[:, :rank] == 7.0).all())
    assert bool(((got[:, rank:] - want).abs() <= 2.0 ** -20 * (want.abs() + 4.0)).all())


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("H,rank", [(3, 64), (33, 512)])
def test_output_rows_that_begin_anywhere(shift, H, rank):
    """The same bits as at an aligned address, and nothing beside them."""
    o, W, bs, L = ops(), rank + 64, 16, 300
    g = torch.Generator().manual_seed(H)
    cache = torch.randn(-(-L // bs), 1, bs, W, generator=g).bfloat16().to(DEV)
    q = torch.randn(2, H * W, generator=g).bfloat16().to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                       # noqa: E731
    table = torch.arange(len(cache), dtype=torch.int32, device=DEV).repeat(2, 1)
    size = 2 * H * rank
    aligned, base = (torch.full((size + 8,), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    for out in (aligned[:size], base[shift:shift + size]):
        o.latent_decode_attention(q, cache, out.view(2, H * rank), i32([L - 1, 40]), i32([0, 1]), table, H, W, rank, bs, W ** -0.5,
                                  0.0, L)
    o.check_device_errors()
    assert torch.equal(base[shift:shift + size], aligned[:size])
    assert bool((base[:shift] == 7.0).all()) and bool((base[shift + size:] == 7.0).all())


@pytest.mark.parametrize("H,rank,r", [(3, 250, 64), (16, 512, 64), (2, 1100, 32)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_many_tokens_are_stored_as_few_are(H, rank, r, dt):
    """One block a token, some, and as many as its queries fill: the same bits."""
    o, n, dq, bs, W = ops(), 1300, 8, 32, rank + r
    g = torch.Generator(device=DEV).manual_seed(rank)
    q = torch.randn(n, H * (dq + r), generator=g, device=DEV).to(dt)
    kv, w = torch.randn(n, W, generator=g, device=DEV), torch.randn(rank, generator=g, device=DEV)
    cs = torch.randn(n, r // 2, 2, generator=g, device=DEV)
    slots = torch.randperm(n, generator=g, device=DEV).to(torch.int32)
    slots[5] = slots[1111] = -1
    got = []
    for step in (n, 700, 100):
        q_att = torch.full((n, H * W), 7.0, dtype=dt, device=DEV)
        cache = torch.full((-(-n // bs), 1, bs, W), 7.0, dtype=dt, device=DEV)
        for a in range(0, n, step):
            b = min(n, a + step)
            o.latent_rope_store(q[a:b], kv[a:b], w, cs[a:b], 1.25, slots[a:b], q_att[a:b], cache, H, dq, r, rank, bs, 1e-6)
        got.append((q_att, cache))
    o.check_device_errors()
    assert all(torch.equal(x, y) for other in got[1:] for x, y in zip(got[0], other))
