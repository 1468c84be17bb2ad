"""Decode attention around the number of blocks where its CTAs have one warp or four, and splits whose keys do not fill
all warps."""
import pytest
import torch

from test_f32_path_gpu import DEV, Step, attend64, ops, rnd

pytestmark = pytest.mark.gpu


def blocks(o, step, H, K, window, keep, chunk):
    """CTAs of the decode launch; with at most three per SM they have four warps."""
    plan = o.AttentionPlan(step, H, K, window, torch.device(DEV), chunk)
    assert plan.n_pre == 0
    return plan.n_dec * K * plan.chunks_d * (plan.n_splits + (1 if keep else 0))


@pytest.mark.parametrize("hd,H,K,bs,many", [(128, 16, 8, 32, 6), (64, 6, 2, 16, 18), (128, 40, 4, 8, 6)])
@pytest.mark.parametrize("form", ["all", "window", "kept", "chunk", "extras"])
@pytest.mark.parametrize("copied", [False, True])
def test_decode(hd, H, K, bs, form, many, copied):
    """`many` times the same requests: beyond three blocks an SM the one-warp kernel runs.  Bound: weights and result are each
    rounded to 9 bits, so 2^-8 of the largest value, and as much again for the exponentials and the sums."""
    copies = many if copied else 1
    lens, q_lens = [1, 15, 16, 17, 33, 128, 129, 300, 515] * copies, [1, 1, 1, 1, 8, 1, 2, 1, 3] * copies
    window, keep, chunk, cap, sink, slopes = 0, 0, 0, 0.0, None, None
    if form in ("window", "kept"):
        window, keep = 70, (150 if form == "kept" else 0)
    if form == "chunk":
        chunk = 100
    if form == "extras":
        cap, sink, slopes = 5.0, rnd(H, seed=9), rnd(H, seed=10).abs() * 0.05
    step = Step(lens, q_lens)
    step.start_pos = [L - k for L, k in zip(lens, q_lens)]
    bf = lambda *s, seed: rnd(*s, seed=seed).bfloat16()                                  # noqa: E731
    q = bf(sum(q_lens[:9]), H, hd, seed=6).repeat(copies, 1, 1)
    pages = sum(-(-L // bs) for L in lens)
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(7)).tolist()
    kc, vc = (torch.zeros(pages, K, bs, hd, dtype=torch.bfloat16) for _ in range(2))
    table = torch.zeros(len(lens), -(-max(lens) // bs), dtype=torch.int32)
    ks, vs = [], []
    for r, L in enumerate(lens):
        k, v = bf(L, K, hd, seed=20 + r % 9), bf(L, K, hd, seed=50 + r % 9)
        ks.append(k), vs.append(v)
        for b in range(-(-L // bs)):
            page = table[r, b] = perm.pop()
            a, e = b * bs, min(L, (b + 1) * bs)
            kc[page, :, :e - a], vc[page, :, :e - a] = k[a:e].transpose(0, 1), v[a:e].transpose(0, 1)
    n = sum(q_lens[:9])
    want = attend64(q[:n], ks, vs, step.where[:n], hd ** -0.5, window, keep, chunk, cap, sink, slopes).repeat(copies, 1)
    dev = lambda x: None if x is None else x.to(DEV)                                     # noqa: E731
    out = torch.full((step.n_tokens, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    o = ops()
    assert (blocks(o, step, H, K, window, keep, chunk) > 3 * o.sm_count(DEV)) or not copied
    o.paged_attention(q.view(-1, H * hd).to(DEV), kc.to(DEV), vc.to(DEV), out, step, table.to(DEV), H, K, hd, bs, hd ** -0.5,
                      window, keep, None, chunk, cap, dev(sink), dev(slopes))
    o.check_device_errors()
    top = max(float(v.abs().max()) for v in vs)
    assert float((out.cpu().double() - want).abs().max()) < 2.0 ** -7 * top
    # a request alone (four warps a CTA) and in the batch (copied: one warp): the same bits
    at = 0
    for r in range(9):
        one = Step([lens[r]], [q_lens[r]])
        one.start_pos = [lens[r] - q_lens[r]]
        assert blocks(o, one, H, K, window, keep, chunk) <= 3 * o.sm_count(DEV)
        alone = torch.empty(q_lens[r], H * hd, dtype=torch.bfloat16, device=DEV)
        o.paged_attention(q[at:at + q_lens[r]].reshape(q_lens[r], -1).to(DEV), kc.to(DEV), vc.to(DEV), alone, one, table[r:r + 1].to(DEV), H,
                          K, hd, bs, hd ** -0.5, window, keep, None, chunk, cap, dev(sink), dev(slopes))
        assert torch.equal(alone, out[at:at + q_lens[r]])
        at += q_lens[r]
    for c in range(1, copies):
        assert torch.equal(out[:n], out[c * n:(c + 1) * n])
