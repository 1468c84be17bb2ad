"""Windows that keep the first keys, bfloat16: the tcgen05 kernel's two runs of key tiles at their edges."""
import pytest
import torch

from test_f32_path_gpu import DEV, Step, attend64, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", [1, 8, 127, 128, 129, 300])
@pytest.mark.parametrize("H,K,bs,window", [(4, 1, 32, 160), (8, 8, 16, 40), (2, 1, 128, 128)])
def test_kept_keys(keep, H, K, bs, window):
    """Portions at the edges of tiles (128 rows, 128 keys).  Pages that hold neither a kept key nor one of a window are
    someone else's: they hold huge values.  Bound: weights and result are each rounded to 9 bits, so 2^-8 of the largest
    value, and as much again for the special-function unit's exponentials and the sums."""
    hd, lens, q_lens = 128, [700, 45, 129, 513], [700, 45, 100, 9]
    step = Step(lens, q_lens)
    bf = lambda *s, seed: rnd(*s, seed=seed).bfloat16()                                  # noqa: E731
    q = bf(step.n_tokens, H, hd, seed=6)
    pages = sum(-(-L // bs) for L in lens) + 2
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(7)).tolist()
    kc, vc = (torch.full((pages, K, bs, hd), 1e4, dtype=torch.bfloat16) for _ in range(2))
    table = torch.zeros(len(lens), -(-max(lens) // bs), dtype=torch.int32)
    ks, vs = [], []
    for r, (L, ql) in enumerate(zip(lens, q_lens)):
        k, v = bf(L, K, hd, seed=20 + r), bf(L, K, hd, seed=50 + r)
        ks.append(k), vs.append(v)
        lo = max(0, L - ql + 1 - window)
        for b in range(-(-L // bs)):
            page = table[r, b] = perm.pop()
            a, e = b * bs, min(L, (b + 1) * bs)
            if e > lo or a < keep:
                kc[page, :, :e - a], vc[page, :, :e - a] = k[a:e].transpose(0, 1), v[a:e].transpose(0, 1)
    want = attend64(q, ks, vs, step.where, hd ** -0.5, window, keep, 0, 0.0, None, None)
    o = ops()
    step.start_pos = [L - k for L, k in zip(lens, q_lens)]
    out = torch.full((step.n_tokens, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    o.paged_attention(q.view(-1, H * hd).to(DEV), kc.to(DEV), vc.to(DEV), out, step, table.to(DEV), H, K, hd, bs, hd ** -0.5,
                      window, keep)
    o.check_device_errors()
    top = max(float(v.abs().max()) for v in vs)
    assert float((out.cpu().double() - want).abs().max()) < 2.0 ** -7 * top
