"""Which requests of a float32 step go in tiles and which token by token (the results are the same)."""
import pytest
import torch

from rllm_b200.csrc import ops


class Step:
    def __init__(self, q_lens):
        self.q_lens = q_lens


def plan(monkeypatch, q_lens, H, K, hd, span):
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    return ops.F32AttentionPlan(Step(q_lens), H, K, hd, span, torch.device("cpu"))


@pytest.mark.parametrize("q_lens,H,K,hd,span,tiles", [
    ([1, 8, 3], 16, 8, 128, 4096, False),               # few tokens
    ([9], 16, 8, 128, 32, False), ([16], 4, 4, 64, 32, False), ([64], 16, 8, 128, 64, False),
    ([64], 16, 8, 128, 4096, False),                    # few tiles, each a long chain of keys on one SM
    ([64], 1, 1, 128, 4096, False), ([12] * 4, 3, 1, 128, 2016, False),
    ([461], 16, 8, 128, 480, True), ([300, 300], 32, 8, 128, 320, True), ([512], 32, 8, 128, 2048, True),
    ([1, 300, 300], 16, 8, 128, 320, True),
])
def test_tiles_or_tokens(monkeypatch, q_lens, H, K, hd, span, tiles):
    p = plan(monkeypatch, q_lens, H, K, hd, span)
    assert (p.n_tiles > 0) == tiles
    # every token once: alone or as a place of a tile
    got, cu = list(p.tokens.tolist()), [0]
    for k in q_lens:
        cu.append(cu[-1] + k)
    for r, t0 in zip(p.t_req.tolist(), p.t_tok.tolist()):
        got += range(t0, min(t0 + p.TT, cu[r + 1]))
    assert sorted(got) == list(range(sum(q_lens))) and p.TT * p.GH <= 32 and p.GH * p.chunks >= H // K
