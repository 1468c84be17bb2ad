"""The sampler's two forms, a cluster of blocks per row and one block per row: equal draws, and those of the plain sampler, at
vocabularies of every kind of slice (shorter than a warp, than a block, kept in shared memory, read from memory)."""
import pytest
import torch

import plain_impl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# (temperature, top_k, top_p)
FORMS = [(0.0, 0, 1.0), (0.8, 0, 1.0), (1.0, 5, 1.0), (0.7, 0, 0.9), (1.3, 40, 0.7), (0.5, 1, 1.0), (1.0, 0, 0.999), (2.0, 1000, 0.95)]


def ops():
    from rllm_b200.csrc import ops as o
    return o


def draw(logits, forms, seeds):
    t = lambda x, dt: torch.tensor(x, dtype=dt, device=DEV)                              # noqa: E731
    ids = torch.full((logits.shape[0],), -7, dtype=torch.int32, device=DEV)
    ops().sample_rows(logits.to(DEV), ids, t([f[0] for f in forms], torch.float32), t([f[1] for f in forms], torch.int32),
                      t([f[2] for f in forms], torch.float32), t(seeds, torch.int64), t([100 + s for s in seeds], torch.int64))
    return ids.tolist()


def rows_of(V, n, seed):
    g = torch.Generator().manual_seed(seed)
    x = 3.0 * torch.randn(n, V, generator=g)
    if V > 1:
        x[1::4, :: 3] = float("-inf")                # banned tokens
        x[2::4, V // 9] = x[2::4, V - 1] = x[2::4].max(1).values + 1          # a tie whose entries lie in unlike slices
    return x


@pytest.mark.parametrize("V", [1, 7, 40, 257, 8191, 8193, 32768, 51201, 151936, 409601])
def test_rows_alone_and_in_a_batch(V):
    """A request's draw does not depend on its batch: 160 rows of a launch (one block a row) against launches of a few (a cluster
    a row at the larger vocabularies), every form of sampling beside the others."""
    base = rows_of(V, 8, seed=V)
    n = 160 if V < 100000 else 40
    logits = base.repeat(n // 8, 1)
    forms, seeds = [FORMS[(r + r // 8) % 8] for r in range(n)], [7919 * r + 4 for r in range(n)]
    got = draw(logits, forms, seeds)
    assert all(0 <= t < V for t in got)
    for lo, hi in ((0, 1), (1, 4), (4, 16), (n - 5, n)):
        assert draw(logits[lo:hi], forms[lo:hi], seeds[lo:hi]) == got[lo:hi]
    ids = [torch.full((m,), -7, dtype=torch.int32, device=DEV) for m in (n, 3)]
    for o in ids:
        ops().sample_rows(logits[:len(o)].to(DEV), o)
    assert ids[0].tolist() == base.argmax(1).tolist() * (n // 8) and ids[1].tolist() == ids[0].tolist()[:3]


@pytest.mark.parametrize("V", [1531, 151936, 409601])
@pytest.mark.parametrize("rows", [8, 24])
def test_draws_of_the_plain_sampler(V, rows):
    """Both forms against the plain sampler; the rounding of log, exp and the sums may flip a near tie."""
    logits = rows_of(V, 8, seed=V + 1).repeat(rows // 8, 1)
    forms, seeds = [FORMS[(r + r // 8) % 8] for r in range(rows)], [31 * r + 5 for r in range(rows)]
    got = draw(logits, forms, seeds)
    want = [plain_impl.sample_row(logits[r].numpy(), *forms[r], seeds[r], 100 + seeds[r]) for r in range(rows)]
    assert sum(a == b for a, b in zip(got, want)) >= rows - 1, (got, want)
