"""Captures of one engine while what is left of another one is collected."""
import gc

import pytest
import torch

import helpers
from helpers import TINY
from test_replay_gpu import STD, make_engine

pytestmark = pytest.mark.gpu


def decode(eng, tokens):
    out = []
    for i, t in enumerate(tokens):
        out.append(eng.step([item("r", [t])]).clone())
    eng.finish("r")
    return torch.cat(out)


def item(rid, tokens):
    from rllm_b200.engine import StepItem
    return StepItem(rid, tokens, [len(tokens) - 1])


def test_a_dead_engine_is_collected_around_a_capture(tmp_path):
    """An engine with graphs in a reference cycle becomes garbage in the middle of another engine's capture, and the collector is
    made to run at the next few allocations: the capture goes through and its graph gives the eager step's logits."""
    helpers.make_model_dir(tmp_path, TINY["A"], seed=5, dtype=torch.float32, std=STD)
    tokens = helpers.random_tokens(6, TINY["A"]["vocab_size"], 3)
    dead = make_engine(tmp_path, "float32", max_tokens=64)
    want = decode(dead, tokens)
    assert dead.stats["graphs_captured"] >= 1
    dead.itself = dead
    box = [dead]
    del dead
    eng = make_engine(tmp_path, "float32", max_tokens=64)
    forward, dropped = eng.model.forward, []

    def dropping(ctx, views):
        if torch.cuda.is_current_stream_capturing() and box:
            box.clear()
            dropped.append([[] for _ in range(5000)])
        return forward(ctx, views)

    eng.model.forward = dropping
    old = gc.get_threshold()
    gc.collect()
    gc.set_threshold(50, 1, 1)
    try:
        got = decode(eng, tokens)
    finally:
        gc.set_threshold(*old)
    assert dropped and gc.isenabled() and eng.stats["graphs_captured"] >= 1 and torch.equal(got, want)
