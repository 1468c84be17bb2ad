"""The work that a user of this package has it do, as cases that can be timed and compared.

Every case is a model of one of the package's architectures in full depth with random weights, an engine that
holds its cache, and one pass through ``Engine.step``: a prompt read in one step (prefill), steps of one token for
every running request (decode), decoding requests beside a portion of a new prompt in the same step (mixed), or whole
short requests from the prompt to the last decoded token (chat).  Tokens are given from outside, as in a comparison, a
perplexity run or a replayed trace, so that the logits of two implementations can be held against one another.

Sizes: the Qwen3 shapes that the benchmark and the published numbers of the reference are quoted on (8B, 0.6B), the
prompt lengths 16..2,048 and the batches 1..64 of the serving workload, contexts up to 4,096, and the Falalix and
Govopel shapes of the benchmark at widths 2,048 and 4,096.  Architectures with routed experts are not among the
cases: in bfloat16 a rounding difference may choose another expert, and no tolerance tells that from a wrong result.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from rllm_b200.config import config_from_dict
from rllm_b200.engine import Engine, StepItem
from rllm_b200.models.model import DecoderModel, expected_tensors, parse_dtype
from rllm_b200.parts import Runtime
from rllm_b200.sampling.device import sample_rows
from rllm_b200.sampling.params import SamplingParams

DEVICE = "cuda:0"
PAGE = 32                       # tokens per page of the cache, the default of LLM(...)
PREPARE_TOKENS = 2048           # tokens of a step that fills the cache before a decode case


# ---------------------------------------------------------------- the models

def _qwen3(layers, hidden, heads, ff, tied):
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=layers, hidden_size=hidden,
                num_attention_heads=heads, num_key_value_heads=8, head_dim=128, intermediate_size=ff,
                vocab_size=151936, rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=tied,
                max_position_embeddings=40960, use_sliding_window=False)


def _falalix(width):
    heads = max(8, width // 128)
    mamba = {"type": "mamba1", "mixer": {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}, "mlp": None}
    par = {"type": "parallel",
           "mixer": {"left": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128,
                              "mask": {"size": 1024, "keep_first": 8}, "scale": 128 ** -0.5},
                     "right": {"heads": width // 64, "dim": 64, "decay_rank": 64},
                     "left_scale": 0.7, "right_scale": 0.8},
           "mlp": {"kind": "dense", "ff": 3 * width}}
    return {"architecture": "Falalix", "vocab": 32768, "width": width, "layers": [par, par, mamba, par, par, mamba],
            "loop": {"start": 0, "stop": 3, "times": 2}, "norm": {"eps": 1e-6}, "residual_mult": 0.5}


def _govopel(width):
    heads = max(8, width // 128)
    mlp = {"kind": "dense", "ff": 3 * width, "limit": 7.0}
    latent = {"type": "latent_attention",
              "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
                        "q_rank": min(1536, 3 * width // 4), "rot": {"dims": 64, "base": 10000.0}, "scale": 192 ** -0.5},
              "mlp": mlp}
    chunked = {"type": "attention",
               "mixer": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "mask": {"size": 1024},
                         "rot": {"dims": 64, "base": 500000.0,
                                 "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}},
                         "scale": 12.0 / 128, "softcap": 50.0},
               "mlp": mlp}
    return {"architecture": "Govopel", "vocab": 32768, "width": width, "layers": [latent, chunked, chunked, latent] * 2,
            "norm": {"eps": 1e-6}, "logit_softcap": 30.0}


MODELS = {"qwen3-8b": lambda: _qwen3(36, 4096, 32, 12288, False), "qwen3-0.6b": lambda: _qwen3(28, 1024, 16, 3072, True),
          "falalix-4k": lambda: _falalix(4096), "falalix-2k": lambda: _falalix(2048),
          "govopel-4k": lambda: _govopel(4096), "govopel-2k": lambda: _govopel(2048)}


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # The smallest call: one user's request on the small model, a token at a time (the reference's tg128).
        dict(name="small-decode-1", model="qwen3-0.6b", dtype="bfloat16", kind="decode", requests=1, tokens=128, steps=16),
        # The reference's pp512 on the small model: one prompt in one step.
        dict(name="small-prefill-512", model="qwen3-0.6b", dtype="bfloat16", kind="prefill", requests=1, tokens=512),
        # The 32-bit path that answers are checked with: two requests in float32, sampled tokens and all.
        dict(name="small-float32-chat-2", model="qwen3-0.6b", dtype="float32", kind="chat", requests=2, tokens=300, steps=8),
        # Chat with one user on the large model.
        dict(name="large-decode-1", model="qwen3-8b", dtype="bfloat16", kind="decode", requests=1, tokens=700, steps=8),
        # The headline of the benchmark: eight requests behind prompts of 2,048 tokens.
        dict(name="large-decode-8", model="qwen3-8b", dtype="bfloat16", kind="decode", requests=8, tokens=2048, steps=8),
        # A busy server: requests of unlike lengths decode together.
        dict(name="large-decode-40-ragged", model="qwen3-8b", dtype="bfloat16", kind="decode", requests=40, tokens=900, steps=4),
        # A short message to the large model: the time to the first token.
        dict(name="large-prefill-77", model="qwen3-8b", dtype="bfloat16", kind="prefill", requests=1, tokens=77),
        # A long prompt in one step, the benchmark's prefill point.
        dict(name="large-prefill-2048", model="qwen3-8b", dtype="bfloat16", kind="prefill", requests=1, tokens=2048),
        # Continuous batching: a portion of 488 tokens of a new prompt beside 24 decoding requests.
        dict(name="large-mixed-24", model="qwen3-8b", dtype="bfloat16", kind="mixed", requests=24, tokens=600, portion=488),
        # Recurrent mixers beside windowed attention: a long prompt, and eight short requests from start to end.
        dict(name="falalix-prefill-2048", model="falalix-4k", dtype="bfloat16", kind="prefill", requests=1, tokens=2048),
        dict(name="falalix-chat-8", model="falalix-4k", dtype="bfloat16", kind="chat", requests=8, tokens=200, steps=24),
        # Latent and chunked attention: four longer requests from start to end.
        dict(name="govopel-chat-4", model="govopel-4k", dtype="bfloat16", kind="chat", requests=4, tokens=1100, steps=24),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    dtype = "bfloat16"
    model, kind = rng.choice([
        ("qwen3-8b", "decode"), ("qwen3-8b", "decode"), ("qwen3-8b", "prefill"), ("qwen3-8b", "prefill"), ("qwen3-8b", "mixed"),
        ("qwen3-0.6b", "decode"), ("qwen3-0.6b", "prefill"), ("qwen3-0.6b", "float32"),
        ("falalix-4k", "prefill"), ("falalix-4k", "chat"), ("falalix-2k", "chat"), ("falalix-2k", "prefill"),
        ("govopel-4k", "chat"), ("govopel-4k", "prefill"), ("govopel-2k", "chat")])
    if kind == "float32":
        kind, dtype = "chat", "float32"
    case = dict(model=model, dtype=dtype, kind=kind)
    if kind == "prefill":
        requests = rng.choice((1, 1, 2, 4))
        return dict(case, requests=requests, tokens=_log_uniform(rng, 16, 2048 // requests))
    if kind == "decode":
        requests = _log_uniform(rng, 1, 64)
        return dict(case, requests=requests, tokens=_log_uniform(rng, 48, min(4000, 40000 // requests)), steps=rng.choice((4, 6)))
    if kind == "mixed":
        requests = _log_uniform(rng, 2, 31)
        return dict(case, requests=requests, tokens=_log_uniform(rng, 48, 1200), portion=_log_uniform(rng, 16, 512 - requests))
    requests = _log_uniform(rng, 1, 4 if dtype == "float32" else 12)
    most = (600 if dtype == "float32" else 4000) // requests
    return dict(case, requests=requests, tokens=_log_uniform(rng, 24, min(1200, most)), steps=rng.randint(6, 20))


def _lengths(case):
    """Prompt length of every request: the longest has `tokens`, more requests than 16 and the whole requests of a chat
    have unlike lengths between a quarter and all of it; the same for every seed."""
    n, top = case["requests"], case["tokens"]
    if n <= 16 and case["kind"] != "chat":
        return [top] * n
    return [max(1, round(top * (1.0 - 0.75 * ((i * 0.618034) % 1.0)))) for i in range(n)]


def _steps(case):
    return case.get("steps", 0)


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 17)


def _weights(config, seed, dtype):
    """Name -> tensor of a model's storage type.  Matrices are N(0, 0.02), as the package's random weights are; those of
    the deep Qwen3 shapes are N(0, 2 / (5 width)) (0.02 at a width of 1,024), a sublayer's last one smaller by the root of
    the number of sublayers, as models are initialised: the stream keeps its size and a rounding is not amplified from
    layer to layer.  Norm weights lie around 1.  The recurrent mixers have memories of unlike length, as trained ones
    have: step sizes 0.001 to 0.1 and rates 1 to N of the selective scan, decays of a step between 0.5 and 0.999 of the
    time mixing."""
    g = _generator(seed)
    out = {}
    spec = config.model_spec()
    std, last = 0.02, 1.0
    if config.architecture.startswith("Qwen3"):
        std, last = (0.4 / spec.hidden_size) ** 0.5, (2 * len(spec.run_order)) ** -0.5
    for name, (shape, role) in expected_tensors(spec).items():
        t = torch.randn(shape, generator=g, dtype=dtype if role == "matrix" else torch.float32, device=DEVICE)
        if role == "norm":
            t = 1.0 + 0.1 * t
        elif role == "mix":
            t = torch.sigmoid(t)
        elif role == "conv":
            t = t / shape[-1] ** 0.5
        else:
            t *= std
            if name.endswith(("o_proj.weight", "down_proj.weight")):
                t *= last
        if name.endswith(".A_log"):
            t = t + torch.log(torch.arange(1, shape[1] + 1, device=DEVICE, dtype=torch.float32))
        elif name.endswith(".dt.b"):
            step = torch.exp(torch.empty(shape, device=DEVICE).uniform_(math.log(1e-3), math.log(0.1), generator=g))
            t = step + torch.log(-torch.expm1(-step))
        elif name.endswith(".w0"):
            t = t + torch.empty(shape, device=DEVICE).uniform_(-6.9, -0.4, generator=g)
        elif name.endswith(".u"):
            t = 25.0 * t
        out[name] = t.to(dtype)
    return out


def _tokens(case, seed, vocab):
    """Per request: its prompt and the tokens that its decode steps are given (and, last, the mixed case's new prompt)."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 18)
    n = [a + _steps(case) + (1 if case["kind"] == "mixed" else 0) for a in _lengths(case)]
    if case["kind"] == "mixed":
        n.append(case["tokens"] // 2 + case["portion"])
    return [torch.randint(0, vocab, (k,), generator=g).tolist() for k in n]


class _State:
    pass


def prepare(case, seed):
    config = config_from_dict(MODELS[case["model"]]())
    dtype = parse_dtype(case["dtype"])
    s = _State()
    s.kind, s.steps, s.lengths = case["kind"], _steps(case), _lengths(case)
    model = DecoderModel(config.model_spec(), Runtime(torch.device(DEVICE), dtype))
    model.load_tensors(_weights(config, seed, dtype))
    s.tokens = _tokens(case, seed, model.spec.vocab_size)
    s.sample = SamplingParams(0.8, 0, 0.95, 11) if case["dtype"] == "float32" else None
    room = sum(-(-len(t) // PAGE) * PAGE + PAGE for t in s.tokens)
    s.engine = Engine(model, block_size=PAGE, max_tokens=room, max_requests=len(s.tokens))
    if s.kind in ("decode", "mixed"):
        fill = [(r, s.tokens[r][:n]) for r, n in enumerate(s.lengths)]
        if s.kind == "mixed":
            s.start = case["tokens"] // 2
            if s.start:
                fill.append((len(s.lengths), s.tokens[-1][:s.start]))
        items, size = [], 0
        for r, toks in fill:
            if items and size + len(toks) > PREPARE_TOKENS:
                s.engine.step(items)
                items, size = [], 0
            for at in range(0, len(toks), PREPARE_TOKENS):
                if at:
                    s.engine.step(items)
                    items, size = [], 0
                items.append(StepItem(r, toks[at:at + PREPARE_TOKENS], []))
                size += len(items[-1].tokens)
        s.engine.step(items)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    return {"prefill": _run_prefill, "decode": _run_decode, "mixed": _run_mixed, "chat": _run_chat}[s.kind](s)


def _run_prefill(s):
    """The prompts in one step, the logits behind each; the requests end."""
    logits = s.engine.step([StepItem(r, s.tokens[r], [n - 1]) for r, n in enumerate(s.lengths)])
    for r in range(len(s.lengths)):
        s.engine.finish(r)
    return logits


def _run_decode(s):
    """A few steps of every request; then the requests are taken back to their prompts, as for another continuation
    (a step's logits are valid until the next step, so a caller that wants them all keeps copies)."""
    out = []
    for j in range(s.steps):
        logits = s.engine.step([StepItem(r, [s.tokens[r][n + j]], [0]) for r, n in enumerate(s.lengths)])
        out.append(logits.clone())
    for r, n in enumerate(s.lengths):
        s.engine.cache.truncate(r, n)
    return out


def _run_mixed(s):
    """One step: a token of every running request and a portion of a new prompt; then back to where they were."""
    R = len(s.lengths)
    items = [StepItem(r, [s.tokens[r][n]], [0]) for r, n in enumerate(s.lengths)]
    part = s.tokens[R][s.start:]
    logits = s.engine.step(items + [StepItem(R, part, [len(part) - 1])])
    for r, n in enumerate(s.lengths):
        s.engine.cache.truncate(r, n)
    if s.start:
        s.engine.cache.truncate(R, s.start)
    else:
        s.engine.finish(R)
    return logits


def _run_chat(s):
    """Whole requests: their prompts in one step, a token at a time after that, and their end."""
    out = []
    for j in range(s.steps + 1):
        if j == 0:
            items = [StepItem(r, s.tokens[r][:n], [n - 1]) for r, n in enumerate(s.lengths)]
        else:
            items = [StepItem(r, [s.tokens[r][n + j - 1]], [0]) for r, n in enumerate(s.lengths)]
        logits = s.engine.step(items)
        if s.sample is None:
            out.append(logits.clone())
        else:
            out.append([logits.clone(), sample_rows(logits, [s.sample] * len(items), [n + j for n in s.lengths])])
    for r in range(len(s.lengths)):
        s.engine.finish(r)
    return out


# ---------------------------------------------------------------- what a pass cannot do without

def _matrix_elements(spec_tensors, loops):
    """Elements of the layer weights that a token goes through (a looped layer counts once per run; the scalars and
    vectors are left out of the arithmetic, not of the bytes)."""
    once = ran = 0
    for name, (shape, role) in spec_tensors.items():
        if name in ("embed", "head", "model.embed_tokens.weight", "lm_head.weight"):
            continue
        n = math.prod(shape)
        once += n
        if role == "matrix":
            ran += n * loops(name)
    return once, ran


def work(case):
    d = MODELS[case["model"]]()
    tensors = expected_tensors(config_from_dict(d).model_spec())
    e = 4 if case["dtype"] == "float32" else 2
    lengths, steps = _lengths(case), _steps(case)
    vocab = d.get("vocab_size") or d["vocab"]
    width = d.get("hidden_size") or d["width"]
    loop = d.get("loop") or {"start": 0, "stop": 0, "times": 1}

    def runs(name):
        if name == "loop.in":
            return loop["times"]
        layer = int(name.split(".")[0][1:]) if name[0] == "l" and name[1].isdigit() else -1
        return loop["times"] if loop["start"] <= layer < loop["stop"] else 1

    once, ran = _matrix_elements(tensors, runs)
    head = vocab * width
    # layers: (times run, key and value entries kept per token, query-key and probability-value multiply-adds per pair,
    # window, float32 entries of the state, multiply-adds of the recurrence per token)
    layers = []
    if "num_hidden_layers" in d:
        layers = [(1, 2 * d["num_key_value_heads"] * 128, 2 * d["num_attention_heads"] * 128, 0, 0, 0)] * d["num_hidden_layers"]
    else:
        for i, layer in enumerate(d["layers"]):
            m, t = layer["mixer"], runs("l%d." % i)
            if layer["type"] == "mamba1":
                layers.append((t, 0, 0, 0, m["inner"] * (m["state"] + m["conv"] - 1), 3 * m["inner"] * m["state"]))
            elif layer["type"] == "parallel":
                a, b = m["left"], m["right"]
                layers.append((t, a["kv_heads"] * (a["dim"] + a["vdim"]), a["heads"] * (a["dim"] + a["vdim"]), a["mask"]["size"],
                               b["heads"] * b["dim"] * b["dim"] + width, 3 * b["heads"] * b["dim"] * b["dim"]))
            elif layer["type"] == "latent_attention":
                layers.append((t, m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), 0, 0, 0))
            else:
                layers.append((t, 2 * m["kv_heads"] * m["dim"], 2 * m["heads"] * m["dim"], m["mask"]["size"], 0, 0))
    total_bytes = total_flops = 0

    def one_step(items):
        """items: (tokens before, new tokens)."""
        nonlocal total_bytes, total_flops
        new, rows = sum(k for _, k in items), len(items)
        total_bytes += (once + head) * e + new * width * e + rows * vocab * 4
        total_flops += 2 * ran * new + 2 * head * rows
        for t, kept, pair, window, state, rec in layers:
            for before, k in items:
                total_bytes += t * (min(before, window or before) * kept * e + k * kept * e + 2 * state * 4)
                if window:
                    seen = sum(min(before + j + 1, window) for j in range(k))
                else:
                    seen = k * before + k * (k + 1) // 2
                total_flops += t * (2 * pair * seen + 2 * rec * k)

    if case["kind"] in ("prefill", "chat"):
        one_step([(0, n) for n in lengths])
    if case["kind"] in ("decode", "chat"):
        for j in range(steps):
            one_step([(n + j, 1) for n in lengths])
    if case["kind"] == "mixed":
        one_step([(n, 1) for n in lengths] + [(case["tokens"] // 2, case["portion"])])
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    """Four times what lies between the cases and their float64 values: 2.6e-6 in float32, 0.5 to 1.3 % in bfloat16 (one
    rounding is up to 0.4 %, and every sublayer reads and returns rounded rows)."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.005}
    return {"rel": 0.03, "max": 0.3}


# ---------------------------------------------------------------- the same in 64 bits

F64 = torch.float64


def _lin(w, a, b=None):
    y = a @ w.to(F64).T
    return y if b is None else y + b.to(F64)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _norm(x, w, eps):
    return _unit(x, eps) * w.to(F64)


def _rotate(x, positions, freq, mult=1.0):
    """x [T, heads, d]: pair (i, i + half) of the first 2 * half entries turned by positions * freq[i]."""
    half = freq.numel()
    ang = positions.to(F64)[:, None, None] * freq
    c, s = torch.cos(ang) * mult, torch.sin(ang) * mult
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _frequencies(rot):
    dims, base = rot["dims"], rot["base"]
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)
    sc = rot.get("scaling")
    if not sc:
        return f, 1.0
    at = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _attend(q, k, v, scale, visible, cap=0.0):
    """q [T, H, d], k [T, G, d], v [T, G, e]; one key/value head after the other."""
    T, H = q.shape[:2]
    per = H // k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=DEVICE)
    for g in range(k.shape[1]):
        s = torch.einsum("thd,sd->hts", q[:, g * per:(g + 1) * per], k[:, g]) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s.masked_fill_(~visible, -math.inf)
        out[:, g * per:(g + 1) * per] = torch.einsum("hts,se->the", torch.softmax(s, -1), v[:, g])
    return out.reshape(T, -1)


def _pairs(T):
    i = torch.arange(T, device=DEVICE)
    return i[:, None], i[None, :]


def _each(x, cuts, fn):
    """fn on the rows of every request by itself."""
    return torch.cat([fn(p) for p in torch.split(x, cuts)], 0)


def _logits_qwen3(d, t, tokens, cuts, rows):
    eps, H, G = d["rms_norm_eps"], d["num_attention_heads"], d["num_key_value_heads"]
    freq = d["rope_theta"] ** (-2.0 * torch.arange(64, dtype=F64, device=DEVICE) / 128)
    x = t["model.embed_tokens.weight"][tokens].to(F64)

    def mix(h, p):
        T = h.shape[0]
        pos = torch.arange(T, device=DEVICE)
        q = _rotate(_norm(_lin(t[p + "q_proj.weight"], h).view(T, H, 128), t[p + "q_norm.weight"], eps), pos, freq)
        k = _rotate(_norm(_lin(t[p + "k_proj.weight"], h).view(T, G, 128), t[p + "k_norm.weight"], eps), pos, freq)
        i, j = _pairs(T)
        return _attend(q, k, _lin(t[p + "v_proj.weight"], h).view(T, G, 128), 128 ** -0.5, j <= i)

    for n in range(d["num_hidden_layers"]):
        p = "model.layers.%d." % n
        h = _norm(x, t[p + "input_layernorm.weight"], eps)
        x = x + _lin(t[p + "self_attn.o_proj.weight"], _each(h, cuts, lambda r: mix(r, p + "self_attn.")))
        h = _norm(x, t[p + "post_attention_layernorm.weight"], eps)
        a = F.silu(_lin(t[p + "mlp.gate_proj.weight"], h)) * _lin(t[p + "mlp.up_proj.weight"], h)
        x = x + _lin(t[p + "mlp.down_proj.weight"], a)
    h = _norm(x[rows], t["model.norm.weight"], eps)
    return _lin(t["model.embed_tokens.weight" if d["tie_word_embeddings"] else "lm_head.weight"], h)


def _logits_falalix(d, t, tokens, cuts, rows):
    eps, m = d["norm"]["eps"], d["residual_mult"]

    def attention(h, p, c):
        T, H, G = h.shape[0], c["heads"], c["kv_heads"]
        q = _norm(_lin(t[p + "q"], h, t[p + "q.b"]), t[p + "q.norm"], eps).view(T, H, -1)
        k = _norm(_lin(t[p + "k"], h, t[p + "k.b"]), t[p + "k.norm"], eps).view(T, G, -1)
        i, j = _pairs(T)
        see = (j <= i) & ((i - j < c["mask"]["size"]) | (j < c["mask"]["keep_first"]))
        o = _attend(q, k, _lin(t[p + "v"], h, t[p + "v.b"]).view(T, G, -1), c["scale"], see)
        return _lin(t[p + "o"], o * torch.sigmoid(_lin(t[p + "g"], h)))

    def time_mix(h, p, c):
        (T, w), H, D = h.shape, c["heads"], c["dim"]
        prev = torch.cat([torch.zeros(1, w, dtype=F64, device=DEVICE), h[:-1]], 0)
        mixed = {s: h + (prev - h) * t[p + "mu." + s].to(F64) for s in "rkvgw"}
        r, k, v = (_lin(t[p + s], mixed[s]).view(T, H, D) for s in "rkv")
        gate = F.silu(_lin(t[p + "g"], mixed["g"]))
        dec = _lin(t[p + "w2"], torch.tanh(_lin(t[p + "w1"], mixed["w"]))) + t[p + "w0"].to(F64)
        dec = torch.exp(-torch.exp(dec)).view(T, H, D)
        u = t[p + "u"].to(F64)
        S = torch.zeros(H, D, D, dtype=F64, device=DEVICE)
        o = torch.empty(T, H, D, dtype=F64, device=DEVICE)
        for i in range(T):
            kv = k[i][:, :, None] * v[i][:, None, :]
            o[i] = torch.bmm(r[i][:, None, :], torch.addcmul(S, u[:, :, None], kv))[:, 0]
            S = torch.addcmul(kv, dec[i][:, :, None], S)
        o = _unit(o, eps).reshape(T, H * D) * t[p + "norm"].to(F64) * gate
        return _lin(t[p + "o"], o)

    def mamba(h, p, c):
        T, I, N, R, taps = h.shape[0], c["inner"], c["state"], c["dt_rank"], c["conv"]
        xz = _lin(t[p + "in"], h)
        x, z = xz[:, :I], xz[:, I:]
        pad = torch.cat([torch.zeros(taps - 1, I, dtype=F64, device=DEVICE), x], 0)
        x = F.silu(sum(pad[j:j + T] * t[p + "conv"][:, j].to(F64) for j in range(taps)) + t[p + "conv.b"].to(F64))
        low = _lin(t[p + "x"], x)
        step, B, C = F.softplus(_lin(t[p + "dt"], low[:, :R], t[p + "dt.b"])), low[:, R:R + N], low[:, R + N:]
        A = -torch.exp(t[p + "A_log"].to(F64))
        S = torch.zeros(I, N, dtype=F64, device=DEVICE)
        y = torch.empty(T, I, dtype=F64, device=DEVICE)
        for i in range(T):
            S = torch.exp(step[i][:, None] * A) * S + (step[i] * x[i])[:, None] * B[i]
            y[i] = S @ C[i]
        return _lin(t[p + "o"], (y + x * t[p + "D"].to(F64)) * F.silu(z))

    x = x0 = t["embed"][tokens].to(F64)
    loop = d["loop"]
    order = [(i, n if i == loop["start"] else None) for n in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    for i, opens in order + [(i, None) for i in range(loop["stop"], len(d["layers"]))]:
        if opens is not None:
            x = _lin(t["loop.in"], torch.cat([x, x0], -1)) + t["loop.step"][opens].to(F64)
        layer, p = d["layers"][i], "l%d." % i
        c = layer["mixer"]
        h = _norm(x, t[p + "norm1"], eps)
        if layer["type"] == "mamba1":
            x = x + m * _each(h, cuts, lambda r: mamba(r, p + "mix.", c))
        else:
            x = x + m * _each(h, cuts, lambda r: c["left_scale"] * attention(r, p + "mix.left.", c["left"])
                              + c["right_scale"] * time_mix(r, p + "mix.right.", c["right"]))
        if layer["mlp"] is not None:
            a = torch.relu(_lin(t[p + "mlp.up"], _norm(x, t[p + "norm2"], eps)))
            x = x + m * _lin(t[p + "mlp.down"], a * a)
    return _lin(t["head"], _norm(x[rows], t["final.norm"], eps))


def _logits_govopel(d, t, tokens, cuts, rows):
    eps = d["norm"]["eps"]

    def chunked(h, p, c):
        T, H, G = h.shape[0], c["heads"], c["kv_heads"]
        pos = torch.arange(T, device=DEVICE)
        freq, mult = _frequencies(c["rot"])
        k = _lin(t[p + "k"], h).view(T, G, -1)
        q = _unit(_rotate(_lin(t[p + "q"], h).view(T, H, -1), pos, freq, mult), eps)
        i, j = _pairs(T)
        size = c["mask"]["size"]
        return _attend(q, _unit(_rotate(k, pos, freq, mult), eps), k, c["scale"], (j <= i) & (i // size == j // size), c["softcap"])

    def latent(h, p, c):
        T, H, n, r, rank = h.shape[0], c["heads"], c["dim"], c["rot_dim"], c["kv_rank"]
        pos = torch.arange(T, device=DEVICE)
        freq, mult = _frequencies(c["rot"])
        q = _lin(t[p + "uq"], _norm(_lin(t[p + "dq"], h), t[p + "dq.norm"], eps)).view(T, H, n + r)
        low = _lin(t[p + "dkv"], h)
        lat = _norm(low[:, :rank], t[p + "dkv.norm"], eps)
        k_rot = _rotate(low[:, rank:].reshape(T, 1, r), pos, freq, mult).expand(T, H, r)
        q = torch.cat([q[..., :n], _rotate(q[..., n:], pos, freq, mult)], -1)
        k = torch.cat([_lin(t[p + "uk"], lat).view(T, H, n), k_rot], -1)
        i, j = _pairs(T)
        return _attend(q, k, _lin(t[p + "uv"], lat).view(T, H, -1), c["scale"], j <= i)

    x = _norm(t["embed"][tokens].to(F64), t["embed.norm"], eps)
    for i, layer in enumerate(d["layers"]):
        p, c, mlp = "l%d." % i, layer["mixer"], layer["mlp"]
        mix = latent if layer["type"] == "latent_attention" else chunked
        x = x + _norm(_lin(t[p + "mix.o"], _each(x, cuts, lambda r: mix(r, p + "mix.", c))), t[p + "norm1"], eps)
        gate = _lin(t[p + "mlp.gate"], x).clamp(max=mlp["limit"])
        up = _lin(t[p + "mlp.up"], x).clamp(-mlp["limit"], mlp["limit"])
        x = x + _norm(_lin(t[p + "mlp.down"], gate * torch.sigmoid(1.702 * gate) * (up + 1.0)), t[p + "norm2"], eps)
    y = _lin(t["embed"], _norm(x[rows], t["final.norm"], eps))
    return d["logit_softcap"] * torch.tanh(y / d["logit_softcap"])


def exact(case, seed):
    """What run() returns, from whole sequences in float64 (None where that would take too long)."""
    if case["kind"] == "mixed":
        flops = work(dict(case, kind="prefill", requests=1, tokens=sum(_lengths(case)) + case["tokens"] // 2 + case["portion"]))["flops"]
    else:
        flops = work(dict(case, kind="prefill"))["flops"]
    if flops > 4e14:
        return None
    d = MODELS[case["model"]]()
    config = config_from_dict(d)
    t = _weights(config, seed, parse_dtype(case["dtype"]))
    seqs = _tokens(case, seed, d.get("vocab_size") or d["vocab"])
    lengths, steps = _lengths(case), _steps(case)
    starts = [sum(len(q) for q in seqs[:i]) for i in range(len(seqs))]
    if case["kind"] == "prefill":
        wanted = [[s + n - 1 for s, n in zip(starts, lengths)]]
    elif case["kind"] == "decode":
        wanted = [[s + n + j for s, n in zip(starts, lengths)] for j in range(steps)]
    elif case["kind"] == "mixed":
        wanted = [[s + n for s, n in zip(starts, lengths)] + [starts[-1] + len(seqs[-1]) - 1]]
    else:
        wanted = [[s + n + j - 1 for s, n in zip(starts, lengths)] for j in range(steps + 1)]
    fn = _logits_qwen3 if "num_hidden_layers" in d else _logits_falalix if d["architecture"] == "Falalix" else _logits_govopel
    tokens = torch.tensor([k for q in seqs for k in q], device=DEVICE)
    rows = torch.tensor([r for w in wanted for r in w], device=DEVICE)
    got = list(torch.split(fn(d, t, tokens, [len(q) for q in seqs], rows), len(wanted[0])))
    if case["kind"] in ("prefill", "mixed"):
        return got[0]
    return [[g, None] for g in got] if case["dtype"] == "float32" else got
