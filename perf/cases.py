"""The work that this engine is timed on: requests served through the step function.

A case is a batch of requests that arrive together.  Their prompts go in as portions under a token
budget a step, beside one token a step of every request that is already generating (which is how the
scheduler fills its steps), until each request has had ``new`` next-token distributions.  The tokens
are given, as in a trace replay or when continuations are scored, so that a pass's work and its logits
do not hang on a tie between two tokens.  A pass takes in every request, runs all of its steps, keeps
the logits of every wanted place and gives the requests' pages back.

Keys of a case: ``model`` (a name of ``GPT2`` or ``LEBEDRA``), ``dtype`` (of the engine), ``requests``,
``shortest`` / ``longest`` (prompt lengths, spread evenly between the two), ``new`` (logits a request),
``portion`` (the longest piece of a prompt in a step).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rosellm_b200.config import EngineConfig, GPT2Config
from rosellm_b200.config.base import resolve_architecture
from rosellm_b200.config.lebedra import LebedraConfig
from rosellm_b200.engine.runner import ModelRunner, StepEntry
from rosellm_b200.models.model import named_params_of_spec

BUDGET = 2048      # tokens a step
MAX_REQUESTS = 64  # requests live at once, the engine's default
POSITIONS = 1024
STD = 0.02         # of random weights

GPT2 = {
    "gpt2-124M": dict(n_layer=12, n_embd=768, n_head=12, n_inner=3072),
    "gpt2-355M": dict(n_layer=24, n_embd=1024, n_head=16, n_inner=4096),
    "gpt2-1.5B": dict(n_layer=48, n_embd=1600, n_head=25, n_inner=6400),
}
GPT2_VOCAB = 50257

# Latent attention (one cached row a token), gated feed-forwards, norms on the sublayers' outputs.  All
# feed-forwards are dense: the choice of experts turns on ties that bfloat16 decides either way.
LEBEDRA = {
    "lebedra-2048": dict(layers=4, vocab=32000, width=2048, heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, ff=8192,
                         side=128),
}


def listed():
    def case(name, model, requests, shortest, longest, new, dtype="bfloat16", portion=512):
        return dict(name=name, model=model, dtype=dtype, requests=requests, shortest=shortest, longest=longest, new=new,
                    portion=portion)

    return [
        # the least a user asks for: the first token after a short prompt (latency, launches)
        case("first token 124M", "gpt2-124M", 1, 33, 33, 1),
        # one person reading along: decode at batch 1
        case("one request 124M", "gpt2-124M", 1, 512, 512, 65),
        # the headline workload: decode at batch 8 after 512 tokens
        case("8 requests 124M", "gpt2-124M", 8, 512, 512, 65),
        # a full engine of the small model, prompts of all lengths
        case("64 requests 124M", "gpt2-124M", 64, 17, 511, 33),
        # prompts alone (scoring, first tokens): 2,048 tokens in one step
        case("prompts 124M", "gpt2-124M", 2, 1024, 1024, 1, portion=1024),
        # the 32-bit path, which users check results with
        case("8 requests 124M fp32", "gpt2-124M", 8, 41, 397, 17, dtype="float32"),
        # continuous batching: portions of prompts beside decoded rows in most steps
        case("64 requests 355M", "gpt2-355M", 64, 16, 959, 33),
        # the large model: one reader, a few, a full engine, and prompts alone
        case("one request 1.5B", "gpt2-1.5B", 1, 896, 896, 33),
        case("8 requests 1.5B", "gpt2-1.5B", 8, 301, 895, 33),
        case("64 requests 1.5B", "gpt2-1.5B", 64, 63, 511, 17),
        case("prompts 1.5B", "gpt2-1.5B", 2, 1024, 1024, 1, portion=1024),
        # latent attention and gated feed-forwards
        case("8 requests latent", "lebedra-2048", 8, 512, 512, 33),
    ]


def draw(rng):
    """Another case of the same ranges; none costs more than the largest listed one."""
    def spread(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))

    limit = max(_cost(c) for c in listed())
    while True:
        model = rng.choice([*GPT2, *GPT2, *LEBEDRA])
        dtype = "float32" if model == "gpt2-124M" and rng.random() < 0.3 else "bfloat16"
        new = spread(1, 65)
        longest = spread(5, POSITIONS + 1 - new)
        case = dict(model=model, dtype=dtype, requests=spread(1, MAX_REQUESTS), shortest=rng.randint(min(longest, 3), longest),
                    longest=longest, new=new, portion=rng.choice([256, 512, 512, 1024]))
        if _cost(case) <= limit and (dtype == "bfloat16" or _tokens(case) <= 4096):
            return case


# ---- sizes -------------------------------------------------------------------------------------------------
def _config(case):
    if case["model"] in GPT2:
        return GPT2Config(**GPT2[case["model"]], vocab_size=GPT2_VOCAB, n_positions=POSITIONS, layer_norm_epsilon=1e-5,
                          activation_function="gelu_new")
    z = LEBEDRA[case["model"]]
    mixer = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot_dim"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
             "scale": (z["dim"] + z["rot_dim"]) ** -0.5, "rot": {"dims": z["rot_dim"], "base": 10000.0}}
    return LebedraConfig.from_dict({
        "architecture": "Lebedra", "vocab": z["vocab"], "width": z["width"], "residual_mult": 0.5, "norm": {"eps": 1e-6},
        "token_side": {"dim": z["side"]}, "max_positions": POSITIONS,
        "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": z["ff"]}}] * z["layers"]})


def _lengths(case):
    return [int(round(x)) for x in np.linspace(case["shortest"], case["longest"], case["requests"])]


def _tokens(case):
    return sum(_lengths(case)) + case["requests"] * (case["new"] - 1)


def _plan(lengths, new, portion):
    """The steps of a pass: lists of (request, first token, tokens, whether its last token's logits are wanted)."""
    done = [0] * len(lengths)
    end = [n + new - 1 for n in lengths]
    steps = []
    while any(d < e for d, e in zip(done, end)):
        step, room = [], BUDGET
        for r, n in enumerate(lengths):  # requests that generate: a token each
            if n <= done[r] < end[r] and room:
                step.append((r, done[r], 1, True))
                room -= 1
        for r, n in enumerate(lengths):  # then portions of prompts, first come first served
            take = min(n - done[r], portion, room)
            if take > 0:
                step.append((r, done[r], take, done[r] + take == n))
                room -= take
        for r, _, take, _ in step:
            done[r] += take
        steps.append(step)
    return steps


def _spec(case):
    cfg = _config(case)
    return resolve_architecture(cfg.to_dict()).build_spec(cfg)


def work(case):
    """Every step reads the weights that its tokens use and the cached rows of its requests once, and writes its
    tokens' rows and the wanted logits; products and attention over the visible keys."""
    size = 4 if case["dtype"] == "float32" else 2
    if case["model"] in GPT2:
        z = GPT2[case["model"]]
        layers, width, vocab = z["n_layer"], z["n_embd"], GPT2_VOCAB
        layer_weights = width * (4 * width + 2 * z["n_inner"])
        row = 2 * width                 # cached values a token and layer
        seen = 4 * width                # operations a token, layer and visible key
    else:
        z = LEBEDRA[case["model"]]
        layers, width, vocab = z["layers"], z["width"], z["vocab"]
        q, kv = z["heads"] * (z["dim"] + z["rot_dim"]), z["kv_rank"] * z["heads"] * (z["dim"] + z["vdim"])
        layer_weights = (width * (q + z["kv_rank"] + z["rot_dim"] + z["heads"] * z["vdim"] + 3 * z["ff"] + 2 * z["side"]) + kv)
        row = z["kv_rank"] + z["rot_dim"]
        seen = 2 * z["heads"] * (z["dim"] + z["rot_dim"] + z["vdim"])
    nbytes = flops = 0
    for step in _plan(_lengths(case), case["new"], case["portion"]):
        tokens = sum(n for _, _, n, _ in step)
        rows = sum(w for _, _, _, w in step)
        keys = sum(first + n for _, first, n, _ in step)
        pairs = sum(n * first + n * (n + 1) // 2 for _, first, n, _ in step)
        nbytes += size * (layers * (layer_weights + row * (keys + tokens)) + 2 * width * tokens)
        nbytes += (size * vocab * width if rows else 0) + 4 * vocab * rows
        flops += 2 * (layers * layer_weights * tokens + vocab * width * rows) + layers * seen * pairs
    return {"bytes": nbytes, "flops": flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# ---- inputs ------------------------------------------------------------------------------------------------
def _weights(case, seed):
    """Random weights by file name, on the GPU: N(0, 0.02) matrices in bfloat16, norm scales about one."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = {}
    for p in named_params_of_spec(_spec(case)):
        for name, shape in p.sources():
            t = torch.randn(shape, generator=g, device="cuda") * STD
            if p.spec.init == "ones":
                t += 1.0
            out[name] = t.to(torch.bfloat16) if p.spec.kind == "matrix" else t
    return out


def _prompts(case, seed):
    """The requests' given tokens (prompt and continuation), in an order of the seed's; and their prompts' lengths."""
    rng = np.random.default_rng(seed)
    lengths = [int(n) for n in rng.permutation(_lengths(case))]
    vocab = GPT2_VOCAB if case["model"] in GPT2 else LEBEDRA[case["model"]]["vocab"]
    return lengths, [rng.integers(0, vocab, n + case["new"] - 1).astype(np.int32) for n in lengths]


def prepare(case, seed):
    lengths, tokens = _prompts(case, seed)
    engine = EngineConfig(dtype=case["dtype"], max_num_seqs=MAX_REQUESTS, max_num_batched_tokens=BUDGET,
                          prefill_chunk_size=case["portion"], max_model_len=POSITIONS,
                          kv_cache_tokens=case["requests"] * (case["longest"] + case["new"] + 16))
    runner = ModelRunner(_config(case), _weights(case, seed), engine)
    runner.capture_graphs()
    steps = []
    for step in _plan(lengths, case["new"], case["portion"]):
        # a long portion as an int32 array and a single token as a list, as the scheduler hands them over
        pieces = [(r, tokens[r][first:first + n] if n > 16 else tokens[r][first:first + n].tolist(), [n - 1] if want else [])
                  for r, first, n, want in step]
        steps.append((pieces, sum(want for _, _, _, want in step)))
    logits = torch.empty((case["requests"] * case["new"], runner.spec.vocab_size), device="cuda")
    return {"runner": runner, "requests": case["requests"], "steps": steps, "logits": logits}


def run(state):
    """One pass: every request served and ended.  Returns the logits ``[wanted places, vocabulary]`` in the order of
    the steps and of the requests in a step."""
    runner, logits = state["runner"], state["logits"]
    slots = [runner.cache.new_request() for _ in range(state["requests"])]
    at = 0
    for pieces, rows in state["steps"]:
        got = runner.step([StepEntry(slots[r], ids, want) for r, ids, want in pieces])
        if rows:  # the step's logits are scratch of the next one
            logits[at:at + rows].copy_(got)
            at += rows
    for slot in slots:
        runner.cache.release(slot)
    return logits


def tolerance(case):
    """Against 64 bits the paths measure 7e-7 (32-bit) and 4e-3 to 7e-3 (bfloat16); two bfloat16 passes that add up in
    another order differ by up to 4e-3, and at most 0.021 in one logit."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 2e-2, "max": 1e-1}


# ---- the same logits in 64 bits ------------------------------------------------------------------------------
def exact(case, seed):
    """Whole sequences, no cache: every wanted place's logits from one plain forward pass over its request."""
    lengths, tokens = _prompts(case, seed)
    w = {name: t.double() for name, t in _weights(case, seed).items()}
    model = _gpt2_logits if case["model"] in GPT2 else _lebedra_logits
    z = GPT2[case["model"]] if case["model"] in GPT2 else LEBEDRA[case["model"]]
    per_request = [model(z, w, torch.from_numpy(t).long().cuda(), n - 1) for t, n in zip(tokens, lengths)]
    rows, taken = [], [0] * len(lengths)
    for step in _plan(lengths, case["new"], case["portion"]):
        for r, _, _, want in step:
            if want:
                rows.append(per_request[r][taken[r]])
                taken[r] += 1
    return torch.stack(rows)


def _causal(scores):
    n = scores.shape[-1]
    hidden = torch.ones((n, n), dtype=torch.bool, device=scores.device).triu(1)
    return scores.masked_fill(hidden, float("-inf"))


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _gpt2_logits(z, w, tokens, first):
    """Logits of the places from ``first`` on."""
    n, width, heads = len(tokens), z["n_embd"], z["n_head"]

    def norm(x, name):
        return torch.nn.functional.layer_norm(x, (width,), w[name + ".weight"], w[name + ".bias"], 1e-5)

    def linear(x, name):
        return x @ w[name + ".weight"] + w[name + ".bias"]

    x = w["wte.weight"][tokens] + w["wpe.weight"][:n]
    for i in range(z["n_layer"]):
        p = f"h.{i}."
        q, k, v = (t.view(n, heads, -1).transpose(0, 1) for t in linear(norm(x, p + "ln_1"), p + "attn.c_attn").split(width, -1))
        prob = torch.softmax(_causal(q @ k.transpose(1, 2) / math.sqrt(width // heads)), -1)
        x = x + linear((prob @ v).transpose(0, 1).reshape(n, width), p + "attn.c_proj")
        x = x + linear(_gelu(linear(norm(x, p + "ln_2"), p + "mlp.c_fc")), p + "mlp.c_proj")
    return norm(x[first:], "ln_f") @ w["wte.weight"].T


def _lebedra_logits(z, w, tokens, first):
    """Logits of the places from ``first`` on."""
    n, heads, dim, rot, rank = len(tokens), z["heads"], z["dim"], z["rot_dim"], z["kv_rank"]

    def norm(x, name):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w[name]

    def turned(v):  # pairs (2i, 2i+1) by the angle position * base^(-2i/rot)
        angle = (torch.arange(n, device=v.device).double()[:, None]
                 * 10000.0 ** (-torch.arange(0, rot, 2, device=v.device).double() / rot))
        c, s = (f(angle).view([n] + [1] * (v.dim() - 2) + [rot // 2]) for f in (torch.cos, torch.sin))
        a, b = v[..., 0::2], v[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)

    x = w["embed"][tokens]
    for i in range(z["layers"]):
        p = f"l{i}."
        q = (x @ w[p + "mix.q"].T).view(n, heads, dim + rot)
        latent, k_rot = (x @ w[p + "mix.dkv"].T).split([rank, rot], -1)
        latent = norm(latent, p + "mix.dkv.norm")
        k = (latent @ w[p + "mix.uk"].T).view(n, heads, dim)
        v = (latent @ w[p + "mix.uv"].T).view(n, heads, z["vdim"])
        scores = torch.einsum("qhd,khd->hqk", q[..., :dim], k) + torch.einsum("qhr,kr->hqk", turned(q[..., dim:]), turned(k_rot))
        scores = _causal(scores * (dim + rot) ** -0.5)
        sink = w[p + "mix.sink"].view(-1, 1, 1).expand(heads, n, 1)  # one more score in the denominator, without a value
        prob = torch.softmax(torch.cat([scores, sink], -1), -1)[..., :n]
        x = x + 0.5 * norm(torch.einsum("hqk,khv->qhv", prob, v).reshape(n, -1) @ w[p + "mix.o"].T, p + "norm1")
        inner = torch.relu(x @ w[p + "mlp.gate"].T) * (x @ w[p + "mlp.up"].T)
        x = x + 0.5 * norm(inner @ w[p + "mlp.down"].T, p + "norm2")
        side = w["side.embed"][tokens][:, i * z["side"]:(i + 1) * z["side"]]
        x = x + 0.5 * norm((_gelu(x @ w[p + "side.gate"].T) * side) @ w[p + "side.proj"].T, p + "side.norm")
    return norm(x[first:], "final.norm") @ w["head"].T
