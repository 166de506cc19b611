"""What a user of this engine has it do, as cases that can be timed and checked.

Every case is the Qwen3 dense decoder at layer sizes that bench.py and the tests use, random weights of the
distributions of `weights/random_init.py`, driven through `ModelRunner.step` (the one path from tokens to logits: trace
replay, the scheduler and the Python entry point all call it) or through `Engine.generate`.  The kinds of pass:

  decode    some single-token steps of every live request, tokens given, behind prompts that are in the cache already
  prefill   new requests, their prompts in portions, logits of the last token of each, requests ended
  mixed     a new request's prompt in portions beside single tokens of live requests
  serve     `Engine.generate`: token ids in, token ids out, continuous batching with portions beside decoding

Where a pass of the full depth would hold too much memory for several states at once, a model has fewer layers of the
same sizes.
"""
from __future__ import annotations

import hashlib
import json
import math
import random

import torch

from inferloop_b200.config.registry import read_model_config
from inferloop_b200.engine.batch import StepEntry
from inferloop_b200.engine.engine import Engine
from inferloop_b200.engine.runner import ModelRunner
from inferloop_b200.sampling.params import SamplingParams

# hidden, query heads, kv heads, head size, feed-forward, vocabulary, positions
SIZES = {
    "tiny": (96, 6, 2, 32, 224, 320, 256),               # the tests' odd sizes, on the general-purpose kernels
    "small": (256, 8, 2, 128, 384, 1000, 2048),          # the tests' smallest model at the serving geometry
    "8b": (4096, 32, 8, 128, 12288, 151936, 4096),
    "14b": (5120, 40, 8, 128, 17408, 151936, 4096),
    "32b": (5120, 64, 8, 128, 25600, 151936, 16384),
}
F64 = torch.float64
DEVICE = "cuda:0"


def _case(name, kind, model, layers, dtype="bfloat16", page=16, batch=1, prompt=0, steps=0, portion=0, tie=False, bias=False,
          window=0, sampled=False):
    """batch, prompt: live requests and the tokens each has in the cache before the pass (about: lengths are ragged);
    steps: single-token steps (mixed: steps with a portion) of a pass; portion: tokens of a new prompt a step takes;
    serve: `batch` requests at most live, twice as many submitted, `steps` new tokens each; prefill: `batch` new prompts
    of about `prompt` tokens; window: every second layer sees that many keys only (0: none)."""
    c = dict(kind=kind, model=model, layers=layers, dtype=dtype, page=page, batch=batch, prompt=prompt, steps=steps,
             portion=portion, tie=tie, bias=bias, window=window, sampled=sampled)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a toy model, one request; launches and latency are all there is
        _case("small decode 1", "decode", "small", 2, batch=1, prompt=70, steps=8),
        # one user at a prompt: latency per token
        _case("8b decode 1", "decode", "8b", 36, batch=1, prompt=1024, steps=4),
        # the headline: a few users decoding together
        _case("8b decode 8", "decode", "8b", 36, batch=8, prompt=1024, steps=4),
        # a busy server
        _case("8b decode 64", "decode", "8b", 36, batch=64, prompt=1024, steps=2),
        # a batch that no recorded size fits exactly, other layer sizes
        _case("14b decode 19", "decode", "14b", 20, batch=19, prompt=700, steps=4),
        # few long conversations
        _case("32b decode 2 long", "decode", "32b", 12, batch=2, prompt=6000, steps=4),
        # one prompt to its first token
        _case("8b prefill 2048", "prefill", "8b", 36, batch=1, prompt=2048, portion=2048),
        # a long document in portions
        _case("32b prefill 7000", "prefill", "32b", 12, batch=1, prompt=7000, portion=2048),
        # continuous batching: a prompt in portions beside decoding requests
        _case("14b mixed 24", "mixed", "14b", 20, batch=24, prompt=1000, steps=3, portion=384),
        # a whole job through the Python entry point
        _case("8b serve 8", "serve", "8b", 36, batch=8, prompt=300, steps=24, portion=512),
        # the 32-bit path, which checks and trace replay against another implementation use
        _case("8b float32 decode 4", "decode", "8b", 4, dtype="float32", batch=4, prompt=100, steps=4),
        _case("8b float32 prefill 200", "prefill", "8b", 4, dtype="float32", batch=1, prompt=200, portion=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed", "mixed", "serve"])
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    model = rng.choice(["small", "8b", "8b", "14b", "32b"]) if rng.random() < 0.9 else "tiny"
    small = model in ("tiny", "small")
    layers = _log(rng, 2, 3 if dtype == "float32" else 12)
    page = rng.choice([16, 16, 32, 64])
    tie, bias = rng.random() < 0.3, rng.random() < 0.15
    window = rng.choice([40, 500]) if rng.random() < 0.1 else 0
    most = {"tiny": 120, "small": 1500}.get(model, 3000)
    if dtype == "float32":
        most = min(most, 300)
    if kind == "decode":
        batch = _log(rng, 1, 24 if dtype == "float32" else 100)
        prompt = _log(rng, 16, max(16, min(most, 40000 // batch)))
        return _case(None, kind, model, layers, dtype, page, batch, prompt, 4, 0, tie, bias, window)
    if kind == "prefill":
        batch = _log(rng, 1, 6)
        prompt = _log(rng, 16, max(16, min(most, 4000 // batch)))
        return _case(None, kind, model, layers, dtype, page, batch, prompt, 0, rng.choice([256, 512, 2048]), tie, bias, window)
    if kind == "mixed":
        batch = _log(rng, 1, 40)
        prompt = _log(rng, 16, max(16, min(most, 20000 // batch)))
        portion = _log(rng, 20, 30 if model == "tiny" else 100 if dtype == "float32" else 500)
        return _case(None, kind, model, layers, dtype, page, batch, prompt, 3, portion, tie, bias, window)
    batch = _log(rng, 2, 24)
    prompt = _log(rng, 16, min(most // 2, 400))
    return _case(None, kind, model, layers, "bfloat16" if not small else dtype, page, batch, prompt, _log(rng, 8, 24),
                 rng.choice([128, 512]), False, False, window, rng.random() < 0.3)


# ------------------------------------------------------------------ weights and inputs
def _config(case):
    hidden, nq, nkv, d, inter, vocab, positions = SIZES[case["model"]]
    c = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=case["layers"], hidden_size=hidden,
             num_attention_heads=nq, num_key_value_heads=nkv, head_dim=d, intermediate_size=inter, vocab_size=vocab,
             rope_theta=1000000.0, rms_norm_eps=1e-6, attention_bias=case["bias"], tie_word_embeddings=case["tie"],
             max_position_embeddings=positions, hidden_act="silu")
    if case["window"]:
        c["layer_types"] = ["sliding_attention" if i % 2 else "full_attention" for i in range(case["layers"])]
        c["sliding_window"] = case["window"]
    return c


def _generator(seed, name):
    h = hashlib.sha256(f"{seed}:{name}".encode()).digest()
    return torch.Generator(device=DEVICE).manual_seed(int.from_bytes(h[:7], "little"))


def _successor(case, seed):
    """serve: the token that the model answers each token with."""
    return torch.randperm(SIZES[case["model"]][5], generator=_generator(seed, "successor"), device=DEVICE)


def _weight(case, seed, name, shape):
    """One tensor by its name in the checkpoint, as the engine holds it: matrices N(0, 0.02) in the case's dtype, norm
    weights 1 + N(0, 0.1) and biases in 32 bits; the two matrices of a layer that write into the residual stream divided
    by sqrt(2 layers) and embeddings N(0, 1), as models are initialised so that the stream keeps its size over the depth
    (without it every layer's rounding is the next one's signal, and logits of 36 layers in bfloat16 are 4 % off).  For
    `serve` the output matrix answers each token with one successor (random matrices alone give logits whose two best
    are nearly equal; a trained model's are not)."""
    if case["kind"] == "serve" and name == "lm_head.weight":
        rows = torch.randn(shape, generator=_generator(seed, "embed_tokens.weight"), device=DEVICE, dtype=torch.bfloat16)
        out = torch.empty_like(rows)
        out[_successor(case, seed)] = rows.mul_(0.02)
        return out.to(getattr(torch, case["dtype"]))
    matrix = len(shape) == 2
    dt = getattr(torch, case["dtype"]) if matrix else torch.float32
    if name == "embed_tokens.weight":
        return torch.randn(shape, generator=_generator(seed, name), device=DEVICE, dtype=torch.bfloat16).to(dt)
    t = torch.randn(shape, generator=_generator(seed, name), device=DEVICE, dtype=dt)
    if "norm" in name:
        return t.mul_(0.1).add_(1.0)
    return t.mul_(0.02 / math.sqrt(2 * case["layers"]) if name.endswith(("o_proj.weight", "down_proj.weight")) else 0.02)


def _shapes(case):
    """{name: shape} of the checkpoint's tensors."""
    hidden, nq, nkv, d, inter, vocab, _ = SIZES[case["model"]]
    out = {"embed_tokens.weight": (vocab, hidden), "norm.weight": (hidden,)}
    if not case["tie"]:
        out["lm_head.weight"] = (vocab, hidden)
    for i in range(case["layers"]):
        out.update(_layer_shapes(case, i))
    return out


def _layer_shapes(case, i):
    hidden, nq, nkv, d, inter, _, _ = SIZES[case["model"]]
    p = f"layers.{i}."
    out = {p + "input_layernorm.weight": (hidden,), p + "post_attention_layernorm.weight": (hidden,),
           p + "self_attn.q_proj.weight": (nq * d, hidden), p + "self_attn.k_proj.weight": (nkv * d, hidden),
           p + "self_attn.v_proj.weight": (nkv * d, hidden), p + "self_attn.o_proj.weight": (hidden, nq * d),
           p + "self_attn.q_norm.weight": (d,), p + "self_attn.k_norm.weight": (d,),
           p + "mlp.gate_proj.weight": (inter, hidden), p + "mlp.up_proj.weight": (inter, hidden),
           p + "mlp.down_proj.weight": (hidden, inter)}
    if case["bias"]:
        out.update({p + "self_attn.q_proj.bias": (nq * d,), p + "self_attn.k_proj.bias": (nkv * d,),
                    p + "self_attn.v_proj.bias": (nkv * d,), p + "self_attn.o_proj.bias": (hidden,)})
    return out


def _lengths(case):
    """Ragged lengths of the live requests' prompts (of the new ones, for prefill and serve): the first is `prompt`, the
    others between half of it and all of it.  They belong to the case and not to the seed: every state has equal work."""
    rng = random.Random(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True))
    n = case["batch"] * (2 if case["kind"] == "serve" else 1)
    lo = case["prompt"] // 4 if case["kind"] == "serve" else case["prompt"] // 2
    return [case["prompt"]] + [rng.randint(max(1, lo), case["prompt"]) for _ in range(n - 1)]


def _tokens(case, seed, key, n):
    rng = random.Random(f"{seed}:{key}")
    vocab = SIZES[case["model"]][5]
    return [rng.randrange(vocab) for _ in range(n)]


def _room(case):
    """Tokens a live request may grow to before the pass starts over."""
    return min(SIZES[case["model"]][6], case["prompt"] + (200 if case["model"] == "tiny" else 1500))


def prepare(case, seed):
    """The model with its weights bound, requests' prompts in the cache, the decode step of this batch recorded."""
    config = _config(case)
    _, _, spec = read_model_config(json.dumps(config))
    tensors = {n: _weight(case, seed, n, s) for n, s in _shapes(case).items()}
    lengths = _lengths(case)
    live = case["batch"] if case["kind"] != "prefill" else len(lengths)
    room = {"decode": _room(case), "mixed": _room(case), "prefill": case["prompt"],
            "serve": case["prompt"] + case["steps"] + 1}[case["kind"]]
    pages = live * (-(-room // case["page"]) + 1)
    if case["kind"] == "mixed":
        pages += -(-case["steps"] * case["portion"] // case["page"]) + 1
    runner = ModelRunner(spec, tensors, getattr(torch, case["dtype"]), torch.device(DEVICE), case["page"], pages + 8, live + 1)
    state = {"case": case, "seed": seed, "runner": runner, "lengths": lengths, "passes": 0}
    if case["kind"] == "serve":
        state["engine"] = Engine(config, runner=runner, block_size=case["page"], max_num_seqs=case["batch"],
                                 prefill_chunk_tokens=case["portion"])
        state["prompts"] = [_tokens(case, seed, f"prompt {i}", n) for i, n in enumerate(lengths)]
        # the shared recorded steps and scratch buffers of a program that serves already
        state["engine"].generate(state["prompts"][:case["batch"]], SamplingParams(), 3)
    elif case["kind"] == "prefill":
        state["prompts"] = [_tokens(case, seed, f"prompt {i}", n) for i, n in enumerate(lengths)]
    else:
        state["portions"] = [_tokens(case, seed, f"portion {i}", case["portion"]) for i in range(case["steps"])] \
            if case["kind"] == "mixed" else []
        _start(state)
    return state


def _start(state):
    """The live requests' prompts into the cache, in portions, and one decode step."""
    case, runner = state["case"], state["runner"]
    for i, n in enumerate(state["lengths"]):
        toks = _tokens(case, state["seed"], f"prompt {i}", n)
        runner.begin(i)
        for a in range(0, n, 2048):
            runner.step([StepEntry(i, toks[a:a + 2048], [])])
    first = _tokens(case, state["seed"], "first", len(state["lengths"]))
    runner.step([StepEntry(i, [t], [0]) for i, t in enumerate(first)], draw_greedy=True)
    state["at"] = case["prompt"] + 1


def _given(case, seed, k, n):
    """The tokens of step k of a decode or mixed pass."""
    return _tokens(case, seed, f"step {k}", n)


# ------------------------------------------------------------------ one pass
def run(state):
    case, runner = state["case"], state["runner"]
    kind = case["kind"]
    if kind == "serve":
        params = [SamplingParams(temperature=0.7, top_p=0.95, seed=i) if case["sampled"] and i % 2 else SamplingParams()
                  for i in range(len(state["prompts"]))]
        out = state["engine"].generate(state["prompts"], params, case["steps"])
        state["engine"].take_completed()
        return torch.tensor(out)
    if kind == "prefill":
        prompts, done = state["prompts"], [0] * len(state["prompts"])
        logits = [None] * len(prompts)
        for i in range(len(prompts)):
            runner.begin(i)
        while any(done[i] < len(p) for i, p in enumerate(prompts)):
            entries, last, left = [], [], case["portion"]
            for i, p in enumerate(prompts):
                n = min(left, len(p) - done[i])
                if n > 0:
                    entries.append(StepEntry(i, p[done[i]:done[i] + n], [n - 1] if done[i] + n == len(p) else []))
                    if done[i] + n == len(p):
                        last.append(i)
                    done[i] += n
                    left -= n
            got = runner.step(entries)
            for row, i in enumerate(last):
                logits[i] = got[row].clone()
        for i in range(len(prompts)):
            runner.end(i)
        return logits
    B = len(state["lengths"])
    if state["at"] + case["steps"] > _room(case):         # the conversations are as long as they may get: new ones
        for i in range(B):
            runner.end(i)
        _start(state)
    out = []
    if kind == "mixed":
        runner.begin("new")
    for k in range(case["steps"]):
        entries = [StepEntry(i, [t], [0]) for i, t in enumerate(_given(case, state["seed"], k, B))]
        if kind == "mixed":
            entries.append(StepEntry("new", state["portions"][k], [case["portion"] - 1] if k + 1 == case["steps"] else []))
        logits, drawn = runner.step(entries, draw_greedy=True)
        out.append(logits.clone())
    if kind == "mixed":
        runner.end("new")
    state["at"] += case["steps"]
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _sequences(case):
    """(tokens in the cache before the pass, tokens of the pass, logits rows of the pass) of each request."""
    lengths = _lengths(case)
    if case["kind"] == "decode":
        return [(n + 1, case["steps"], case["steps"]) for n in lengths]
    if case["kind"] == "mixed":
        return [(n + 1, case["steps"], case["steps"]) for n in lengths] + [(0, case["steps"] * case["portion"], 1)]
    if case["kind"] == "prefill":
        return [(0, n, 1) for n in lengths]
    return [(0, n + case["steps"] - 1, case["steps"]) for n in lengths]


def _steps(case):
    """How many steps a pass needs at least: the weights are read once in each."""
    lengths = _lengths(case)
    if case["kind"] in ("decode", "mixed"):
        return case["steps"]
    if case["kind"] == "prefill":
        return -(-sum(lengths) // case["portion"])
    return 2 * case["steps"]                              # two rounds of `batch` live requests


def work(case):
    hidden, nq, nkv, d, inter, vocab, _ = SIZES[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    layer = (nq + 2 * nkv) * d * hidden + nq * d * hidden + 3 * inter * hidden
    seqs, L = _sequences(case), case["layers"]
    tokens, rows = sum(n for _, n, _ in seqs), sum(r for _, _, r in seqs)
    weights = (layer * L + vocab * hidden) * size
    kv, pairs = 0, 0
    for at, n, _ in seqs:
        own = n * (n + 1) // 2 if case["kind"] in ("prefill", "serve") or n == case["portion"] * case["steps"] else 0
        if own:                                           # a prompt: read and written once
            kv, pairs = kv + n, pairs + own
        else:                                             # single tokens: every key of the request each time
            kv, pairs = kv + sum(at + k + 1 for k in range(n)), pairs + sum(at + k + 1 for k in range(n))
    full = L - (L // 2 if case["window"] else 0)          # (layers with a window count as nothing: a lower bound)
    moved = weights * _steps(case) + kv * 2 * nkv * d * size * full + rows * vocab * 4 + tokens * hidden * size
    flops = 2 * tokens * layer * L + 4 * pairs * nq * d * full + 2 * rows * vocab * hidden
    return {"bytes": float(moved), "flops": float(flops)}


def tolerance(case):
    if case["kind"] == "serve":
        return {"rel": 0.0, "differ": 0.01}               # token ids whose logits stand apart: only a tie may differ
    if case["dtype"] == "float32":
        return {"rel": 2e-6}                               # (measured against 64 bits: 3e-7 to 5e-7)
    return {"rel": 0.025}                                  # (against 64 bits 5e-3 to 7e-3; twice the same inputs: 6e-3)


# ------------------------------------------------------------------ in 64 bits
def _rms(x, w, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, positions, theta=1000000.0):
    half = x.shape[-1] // 2
    freq = theta ** (-torch.arange(half, device=x.device, dtype=F64) / half)
    angle = positions.to(F64)[:, None, None] * freq
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _logits(case, seed, sequences, wanted):
    """Logits [rows, vocab] of each sequence at its wanted positions, whole sequences from position 0."""
    hidden, nq, nkv, d, inter, vocab, _ = SIZES[case["model"]]
    get = lambda name, shape: _weight(case, seed, name, shape)
    table = get("embed_tokens.weight", (vocab, hidden))
    lens = [len(s) for s in sequences]
    x = table[torch.tensor([t for s in sequences for t in s], device=DEVICE)].to(F64)
    pos = torch.cat([torch.arange(n, device=DEVICE) for n in lens])
    for li in range(case["layers"]):
        w = {n.split(".", 2)[2]: get(n, s).to(F64) for n, s in _layer_shapes(case, li).items()}
        b = {k: (w[f"self_attn.{k}_proj.bias"] if case["bias"] else 0.0) for k in "qkvo"}
        h = _rms(x, w["input_layernorm.weight"])
        q = _rms((h @ w["self_attn.q_proj.weight"].T + b["q"]).view(-1, nq, d), w["self_attn.q_norm.weight"])
        k = _rms((h @ w["self_attn.k_proj.weight"].T + b["k"]).view(-1, nkv, d), w["self_attn.k_norm.weight"])
        v = (h @ w["self_attn.v_proj.weight"].T + b["v"]).view(-1, nkv, d)
        q, k = _rotate(q, pos), _rotate(k, pos)
        o = torch.empty_like(q)
        a = 0
        for n in lens:
            i = torch.arange(n, device=DEVICE)
            sees = i[:, None] >= i[None, :]
            if case["window"] and li % 2:
                sees &= i[:, None] - i[None, :] < case["window"]
            for g in range(nkv):
                heads = slice(g * (nq // nkv), (g + 1) * (nq // nkv))
                step = max(1, (1 << 27) // (n * (nq // nkv)))
                for r in range(0, n, step):
                    s = torch.einsum("thd,sd->hts", q[a + r:a + min(n, r + step), heads], k[a:a + n, g]) / math.sqrt(d)
                    p = torch.softmax(s.masked_fill_(~sees[r:r + step], -math.inf), -1)
                    o[a + r:a + min(n, r + step), heads] = torch.einsum("hts,sd->thd", p, v[a:a + n, g])
                    del s, p
            a += n
        x = x + (o.reshape(-1, nq * d) @ w["self_attn.o_proj.weight"].T + b["o"])
        h = _rms(x, w["post_attention_layernorm.weight"])
        for r in range(0, h.shape[0], 4096):
            z = h[r:r + 4096] @ w["mlp.gate_proj.weight"].T
            x[r:r + 4096] += (z * torch.sigmoid(z) * (h[r:r + 4096] @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T
        del w
    final = get("norm.weight", (hidden,)).to(F64)
    out, a, rows = [], 0, []
    for n, want in zip(lens, wanted):
        rows.append(x[a + torch.tensor(want, device=DEVICE)])
        a += n
    normed = _rms(torch.cat(rows), final)
    head = table if case["tie"] else get("lm_head.weight", (vocab, hidden))
    logits = torch.cat([normed @ head[r:r + 16384].to(F64).T for r in range(0, vocab, 16384)], -1)
    a = 0
    for want in wanted:
        out.append(logits[a:a + len(want)])
        a += len(want)
    return out


def exact(case, seed):
    lengths, B = _lengths(case), len(_lengths(case))
    if case["kind"] == "serve":
        return None                                       # whole numbers: token ids
    # (about 25 TFLOP/s in 64 bits)
    total = sum(a + n for a, n, _ in _sequences(case))
    hidden, nq, nkv, d, inter, vocab, _ = SIZES[case["model"]]
    if 2.0 * total * (2 * (nq + nkv) * d + 3 * inter) * hidden * case["layers"] > 3.0e14:
        return None
    if case["kind"] == "prefill":
        seqs = [_tokens(case, seed, f"prompt {i}", n) for i, n in enumerate(lengths)]
        return [x[0] for x in _logits(case, seed, seqs, [[len(s) - 1] for s in seqs])]
    first = _tokens(case, seed, "first", B)
    given = [_given(case, seed, k, B) for k in range(case["steps"])]
    seqs = [_tokens(case, seed, f"prompt {i}", n) + [first[i]] + [g[i] for g in given] for i, n in enumerate(lengths)]
    wanted = [list(range(n + 1, n + 1 + case["steps"])) for n in lengths]
    if case["kind"] == "mixed":
        seqs.append([t for k in range(case["steps"]) for t in _tokens(case, seed, f"portion {k}", case["portion"])])
        wanted.append([len(seqs[-1]) - 1])
    rows = _logits(case, seed, seqs, wanted)
    out = [torch.stack([rows[i][k] for i in range(B)]) for k in range(case["steps"])]
    if case["kind"] == "mixed":
        out[-1] = torch.cat([out[-1], rows[B]])
    return out
