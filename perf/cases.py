"""What the engine is timed on: batches of requests that it opens, reads, decodes and closes.

Every case is a small model of one of the framework's designs with the layer sizes of a real one, and a
batch of requests that go through ``ModelRunner`` turn by turn, as the scheduler and the trace runner
drive it: a turn holds the next portion of every request that still has prompt to read and the next
token of every other, and gives the logits of each request's last prompt token and of each of its later
tokens.  The tokens are given (a trace is replayed), so the same inputs give the same logits whatever
is sampled.  ``cached`` tokens of a request stand in the prefix cache already, as a shared system
prompt or the turns of a conversation so far do; ``prompt`` new ones are read, ``steps`` decoded.
"""
from __future__ import annotations

import gc
import itertools
import json
import math

import numpy as np
import torch

from lgml_b200.config import config_from_dict
from lgml_b200.engine import ModelRunner, Runtime
from lgml_b200.models import build_model

DEVICE = "cuda:0"
PAGE = 64
BUDGET = 2048            # most tokens of one turn
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
WINDOW = 1024            # of the windowed attention layers


# ---- the cases ---------------------------------------------------------------------------------------

def _case(name, family, dtype, width, heads, kv_heads, head_dim, inner, layers, vocab, requests, cached, prompt, ragged, steps):
    return {"name": name, "family": family, "dtype": dtype, "width": width, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "inner": inner, "layers": layers, "vocab": vocab, "requests": requests, "cached": cached, "prompt": prompt, "ragged": ragged,
            "steps": steps}


def listed():
    return [
        # the smallest model (the tests' tiny configuration): a short prompt and a few tokens, all launches and latency
        _case("llama_tiny_b1", "llama", "bfloat16", 96, 6, 2, 32, 256, 3, 320, 1, 0, 19, False, 12),
        # one user's next turn in a conversation: a short question behind 2,048 cached tokens, then the answer
        _case("llama_8b_turn_b1", "llama", "bfloat16", 4096, 32, 8, 128, 14336, 2, 32000, 1, 2048, 37, False, 16),
        # decoding eight requests behind 2,048 tokens: the benchmark's own workload
        _case("llama_8b_decode_b8", "llama", "bfloat16", 4096, 32, 8, 128, 14336, 2, 32000, 8, 2048, 1, False, 16),
        # a busy server: 64 requests decode
        _case("llama_8b_decode_b64", "llama", "bfloat16", 4096, 32, 8, 128, 14336, 2, 32000, 64, 1536, 1, False, 24),
        # one long prompt, read at once
        _case("llama_8b_prompt", "llama", "bfloat16", 4096, 32, 8, 128, 14336, 2, 32000, 1, 0, 2048, False, 0),
        # prompts of many lengths arrive together: portions beside decodes
        _case("llama_3b_mixed", "llama", "bfloat16", 3072, 24, 8, 128, 8192, 2, 32000, 8, 0, 1500, True, 8),
        # as many key heads as query heads, long contexts
        _case("llama_13b_decode_b16", "llama", "bfloat16", 5120, 40, 40, 128, 13824, 2, 32000, 16, 3584, 1, False, 16),
        # the 32-bit mode, which traces are checked with: reading prompts, and decoding
        _case("llama_f32_prompt", "llama", "float32", 2048, 16, 4, 128, 5632, 2, 32000, 2, 0, 600, True, 2),
        _case("llama_f32_decode_b4", "llama", "float32", 2048, 16, 4, 128, 5632, 2, 32000, 4, 1024, 1, False, 8),
        # designs with recurrences: two prompts of different length, then a few tokens each
        _case("lefulorn_prompt", "lefulorn", "bfloat16", 2048, 16, 4, 128, 8192, 2, 32000, 2, 0, 2000, True, 4),
        _case("dizepel_prompt", "dizepel", "bfloat16", 2048, 16, 4, 128, 8192, 2, 32000, 2, 0, 1000, True, 4),
        # experts, latent attention and a gated recurrence: eight requests read and decode
        _case("nelosun_b8", "nelosun", "bfloat16", 2048, 16, 4, 128, 5632, 3, 32000, 8, 0, 200, True, 12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A model and a batch of the listed kinds: any design and type, widths of 96 to 5,120 (odd multiples of 8 among
    them), 1 to 64 requests, contexts up to 3,584 cached tokens, prompts of 1 to 2,048 tokens."""
    caps = [_cost(c) for c in listed()]
    while True:
        family = rng.choice(["llama"] * 6 + ["lefulorn", "dizepel", "nelosun"])
        dtype = "float32" if family == "llama" and rng.random() < 0.3 else "bfloat16"
        head_dim = rng.choice([64, 128, 128])
        if family == "llama":
            kv_heads = rng.choice([1, 2, 4, 5, 8, 8])
            heads = kv_heads * rng.choice([1, 2, 3, 4, 5])
            width = 8 * _log(rng, 64 if dtype == "float32" else 96, 256 if dtype == "float32" else 640)
        else:
            kv_heads = rng.choice([2, 4, 8])
            heads = kv_heads * rng.choice([2, 4])
            head_dim, width = 128, 256 * rng.randint(3, 16)
        inner = 8 * max(8, int(width * rng.uniform(2.0, 4.0)) // 8) if family != "nelosun" else 1024 * rng.randint(2, 9)
        layers = 3 if family == "nelosun" else rng.choice([1, 2, 3]) if family != "lefulorn" else 2
        requests = _log(rng, 1, 64 if dtype == "bfloat16" else 8)
        steps = rng.randint(1, 12)
        cached = PAGE * rng.randint(1, 56) if family == "llama" and rng.random() < 0.55 else 0
        prompt = 1 if cached and rng.random() < 0.6 else _log(rng, 2, 2048)
        ragged = prompt > 4 and requests > 1 and rng.random() < 0.6
        case = _case("", family, dtype, width, heads, kv_heads, head_dim, inner, layers, rng.choice([320, 8000, 32000]), requests, cached, prompt,
                     ragged, steps)
        del case["name"]
        if requests * (cached + prompt) <= 64 * 1600 and _cost(case) <= max(caps):
            return case


# ---- the models --------------------------------------------------------------------------------------

def _model_dict(case):
    """The configuration (config.json as a dictionary): the benchmark's layers of each design at the case's sizes."""
    W, H, G, D, F, L, V = (case[k] for k in ("width", "heads", "kv_heads", "head_dim", "inner", "layers", "vocab"))
    if case["family"] == "llama":
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": L, "hidden_size": W, "num_attention_heads": H,
                "num_key_value_heads": G, "head_dim": D, "intermediate_size": F, "vocab_size": V, "rope_theta": 500000.0, "rope_scaling": None,
                "rms_norm_eps": 1e-5, "tie_word_embeddings": False, "attention_bias": False, "mlp_bias": False, "max_position_embeddings": 4096,
                "hidden_act": "silu"}
    if case["family"] == "lefulorn":       # attention with a window, a sink and distance slopes, then the delta rule with a decay per channel
        att = {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5, "mask": {"size": WINDOW},
                                              "q_temp": {"coef": 0.1, "every": 256}}, "mlp": {"kind": "dense", "ff": F}}
        dl = {"type": "channel_delta", "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "conv": 4, "rank_a": 64, "rank_g": 64},
              "mlp": {"kind": "dense", "ff": F}}
        return {"architecture": "Lefulorn", "vocab": V, "width": W, "norm": {"eps": 1e-6}, "logit_scale": 1.0,
                "layers": [dict(att if i % 2 == 0 else dl) for i in range(L)]}
    if case["family"] == "dizepel":        # capped attention over convolved keys beside a state-space recurrence
        left = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "conv": 4, "scale": D ** -0.5, "softcap": 30.0,
                "rot": {"base": 500000.0, "dims": D // 2, "scaling": {"factor": 4.0, "original": 2048, "fast": 16.0, "slow": 1.0}}}
        right = {"heads": W // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
        layer = {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": {"kind": "dense", "ff": F}}
        return {"architecture": "Dizepel", "vocab": V, "width": W, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "canon": {"taps": 4},
                "layers": [dict(layer) for _ in range(L)]}
    # Nelosun: attention with a one in its denominator, latent attention and a gated linear recurrence, each beside experts by table
    mlp = {"kind": "moe", "expert": {"ff": F // 4, "limit": 7.0}, "router": {"experts": 8, "top": 2}}
    att = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5, "q_temp": {"coef": 0.1, "every": 1024}}
    lat = {"heads": H, "dim": D // 2, "rot_dim": 32, "vdim": D // 2, "q_rank": W // 4, "kv_rank": 96, "scale": (D // 2 + 32) ** -0.5,
           "rot": {"base": 10000.0, "dims": 32}}
    kinds = [("attention", att), ("latent_attention", lat), ("rglru", {"width": W, "blocks": W // 256, "conv": 4})]
    return {"architecture": "Nelosun", "vocab": V, "width": W, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
            "layers": [{"type": kinds[i % 3][0], "mixer": dict(kinds[i % 3][1]), "mlp": mlp} for i in range(L)]}


# Where the plain N(mean, 0.02 scale) of random weights would make a recurrence forget all at the same pace: decays from almost none
# to almost all, steps of a state-space recurrence around 0.05.
_SPREAD = {"lefulorn": {".A_log": (-0.5, 0.7), ".dt_bias": (-1.0, 1.0)}, "dizepel": {".A_log": (0.5, 0.7), ".dt_bias": (-3.0, 1.0)}}


def _weights(case, specs):
    """Random weights by name, on the device; the same for every seed (a user's program loads one model)."""
    g = torch.Generator(device=DEVICE).manual_seed(17)
    out = {}
    for s in specs:
        if s.kind == "int":            # every token's row of an expert table: different experts
            out[s.name] = torch.argsort(torch.rand(s.shape[0], s.below, device=DEVICE, generator=g), dim=1)[:, :s.shape[1]].to(torch.int32).contiguous()
            continue
        mean, sd = s.init[0], 0.02 * s.init[1]
        for end, spread in _SPREAD.get(case["family"], {}).items():
            if s.name.endswith(end):
                mean, sd = spread
        t = torch.randn(s.shape, device=DEVICE, generator=g) * sd + mean
        out[s.name] = t.to(DTYPES[case["dtype"]] if s.kind == "matrix" else torch.float32)
    return out


_kept = {}          # the one model in hand
_number = itertools.count()


def _model_key(case):
    return json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)


def _runner(case):
    """The engine's runner with its weights, its cache and the captured steps of earlier passes: a program keeps it."""
    key = _model_key(case)
    if key not in _kept:
        _kept.clear()
        gc.collect()
        torch.cuda.empty_cache()
        rt = Runtime(DEVICE, DTYPES[case["dtype"]])
        model = build_model(config_from_dict(_model_dict(case)))
        model.bind(_weights(case, [s for s in model.tensor_specs() if not s.optional]), rt)
        pages = -(-(case["cached"] + case["prompt"] + case["steps"]) // PAGE) + 1
        several = 6 if case["cached"] else 1            # cached prefixes of several batches stand side by side
        runner = ModelRunner(model, rt, n_pages=several * case["requests"] * pages + 8, max_slots=case["requests"], max_step_tokens=BUDGET,
                             prefix_cache=bool(case["cached"]))
        _kept[key] = runner
        state = _state(case, runner, 1)
        for _ in range(3):             # the kernels are loaded and the steps captured
            run(state)
    return _kept[key]


# ---- a batch of requests, turn by turn ---------------------------------------------------------------

def _prompts(case):
    """How many new tokens each request brings."""
    n, p = case["requests"], case["prompt"]
    return [max(1, p * (i + 1) // n) if case["ragged"] else p for i in range(n)]


def _turns(case):
    """Turn by turn: a list of (request, first new token, behind the last, are the last one's logits wanted)."""
    done, prompts = [0] * case["requests"], _prompts(case)
    while True:
        room, turn = BUDGET, []
        for r, p in enumerate(prompts):
            if p <= done[r] < p + case["steps"]:
                turn.append((r, done[r], done[r] + 1, True))
                room -= 1
        for r, p in enumerate(prompts):
            n = min(p - done[r], 512 if case["requests"] > 1 else BUDGET, room)
            if done[r] < p and n > 0:
                turn.append((r, done[r], done[r] + n, done[r] + n == p))
                room -= n
        if not turn:
            return
        for r, _, end, _ in turn:
            done[r] = end
        yield turn


def _ids(case, seed):
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, case["vocab"], (case["cached"] + p + case["steps"],), generator=g).tolist() for p in _prompts(case)]


def _state(case, runner, seed):
    ids = _ids(case, seed)
    for tokens in ids if case["cached"] else ():        # what a conversation so far left in the prefix cache
        req = runner.open(("prefix", next(_number)), None)
        for at in range(0, case["cached"], BUDGET):
            runner.step([(req, tokens[at:min(at + BUDGET, case["cached"])], [])])
        runner.cache.publish(req, tokens)
        runner.close(req)
    turns = list(_turns(case))
    return {"runner": runner, "ids": ids, "turns": turns, "rows": sum(want for t in turns for *_, want in t), "cached": case["cached"],
            "vocab": case["vocab"]}


def prepare(case, seed):
    return _state(case, _runner(case), seed)


def run(state):
    """Every request opened, read, decoded and closed; float32 logits, a row per wanted token, turn by turn."""
    runner, ids, cached = state["runner"], state["ids"], state["cached"]
    reqs = [runner.open(("pass", next(_number)), tokens if cached else None) for tokens in ids]
    if any(r.n_tokens != cached for r in reqs):
        raise RuntimeError("a cached prefix is gone")
    out = torch.empty((state["rows"], state["vocab"]), dtype=torch.float32, device=DEVICE)
    row = 0
    for turn in state["turns"]:
        logits = runner.step([(reqs[r], ids[r][cached + a:cached + b], [b - a - 1] if want else []) for r, a, b, want in turn])
        n = logits.shape[0]
        out[row:row + n].copy_(logits)
        row += n
    for r in reqs:
        runner.close(r)
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------

def work(case):
    """Of every turn: the weights it uses read once, the keys and values its tokens look at read once a request, what it
    adds to the cache written, a row of the embedding per token in, logits out.  Two operations per weight and token, four per
    visible key, head entry and token; the recurrences' own by their formulas."""
    size = 4 if case["dtype"] == "float32" else 2
    model = build_model(config_from_dict(_model_dict(case)))
    W, H, D, V, F, L, fam = (case[k] for k in ("width", "heads", "head_dim", "vocab", "inner", "layers", "family"))
    specs = [s for s in model.tensor_specs() if s.kind == "matrix" and "embed" not in s.name and "head" not in s.name]
    expert = lambda s: ".mlp.e" in s.name
    dense = sum(math.prod(s.shape) for s in specs if not expert(s))
    one_expert = 3 * W * (F // 4)
    byts = flops = 0.0
    for turn in _turns(case):
        new = [b - a for _, a, b, _ in turn]
        rows = sum(want for *_, want in turn)
        n = sum(new)
        weights = dense + (L * min(8, 2 * n) * one_expert if fam == "nelosun" else 0)
        byts += size * (weights + (V * W if rows else 0) + n * W) + 4 * rows * V
        flops += 2.0 * n * (dense + (L * 2 * one_expert if fam == "nelosun" else 0)) + 2.0 * rows * V * W
        for r, a, b, _ in turn:
            start, end = case["cached"] + a, case["cached"] + b
            pairs = (end * (end + 1) - start * (start + 1)) / 2.0          # (token, visible key) pairs
            if fam == "llama":
                byts += size * L * 2 * case["kv_heads"] * D * (end + (b - a))
                flops += 4.0 * H * D * L * pairs
            elif fam == "lefulorn":
                seen = min(pairs, float(WINDOW) * (b - a))
                byts += size * 2 * case["kv_heads"] * D * (min(end, WINDOW + b - a) + (b - a)) + 8.0 * H * D * D
                flops += 4.0 * H * D * seen + 6.0 * H * D * D * (b - a)
            elif fam == "dizepel":
                byts += L * (size * 2 * case["kv_heads"] * D * (end + (b - a)) + 8.0 * W * 128)
                flops += L * (4.0 * H * D * pairs + 4.0 * W * 128 * (b - a))
            else:
                byts += size * (2 * case["kv_heads"] * D + 128) * (end + (b - a)) + 8.0 * W
                flops += (4.0 * H * D + 2.0 * H * (D + 32)) * pairs + 4.0 * W * 256 * (b - a)
    return {"bytes": byts, "flops": flops}


def _cost(case):
    """Roughly the seconds that the work takes."""
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / (4e13 if case["dtype"] == "float32" else 1e15)


def tolerance(case):
    """Logits of a stack of one to three layers.  bfloat16: every product's inputs are rounded to 8 bits, and a change of any
    sum's order moves such roundings through all that follows; measured against 64 bits 0.003 to 0.015 off.  float32: 2e-6
    to 4e-6 off."""
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 2e-4}
    return {"rel": 0.025, "max": 0.25}


# ---- the same in 64 bits -----------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w


def _silu(z):
    return z * torch.sigmoid(z)


def _conv(u, w):
    """Causal, channel by channel; the last column of w weighs the current row."""
    taps = w.shape[1]
    padded = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=u.dtype, device=u.device), u])
    return sum(padded[j:j + u.shape[0]] * w[:, j] for j in range(taps))


def _turned(x, freq, factor=1.0):
    """Rotary positions on the first 2 * len(freq) entries of the last axis of x [T, heads, n]: entry i with entry i + half."""
    half = freq.numel()
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * freq
    c, s = (torch.cos(a) * factor)[:, None], (torch.sin(a) * factor)[:, None]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _freq(base, dims):
    return float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)


def _attend(q, k, v, scale, window=None, slopes=None, cap=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv]; ``sink`` [H]: one more score in each denominator, without a value."""
    T, H, _ = q.shape
    i, j = torch.arange(T, device=q.device)[:, None], torch.arange(T, device=q.device)[None]
    hidden = (j > i) | ((i - j >= window) if window else False)
    out = []
    for h in range(H):
        g = h // (H // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * (i - j)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, g])
    return torch.stack(out, 1).reshape(T, -1)


def _llama_layer(x, w, i, case):
    H, G, D, T = case["heads"], case["kv_heads"], case["head_dim"], x.shape[0]
    p = f"model.layers.{i}."
    h = _rms(x, 1e-5) * w(p + "input_layernorm.weight")
    q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).view(T, -1, D) for n in "qkv")
    f = _freq(500000.0, D)
    x = x + _attend(_turned(q, f), _turned(k, f), v, D ** -0.5) @ w(p + "self_attn.o_proj.weight").T
    h = _rms(x, 1e-5) * w(p + "post_attention_layernorm.weight")
    return x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T


def _lefulorn_layer(x, w, i, case):
    H, G, D, T = case["heads"], case["kv_heads"], case["head_dim"], x.shape[0]
    p = f"l{i}.mix."
    h = _rms(x, 1e-6) * w(f"l{i}.norm1")
    if i % 2 == 0:
        q, k, v = ((h @ w(p + n).T + w(p + n + ".b")).view(T, -1, D) for n in "qkv")
        steps = torch.div(torch.arange(T, device=DEVICE) + 1, 256, rounding_mode="floor").double()
        q = q * (1.0 + 0.1 * torch.log(steps + 1.0))[:, None, None]
        slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device=DEVICE) / H)
        o = _attend(q, k, v, D ** -0.5, WINDOW, slopes, sink=w(p + "sink")) * torch.sigmoid(h @ w(p + "g").T)
    else:
        q, k, v = (_silu(_conv(h @ w(p + n).T, w(p + n + ".conv"))).view(T, -1, D) for n in "qkv")
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q * D ** -0.5, k))
        beta = torch.sigmoid(h @ w(p + "b").T)
        a = (h @ w(p + "a1").T @ w(p + "a2").T + w(p + "dt_bias")).view(T, H, D)
        decay = torch.exp(-torch.exp(w(p + "A_log"))[:, None] * torch.nn.functional.softplus(a))
        S, o = torch.zeros(H, D, D, dtype=torch.float64, device=DEVICE), []
        for t in range(T):
            S = S * decay[t, :, :, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o.append(torch.bmm(q[t][:, None], S)[:, 0])
        o = _rms(torch.stack(o), 1e-6) * w(p + "norm")
        o = o.reshape(T, -1) * torch.sigmoid(h @ w(p + "g1").T @ w(p + "g2").T)
    x = x + o @ w(p + "o").T
    h = _rms(x, 1e-6) * w(f"l{i}.norm2")
    return x + torch.relu(h @ w(f"l{i}.mlp.up").T + w(f"l{i}.mlp.up.b")).square() @ w(f"l{i}.mlp.down").T + w(f"l{i}.mlp.down.b")


def _dizepel_layer(x, w, i, case):
    H, D, W, T = case["heads"], case["head_dim"], case["width"], x.shape[0]
    p = f"l{i}.mix"
    h = _layer_norm(x, w(f"l{i}.norm1"), 1e-6)
    h = h + _conv(h, w(f"l{i}.canon1"))
    q, k = (_conv(h @ w(f"{p}.left.{n}").T + w(f"{p}.left.{n}.b"), w(f"{p}.left.{n}.conv")).view(T, -1, D) for n in "qk")
    dims, base = D // 2, 500000.0
    at = lambda t: dims * math.log(2048.0 / (2.0 * math.pi * t)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(16.0)), 0), min(math.ceil(at(1.0)), dims - 1)
    r = ((torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f = _freq(base, dims)
    f, factor = f / 4.0 * r + f * (1.0 - r), 0.1 * math.log(4.0) + 1.0
    left = _attend(_turned(q, f, factor), _turned(k, f, factor), k, D ** -0.5, cap=30.0, sink=w(p + ".left.sink")) @ w(p + ".left.o").T
    z, xbc, dt = (h @ w(p + ".right.in").T).split([W, W + 256, W // 64], 1)
    u, B, C = _silu(_conv(xbc, w(p + ".right.conv")) + w(p + ".right.conv.b")).split([W, 128, 128], 1)
    u, dt = u.view(T, -1, 64), torch.nn.functional.softplus(dt + w(p + ".right.dt_bias"))
    keep, push = torch.exp(-torch.exp(w(p + ".right.A_log")) * dt), dt[:, :, None] * u
    S, y = torch.zeros(W // 64, 128, 64, dtype=torch.float64, device=DEVICE), []
    for t in range(T):
        S = keep[t, :, None, None] * S + B[t][:, None] * push[t][:, None]
        y.append(torch.matmul(C[t], S))
    y = (torch.stack(y) + w(p + ".right.D")[:, None] * u).reshape(T, W)
    right = _rms(y * _silu(z), 1e-6) * w(p + ".right.norm") @ w(p + ".right.o").T
    d = 0.5 * (_rms(left, 1e-6) * w(p + ".left.out") + _rms(right, 1e-6) * w(p + ".right.out"))
    x = x + _layer_norm(d, w(f"l{i}.norm1b"), 1e-6)
    h = _layer_norm(x, w(f"l{i}.norm2"), 1e-6)
    z = (h + _conv(h, w(f"l{i}.canon2"))) @ w(f"l{i}.mlp.up").T
    a, b, c, e = w(f"l{i}.mlp.act")
    return x + _layer_norm((a * _rms(z, 1e-6) + b * _rms(z * z, 1e-6) + c * _rms(z ** 3, 1e-6) + e) @ w(f"l{i}.mlp.down").T, w(f"l{i}.norm2b"), 1e-6)


def _nelosun_layer(x, w, i, case, ids):
    H, D, W, T = case["heads"], case["head_dim"], case["width"], x.shape[0]
    p = f"l{i}.mix."
    h = _rms(x, 1e-6) * w(f"l{i}.norm1")
    if i % 3 == 0:
        q, k, v = ((h @ w(p + n).T + w(p + n + ".b")).view(T, -1, D) for n in "qkv")
        steps = torch.div(torch.arange(T, device=DEVICE) + 1, 1024, rounding_mode="floor").double()
        q = q * (1.0 + 0.1 * torch.log(steps + 1.0))[:, None, None]
        o = _attend(q, k, v, D ** -0.5, sink=torch.zeros(H, dtype=torch.float64, device=DEVICE)).view(T, H, D)
        d = (o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(T, -1) @ w(p + "o").T + w(p + "o.b")
    elif i % 3 == 1:
        n, f = D // 2, _freq(10000.0, 32)
        q = ((_rms(h @ w(p + "dq").T, 1e-6) * w(p + "dq.norm")) @ w(p + "uq").T).view(T, H, n + 32)
        down = h @ w(p + "dkv").T
        c = _rms(down[:, :96], 1e-6) * w(p + "dkv.norm")
        k_rot = _turned(down[:, None, 96:], f).expand(T, H, 32)
        k = torch.cat([(c @ w(p + "uk").T).view(T, H, n), k_rot], -1)
        q = torch.cat([q[..., :n], _turned(q[..., n:], f)], -1)
        d = _attend(q, k, (c @ w(p + "uv").T).view(T, H, n), (n + 32) ** -0.5) @ w(p + "o").T
    else:
        y = torch.nn.functional.gelu(h @ w(p + "y").T + w(p + "y.b"), approximate="tanh")
        u = _conv(h @ w(p + "x").T + w(p + "x.b"), w(p + "conv")) + w(p + "conv.b")
        gate = lambda n: torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, -1, 256), w(p + n)) + w(p + n + ".b")).reshape(T, W)
        log_a = -8.0 * gate("ra") * torch.nn.functional.softplus(w(p + "lam"))
        a, push = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * gate("ri") * u
        S, out = torch.zeros(W, dtype=torch.float64, device=DEVICE), []
        for t in range(T):
            S = a[t] * S + push[t]
            out.append(S)
        d = (torch.stack(out) * y) @ w(p + "o").T
    d = d * w(f"l{i}.ls1")
    named, e_out = w(f"l{i}.mlp.table")[torch.tensor(ids, device=DEVICE)], torch.zeros_like(x)
    for e in range(8):
        at = (named == e).any(1).nonzero()[:, 0]
        m, he = f"l{i}.mlp.e{e}.", h[at]
        g, u = (he @ w(m + "gate").T).clamp(max=7.0), (he @ w(m + "up").T).clamp(-7.0, 7.0)
        e_out[at] += 0.5 * (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(m + "down").T
    return x + d + e_out * w(f"l{i}.ls2")


def _logits64(case, w, ids, places):
    """Logits of the tokens at ``places`` of one whole sequence."""
    fam = case["family"]
    x = w("model.embed_tokens.weight" if fam == "llama" else "embed")[torch.tensor(ids, device=DEVICE)]
    for i in range(case["layers"]):
        if fam == "llama":
            x = _llama_layer(x, w, i, case)
        elif fam == "lefulorn":
            x = _lefulorn_layer(x, w, i, case)
        elif fam == "dizepel":
            x = _dizepel_layer(x, w, i, case)
        else:
            x = _nelosun_layer(x, w, i, case, ids)
    x = x[torch.tensor(places, device=DEVICE)]
    if fam == "llama":
        return (_rms(x, 1e-5) * w("model.norm.weight")) @ w("lm_head.weight").T
    if fam == "dizepel":
        return _layer_norm(x, w("final.norm"), 1e-6) @ w("head").T
    return (_rms(x, 1e-6) * w("final.norm")) @ w("embed" if fam == "nelosun" else "head").T


def exact(case, seed):
    if any(case["family"] == f and case["requests"] * case["prompt"] > 30000 for f in ("lefulorn", "dizepel", "nelosun")):
        return None            # token by token in 64 bits: over a minute
    model = build_model(config_from_dict(_model_dict(case)))
    plain = _weights(case, [s for s in model.tensor_specs() if not s.optional])
    wide = {}

    def w(name):               # in 64 bits, once
        if name not in wide:
            wide[name] = plain.pop(name).long() if name.endswith(".table") else plain.pop(name).double()
        return wide[name]

    ids, at, rows = _ids(case, seed), {}, 0
    for turn in _turns(case):
        for r, _, end, want in turn:
            if want:
                at.setdefault(r, []).append((rows, case["cached"] + end - 1))
                rows += 1
    out = torch.empty((rows, case["vocab"]), dtype=torch.float64, device=DEVICE)
    for r, wanted in at.items():
        out[torch.tensor([row for row, _ in wanted], device=DEVICE)] = _logits64(case, w, ids[r], [place for _, place in wanted])
    return out.cpu().numpy().astype(np.float64)
