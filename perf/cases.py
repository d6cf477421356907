"""What this framework is timed on: the calls that a program which serves its models makes, over the range of sizes that
the repository's own configurations, benchmark and tests name.

Qwen2 decoders through `JacobiRuntime` (one draft block, device-resident Jacobi runs of one and of many sequences, prompt
chunks) and the layered hybrid decoders through `HybridRuntime` (prompt portions of one or two layers, where the result is
the layer's own, and whole requests: prompt, then one sampled token per step).

An engine (weights, caches, workspace) is kept for the case that is being measured, as a program keeps its model; prompts,
drafts and cached contexts are made from the seed.  Random weights have two structures that trained ones have and plain
noise lacks, so that rounding does not decide discrete choices: an embedding names the experts its token goes to, and the
output head ranks one next token clearly first."""
from __future__ import annotations

import math
import random

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64

# ---------------------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: one draft block of eight tokens of the 0.5B shape, verified at a short context (an interactive
        # session on the small model; launch and barrier latency count, the weights are read once)
        {"name": "qwen05b_block8", "kind": "block", "model": "qwen2-0.5b", "rows": 8, "ctx": 100},
        # the headline use: greedy Jacobi decoding of the 7B shape, one sequence, blocks of 32, after a 512-token prompt
        {"name": "qwen7b_jacobi", "kind": "jacobi", "model": "qwen2.5-coder-7b", "batch": 1, "n": 32, "mode": "single", "prompt": 512, "new": 32},
        # eight sequences with lookahead blocks and rejection recycling (prompts of unequal length)
        {"name": "qwen7b_multi8", "kind": "jacobi", "model": "qwen2.5-coder-7b", "batch": 8, "n": 32, "mode": "multiblock", "prompt": 300, "new": 16},
        # time to the first token: the prompt of a request in one chunk
        {"name": "qwen7b_prompt", "kind": "chunk", "model": "qwen2.5-coder-7b", "rows": 1000, "ctx": 0},
        # a chat request on a hybrid decoder: prompt of 512 tokens, then sampled tokens one step each, batch 1
        {"name": "kinetar_request", "kind": "request", "family": "kinetar", "batch": 1, "prompt": 512, "new": 24},
        # a batch of eight requests with unequal prompts on a decoder with routed experts in every layer
        {"name": "mafalorn_batch8", "kind": "request", "family": "mafalorn", "batch": 8, "prompt": 200, "new": 16},
        # prompt portions (2048 tokens a step is the benchmark's and the scheduler's default), by mixer
        {"name": "kinetar_portion", "kind": "portion", "layers": "parallel,delta", "width": 2048, "dtype": "bfloat16", "tokens": 2048, "entries": 1, "ctx": 0},
        {"name": "famepel_portion", "kind": "portion", "layers": "ssd,glr", "width": 1024, "dtype": "bfloat16", "tokens": 2048, "entries": 1, "ctx": 0},
        # the second portion of a long prompt: attention over what the first one left in the pages
        {"name": "latent_portion", "kind": "portion", "layers": "latent", "width": 2048, "dtype": "bfloat16", "tokens": 1531, "entries": 1, "ctx": 2048},
        # several requests' prompts in one step, odd lengths
        {"name": "mafalorn_portion", "kind": "portion", "layers": "retention,side", "width": 1024, "dtype": "bfloat16", "tokens": 1999, "entries": 5, "ctx": 0},
        {"name": "kisadra_portion", "kind": "portion", "layers": "gla,chunk", "width": 2048, "dtype": "bfloat16", "tokens": 2048, "entries": 2, "ctx": 0},
        # the fp32 build, as a program that checks a checkpoint runs it: a short ragged step
        {"name": "famepel_fp32", "kind": "portion", "layers": "ssd,glr", "width": 256, "dtype": "float32", "tokens": 77, "entries": 3, "ctx": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "jacobi", "chunk", "request", "portion", "portion", "portion", "portion"])
    if kind == "block":
        return {"kind": kind, "model": "qwen2-0.5b", "rows": 8 * rng.randint(1, 4), "ctx": _log(rng, 1, 900)}
    if kind == "jacobi":
        batch = rng.choice([1, 1, 2, 3, 5, 8])
        return {"kind": kind, "model": "qwen2.5-coder-7b", "batch": batch, "n": rng.choice([8, 16, 32]), "mode": rng.choice(["single", "multiblock"]),
                "prompt": _log(rng, 20, 600), "new": rng.randint(8, 16 if batch > 2 else 32)}
    if kind == "chunk":
        return {"kind": kind, "model": "qwen2.5-coder-7b", "rows": _log(rng, 40, 1024), "ctx": rng.choice([0, 0, rng.randint(1, 700)])}
    if kind == "request":
        return {"kind": kind, "family": rng.choice(["kinetar", "mafalorn"]), "batch": rng.choice([1, 2, 4, 8]), "prompt": _log(rng, 10, 512), "new": rng.randint(8, 24)}
    layers = rng.choice(["parallel", "delta", "ssd", "glr", "latent", "retention", "side", "gla", "chunk", "parallel,delta", "ssd,glr"])
    f32 = rng.random() < 0.15
    tokens = _log(rng, 20, 150) if f32 else _log(rng, 16, 2048)
    return {"kind": kind, "layers": layers, "width": 256 if f32 else 1024 if layers[:3] in ("ssd", "glr", "ret", "sid") else rng.choice([1024, 2048]),
            "dtype": "float32" if f32 else "bfloat16", "tokens": tokens, "entries": rng.choice([1, 1, 2, max(1, min(8, tokens // 10))]),
            "ctx": rng.randint(1, 2048) if layers == "latent" and not f32 else 0}


# ---------------------------------------------------------------------------------------------------------------------------
# shared pieces
# ---------------------------------------------------------------------------------------------------------------------------
_kept = {"key": None, "engine": None}


def engine(key, make):
    """The engine of the case that is being measured; another case's is let go first."""
    if _kept["key"] != key:
        _kept.update(key=None, engine=None)
        _kept.update(engine=make(), key=key)
    return _kept["engine"]


class Pages:
    """Pages (or slots) that a state holds, given back with it."""

    def __init__(self, free, count):
        if len(free) < count:
            raise MemoryError("out of memory: no pages left for another state")
        self.free, self.ids = free, [free.pop() for _ in range(count)]

    def __del__(self):
        self.free.extend(reversed(self.ids))


def noise(seed, *shape):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32)


def following(tokens, vocab):
    """The token that the output head of these models ranks first behind a token."""
    return (tokens * 7 + 11) % vocab


def lengths(total, parts):
    """`total` cut into `parts` unequal lengths."""
    w = [3 + (5 * i) % 7 for i in range(parts)]
    cut = [max(1, total * x // sum(w)) for x in w]
    cut[0] += total - sum(cut)
    return cut


def prompts_of(seed, vocab, lens):
    rng = np.random.default_rng(seed + 17)
    return [[int(t) for t in rng.integers(0, vocab, n)] for n in lens]


# ---------------------------------------------------------------------------------------------------------------------------
# Qwen2
# ---------------------------------------------------------------------------------------------------------------------------
QWEN = {
    "qwen2.5-coder-7b": dict(hidden_size=3584, num_hidden_layers=28, num_attention_heads=28, num_key_value_heads=4, head_dim=128,
                             intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False, rope_theta=1e6,
                             max_position_embeddings=32768, rms_norm_eps=1e-6),
    "qwen2-0.5b": dict(hidden_size=896, num_hidden_layers=24, num_attention_heads=14, num_key_value_heads=2, head_dim=64,
                       intermediate_size=4864, vocab_size=151936, tie_word_embeddings=True, rope_theta=1e6,
                       max_position_embeddings=32768, rms_norm_eps=1e-6),
}
PAGE = 256


def qwen_tensor(cfg, name, shape):
    if name.endswith("norm.weight") or name.endswith("layernorm.weight"):
        return torch.ones(shape, device=DEV, dtype=torch.bfloat16)
    if name == "lm_head.weight":                                           # row following(t) is token t's embedding
        e = qwen_tensor(cfg, "model.embed_tokens.weight", shape)
        t = torch.arange(shape[0], device=DEV)
        out = torch.empty_like(e)
        out[following(t, shape[0])] = (e.float() * (0.02 / 8.0)).to(torch.bfloat16)
        return out
    scale = 8.0 if name == "model.embed_tokens.weight" and not cfg["tie_word_embeddings"] else 0.02
    return (noise(sum(ord(c) * (i + 1) for i, c in enumerate(name)), *shape) * scale).to(torch.bfloat16)


def qwen_shapes(cfg):
    h, inter, v = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
    q, kv = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
    s = {"model.embed_tokens.weight": (v, h), "model.norm.weight": (h,)}
    if not cfg["tie_word_embeddings"]:
        s["lm_head.weight"] = (v, h)
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        s.update({p + "self_attn.q_proj.weight": (q, h), p + "self_attn.k_proj.weight": (kv, h), p + "self_attn.v_proj.weight": (kv, h),
                  p + "self_attn.q_proj.bias": (q,), p + "self_attn.k_proj.bias": (kv,), p + "self_attn.v_proj.bias": (kv,),
                  p + "self_attn.o_proj.weight": (h, q), p + "mlp.gate_proj.weight": (inter, h), p + "mlp.up_proj.weight": (inter, h),
                  p + "mlp.down_proj.weight": (h, inter), p + "input_layernorm.weight": (h,), p + "post_attention_layernorm.weight": (h,)})
    return s


def qwen_engine(model):
    def make():
        from jacobiforcing_b200.runtime import JacobiRuntime
        cfg = QWEN[model]
        rt = JacobiRuntime(cfg, max_rows=1024, max_seqs=8, num_kv_pages=288, max_pages_per_seq=8)
        for name, shape in qwen_shapes(cfg).items():
            rt.load_tensor(name, qwen_tensor(cfg, name, shape))
        rt.finalize()
        torch.cuda.empty_cache()
        return rt
    return engine(model, make)


class Sequences:
    """Sequences of the runtime that a state holds, released with it."""

    def __init__(self, rt, count):
        self.rt, self.all = rt, [rt.new_sequence() for _ in range(count)]

    def __del__(self):
        for s in self.all:
            self.rt.release(s)


def qwen_cached(rt, seq, tokens):
    """`tokens` through the model in chunks, their keys and values committed to the sequence's pages."""
    rt.ensure_capacity(seq, len(tokens) + rt.max_rows // 4)
    for a in range(0, len(tokens), rt.max_rows):
        part = tokens[a:a + rt.max_rows]
        rt.forward(part, [(0, len(part), 0, a)], [seq], 0, 0, [(i, 0, a + i) for i in range(len(part))])
    seq.tokens, seq.ctx = list(tokens), len(tokens)


def qwen_prepare(case, seed):
    from jacobiforcing_b200.policy import MODES, PolicyKnobs, draw_prefill_draft, mt_state_words
    cfg = QWEN[case["model"]]
    rt, v = qwen_engine(case["model"]), cfg["vocab_size"]
    st = {"rt": rt, "kind": case["kind"]}
    if case["kind"] == "jacobi":
        lens = [max(4, case["prompt"] - 13 * i) for i in range(case["batch"])]
        held = Sequences(rt, case["batch"])
        firsts, calls, words = [], [], []
        prompts = prompts_of(seed, v, lens)
        for i, (s, p) in enumerate(zip(held.all, prompts)):
            rng = random.Random(seed * 31 + i)
            first, drafted, _ = rt.prefill(s, p, draw_prefill_draft(rng, p, case["n"]))
            firsts.append(first)
            calls.append(drafted)
            words.append(mt_state_words(rng))
        knobs = PolicyKnobs(mode=MODES[case["mode"]], n=case["n"], K=2, r=0.85, n_gram_pool_size=4, pad=0, max_new_tokens=case["new"],
                            max_calls=64, vocab=v)
        return dict(st, held=held, prompts=prompts, knobs=knobs, firsts=firsts, calls=calls, words=words, block=prompts_of(seed + 1, v, [8])[0])
    ctx, part = prompts_of(seed, v, [case["ctx"], case["rows"]])
    held = Sequences(rt, 1)
    if ctx:
        qwen_cached(rt, held.all[0], ctx)
    rt.ensure_capacity(held.all[0], case["ctx"] + case["rows"])
    rows = case["rows"]
    row0 = 0 if case["kind"] == "block" else (rows - 8) // 8 * 8
    commits = [] if case["kind"] == "block" else [(i, 0, case["ctx"] + i) for i in range(rows)]
    return dict(st, held=held, tokens=part, ctx=case["ctx"], row0=row0, commits=commits)


def qwen_run(st):
    rt, seqs = st["rt"], st["held"].all
    if st["kind"] == "jacobi":
        for s, p in zip(seqs, st["prompts"]):                               # the caches hold the prompts: generate behind them
            s.tokens, s.ctx = list(p), len(p)
        results, _ = rt.jacobi_run(seqs, st["knobs"], st["firsts"], st["calls"], rng_states=st["words"])
        check = rt.forward(st["block"], [(0, 8, 0, len(st["prompts"][0]))], seqs[:1], 0, 8, want_logits=True)
        return {"tokens": np.array([t for r in results for t in r.tokens], dtype=np.int32), "logits": check["logits"]}
    n = len(st["tokens"])
    return rt.forward(st["tokens"], [(0, n, 0, st["ctx"])], seqs, st["row0"], n - st["row0"], st["commits"], want_logits=True)["logits"]


def qwen_exact(case, seed):
    cfg = QWEN[case["model"]]
    v, d, heads, kvh, h = cfg["vocab_size"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["hidden_size"]
    if case["kind"] == "jacobi":
        tokens = prompts_of(seed, v, [max(4, case["prompt"] - 13 * i) for i in range(case["batch"])])[0] + prompts_of(seed + 1, v, [8])[0]
        rows = 8
    else:
        ctx, part = prompts_of(seed, v, [case["ctx"], case["rows"]])
        tokens = ctx + part
        rows = case["rows"] - (0 if case["kind"] == "block" else (case["rows"] - 8) // 8 * 8)
    shapes = qwen_shapes(cfg)
    w = lambda name: qwen_tensor(cfg, name, shapes[name])                    # noqa: E731
    embed = w("model.embed_tokens.weight")
    x = embed[torch.tensor(tokens, device=DEV)].to(F64)
    t = len(tokens)
    inv = cfg["rope_theta"] ** (-torch.arange(0, d, 2, device=DEV, dtype=F64) / d)
    ang = torch.arange(t, device=DEV, dtype=F64)[:, None] * inv[None]
    cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def turn(u):
        a, b = u[..., :d // 2], u[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def lin(u, name, bias=False):
        y = u @ w(name + ".weight").to(F64).T
        return y + w(name + ".bias").to(F64) if bias else y
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        u = unit_rms(x, cfg["rms_norm_eps"])
        q = turn(lin(u, p + "self_attn.q_proj", True).view(t, heads, d))
        k = turn(lin(u, p + "self_attn.k_proj", True).view(t, kvh, d))
        val = lin(u, p + "self_attn.v_proj", True).view(t, kvh, d)
        x = x + lin(attend(q, k, val, d ** -0.5).reshape(t, heads * d), p + "self_attn.o_proj")
        u = unit_rms(x, cfg["rms_norm_eps"])
        x = x + lin(silu(lin(u, p + "mlp.gate_proj")) * lin(u, p + "mlp.up_proj"), p + "mlp.down_proj")
    x = unit_rms(x[-rows:], cfg["rms_norm_eps"])
    head = embed if cfg["tie_word_embeddings"] else w("lm_head.weight")
    logits = torch.cat([x @ head[a:a + 16384].to(F64).T for a in range(0, v, 16384)], 1)
    return {"tokens": None, "logits": logits} if case["kind"] == "jacobi" else logits


def qwen_work(case):
    cfg = QWEN[case["model"]]
    h, inter, v, n_layers = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["num_hidden_layers"]
    q, kv = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
    body = n_layers * (h * (q + 2 * kv) + q * h + 3 * h * inter)

    def forward(rows, groups, ctx, head_rows, new_bytes):
        cached = n_layers * 2 * kv * 2
        b = 2 * (body + v * h) + groups * ctx * cached + rows * (cached + 2 * h) + new_bytes
        return b, 2.0 * (rows * body + head_rows * v * h) + 4.0 * n_layers * rows * q * (ctx + rows / (2.0 * groups))
    if case["kind"] != "jacobi":
        rows = case["rows"]
        head = rows if case["kind"] == "block" else rows - (rows - 8) // 8 * 8
        b, f = forward(rows, 1, case["ctx"], head, 4 * head * v)
        return {"bytes": b, "flops": f}
    # greedy decoding of these weights accepts about one token a forward; a forward holds the rest of the block (and, with
    # lookahead blocks, candidate rows of about its size again)
    rows = case["batch"] * case["n"] * (0.75 if case["mode"] == "single" else 0.65)
    b, f = forward(rows, case["batch"], case["prompt"], rows, 0)
    b8, f8 = forward(8, 1, case["prompt"], 8, 32 * v)
    return {"bytes": case["new"] * b + b8, "flops": case["new"] * f + f8}


# ---------------------------------------------------------------------------------------------------------------------------
# plain 64-bit pieces
# ---------------------------------------------------------------------------------------------------------------------------


def unit_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(z):
    return z * torch.sigmoid(z)


def softplus(z):
    return torch.clamp(z, min=0.0) + torch.log1p(torch.exp(-z.abs()))


def attend(q, k, v, scale, seen=None, lower=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv]; seen(i, j): what a position sees (default: all j <= i); lower(head, i, j): what
    is taken off a score; sink [H]: a logit without key and value."""
    t, heads, per = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    at = torch.arange(t, device=q.device)
    i, j = at[:, None], at[None, :]
    ok = j <= i if seen is None else seen(i, j)
    out = []
    for hh in range(heads):
        s = q[:, hh] @ k[:, hh // per].T * scale
        if lower is not None:
            s = s - lower(hh, i, j)
        s = s.masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[hh].expand(t, 1)], 1)
        out.append(torch.softmax(s, 1)[:, :t] @ v[:, hh // per])
    return torch.stack(out, 1)


def recur(q, k, v, decay, beta=None):
    """S <- decay S + k v' token by token (with `beta` the delta rule: v - S'k, scaled), read with q behind the write.
    q, k, decay [T, H, D], v [T, H, Dv], beta [T, H]."""
    t, heads, d = k.shape
    s = torch.zeros(heads, d, v.shape[2], device=k.device, dtype=k.dtype)
    out = []
    for n in range(t):
        s = s * decay[n][:, :, None]
        u = v[n] if beta is None else beta[n][:, None] * (v[n] - torch.einsum("hd,hdv->hv", k[n], s))
        s = torch.baddbmm(s, k[n][:, :, None], u[:, None])
        out.append(torch.einsum("hd,hdv->hv", q[n], s))
    return torch.stack(out)


def short_conv(u, w, bias=None):
    taps = w.shape[1]
    y = torch.zeros_like(u)
    for a in range(taps):
        back = taps - 1 - a
        y[back:] += u[:u.shape[0] - back] * w[:, a]
    return y if bias is None else y + bias


def frequencies(rot):
    dims, base = rot["dims"], rot["base"]
    f = base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=F64) / dims)
    sc = rot.get("scaling")
    if not sc:
        return f, 1.0
    at = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))   # noqa: E731
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
    ramp = torch.clamp((torch.arange(dims // 2, device=DEV, dtype=F64) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def rotate(x, rot, halves):
    """x [T, ..., n]: row t turns by its position; pairs (i, i + dims / 2) or neighbours over the first dims dimensions."""
    f, mag = frequencies(rot)
    dims = rot["dims"]
    ang = torch.arange(x.shape[0], device=DEV, dtype=F64).view([-1] + [1] * (x.dim() - 1)) * f
    c, s = torch.cos(ang) * mag, torch.sin(ang) * mag
    out = x.clone()
    one, two = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., one] = x[..., one] * c - x[..., two] * s
    out[..., two] = x[..., two] * c + x[..., one] * s
    return out


def unit_vector(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


# ---------------------------------------------------------------------------------------------------------------------------
# hybrid decoders: descriptions and weights
# ---------------------------------------------------------------------------------------------------------------------------
FAMILY = {"parallel": "Kinetar", "delta": "Kinetar", "ssd": "Famepel", "glr": "Famepel", "latent": "Famepel", "retention": "Mafalorn",
          "side": "Mafalorn", "gla": "Kisadra", "chunk": "Kisadra"}
LOW, VOCAB = 64, {"request": 32000, "portion": 4096}


def layer_of(name, w):
    """A layer in the proportions of the repository's benchmark (heads of 128; feed-forward 4 width, in routed layers 32 experts,
    4 per token) at width `w`."""
    heads = w // 128
    moe = {"kind": "moe", "expert": {"ff": w // 2}, "router": {"experts": 32, "top": 4, "groups": {"count": 4, "keep": 2}}}
    interpolated = {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    if name == "parallel":
        return {"type": "parallel",
                "mixer": {"left": {"conv": 4, "dim": 128, "heads": heads, "kv_heads": max(1, heads // 4), "q_temp": {"coef": 0.5, "every": 1024},
                                   "scale": 128 ** -0.5, "vdim": 128}, "left_scale": 0.7,
                          "right": {"conv": 4, "dt_rank": w // 16, "inner": 2 * w, "state": 16}, "right_scale": 0.7}, "mlp": {"ff": 4 * w, "kind": "dense"}}
    if name == "delta":
        return {"type": "channel_delta", "mixer": {"conv": 4, "dim": 128, "heads": heads, "kv_heads": max(1, heads // 2), "vdim": 128},
                "mlp": {"ff": 4 * w, "kind": "dense"}}
    if name in ("ssd", "glr", "latent"):
        moe["router"]["scale"] = 2.5
        mixer = {"ssd": {"heads": 2 * w // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8},
                 "glr": {"heads": heads, "dim": 128, "vdim": 128},
                 "latent": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 3 * w // 4, "scale": 192 ** -0.5,
                            "rot": {"base": 10000.0, "dims": 64, "scaling": interpolated}}}[name]
        return {"type": {"ssd": "mamba2", "glr": "hgrn2", "latent": "latent_attention"}[name], "mixer": mixer, "mlp": None if name == "latent" else moe}
    if name in ("retention", "side"):
        moe["router"]["identity"] = 4
        if name == "retention":
            return {"type": "retention", "mlp": moe,
                    "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5.0 - 4.0 * h / heads) for h in range(heads)],
                              "rot": {"base": 10000.0, "dims": 128}}}
        return {"type": "parallel", "mlp": moe,
                "mixer": {"left": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                   "rot": {"base": 10000.0, "dims": 64, "scaling": dict(interpolated, factor=4.0)}}, "left_scale": 0.7,
                          "right": {"heads": heads, "kv_heads": max(1, heads // 2), "dim": 128, "vdim": 128, "conv": 4}, "right_scale": 0.7}}
    dense = {"kind": "dense", "ff": 4 * w}
    if name == "gla":
        return {"type": "gla", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "tau": 16.0}, "mlp": dense}
    return {"type": "attention", "mlp": dense,
            "mixer": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "mask": {"size": 1024}, "scale": 128 ** -0.5}}


def describe(case):
    if case["kind"] == "request":
        names = {"kinetar": "parallel,delta,parallel,delta", "mafalorn": "retention,side,retention,side"}[case["family"]].split(",")
        w = 1024
    else:
        names, w = case["layers"].split(","), case["width"]
    d = {"architecture": FAMILY[names[0]], "embedding": {"scale": 1.0}, "layers": [layer_of(n, w) for n in names], "logit_scale": 1.0,
         "norm": {"eps": 1e-6}, "vocab": VOCAB[case["kind"]], "width": w}
    return names, d


def token_experts(tokens, groups, per):
    """Four router outputs of a token: two in each of two groups."""
    g = torch.stack([tokens % groups, (tokens + 1 + (tokens // groups) % (groups - 1)) % groups], 1)
    a = (tokens // 12) % per
    b = (a + 1 + (tokens // (12 * per)) % (per - 1)) % per
    return torch.cat([g * per + a[:, None], g * per + b[:, None]], 1)


def hybrid_weights(case):
    names, d = describe(case)
    w, v = d["width"], d["vocab"]
    out, count = {}, [1000]

    def rnd(*shape):
        count[0] += 1
        return noise(count[0], *shape)

    def lin(n, k):
        return rnd(n, k) / math.sqrt(k)

    def vec(n, s=0.1, b=0.0):
        return rnd(n) * s + b
    plain = rnd(v, w)
    big = 4.0 if case["kind"] == "request" else 1.0
    embed = plain.clone()
    router = None
    first = next((lc["mlp"]["router"] for lc in d["layers"] if lc["mlp"] and lc["mlp"]["kind"] == "moe"), None)
    if first:
        n = first["experts"] + first.get("identity", 0)
        router = rnd(n, w)
        embed += router[token_experts(torch.arange(v, device=DEV), first["groups"]["count"], n // first["groups"]["count"])].sum(1)
        big /= 2.0
    out["embed"] = embed * big
    head = torch.empty_like(plain)
    head[following(torch.arange(v, device=DEV), v)] = plain / math.sqrt(w)
    out["head"] = head
    tanh = d["architecture"] == "Famepel"

    def norm(name):
        out[name] = vec(w, 0.1, 0.0 if d["architecture"] == "Kinetar" else 1.0)
        if tanh:
            out[name + ".b"], out[name + ".alpha"] = vec(w), torch.full((), 0.7, device=DEV)
    norm("final.norm")
    for i, (name, lc) in enumerate(zip(names, d["layers"])):
        p, m, x = "l%d." % i, "l%d.mix." % i, lc["mixer"]
        mlp = lc["mlp"]
        norm(p + "norm1")
        if d["architecture"] in ("Famepel", "Mafalorn"):
            for n in ("norm1b", "norm2", "norm2b") if mlp else ("norm1b",):
                norm(p + n)
            if tanh:
                out[p + "ls1"] = vec(w, 0.1, 0.7)
                if mlp:
                    out[p + "ls2"] = vec(w, 0.1, 0.7)
        if name == "parallel":
            a, s = x["left"], x["right"]
            nq, nk, inner, ns, r = a["heads"] * 128, a["kv_heads"] * 128, s["inner"], s["state"], s["dt_rank"]
            lm, rm = m + "left.", m + "right."
            out.update({lm + "q": lin(nq, w), lm + "k": lin(nk, w), lm + "q.conv": rnd(nq, 4) * 0.5, lm + "k.conv": rnd(nk, 4) * 0.5,
                        lm + "sink": vec(a["heads"], 1.0), lm + "g": lin(nq, w), lm + "o": lin(w, nq), rm + "in": lin(2 * inner, w),
                        rm + "conv": rnd(inner, 4) * 0.5, rm + "conv.b": vec(inner), rm + "x": lin(r + 2 * ns, inner), rm + "dt": lin(inner, r),
                        rm + "dt.b": vec(inner, 0.5, -1.0), rm + "A_log": rnd(inner, ns) * 0.5 - 0.3, rm + "D": vec(inner, 0.3, 1.0), rm + "o": lin(w, inner)})
        elif name == "delta":
            nq, nv, h = x["kv_heads"] * 128, x["heads"] * 128, x["heads"]
            out.update({m + "q": lin(nq, w), m + "k": lin(nq, w), m + "v": lin(nv, w), m + "q.conv": rnd(nq, 4) * 0.5, m + "k.conv": rnd(nq, 4) * 0.5,
                        m + "v.conv": rnd(nv, 4) * 0.5, m + "b": lin(h, w), m + "A_log": vec(h, 0.5, -0.7), m + "norm": vec(128, 0.2, 1.0),
                        m + "a1": lin(LOW, w), m + "a2": lin(nv, LOW), m + "dt_bias": vec(nv, 0.5, -1.0), m + "g1": lin(LOW, w), m + "g2": lin(nv, LOW),
                        m + "o": lin(w, nv)})
        elif name == "ssd":
            h, inner, gn = x["heads"], x["heads"] * x["vdim"], x["groups"] * x["state"]
            out.update({m + "in": lin(2 * inner + 2 * gn + h, w), m + "conv": rnd(inner + 2 * gn, 4) * 0.5, m + "conv.b": vec(inner + 2 * gn),
                        m + "dt_bias": vec(h, 0.5, -1.0), m + "A_log": vec(h, 0.5, -0.3), m + "D": vec(h, 0.3, 1.0), m + "norm": vec(inner, 0.1, 1.0),
                        m + "o": lin(w, inner)})
        elif name == "glr":
            n = x["heads"] * 128
            out.update({m + "q": lin(n, w), m + "f": lin(n, w), m + "f.b": vec(n, 0.5), m + "lower": torch.sigmoid(rnd(n)) * 0.9, m + "v": lin(n, w),
                        m + "norm": vec(128, 0.1, 1.0), m + "o": lin(w, n)})
        elif name == "latent":
            h, r = x["heads"], x["kv_rank"]
            out.update({m + "dq": lin(x["q_rank"], w), m + "dq.norm": vec(x["q_rank"], 0.1, 1.0), m + "uq": lin(h * 192, x["q_rank"]),
                        m + "uk": lin(h * 128, r), m + "uv": lin(h * 128, r), m + "sink": vec(h, 1.0), m + "o": lin(w, h * 128),
                        m + "dkv": lin(r + 64, w), m + "dkv.norm": vec(r, 0.1, 1.0)})
        elif name == "retention":
            n = x["heads"] * 128
            out.update({m + "q": lin(n, w), m + "k": lin(n, w), m + "v": lin(n, w), m + "g": lin(n, w), m + "o": lin(w, n)})
        elif name == "side":
            a, s = x["left"], x["right"]
            nq, h, nk, nv, lm, rm = a["heads"] * 128, s["heads"], s["kv_heads"] * 128, s["heads"] * 128, m + "left.", m + "right."
            out.update({lm + "q": lin(nq, w), lm + "k": lin(a["kv_heads"] * 128, w), lm + "g": lin(a["heads"], w), lm + "o": lin(w, nq),
                        rm + "q": lin(nk, w), rm + "k": lin(nk, w), rm + "v": lin(nv, w), rm + "q.conv": rnd(nk, 4) * 0.5, rm + "k.conv": rnd(nk, 4) * 0.5,
                        rm + "v.conv": rnd(nv, 4) * 0.5, rm + "b": lin(h, w), rm + "a": lin(h, w), rm + "A_log": vec(h, 0.5, -0.7),
                        rm + "dt_bias": vec(h, 0.5, -1.0), rm + "norm": vec(128, 0.2, 1.0), rm + "g": lin(nv, w), rm + "o": lin(w, nv)})
        elif name == "gla":
            n = x["heads"] * 128
            out.update({m + "q": lin(n, w), m + "k": lin(n, w), m + "v": lin(n, w), m + "g": lin(n, w), m + "norm": vec(128, 0.1, 1.0), m + "a1": lin(16, w),
                        m + "a2": lin(n, 16), m + "a2.b": vec(n, 0.5, 1.0), m + "o": lin(w, n)})
        else:
            nq, nk = x["heads"] * 128, x["kv_heads"] * 128
            out.update({m + "q": lin(nq, w), m + "k": lin(nk, w), m + "v": lin(nk, w), m + "q.norm": vec(nq, 0.1, 1.0), m + "k.norm": vec(nk, 0.1, 1.0),
                        m + "o": lin(w, nq)})
        q = p + "mlp."
        if mlp and mlp["kind"] == "dense":
            if d["architecture"] == "Kisadra":
                out[q + "gate"] = lin(mlp["ff"], w)
            out[q + "up"], out[q + "down"] = lin(mlp["ff"], w), lin(w, mlp["ff"])
        elif mlp:
            ff = mlp["expert"]["ff"]
            out[q + "router"] = router * (0.5 / math.sqrt(w))
            if d["architecture"] == "Mafalorn":
                out[q + "correction"] = vec(router.shape[0], 0.01)
            for e in range(mlp["router"]["experts"]):
                out[q + "e%d.gate" % e], out[q + "e%d.up" % e], out[q + "e%d.down" % e] = lin(ff, w), lin(ff, w), lin(w, ff)
    return {k: t.to(torch.bfloat16) for k, t in out.items()}


# ---------------------------------------------------------------------------------------------------------------------------
# hybrid decoders: states and passes
# ---------------------------------------------------------------------------------------------------------------------------
KV_PAGE, MOST_TOKENS = 64, 2048


def hybrid_engine(case):
    key = (case["kind"], case.get("family"), case.get("layers"), case.get("width"), case.get("dtype", "bfloat16"))

    def make():
        from jacobiforcing_b200.hybrid_config import HybridConfig
        from jacobiforcing_b200.hybrid_runtime import HybridRuntime
        _, d = describe(case)
        w = hybrid_weights(case)
        rt = HybridRuntime(HybridConfig.from_dict(d, {k: tuple(t.shape) for k, t in w.items()}), dtype=case.get("dtype", "bfloat16"),
                           max_step_tokens=MOST_TOKENS, max_step_entries=16, page_size=KV_PAGE, num_pages=1024, max_pages_per_seq=80, num_slots=128,
                           max_want=64)
        rt.load_state_dict(w)
        del w
        torch.cuda.empty_cache()
        rt.free, rt.free_slots = list(range(1024)), list(range(128))
        return rt
    return engine(key, make)


def hybrid_lengths(case):
    if case["kind"] == "request":
        return [max(4, case["prompt"] + (37 * i) % 101 - 13 * i) for i in range(case["batch"])]
    return lengths(case["tokens"], case["entries"])


def wanted(case, lens):
    """Rows whose logits a portion returns: the last of every request (where its next token is sampled) and, as in scoring, a
    spread of others (from the eighth on: a matrix state of one or two tokens can be read out near zero, and the norm behind
    it then shows nothing but rounding)."""
    start, rows = 0, set()
    for n in lens:
        rows.add(start + n - 1)
        start += n
    rows.update(range(min(7, start - 1), start, max(1, start // 16)))
    return sorted(rows)


def hybrid_prepare(case, seed):
    rt, lens = hybrid_engine(case), hybrid_lengths(case)
    more = case["new"] if case["kind"] == "request" else case["ctx"]
    prompts = prompts_of(seed, VOCAB[case["kind"]], [n + (case["ctx"] if case["kind"] == "portion" else 0) for n in lens])
    pages = [Pages(rt.free, (n + more + KV_PAGE - 1) // KV_PAGE) for n in lens]
    slots = Pages(rt.free_slots, len(lens))
    st = {"rt": rt, "kind": case["kind"], "pages": pages, "slots": slots, "prompts": prompts, "new": case.get("new", 0), "pos0": 0}
    if case["kind"] == "portion":
        st["want"], st["pos0"] = wanted(case, lens), case["ctx"]
        for i, p in enumerate(prompts):                                     # the earlier portion of each prompt
            if case["ctx"]:
                rt.step([(p[:case["ctx"]], 0, slots.ids[i], pages[i].ids)])
        st["prompts"] = [p[case["ctx"]:] for p in prompts]
    return st


def hybrid_run(st):
    rt, pages, slots = st["rt"], st["pages"], st["slots"].ids
    entries = [(p, st["pos0"], slots[i], pages[i].ids) for i, p in enumerate(st["prompts"])]
    if st["kind"] == "portion":
        return rt.step(entries, st["want"])["logits"]
    # prompts that fit a step together run in one, as the scheduler packs them
    logits, tokens, at = [], [], [len(p) for p in st["prompts"]]
    last, group, used = [], [], 0
    for i, e in enumerate(entries + [None]):
        if e is None or used + len(e[0]) > MOST_TOKENS:
            ends = np.cumsum([len(x[0]) for x in group]) - 1
            r = rt.step(group, ends.tolist(), sample=True)
            last.append(r["logits"])
            tokens.extend(int(t) for t in r["sampled"])
            group, used = [], 0
        if e is not None:
            group.append(e)
            used += len(e[0])
    logits.append(np.concatenate(last))
    out = [list(tokens)]
    for _ in range(st["new"]):
        r = rt.step([([t], p, slots[i], pages[i].ids) for i, (t, p) in enumerate(zip(tokens, at))], list(range(len(at))), sample=True)
        tokens, at = [int(t) for t in r["sampled"]], [p + 1 for p in at]
        logits.append(r["logits"])
        out.append(list(tokens))
    return {"logits": logits, "tokens": np.array(out, dtype=np.int32)}


def one_sequence(names, d, w, tokens):
    """The stream behind the last layer for one sequence, in 64 bits."""
    eps, arch = d["norm"]["eps"], d["architecture"]
    tok = torch.tensor(tokens, device=DEV)
    x = w["embed"][tok]
    t, width = len(tokens), d["width"]
    if arch == "Kinetar":
        f = 10000.0 ** (-2.0 * torch.arange(width // 2, device=DEV, dtype=F64) / width)
        ang = torch.arange(t, device=DEV, dtype=F64)[:, None] * f
        x = x + torch.stack([torch.sin(ang), torch.cos(ang)], 2).reshape(t, width)

    def norm(y, name):
        if arch == "Famepel":
            return torch.tanh(w[name + ".alpha"] * y) * w[name] + w[name + ".b"]
        return unit_rms(y, eps) * (w[name] + (1.0 if arch == "Kinetar" else 0.0))

    def spread(u, heads):                                                   # key heads to the heads that share them
        return u.repeat_interleave(heads // u.shape[1], 1)

    def mixer(name, h, g, c):
        def lin(n):
            return h @ g[n].T
        if name == "parallel":
            a, s = c["left"], c["right"]
            q, k = short_conv(lin("left.q"), g["left.q.conv"]), short_conv(lin("left.k"), g["left.k.conv"])
            temp = 1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((torch.arange(t, device=DEV, dtype=F64) + 1) / a["q_temp"]["every"]) + 1.0)
            k = k.view(t, a["kv_heads"], 128)
            y = attend((q * temp[:, None]).view(t, a["heads"], 128), k, k, a["scale"], sink=g["left.sink"]).reshape(t, -1)
            left = (y * torch.sigmoid(lin("left.g"))) @ g["left.o"].T
            inner, n, r = s["inner"], s["state"], s["dt_rank"]
            xz = lin("right.in")
            u = silu(short_conv(xz[:, :inner], g["right.conv"], g["right.conv.b"]))
            low = u @ g["right.x"].T
            dt = softplus(low[:, :r] @ g["right.dt"].T + g["right.dt.b"])
            rate, state, ys = -torch.exp(g["right.A_log"]), torch.zeros(inner, n, device=DEV, dtype=F64), []
            for i in range(t):
                state = torch.exp(dt[i][:, None] * rate) * state + (dt[i] * u[i])[:, None] * low[i, r:r + n]
                ys.append(state @ low[i, r + n:])
            y = (torch.stack(ys) + g["right.D"] * u) * silu(xz[:, inner:])
            return c["left_scale"] * left + c["right_scale"] * (y @ g["right.o"].T)
        if name == "delta":
            nh, nk = c["heads"], c["kv_heads"]
            q = unit_vector(silu(short_conv(lin("q"), g["q.conv"])).view(t, nk, 128)) * 128 ** -0.5
            k = unit_vector(silu(short_conv(lin("k"), g["k.conv"])).view(t, nk, 128))
            v = silu(short_conv(lin("v"), g["v.conv"])).view(t, nh, 128)
            a = (lin("a1") @ g["a2"].T + g["dt_bias"]).view(t, nh, 128)
            decay = torch.exp(-torch.exp(g["A_log"])[None, :, None] * softplus(a))
            o = recur(spread(q, nh), spread(k, nh), v, decay, torch.sigmoid(lin("b")))
            gate = torch.sigmoid(lin("g1") @ g["g2"].T).view(t, nh, 128)
            return (unit_rms(o, eps) * g["norm"] * gate).reshape(t, -1) @ g["o"].T
        if name == "ssd":
            nh, pd, ns, ng = c["heads"], c["vdim"], c["state"], c["groups"]
            inner = nh * pd
            u = lin("in")
            z, dt = u[:, :inner], softplus(u[:, 2 * inner + 2 * ng * ns:] + g["dt_bias"])
            xbc = silu(short_conv(u[:, inner:2 * inner + 2 * ng * ns], g["conv"], g["conv.b"]))
            xs = xbc[:, :inner].view(t, nh, pd)
            b = spread(xbc[:, inner:inner + ng * ns].reshape(t, ng, ns), nh)
            cc = spread(xbc[:, inner + ng * ns:].reshape(t, ng, ns), nh)
            decay = torch.exp(-torch.exp(g["A_log"]) * dt)[:, :, None].expand(t, nh, ns)
            y = recur(cc, b, dt[:, :, None] * xs, decay) + g["D"][None, :, None] * xs
            y = y.reshape(t, inner) * silu(z)
            parts = c["norm_groups"]
            return (unit_rms(y.view(t, parts, inner // parts), eps).reshape(t, inner) * g["norm"]) @ g["o"].T
        if name == "glr":
            nh = c["heads"]
            q, v = silu(lin("q")).view(t, nh, 128), lin("v").view(t, nh, 128)
            f = (g["lower"] + (1.0 - g["lower"]) * torch.sigmoid(lin("f") + g["f.b"])).view(t, nh, 128)
            return (unit_rms(recur(q, 1.0 - f, v, f), eps) * g["norm"]).reshape(t, -1) @ g["o"].T
        if name == "latent":
            nh, r, rot = c["heads"], c["kv_rank"], c["rot"]
            dkv = lin("dkv")
            lat, kr = unit_rms(dkv[:, :r], eps) * g["dkv.norm"], rotate(dkv[:, r:], rot, False)
            q = ((unit_rms(lin("dq"), eps) * g["dq.norm"]) @ g["uq"].T).view(t, nh, 192)
            q = torch.cat([q[..., :128], rotate(q[..., 128:], rot, False)], -1)
            k = torch.cat([(lat @ g["uk"].T).view(t, nh, 128), kr[:, None].expand(t, nh, 64)], -1)
            return attend(q, k, (lat @ g["uv"].T).view(t, nh, 128), c["scale"], sink=g["sink"]).reshape(t, -1) @ g["o"].T
        if name == "retention":
            nh = c["heads"]
            q, k = rotate(lin("q").view(t, nh, 128), c["rot"], True), rotate(lin("k").view(t, nh, 128), c["rot"], True) * 128 ** -0.5
            decay = torch.tensor(c["decay"], device=DEV, dtype=F64)[None, :, None].expand(t, nh, 128)
            o = recur(q, k, lin("v").view(t, nh, 128), decay)
            return (unit_rms(o, eps).reshape(t, -1) * silu(lin("g"))) @ g["o"].T
        if name == "side":
            a, s = c["left"], c["right"]
            k = lin("left.k").view(t, a["kv_heads"], 128)
            y = attend(rotate(lin("left.q").view(t, a["heads"], 128), a["rot"], True), rotate(k, a["rot"], True), k, a["scale"])
            left = (y * torch.sigmoid(lin("left.g"))[:, :, None]).reshape(t, -1) @ g["left.o"].T
            nh, nk = s["heads"], s["kv_heads"]
            q = unit_vector(silu(short_conv(lin("right.q"), g["right.q.conv"])).view(t, nk, 128)) * 128 ** -0.5
            k = unit_vector(silu(short_conv(lin("right.k"), g["right.k.conv"])).view(t, nk, 128))
            v = silu(short_conv(lin("right.v"), g["right.v.conv"])).view(t, nh, 128)
            decay = torch.exp(-torch.exp(g["right.A_log"]) * softplus(lin("right.a") + g["right.dt_bias"]))[:, :, None].expand(t, nh, 128)
            o = recur(spread(q, nh), spread(k, nh), v, decay, torch.sigmoid(lin("right.b")))
            o = (unit_rms(o, eps) * g["right.norm"]).reshape(t, -1) * silu(lin("right.g"))
            return c["left_scale"] * left + c["right_scale"] * (o @ g["right.o"].T)
        if name == "gla":
            nh = c["heads"]
            decay = torch.sigmoid(lin("a1") @ g["a2"].T + g["a2.b"]) ** (1.0 / c["tau"])
            o = recur(lin("q").view(t, nh, 128) * 128 ** -0.5, lin("k").view(t, nh, 128), lin("v").view(t, nh, 128), decay.view(t, nh, 128))
            return ((unit_rms(o, eps) * g["norm"]).reshape(t, -1) * silu(lin("g"))) @ g["o"].T
        nh, nk, size = c["heads"], c["kv_heads"], c["mask"]["size"]
        q = (unit_rms(lin("q"), eps) * g["q.norm"]).view(t, nh, 128)
        k = (unit_rms(lin("k"), eps) * g["k.norm"]).view(t, nk, 128)
        y = attend(q, k, lin("v").view(t, nk, 128), c["scale"], seen=lambda i, j: (j <= i) & (i // size == j // size),
                   lower=lambda hh, i, j: 2.0 ** (-8.0 * (hh + 1) / nh) * (i - j), sink=torch.zeros(nh, device=DEV, dtype=F64))
        return y.reshape(t, -1) @ g["o"].T

    def feed(h, g, mlp):
        if mlp["kind"] == "dense":
            up = h @ g["up"].T
            return (torch.relu(up) ** 2 if arch == "Kinetar" else gelu_tanh(h @ g["gate"].T) * up) @ g["down"].T
        r = mlp["router"]
        z = h @ g["router"].T
        n, groups = z.shape[1], r["groups"]["count"]
        score = torch.sigmoid(z) if arch == "Famepel" else torch.softmax(z, 1)
        choice = score + g["correction"] if arch == "Mafalorn" else score
        by = choice.view(t, groups, n // groups)
        worth = by.topk(2, -1).values.sum(-1) if arch == "Famepel" else by.max(-1).values
        allowed = torch.zeros_like(worth).scatter_(1, worth.topk(r["groups"]["keep"], -1).indices, 1.0).bool()
        ids = choice.masked_fill(~allowed.repeat_interleave(n // groups, 1), -math.inf).topk(r["top"], -1).indices
        wts = score.gather(1, ids)
        if arch == "Famepel":
            wts = wts / (wts.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        y = torch.zeros_like(h)
        for e in range(n):
            at, slot = torch.nonzero(ids == e, as_tuple=True)
            if at.numel():
                he = h[at]
                ye = he if e >= r["experts"] else (silu(he @ g["e%d.gate" % e].T) * (he @ g["e%d.up" % e].T)) @ g["e%d.down" % e].T
                y.index_add_(0, at, ye * wts[at, slot][:, None])
        return y

    for i, (name, lc) in enumerate(zip(names, d["layers"])):
        p, mlp = "l%d." % i, lc["mlp"]
        g = {k[len(p) + 4:]: v for k, v in w.items() if k.startswith(p + "mix.")}
        gm = {k[len(p) + 4:]: v for k, v in w.items() if k.startswith(p + "mlp.")}
        h = norm(x, p + "norm1")
        m = mixer(name, h, g, lc["mixer"])
        if arch in ("Kinetar", "Kisadra"):
            x = x + m + feed(h, gm, mlp)
            continue
        x = x + norm(m, p + "norm1b") * (w[p + "ls1"] if arch == "Famepel" else 1.0)
        if mlp:
            x = x + norm(feed(norm(x, p + "norm2"), gm, mlp), p + "norm2b") * (w[p + "ls2"] if arch == "Famepel" else 1.0)
    return norm(x, "final.norm")


def hybrid_exact(case, seed):
    names, d = describe(case)
    w = {k: v.to(F64) for k, v in hybrid_weights(case).items()}
    lens, v = hybrid_lengths(case), d["vocab"]
    if case["kind"] == "portion":
        prompts = prompts_of(seed, v, [n + case["ctx"] for n in lens])
        rows = torch.cat([one_sequence(names, d, w, p)[case["ctx"]:] for p in prompts])
        return rows[torch.tensor(wanted(case, lens), device=DEV)] @ w["head"].T
    out = []
    for p in prompts_of(seed, v, lens):
        seq = list(p)
        for _ in range(case["new"]):
            seq.append(int(following(seq[-1], v)))
        out.append(one_sequence(names, d, w, seq)[len(p) - 1:] @ w["head"].T)
    every = torch.stack(out, 1)
    return {"logits": list(every), "tokens": None}


def hybrid_work(case):
    names, d = describe(case)
    w, v, lens = d["width"], d["vocab"], hybrid_lengths(case)
    size = 4 if case.get("dtype") == "float32" else 2
    ctx = case.get("ctx", 0)

    def step(tokens, entries, context, want):
        """bytes, flops of a step: `tokens` tokens of `entries` requests behind `context` earlier tokens each."""
        b, f = v * w * size + 4.0 * want * v + tokens * w * size, 2.0 * want * v * w
        pairs = entries * ((tokens / entries) * context + (tokens / entries) ** 2 / 2.0)
        for name, lc in zip(names, d["layers"]):
            x, mlp = lc["mixer"], lc["mlp"]
            n = w // 128 * 128
            if name == "parallel":
                inner, r = x["right"]["inner"], x["right"]["dt_rank"]
                par = w * (3 * n + n // 4) + 3 * inner * w + inner * (2 * r + 32)
                f += pairs * n * 4 + tokens * inner * 16 * 6
                b += entries * (context + tokens / entries) * (n // 4) * size + 2 * entries * inner * 16 * 4
            elif name == "delta":
                par = w * (3 * n) + 2 * LOW * (w + n)
                f += tokens * n * 128 * 8
                b += 2 * entries * n * 128 * 4
            elif name == "ssd":
                inner = 2 * w
                par = w * (3 * inner + 2 * 8 * 128 + inner // 64)
                f += tokens * inner * 128 * 5
                b += 2 * entries * inner * 128 * 4
            elif name in ("glr", "retention", "gla"):
                par = w * (4 if name == "glr" else 5) * n
                f += tokens * n * 128 * 5
                b += 2 * entries * n * 128 * 4
            elif name == "latent":
                q = x["q_rank"]
                par = w * (q + 576) + q * x["heads"] * 192 + 2 * 512 * x["heads"] * 128 + w * n
                f += pairs * x["heads"] * 2 * (192 + 128) + 2.0 * ctx * entries * 512 * 256 * x["heads"]
                b += entries * (context + tokens / entries) * 576 * size
            elif name == "side":
                par = w * (2 * n + n // 4) + w * (4 * n)
                f += pairs * n * 4 + tokens * n * 128 * 8
                b += entries * (context + tokens / entries) * (n // 2) * size + 2 * entries * n * 128 * 4
            else:
                par = w * (2 * n + n // 2)
                f += entries * min(tokens / entries, 1024) * (tokens / entries) / 2 * n * 4
                b += entries * min(context + tokens / entries, 1024) * (n // 2) * size
            b, f = b + par * size, f + 2.0 * tokens * par
            if mlp and mlp["kind"] == "dense":
                one = (3 if d["architecture"] == "Kisadra" else 2) * mlp["ff"] * w
                b, f = b + one * size, f + 2.0 * tokens * one
            elif mlp:
                one, r = 3 * mlp["expert"]["ff"] * w, mlp["router"]
                hit = r["experts"] * (1.0 - (1.0 - 1.0 / r["experts"]) ** (tokens * r["top"]))
                b, f = b + hit * one * size, f + 2.0 * tokens * r["top"] * one
        return b, f
    if case["kind"] == "portion":
        b, f = step(sum(lens), len(lens), ctx, len(wanted(case, lens)))
        return {"bytes": b, "flops": f}
    b, f = step(sum(lens), len(lens), 0, len(lens))
    for i in range(case["new"]):
        bi, fi = step(len(lens), len(lens), sum(lens) / len(lens) + i, len(lens))
        b, f = b + bi, f + fi
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------------------------------------
# entry points
# ---------------------------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    return qwen_prepare(case, seed) if "model" in case else hybrid_prepare(case, seed)


def run(state):
    return hybrid_run(state) if state["kind"] in ("request", "portion") else qwen_run(state)


def exact(case, seed):
    if torch.cuda.is_available():
        _kept.update(key=None, engine=None)
    return qwen_exact(case, seed) if "model" in case else hybrid_exact(case, seed)


def work(case):
    return qwen_work(case) if "model" in case else hybrid_work(case)


def tolerance(case):
    """About four times the distance of the results from the same layers in 64 bits, as measured: 28 layers of bf16 0.019 (all of
    them round the stream), one or two hybrid layers 0.0013 to 0.0052, fp32 6e-7 to 4e-6.  Tokens are the same: the head's first
    choice stands clear of rounding."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    if "model" in case:
        return {"rel": 0.03}
    return {"rel": 0.012 if case["kind"] == "request" else 0.016}
