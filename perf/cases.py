"""The work that the engine's speed is judged by, as cases that can be prepared, run once and compared.

A case names a model, what a step is asked to do and its sizes:

    prefill   prompts (up to 2,048 tokens together: one step) to the logits behind their last tokens, as when
              requests arrive
    decode    one more token of each of several running requests, whose caches are in place
    mixed     the next 512 tokens of a prompt beside one more token of each running request, as when a request arrives
              while others are being answered
    reply     prompts, then a known reply token by token (what an answer costs from arrival to its last token, and how
              a model without an undoable cache is decoded), the logits of every step kept

All of it goes through `ModelRunner.step`, the step function that `Engine` runs, with an engine around random weights;
a pass puts the caches back as they were (`truncate`, `free_request`), so that it can be repeated. The models are the
benchmark's: Qwen2.5 0.5B whole and eight layers of the 3B and 7B sizes (at full depth their random weights carry
bfloat16's rounding to 3 % of the logits, more than a comparison can use), and for the designs with other mixers and
feed-forwards Fezopel (windowed attention with sinks, two linear recurrences, depth averages) and Miforax (latent
attention, experts by table) with eight layers at the 0.5B and 3B widths.
"""
import hashlib
import itertools
import math
import random
import weakref

import torch

import boring_llm_b200 as bl

STEP_TOKENS = 2048            # tokens of one step (the engine's default budget)
PORTION = 512                 # prompt tokens of one request beside running ones (the engine's default portion)
CONTEXT = 4096                # the engine's default context size
WINDOW = 1024                 # of the windowed models
STATES = 5                    # prepared states that may be alive together

QWEN2 = {
    "0.5b": dict(num_hidden_layers=24, hidden_size=896, num_attention_heads=14, num_key_value_heads=2, head_dim=64,
                 intermediate_size=4864, vocab_size=151936, tie_word_embeddings=True),
    "3b": dict(num_hidden_layers=8, hidden_size=2048, num_attention_heads=16, num_key_value_heads=2, head_dim=128,
               intermediate_size=11008, vocab_size=151936, tie_word_embeddings=True),
    "7b": dict(num_hidden_layers=8, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4, head_dim=128,
               intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False),
}
LATENT = {"0.5b": (384, 256, 32), "3b": (768, 512, 64)}       # query rank, key/value rank, rotated part
DESIGN_LAYERS = 8


def listed():
    return [
        # one user at a prompt: the smallest step there is, all launches and latency
        {"name": "decode 1 short", "model": "qwen2-0.5b", "kind": "decode", "requests": 1, "longest": 300, "shortest": 300},
        # the headline: eight users with long contexts
        {"name": "decode 8 long", "model": "qwen2-0.5b", "kind": "decode", "requests": 8, "longest": 4000, "shortest": 4000},
        # a full server, contexts of all lengths
        {"name": "decode 64 ragged", "model": "qwen2-0.5b", "kind": "decode", "requests": 64, "longest": 4003, "shortest": 205},
        # the headline prompt: 2,048 tokens in one step
        {"name": "prefill 2048", "model": "qwen2-0.5b", "kind": "prefill", "requests": 1, "longest": 2048, "shortest": 2048},
        # a prompt arrives at a full server
        {"name": "mixed 512 + 63", "model": "qwen2-0.5b", "kind": "mixed", "requests": 63, "longest": 3600, "shortest": 512},
        # the true 32-bit path: short prompts of odd lengths
        {"name": "prefill 32-bit", "model": "qwen2-0.5b", "kind": "prefill", "dtype": "float32", "requests": 3, "longest": 211,
         "shortest": 33},
        # a larger model: prompts of odd lengths in one step, and a few users
        {"name": "prefill 3b ragged", "model": "qwen2-3b", "kind": "prefill", "requests": 3, "longest": 1001, "shortest": 333},
        {"name": "decode 7b 16", "model": "qwen2-7b", "kind": "decode", "requests": 16, "longest": 901, "shortest": 203},
        # recurrent layers: a long prompt, and eight short questions answered at the larger width
        {"name": "fezopel prefill 2048", "model": "fezopel-0.5b", "kind": "prefill", "requests": 1, "longest": 2048, "shortest": 2048},
        {"name": "fezopel 3b reply", "model": "fezopel-3b", "kind": "reply", "requests": 8, "longest": 401, "shortest": 57, "reply": 6},
        # latent attention and experts: prompts of odd lengths at the larger width, and a few users past the window
        {"name": "miforax 3b prefill", "model": "miforax-3b", "kind": "prefill", "requests": 2, "longest": 1400, "shortest": 600},
        {"name": "miforax decode 8", "model": "miforax-0.5b", "kind": "decode", "requests": 8, "longest": 2001, "shortest": 1501},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model, kinds = rng.choice([
        ("qwen2-0.5b", ("prefill", "decode", "mixed")), ("qwen2-0.5b", ("prefill", "decode", "mixed")),
        ("qwen2-3b", ("prefill", "decode")), ("qwen2-7b", ("decode",)), ("fezopel-0.5b", ("prefill", "reply")),
        ("fezopel-3b", ("prefill", "reply")), ("miforax-0.5b", ("prefill", "decode")), ("miforax-3b", ("prefill", "decode"))])
    kind = rng.choice(kinds)
    case = {"model": model, "kind": kind}
    if kind == "prefill" and model == "qwen2-0.5b" and rng.random() < 0.25:
        case["dtype"] = "float32"
        case["requests"] = rng.randint(1, 4)
        case["longest"] = _log(rng, 8, 211)
    elif kind == "prefill":
        case["requests"] = _log(rng, 1, 8)
        case["longest"] = _log(rng, 24, STEP_TOKENS // case["requests"])
    elif kind == "decode":
        case["requests"] = _log(rng, 1, 16 if model == "qwen2-7b" else 64)
        case["longest"] = _log(rng, 60, min(4000, 32768 // case["requests"]) if model != "qwen2-7b" else 900)
    elif kind == "mixed":
        case["requests"] = _log(rng, 1, 63)
        case["longest"] = _log(rng, 100, 3500)
    else:
        case["requests"] = _log(rng, 1, 12)
        case["longest"] = _log(rng, 20, 400)
        case["reply"] = rng.randint(3, 6)
    case["shortest"] = _log(rng, max(5, case["longest"] // 8), case["longest"]) if case["requests"] > 1 else case["longest"]
    return case


# ---- models ----------------------------------------------------------------------------------------------------------
def _config_dict(model):
    """config.json of a case's model."""
    family, size = model.split("-")
    s = QWEN2[size]
    if family == "qwen2":
        return dict(s, architectures=["Qwen2ForCausalLM"], rope_theta=1000000.0, rms_norm_eps=1e-6, max_position_embeddings=32768)
    d, H, KV, dh, F = (s[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
    common = {"vocab": s["vocab_size"], "width": d, "norm": {"eps": 1e-6}, "max_position_embeddings": 32768}
    if family == "fezopel":
        mixers = {
            "attention": {"heads": H, "kv_heads": KV, "dim": dh, "vdim": dh, "mask": {"size": WINDOW},
                          "rot": {"base": 1000000.0, "dims": dh}, "scale": dh ** -0.5},
            "gla": {"heads": H // 2, "dim": dh, "vdim": 2 * dh, "tau": 16.0, "rank": 16},
            "channel_delta": {"heads": H // 2, "kv_heads": H // 2, "dim": dh, "vdim": 2 * dh, "conv": 4, "rank": 32, "gate_rank": 32},
        }
        pattern = ("attention", "gla", "gla", "channel_delta")
        layers = [{"type": pattern[i % 4], "mixer": mixers[pattern[i % 4]], "mlp": {"kind": "dense", "ff": F}} for i in range(DESIGN_LAYERS)]
        return dict(common, architecture="Fezopel", layers=layers)
    q_rank, kv_rank, rot = LATENT[size]
    layers = []
    for i in range(DESIGN_LAYERS):
        m = {"heads": H, "dim": dh, "rot_dim": rot, "vdim": dh, "q_rank": q_rank, "kv_rank": kv_rank, "scale": (dh + rot) ** -0.5,
             "mask": {"size": WINDOW},
             "rot": {"base": 1000000.0, "dims": rot, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        if i % 2 == 1:
            m["kv_from"] = i - 1
        mlp = {"kind": "dense", "ff": F} if i == 0 else {
            "kind": "moe", "expert": {"ff": F // 4 // 8 * 8, "limit": 7.0}, "router": {"experts": 16, "top": 2},
            "shared": {"ff": F // 2 // 8 * 8, "limit": 7.0}}
        layers.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
    return dict(common, architecture="Miforax", embedding={"scale": 1.0}, layers=layers)


def _config(model):
    cls = {"qwen2": bl.Qwen2Config, "fezopel": bl.FezopelConfig, "miforax": bl.MiforaxConfig}[model.split("-")[0]]
    return cls.from_dict(_config_dict(model))


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


class _Weights:
    """Seeded random tensors by name, made on the GPU when asked for: matrices and biases N(0, 0.02), norm weights
    1 + N(0, 0.02), tables of different numbers in a row."""

    def __init__(self, model, dtype):
        config = _config(model)
        self.specs = bl.build_model(config).tensor_specs()
        self.dtype = dtype

    def __getitem__(self, name):
        spec = self.specs[name]
        g = torch.Generator(device="cuda").manual_seed(int.from_bytes(hashlib.sha256(name.encode()).digest()[:7], "little"))
        if spec.kind == "int_table":
            first = torch.randint(0, spec.high, (spec.shape[0], 1), generator=g, device="cuda")
            return ((first + torch.arange(spec.shape[1], device="cuda")) % spec.high).to(torch.int32)
        x = torch.randn(tuple(spec.shape), generator=g, device="cuda") * 0.02
        return (x + 1.0 if spec.kind == "norm" else x).to(self.dtype)

    def __contains__(self, name):
        return name in self.specs

    def __iter__(self):
        return iter(self.specs)

    def __len__(self):
        return len(self.specs)

    def keys(self):
        return self.specs.keys()


_engines = {}                 # the one engine that is kept, by what it was built for
_names = itertools.count()


def _engine(case):
    """The engine that serves the case's model: a program builds it once and gives it all its requests."""
    key = (case["model"], str(_dtype(case)), case["requests"], case["kind"], case["longest"])
    if key not in _engines:
        _engines.clear()
        torch.cuda.empty_cache()
        config = _config(case["model"])
        model = bl.build_model(config)
        model.load(_Weights(case["model"], _dtype(case)), _dtype(case), torch.device("cuda:0"))
        seqs = STATES * (case["requests"] + 1)
        tokens = STATES * sum(n + 32 for n in _lengths(case) + [3 * PORTION if case["kind"] == "mixed" else 0])
        options = bl.EngineOptions(dtype="float32" if _dtype(case) == torch.float32 else "bfloat16", ctx_size=CONTEXT, max_num_seqs=seqs,
                                   max_tokens=tokens, max_num_batched_tokens=STEP_TOKENS, prefill_chunk=PORTION)
        _engines[key] = bl.Engine.from_model(config, model, options)
    return _engines[key]


# ---- cases -----------------------------------------------------------------------------------------------------------
def _lengths(case):
    """The requests' lengths (of their prompts, or of what is cached), spread evenly from the longest to the shortest."""
    n, hi, lo = case["requests"], case["longest"], case["shortest"]
    out = [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]
    if case["kind"] == "decode" and not case["model"].startswith("qwen2"):
        # one token more would make the window drop a page, and a dropped page cannot be taken back by the next pass
        out = [m + 1 if (m - WINDOW + 2) % 16 == 0 else m for m in out]
    return out


def _tokens(case, seed):
    """(the requests' cached tokens or prompts, what follows them): uniform token ids."""
    vocab = QWEN2[case["model"].split("-")[1]]["vocab_size"]
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)

    def ids(n):
        return torch.randint(0, vocab, (n,), generator=g).tolist()
    before = [ids(n) for n in _lengths(case)]
    if case["kind"] == "prefill":
        return before, [[] for _ in before]
    after = [ids(case.get("reply", 1)) for _ in before]
    if case["kind"] == "mixed":
        before.append(ids(2 * PORTION))
        after.append(ids(PORTION))
    return before, after


def _batches(ids, prompts):
    """Steps of up to STEP_TOKENS tokens that run the prompts: lists of (request, from, to)."""
    out, room = [[]], STEP_TOKENS
    for rid, p in zip(ids, prompts):
        at = 0
        while at < len(p):
            n = min(room, len(p) - at)
            out[-1].append((rid, at, at + n))
            at, room = at + n, room - n
            if room == 0:
                out.append([])
                room = STEP_TOKENS
    return [b for b in out if b]


class _State:
    pass


def _release(runner, ids):
    for rid in ids:
        if runner.has_request(rid):
            runner.free_request(rid)


def prepare(case, seed):
    s = _State()
    s.kind, s.runner = case["kind"], _engine(case).runner
    before, after = _tokens(case, seed)
    s.ids = ["r%d" % next(_names) for _ in before]
    weakref.finalize(s, _release, s.runner, list(s.ids))
    prompts = dict(zip(s.ids, before))
    steps = [[bl.StepEntry(r, prompts[r][a:b], [b - a - 1] if b == len(prompts[r]) else []) for r, a, b in batch]
             for batch in _batches(s.ids, before)]
    if s.kind in ("prefill", "reply"):
        s.steps = steps
        s.replies = [[bl.StepEntry(r, [t[i]], [0]) for r, t in zip(s.ids, after)] for i in range(case.get("reply", 0))]
        return s
    for step in steps:
        s.runner.step([bl.StepEntry(e.request_id, e.tokens) for e in step])
    s.entries = [bl.StepEntry(r, t, [len(t) - 1]) for r, t in zip(s.ids, after)]
    s.lengths = [len(p) for p in before]
    return s


def run(s):
    runner = s.runner
    if s.kind in ("decode", "mixed"):
        logits = runner.step(s.entries)
        for rid, n in zip(s.ids, s.lengths):
            runner.truncate(rid, n)
        return logits
    if s.kind == "prefill":                        # one step: its logits stay until the next
        out = runner.step(s.steps[0])
    else:
        out = [torch.cat([runner.step(step).clone() for step in s.steps])]
        for step in s.replies:
            out.append(runner.step(step).clone())
    for rid in s.ids:
        runner.free_request(rid)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    """Each weight that the pass uses read once (of an embedding the gathered rows; of experts those that the tokens reach),
    cached rows read once by the step that sees them and new ones written, states read and written, logits written;
    two operations a weight and token, the products of attention over the visible keys, three multiply-adds a state
    value and token."""
    model = case["model"]
    cfg, specs = _config_dict(model), bl.build_model(_config(model)).tensor_specs()
    size = 4 if _dtype(case) == torch.float32 else 2
    s = QWEN2[model.split("-")[1]]
    H, KV, dh, V, d = (s[k] for k in ("num_attention_heads", "num_key_value_heads", "head_dim", "vocab_size", "hidden_size"))
    before = _lengths(case)
    if case["kind"] == "decode":
        steps = [[(n, 1) for n in before]]
    elif case["kind"] == "mixed":
        steps = [[(n, 1) for n in before] + [(2 * PORTION, PORTION)]]
    else:
        steps = [[(0, b - a) if a == 0 else (a, b - a) for _, a, b in batch] for batch in _batches(range(len(before)), [range(n) for n in before])]
        steps += [[(n + i, 1) for n in before] for i in range(case.get("reply", 0))]
    rows = len(before) + (case["kind"] == "mixed")
    total_bytes = total_flops = 0.0
    for step in steps:
        T = sum(n for _, n in step)
        for name, spec in specs.items():
            n = math.prod(spec.shape)
            if len(spec.shape) < 2 or spec.kind == "int_table" or name in ("model.embed_tokens.weight", "embed", "lm_head.weight", "head"):
                continue
            share = reach = 1.0
            if ".e" in name and name.split(".e")[1][0].isdigit():
                share = 2 / 16
                reach = 1.0 - (1.0 - share) ** T
            total_bytes += n * reach * size
            total_flops += 2.0 * n * share * T
        total_bytes += V * d * size + rows * V * 4 + T * d * size
        total_flops += 2.0 * V * d * rows
        for i in range(len(cfg["layers"]) if "layers" in cfg else cfg["num_hidden_layers"]):
            kind = cfg["layers"][i]["type"] if "layers" in cfg else "attention"
            m = cfg["layers"][i]["mixer"] if "layers" in cfg else {}
            window = (m.get("mask") or {}).get("size", 1 << 30)
            if kind in ("gla", "channel_delta"):
                state = m["heads"] * m["dim"] * m["vdim"]
                total_bytes += 8.0 * state * len(step)
                total_flops += 6.0 * state * T
                continue
            if kind == "latent_attention":
                row, per_pair = m["kv_rank"] + m["rot_dim"], 2.0 * H * (2 * dh + m["rot_dim"])
            else:
                row, per_pair = 2 * KV * dh, 4.0 * H * dh
            for have, n in step:
                total_bytes += row * size * (min(have, window) + n)
                total_flops += per_pair * sum(min(have + j + 1, window) for j in range(n))
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # four times the error against `exact` (32-bit: 3.7e-6 of the logits; bfloat16: 0.6 to 1.5e-2, held to 0.03)
    return {"rel": 1.5e-5} if case.get("dtype") == "float32" else {"rel": 0.03}


# ---- the same outputs in 64 bits, plainly ----------------------------------------------------------------------------
def _rms(x, w=None, eps=1e-6):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _ln(x, w, b, eps=1e-6):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w + b


def _turn(x, freq, interleaved=False, factor=1.0):
    """x [T, heads, n]: pairs (i, i + n/2), or neighbours, turn by position * freq[i]."""
    a = (torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None] * freq)[:, None]
    c, s = torch.cos(a) * factor, torch.sin(a) * factor
    u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else x.chunk(2, -1)
    parts = (u * c - v * s, v * c + u * s)
    return torch.stack(parts, -1).flatten(-2) if interleaved else torch.cat(parts, -1)


def _frequencies(n, base):
    return base ** (-2.0 * torch.arange(n // 2, device="cuda", dtype=torch.float64) / n)


def _stretched(n, base, sc):
    """Frequencies for longer contexts: fast pairs stay, slow ones are divided by the factor, a ramp between the two."""
    f = _frequencies(n, base)

    def pair(turns):
        return n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), n - 1)
    ramp = ((torch.arange(n // 2, device="cuda", dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _attend(q, k, v, scale, window=0, sink=None):
    """q [T, H, dq], k [T, G, dq], v [T, G, dv]: causal softmax attention, one query head after the other."""
    T, H, _ = q.shape
    i = torch.arange(T, device=q.device)
    hidden = i[None, :] > i[:, None]
    if window:
        hidden |= i[:, None] - i[None, :] >= window
    out = q.new_empty(T, H, v.shape[2])
    for h in range(H):
        g = h // (H // k.shape[1])
        s = (q[:, h] @ k[:, g].T * scale).masked_fill_(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, g]
    return out


def _qwen2(W, cfg, x, tokens, i):
    p = "model.layers.%d." % i
    H, KV, dh = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    # the angles are products in 32 bits by definition of the architecture
    j = torch.arange(dh // 2, dtype=torch.float32)
    freq = (1.0 / torch.pow(torch.tensor(cfg["rope_theta"], dtype=torch.float32), 2.0 * j / dh)).cuda()
    w = {n: W(p + n) for n in ["input_layernorm.weight", "post_attention_layernorm.weight", "self_attn.o_proj.weight"]
         + ["mlp.%s_proj.weight" % n for n in ("gate", "up", "down")] + ["self_attn.%s_proj.%s" % (n, t) for n in "qkv" for t in ("weight", "bias")]}
    out = []
    for y in x:
        T = y.shape[0]
        a32 = (torch.arange(T, dtype=torch.float32, device="cuda")[:, None] * freq).double()[:, None]
        c, s = torch.cos(a32), torch.sin(a32)

        def turn(z):
            u, v = z.chunk(2, -1)
            return torch.cat([u * c - v * s, u * s + v * c], -1)
        h = _rms(y, w["input_layernorm.weight"])
        q, k, v = (h @ w["self_attn.%s_proj.weight" % n].T + w["self_attn.%s_proj.bias" % n] for n in "qkv")
        a = _attend(turn(q.view(T, H, dh)), turn(k.view(T, KV, dh)), v.view(T, KV, dh), dh ** -0.5)
        y = y + a.flatten(1) @ w["self_attn.o_proj.weight"].T
        h = _rms(y, w["post_attention_layernorm.weight"])
        out.append(y + (torch.nn.functional.silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T)
    return out


def _recurrence(q, k, v, decay, beta=None):
    """S <- decay S (rows); u = v, or beta (v - S^T k) where beta is given; S <- S + k u^T; o = S^T q, from S = 0."""
    T, H, dk = q.shape
    S = q.new_zeros(H, dk, v.shape[2])
    out = torch.empty_like(v)
    for t in range(T):
        S *= decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S += k[t][:, :, None] * u[:, None]
        out[t] = (q[t][:, None] @ S)[:, 0]
    return out


def _fezopel_mixer(W, p, kind, m, h):
    T, H, dk, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
    if kind == "attention":
        q, k = (_rms(h @ W(p + n).T, W(p + n + ".norm")).view(T, -1, dk) for n in "qk")
        f = _frequencies(m["rot"]["dims"], m["rot"]["base"])
        o = _attend(_turn(q, f, True), _turn(k, f, True), (h @ W(p + "v").T).view(T, -1, dv), m["scale"], WINDOW, W(p + "sink"))
        return (o * torch.sigmoid(h @ W(p + "g").T)[:, :, None]).flatten(1) @ W(p + "o").T
    if kind == "gla":
        q, k, v = ((h @ W(p + n).T).view(T, H, -1) for n in "qkv")
        decay = torch.sigmoid(h @ W(p + "a1").T @ W(p + "a2").T + W(p + "a2.b")).view(T, H, dk) ** (1.0 / m["tau"])
        o = _rms(_recurrence(q * dk ** -0.5, k, v, decay), W(p + "norm")).flatten(1)
        return (o * torch.nn.functional.silu(h @ W(p + "g").T)) @ W(p + "o").T

    def conv(n):
        x, taps = h @ W(p + n).T, W(p + n + ".conv")
        x = torch.cat([x.new_zeros(taps.shape[1] - 1, x.shape[1]), x])
        return torch.nn.functional.silu(sum(x[j:j + T] * taps[:, j] for j in range(taps.shape[1]))).view(T, H, -1)
    q, k, v = (conv(n) for n in "qkv")
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    z = (h @ W(p + "a1").T @ W(p + "a2").T + W(p + "dt_bias")).view(T, H, dk)
    decay = torch.exp(-torch.exp(W(p + "A_log"))[:, None] * torch.nn.functional.softplus(z))
    o = _rms(_recurrence(q * dk ** -0.5, k, v, decay, torch.sigmoid(h @ W(p + "b").T)), W(p + "norm"))
    return (o * torch.sigmoid(h @ W(p + "g1").T @ W(p + "g2").T).view(T, H, dv)).flatten(1) @ W(p + "o").T


def _fezopel(W, layer, history, x, i):
    p = "l%d." % i
    out = []
    for r, y in enumerate(x):
        h = _ln(y, W(p + "norm1"), W(p + "norm1.b"))
        m = _fezopel_mixer(W, p + "mix.", layer["type"], layer["mixer"], h) * torch.sigmoid(h @ W(p + "rg1").T + W(p + "rg1.b"))
        y = y + _ln(m, W(p + "norm1b"), W(p + "norm1b.b"))
        h = _ln(y, W(p + "norm2"), W(p + "norm2.b"))
        f = torch.nn.functional.gelu(h @ W(p + "mlp.up").T) @ W(p + "mlp.down").T * torch.sigmoid(h @ W(p + "rg2").T + W(p + "rg2.b"))
        history[r].append(y + _ln(f, W(p + "norm2b"), W(p + "norm2b.b")))
        out.append(sum(a * b for a, b in zip(W(p + "dwa"), history[r])))
    return out


def _clamped(W, p, h, limit):
    g, u = (h @ W(p + "gate").T).clamp(max=limit), (h @ W(p + "up").T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(p + "down").T


def _miforax(W, layer, cached, x, tokens, i):
    p, m, f = "l%d." % i, layer["mixer"], layer["mlp"]
    H, dn, dv, rank = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    freq, factor = _stretched(m["rot_dim"], m["rot"]["base"], m["rot"]["scaling"])
    out = []
    for r, y in enumerate(x):
        T = y.shape[0]
        h = _rms(y, W(p + "norm1"))
        q = (_rms(h @ W(p + "mix.dq").T, W(p + "mix.dq.norm")) @ W(p + "mix.uq").T).view(T, H, -1)
        if "kv_from" not in m:
            z = h @ W(p + "mix.dkv").T
            cached[r] = _rms(z[:, :rank], W(p + "mix.dkv.norm")), _turn(z[:, None, rank:], freq, factor=factor)
        latent, turned = cached[r]
        q = torch.cat([q[..., :dn], _turn(q[..., dn:], freq, factor=factor)], -1)
        k = torch.cat([(latent @ W(p + "mix.uk").T).view(T, H, dn), turned.expand(T, H, -1)], -1)
        o = _attend(q, k, (latent @ W(p + "mix.uv").T).view(T, H, dv), m["scale"], WINDOW, W(p + "mix.sink")).flatten(1)
        y = y + (o * torch.sigmoid(h @ W(p + "mix.g").T)) @ W(p + "mix.o").T
        h = _rms(y, W(p + "norm2"))
        p2 = p + "mlp."
        if f["kind"] == "dense":
            a = torch.nn.functional.gelu(h @ W(p2 + "gate").T, approximate="tanh") * (h @ W(p2 + "up").T) @ W(p2 + "down").T
        else:
            a = _clamped(W, p2 + "shared.", h, f["shared"]["limit"])
            chosen = W(p2 + "table")[torch.tensor(tokens[r], device="cuda")]
            for e in range(f["router"]["experts"]):
                at = (chosen == e).any(1).nonzero()[:, 0]
                if len(at):
                    a[at] += _clamped(W, p2 + "e%d." % e, h[at], f["expert"]["limit"]) / f["router"]["top"]
        out.append(y + a)
    return out


@torch.no_grad()
def exact(case, seed):
    """Every request as one whole sequence without a cache; the rows that `run` returns."""
    cfg, made = _config_dict(case["model"]), _Weights(case["model"], _dtype(case))
    if work(dict(case, kind="prefill", requests=1, longest=1, shortest=1))["flops"] * sum(_lengths(case)) > 4e14:
        return None

    layer_weights = {}

    def W(name):                                   # kept for one layer at a time
        if name not in layer_weights:
            t = made[name]
            layer_weights[name] = t.double() if t.is_floating_point() else t
        return layer_weights[name]

    before, after = _tokens(case, seed)
    tokens = [p + t for p, t in zip(before, after)]
    family = case["model"].split("-")[0]
    embed = "model.embed_tokens.weight" if family == "qwen2" else "embed"
    table = made[embed]
    x = [table[torch.tensor(t, device="cuda")].double() for t in tokens]
    history, cached = [[y] for y in x], {}
    for i in range(cfg["num_hidden_layers"] if family == "qwen2" else len(cfg["layers"])):
        layer_weights.clear()
        if family == "qwen2":
            x = _qwen2(W, cfg, x, tokens, i)
        elif family == "fezopel":
            x = _fezopel(W, cfg["layers"][i], history, x, i)
        else:
            x = _miforax(W, cfg["layers"][i], cached, x, tokens, i)
    layer_weights.clear()
    head = W(embed if cfg.get("tie_word_embeddings") else "lm_head.weight" if family == "qwen2" else "head")
    if family == "fezopel":
        x = [_ln(y, W("final.norm"), W("final.norm.b")) for y in x]
    else:
        x = [_rms(y, W("model.norm.weight" if family == "qwen2" else "final.norm")) for y in x]
    if case["kind"] == "reply":
        n = case["reply"]
        return [torch.stack([y[len(y) - 1 - n + i] for y in x]) @ head.T for i in range(n + 1)]
    return torch.stack([y[-1] for y in x]) @ head.T
