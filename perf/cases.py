"""The work that a user of this engine has it do, as cases to be timed and compared.

A case is one pass through the engine's public step function (`Engine.step`, `Engine.finish`), on a model of seeded
random weights at the layer sizes of `bench.py`, with fewer layers so that many models can be made in a row:

* `decode`: `requests` running requests whose contexts (up to `context` tokens, ragged) are cached; the pass is the step
  that brings one more token of each. It can be run again: a step at an earlier position takes the place of what was there.
* `mixed`: the same riders, and in the same step a portion of `rows` tokens of a prompt whose first `rows` tokens are cached.
* `prompt`: `requests` new requests bring `rows` prompt tokens in one step (ragged, or one whole prompt), then `tail` steps of
  one given token each (as trace replay feeds them), then they end and give their pages back.

What comes back is what the step function gives: the logits at the places a generating program asks for (the last row of
every prompt, every decoded row). `exact` computes the same logits in 64 bits from the models' formulas with plain torch.
"""
import hashlib
import math

import torch

from jllm_serve_b200.engine import Engine, Segment

DEVICE = "cuda:0"
PAGE = 16
MAX_STEP_ROWS = 2048


# ---- the cases ----------------------------------------------------------------------------------------------------

def _case(name, kind, model, width, layers, requests, *, context=0, rows=0, tail=0, dtype="bfloat16"):
    out = dict(kind=kind, model=model, width=width, layers=layers, requests=requests, context=context, rows=rows, tail=tail,
               dtype=dtype)
    return dict(out, name=name) if name else out


def listed():
    return [
        # one user's chat: every new token is a step of one row, bound by the weights' stream and by launches
        _case("decode 1", "decode", "qwen3", 4096, 8, 1, context=777),
        # the headline point of the benchmark: eight requests at contexts of up to 4,096 tokens
        _case("decode 8", "decode", "qwen3", 4096, 8, 8, context=4095),
        # a busy server: 64 requests, the cache as large as the weights
        _case("decode 64", "decode", "qwen3", 4096, 8, 64, context=1800),
        # a short question: the smallest prompt step, where the host's launches show
        _case("prompt 47", "prompt", "qwen3", 4096, 8, 1, rows=47),
        # three users' prompts that arrive together, of odd lengths: some hundreds of rows
        _case("prompts 613 of 3", "prompt", "qwen3", 4096, 8, 3, rows=613),
        # the benchmark's prompt: 2,048 tokens at once
        _case("prompt 2048", "prompt", "qwen3", 4096, 8, 1, rows=2048),
        # a long prompt's portion of 512 tokens beside 32 decoding requests, at the 14B layer sizes
        _case("mixed 512+32", "mixed", "qwen3", 5120, 4, 32, context=4096, rows=512),
        # the 32-bit path, which checks the other one: a prompt, then tokens one by one
        _case("prompt 300 fp32", "prompt", "qwen3", 4096, 2, 1, rows=300, tail=4, dtype="float32"),
        # the other designs at the benchmark's first size: a whole prompt ...
        _case("movivik 2048", "prompt", "movivik", 2048, 8, 1, rows=2048),
        _case("guvolix 1536 of 2", "prompt", "guvolix", 2048, 8, 2, rows=1536),
        _case("bozevik 2048", "prompt", "bozevik", 2048, 8, 1, rows=2048),
        # ... and eight short requests answered with two dozen tokens each: mostly decode steps over states of fixed size
        _case("fusazen 777 of 8", "prompt", "fusazen", 2048, 8, 8, rows=777, tail=24),
    ]


def _spread(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "design", "design", "design", "float32"])
    if kind == "decode":
        requests = _spread(rng, 1, 64)
        return _case("", kind, "qwen3", 4096, 8, requests, context=_spread(rng, 100, min(8000, 120000 // requests)))
    if kind == "prompt":
        rows = _spread(rng, 20, 2048)
        return _case("", kind, "qwen3", 4096, 8, rng.randint(1, max(1, min(8, rows // 20))), rows=rows)
    if kind == "mixed":
        requests = _spread(rng, 2, 48)
        return _case("", kind, "qwen3", 5120, 4, requests, context=_spread(rng, 200, min(6000, 120000 // requests)),
                     rows=_spread(rng, 64, 1024))
    if kind == "float32":
        return _case("", "prompt", "qwen3", 4096, 2, rng.randint(1, 4), rows=_spread(rng, 30, 300), tail=rng.randint(0, 4),
                     dtype="float32")
    model, requests = rng.choice(["movivik", "guvolix", "bozevik", "fusazen"]), rng.randint(1, 8)
    return _case("", "prompt", model, 2048, 8, requests, rows=_spread(rng, 30 * requests, 2048), tail=rng.choice([0, 0, rng.randint(1, 16)]))


def _prompt_lengths(case):
    """`rows` tokens over `requests` prompts: shares that grow by a half from the first to the last."""
    n, rows = case["requests"], case["rows"]
    weights = [1.0 + 0.5 * i / max(1, n - 1) for i in range(n)]
    ends = [round(rows * sum(weights[:i + 1]) / sum(weights)) for i in range(n)]
    return [b - a for a, b in zip([0] + ends, ends)]


def _contexts(case):
    """The riders' contexts: from `context` down to seven eighths of it."""
    n, ctx = case["requests"], case["context"]
    return [ctx - (i * 37) % max(1, ctx // 8) for i in range(n)]


# ---- the models ---------------------------------------------------------------------------------------------------

def config(case):
    """config.json of the case's model: the layer sizes of `bench.py`."""
    D, L = case["width"], case["layers"]
    if case["model"] == "qwen3":
        heads, ffn = {4096: (32, 12288), 5120: (40, 17408)}[D]
        return dict(model_type="qwen3", hidden_size=D, num_hidden_layers=L, num_attention_heads=heads, num_key_value_heads=8,
                    head_dim=128, intermediate_size=ffn, vocab_size=151936, rope_theta=1000000.0, rms_norm_eps=1e-6,
                    tie_word_embeddings=False, attention_bias=False, use_sliding_window=False, max_position_embeddings=40960,
                    hidden_act="silu")
    heads, kv_heads, ff, s = D // 128, 8, 4 * D, 128 ** -0.5
    base = {"width": D, "vocab": 32768, "norm": {"eps": 1e-6}}
    att = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": s}
    if case["model"] == "movivik":        # pairs: two layers of chunked attention, two of attention beside linear attention
        chunked = dict(att, mask={"size": 1024}, rot={"base": 500000.0, "dims": 128, "scaling": {
            "factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}})
        decay = [1.0 - 2.0 ** (-2 - 6 * h / (heads - 1)) for h in range(heads)]
        beside = {"left": dict(att, rot={"base": 10000.0, "dims": 64}),
                  "right": {"heads": heads, "dim": 128, "vdim": 128, "decay": decay}}
        mlp = {"kind": "dense", "ff": ff}
        layers = [{"type": "attention", "mixer": chunked, "mlp": mlp}] * 2 + [{"type": "parallel", "mixer": beside, "mlp": mlp}] * 2
        return dict(base, architecture="Movivik", layers=[layers[i % 4] for i in range(L)])
    if case["model"] == "guvolix":        # fours: three of attention beside a state space, one beside a matrix memory
        left = dict(att, rot={"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0}}, mask={"size": 1024, "keep_first": 64})
        left2 = dict(att, rot={"base": 20000.0, "dims": 128, "scaling": {"factor": 4.0, "low": 1.0, "high": 4.0, "original": 4096}},
                     mask={"size": 1024})
        ssm = {"heads": 2 * D // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
        memory = {"heads": D // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}
        mlp = {"kind": "dense", "ff": ff}
        first = {"type": "parallel", "mixer": {"left": left, "right": ssm}, "mlp": mlp}
        last = {"type": "parallel_2", "mixer": {"left": left2, "right": memory, "left_scale": 0.6, "right_scale": 1.1}, "mlp": mlp}
        return dict(base, architecture="Guvolix", norm={"eps": 1e-5}, embedding={"scale": 0.5},
                    layers=[last if i % 4 == 3 else first for i in range(L)])
    if case["model"] == "bozevik":        # attention over a cached latent, every second layer over its neighbour's rows
        mix = {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 192, "q_rank": 768, "rot_dim": 64,
               "rot": {"base": 10000.0, "dims": 64}, "scale": 192 ** -0.5}
        mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
        return dict(base, architecture="Bozevik", logit_scale=1.0, layers=[
            {"type": "latent_attention", "mixer": dict(mix, kv_from=i - 1) if i % 2 else mix, "mlp": mlp} for i in range(L)])
    # fusazen, in fours: attention with norms over all heads, a delta rule, differential attention with keys of its own and
    # with its neighbour's
    mlp = {"kind": "dense", "ff": 6 * D}
    whole = dict(att, mask={"size": 1024})
    delta = {"heads": D // 64, "dim": 64, "decay_rank": 64}
    diff = {"heads": heads, "kv_heads": kv_heads, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "mask": {"size": 1024}, "diff": 0.5,
            "rot": {"base": 10000.0, "dims": 32}}
    kinds = [lambda i: ("attention_2", whole), lambda i: ("general_delta", delta), lambda i: ("attention", diff),
             lambda i: ("attention", dict(diff, kv_from=i - 1))]
    layers = [dict(zip(("type", "mixer"), kinds[i % 4](i)), mlp=mlp) for i in range(L)]
    return dict(base, architecture="Fusazen", canon={"taps": 4}, embedding={"scale": 2.0}, layers=layers)


def shapes(cfg):
    """The model's tensors: name -> (shape, how random weights are drawn)."""
    out = {}

    def put(prefix, init="normal", **sizes):
        for name, shape in sizes.items():
            out[prefix + name.replace("__", ".")] = (shape if isinstance(shape, tuple) else (shape,), init)

    if cfg.get("model_type") == "qwen3":
        D, H, G, hd, F, V = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                              "intermediate_size", "vocab_size"))
        put("", **{"model.embed_tokens.weight": (V, D), "lm_head.weight": (V, D)})
        put("", "gain", **{"model.norm.weight": D})
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            put(p, **{"self_attn.q_proj.weight": (H * hd, D), "self_attn.k_proj.weight": (G * hd, D),
                      "self_attn.v_proj.weight": (G * hd, D), "self_attn.o_proj.weight": (D, H * hd),
                      "mlp.gate_proj.weight": (F, D), "mlp.up_proj.weight": (F, D), "mlp.down_proj.weight": (D, F)})
            put(p, "gain", **{"self_attn.q_norm.weight": hd, "self_attn.k_norm.weight": hd, "input_layernorm.weight": D,
                              "post_attention_layernorm.weight": D})
        return out
    D, V, name = cfg["width"], cfg["vocab"], cfg["architecture"]
    put("", embed=(V, D))
    put("", "gain", final__norm=D)
    if name != "Bozevik":
        put("", head=(V, D))

    def attention(p, m, **more):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        put(p, q=(H * dk, D), k=(G * dk, D), v=(G * dv, D), o=(D, H * dv), **more)

    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        x, kind = p + "mix.", layer["type"]
        if name == "Bozevik":
            H, dk, dv, R, qr, rd = (m[k] for k in ("heads", "dim", "vdim", "kv_rank", "q_rank", "rot_dim"))
            put(x, uk=(H * dk, R), uv=(H * dv, R), o=(D, H * dv), dq=(qr, D), uq=(H * (dk + rd), qr))
            put(x, "gain", dq__norm=qr)
            if "kv_from" not in m:
                put(x, dkv=(R + rd, D))
                put(x, "gain", dkv__norm=R)
            put(p, shift=D)
            put(p, "gain", norm1=D, norm2=D)
            put(p, "average", dwa=i + 2)
        elif name == "Movivik":
            put(p, "gain", norm1=D, norm1b=D, norm2=D, norm2b=D)
            if kind == "attention":
                attention(x, m, g=(m["heads"], D), q__b=m["heads"] * m["dim"], k__b=m["kv_heads"] * m["dim"],
                          v__b=m["kv_heads"] * m["vdim"])
            else:
                attention(x + "left.", m["left"], g=(m["left"]["heads"], D))
                r = m["right"]
                put(x + "right.", q=(r["heads"] * r["dim"], D), k=(r["heads"] * r["dim"], D), v=(r["heads"] * r["vdim"], D),
                    g=(r["heads"] * r["vdim"], D), o=(D, r["heads"] * r["vdim"]))
                put(x + "right.", "gain", norm=r["heads"] * r["vdim"])
                put(x, "gain", left__out=D, right__out=D)
        elif name == "Guvolix":
            put(p, "gain", norm1=D)
            left, r = m["left"], m["right"]
            attention(x + "left.", left, g=(left["heads"] * left["vdim"], D), sink=left["heads"])
            if kind == "parallel":
                inner, ch = r["heads"] * r["vdim"], r["heads"] * r["vdim"] + 2 * r["groups"] * r["state"]
                put(x + "right.", conv=(ch, r["conv"]), conv__b=ch, dt_bias=r["heads"], A_log=r["heads"], o=(D, inner))
                out[x + "right.in"] = ((inner + ch + r["heads"], D), "normal")
                put(x + "right.", "gain", D=r["heads"], norm=inner)
                put(x, "gain", left__out=D, right__out=D)
            else:
                H, dk, dv = r["heads"], r["dim"], r["vdim"]
                put(x + "right.", q=(H * dk, D), k=(H * dk, D), v=(H * dv, D), g=(H * dv, D), o=(D, H * dv), i=(H, D), i__b=H,
                    f=(H, D), f__b=H)
                put(x + "right.", "gain", norm=H * dv)
        else:
            put(p, "gain", norm1=D, norm2=D)
            put(p, canon1=(D, cfg["canon"]["taps"]))
            H, dk = m["heads"], m["dim"]
            if kind == "general_delta":
                put(x, **{n: (H * dk, D) for n in ("r", "k", "v", "g", "a")}, a__b=H * dk, w1=(m["decay_rank"], D),
                    w2=(H * dk, m["decay_rank"]), w0=H * dk, o=(D, H * dk))
                put(x, "gain", norm=H * dk)
            elif kind == "attention_2":
                attention(x, m)
                put(x, "gain", q__norm=H * dk, k__norm=m["kv_heads"] * dk, temp=H)
            else:
                put(x, q=(2 * H * dk, D), o=(D, H * m["vdim"]), lq1=dk, lk1=dk, lq2=dk, lk2=dk)
                if "kv_from" not in m:
                    put(x, k=(2 * m["kv_heads"] * dk, D), v=(m["kv_heads"] * m["vdim"], D))
        F = mlp["ff"]
        put(p + "mlp.", up=(F, D), down=(D, F))
        if name == "Fusazen":
            put(p + "mlp.", up__b=F, down__b=D)
        elif name != "Guvolix":
            put(p + "mlp.", gate=(F, D))
    return out


# ---- the pass -----------------------------------------------------------------------------------------------------

def _tokens(case, seed):
    """Every request's tokens: its context (or prompt) and all that the pass feeds behind it; of a mixed step also the long
    prompt's."""
    g = torch.Generator().manual_seed(seed)
    vocab = 151936 if case["model"] == "qwen3" else 32768
    if case["kind"] == "prompt":
        counts = [n + case["tail"] for n in _prompt_lengths(case)]
    else:
        counts = [n + 1 for n in _contexts(case)] + ([2 * case["rows"]] if case["kind"] == "mixed" else [])
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in counts]


def prepare(case, seed):
    tokens = _tokens(case, seed)
    longest, pages = max(map(len, tokens)), sum(-(-len(t) // PAGE) + 1 for t in tokens)
    engine = Engine(config=config(case), seed=seed, dtype=case["dtype"], ctx=-(-longest // PAGE) * PAGE + PAGE, page_size=PAGE,
                    num_pages=pages, max_batch_tokens=MAX_STEP_ROWS + 64, max_running=len(tokens))
    ids = list(range(len(tokens)))
    if case["kind"] == "prompt":
        lengths = _prompt_lengths(case)
        steps = [[Segment(i, tokens[i][:n], 0, [n - 1]) for i, n in zip(ids, lengths)]]
        steps += [[Segment(i, [tokens[i][n + k]], n + k, [0]) for i, n in zip(ids, lengths)] for k in range(case["tail"])]
        return {"engine": engine, "steps": steps, "ending": ids}
    riders = _contexts(case)
    cached = [Segment(i, tokens[i][:n], 0, []) for i, n in zip(ids, riders)]
    step = [Segment(i, [tokens[i][n]], n, [0]) for i, n in zip(ids, riders)]
    if case["kind"] == "mixed":
        cached.append(Segment(ids[-1], tokens[-1][:case["rows"]], 0, []))
        step.insert(0, Segment(ids[-1], tokens[-1][case["rows"]:], case["rows"], []))
    engine.step(cached)
    return {"engine": engine, "steps": [step], "ending": []}


def run(state):
    engine = state["engine"]
    first = logits = engine.step(state["steps"][0])
    for segments in state["steps"][1:]:
        logits = engine.step(segments)
    for request in state["ending"]:
        engine.finish(request)
    return [first] if logits is first else [first, logits]


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Bytes: every step reads the layers' weights and the head once, its rows of the embedding, the keys and values (or
    states) of its requests, and writes its logits. Operations: two per weight and row, and the attention's two products."""
    cfg = config(case)
    size = 4 if case["dtype"] == "float32" else 2
    table = shapes(cfg)
    qwen = case["model"] == "qwen3"
    vocab, D = (cfg["vocab_size"], cfg["hidden_size"]) if qwen else (cfg["vocab"], cfg["width"])
    layers = sum(math.prod(s) for n, (s, _) in table.items() if "embed" not in n and "head" not in n)
    # per layer: (bytes a cached position has, products' operations per row and key it sees, keys it sees at most, state's bytes)
    runs = []
    if qwen:
        runs = [(2 * 8 * 128 * size, 4 * cfg["num_attention_heads"] * 128, 1 << 40, 0)] * case["layers"]
    else:
        for layer in cfg["layers"]:
            m = layer["mixer"]
            left = m.get("left", m)
            span = left.get("mask", {}).get("size", 1 << 40) if layer["type"] != "general_delta" else 0
            if case["model"] == "bozevik":
                row, ops = 2 * (m["kv_rank"] + m["rot_dim"]), 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            elif layer["type"] == "general_delta":
                row, ops = 0, 0
            else:
                maps = 2 if "diff" in m else 1
                row = 2 * left["kv_heads"] * (maps * left["dim"] + left["vdim"])
                ops = 2 * maps * left["heads"] * (left["dim"] + left["vdim"])
            r = m.get("right", m if layer["type"] == "general_delta" else None)
            state = 0 if r is None else 4 * r["heads"] * r.get("state", r.get("dim", 0)) * r.get("vdim", r.get("dim", 0))
            runs.append((row, ops, span, state))
    nbytes = flops = 0.0

    def step(segments, wanted):        # segments: (first position, rows)
        nonlocal nbytes, flops
        rows = sum(n for _, n in segments)
        nbytes += size * (layers + vocab * D) + rows * D * size + 4 * wanted * vocab
        flops += 2.0 * layers * rows + 2.0 * vocab * D * wanted
        for row, ops, span, state in runs:
            for start, n in segments:
                keys = min(start + n, span + n)
                nbytes += row * keys + (state * 2 if state else 0)
                flops += ops * sum(min(start + k + 1, span) for k in range(n)) + (state / 4) * 4.0 * n

    if case["kind"] == "prompt":
        lengths = _prompt_lengths(case)
        step([(0, n) for n in lengths], len(lengths))
        for k in range(case["tail"]):
            step([(n + k, 1) for n in lengths], len(lengths))
    else:
        segments = [(n, 1) for n in _contexts(case)]
        step(segments + ([(case["rows"], case["rows"])] if case["kind"] == "mixed" else []), len(segments))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 0.03, "max": 0.3}


# ---- the same logits in 64 bits -----------------------------------------------------------------------------------

class _Weights:
    """The random weights of a model, each made when it is asked for: every tensor has a generator of its own, seeded by the
    model's seed and the tensor's name, and is rounded to bfloat16 as the engine's random-weights mode rounds it."""

    def __init__(self, cfg, seed):
        self.table, self.seed, self.prefix = shapes(cfg), seed, ""

    def __getitem__(self, name):
        shape, init = self.table[self.prefix + name]
        digest = hashlib.sha256(f"{self.seed}:{self.prefix + name}".encode()).digest()
        g = torch.Generator(device=DEVICE).manual_seed(int.from_bytes(digest[:8], "little") & 0x7FFFFFFFFFFFFFFF)
        t = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32)
        if init == "average":
            t = (t * 0.1 + 1.0) / max(1, t.numel())
        else:
            t = t * 0.1 + 1.0 if init == "gain" else t * 0.02
        return t.to(torch.bfloat16).double()

    def under(self, prefix):
        w = object.__new__(_Weights)
        w.table, w.seed, w.prefix = self.table, self.seed, self.prefix + prefix
        return w

    def linear(self, x, name, chunk=16384):
        w = self[name]
        return torch.cat([part @ w.T for part in x.split(chunk)])


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _layer_norm(x, gain, eps):
    x = x - x.mean(dim=-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps) * gain


def _silu(z):
    return z * torch.sigmoid(z)


def _frequencies(rot):
    """(frequencies of a head's rotated pairs, amplitude): plain, divided, by wavelength bands, or stretched over a ramp."""
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not s:
        return f, 1.0
    factor = s["factor"]
    if "fast" in s:
        at = [dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base)) for turns in (s["fast"], s["slow"])]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
        return [x / factor * r + x * (1 - r) for x, r in zip(f, ramp)], 0.1 * math.log(factor) + 1.0
    if "original" not in s:
        return [x / factor for x in f], 1.0
    share = [min(max((s["original"] * x / (2 * math.pi) - s["low"]) / (s["high"] - s["low"]), 0.0), 1.0) for x in f]
    return [(1 - r) * x / factor + r * x for x, r in zip(f, share)], 1.0


def _rotate(x, rot, interleaved=False):
    """x [T, heads, dim]: the first rot.dims values of every head turned by the row's position."""
    if rot is None:
        return x
    f, amplitude = _frequencies(rot)
    angle = torch.arange(x.shape[0], device=DEVICE, dtype=torch.float64)[:, None, None] * torch.tensor(f, device=DEVICE, dtype=torch.float64)
    c, s = torch.cos(angle) * amplitude, torch.sin(angle) * amplitude
    out, half = x.clone(), len(f)
    a, b = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _attention(q, k, v, scale, *, window=0, keep=0, chunk=0, sink=None, last_only=False):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv], scale a number or [H] -> [T, H, dv]."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    scale = torch.as_tensor(scale, device=DEVICE, dtype=torch.float64).expand(H)
    out = torch.zeros(T, H, v.shape[2], dtype=torch.float64, device=DEVICE)
    block = max(128, min(T, (1 << 26) // max(1, T * per)))
    for lo in range(0, T, block):
        t = torch.arange(lo, min(T, lo + block), device=DEVICE)[:, None]
        j = torch.arange(int(t[-1]) + 1, device=DEVICE)[None, :]
        hidden = j > t
        if window:
            hidden |= (t - j >= window) & (j >= keep)
        if chunk:
            hidden |= j // chunk != t // chunk
        for g in range(k.shape[1]):
            heads = slice(g * per, (g + 1) * per)
            s = torch.einsum("thd,jd->htj", q[lo:lo + block, heads], k[:j.shape[1], g]) * scale[heads, None, None]
            s.masked_fill_(hidden, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[heads, None, None].expand(per, s.shape[1], 1)], dim=-1)
            s = torch.softmax(s, dim=-1)[..., :j.shape[1]]
            out[lo:lo + block, heads] = torch.einsum("htj,jd->thd", s, v[:j.shape[1], g])
    return out


def _qkv(w, h, m, maps=1, bias=False):
    T, H, G = h.shape[0], m["heads"], m["kv_heads"]
    q, k, v = (w.linear(h, n) + (w[n + ".b"] if bias else 0.0) for n in ("q", "k", "v"))
    return q.view(T, H, maps * m["dim"]), k.view(T, G, maps * m["dim"]), v.view(T, G, m["vdim"])


def _linear_attention(w, h, m, eps):
    T, H = h.shape[0], m["heads"]
    q, k, v = (_silu(w.linear(h, n)).view(T, H, -1) for n in ("q", "k", "v"))
    decay = torch.tensor(m["decay"], device=DEVICE, dtype=torch.float64)[:, None, None]
    S, o = torch.zeros(H, m["dim"], m["vdim"], dtype=torch.float64, device=DEVICE), torch.empty_like(v)
    for t in range(T):
        S = decay * S + k[t][:, :, None] * v[t][:, None, :]
        o[t] = (S * q[t][:, :, None]).sum(dim=1)
    return w.linear(_rms(o.reshape(T, -1), eps) * w["norm"] * torch.sigmoid(w.linear(h, "g")), "o")


def _state_space(w, h, m, eps):
    H, P, N, G, taps, parts = (m[k] for k in ("heads", "vdim", "state", "groups", "conv", "norm_groups"))
    T, inner = h.shape[0], H * P
    z, xbc, dt = w.linear(h, "in").split([inner, inner + 2 * G * N, H], dim=1)
    conv, padded = w["conv"], torch.cat([torch.zeros(taps - 1, xbc.shape[1], dtype=torch.float64, device=DEVICE), xbc])
    x, B, C = _silu(w["conv.b"] + sum(conv[:, r] * padded[r:r + T] for r in range(taps))).split([inner, G * N, G * N], dim=1)
    x = x.reshape(T, H, P)
    B, C = (y.reshape(T, G, 1, N).expand(T, G, H // G, N).reshape(T, H, N) for y in (B, C))
    dt = torch.nn.functional.softplus(dt + w["dt_bias"], threshold=50)
    keep = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, y = torch.zeros(H, N, P, dtype=torch.float64, device=DEVICE), torch.empty_like(x)
    for t in range(T):
        S = keep[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        y[t] = (S * C[t][:, :, None]).sum(dim=1)
    y = ((y + w["D"][:, None] * x).reshape(T, inner) * _silu(z)).view(T, parts, -1)
    return w.linear(_rms(y, eps).reshape(T, inner) * w["norm"], "o")


def _matrix_memory(w, h, m, eps):
    T, H, dk, dv, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = w.linear(h, "q").view(T, H, dk) / math.sqrt(dk), w.linear(h, "k").view(T, H, dk), w.linear(h, "v").view(T, H, dv)
    take, keep = (cap * torch.tanh((w.linear(h, n) + w[n + ".b"]) / cap) for n in ("i", "f"))
    keep = torch.nn.functional.logsigmoid(keep)
    S, n, top = (torch.zeros(*s, dtype=torch.float64, device=DEVICE) for s in ((H, dk, dv), (H, dk), (H,)))
    o = torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(keep[t] + top, take[t])
        a, b, top = torch.exp(keep[t] + top - new), torch.exp(take[t] - new), new
        S = a[:, None, None] * S + (b[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        n = a[:, None] * n + b[:, None] * k[t]
        by = torch.maximum((n * q[t]).sum(dim=1).abs(), torch.exp(-top)) + 1e-6
        o[t] = (S * q[t][:, :, None]).sum(dim=1) / by[:, None]
    return w.linear(_rms(o, eps).reshape(T, -1) * w["norm"] * torch.sigmoid(w.linear(h, "g")), "o")


def _delta(w, h, m, eps):
    T, H, n = h.shape[0], m["heads"], m["dim"]
    r, k, v = (w.linear(h, x).view(T, H, n) for x in ("r", "k", "v"))
    decay = torch.sigmoid(torch.tanh(w.linear(h, "w1")) @ w["w2"].T + w["w0"]).view(T, H, n)
    d, a = torch.exp(-math.exp(-0.5) * decay), torch.sigmoid(w.linear(h, "a") + w["a.b"]).view(T, H, n)
    u = k / torch.sqrt((k * k).sum(dim=-1, keepdim=True) + 1e-6)
    S, o = torch.zeros(H, n, n, dtype=torch.float64, device=DEVICE), torch.empty_like(v)
    for t in range(T):
        read = (S * u[t][:, :, None]).sum(dim=1)
        S = d[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * read[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
        o[t] = (S * r[t][:, :, None]).sum(dim=1)
    return w.linear(_rms(o, eps).reshape(T, -1) * w["norm"] * torch.sigmoid(w.linear(h, "g")), "o")


def _qwen3(cfg, w, rows):
    """Residual rows of all sequences behind the last layer and its norm; `rows`: one [T, width] tensor per sequence."""
    eps, H, G, hd = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    counts, x, rot = [len(r) for r in rows], torch.cat(rows), {"dims": hd, "base": cfg["rope_theta"]}
    for i in range(cfg["num_hidden_layers"]):
        l = w.under(f"model.layers.{i}.")
        h = _rms(x, eps) * l["input_layernorm.weight"]
        qkv, gq, gk = [], l["self_attn.q_norm.weight"], l["self_attn.k_norm.weight"]
        for n in ("q_proj", "k_proj", "v_proj"):
            qkv.append(l.linear(h, f"self_attn.{n}.weight").split(counts))
        out = []
        for q, k, v in zip(*qkv):
            q, k = _rms(q.view(-1, H, hd), eps) * gq, _rms(k.view(-1, G, hd), eps) * gk
            out.append(_attention(_rotate(q, rot), _rotate(k, rot), v.view(-1, G, hd), hd ** -0.5).reshape(len(q), -1))
        x = x + l.linear(torch.cat(out), "self_attn.o_proj.weight")
        del h, qkv, out
        gain, gate, up, down = (l[n] for n in ("post_attention_layernorm.weight", "mlp.gate_proj.weight", "mlp.up_proj.weight",
                                               "mlp.down_proj.weight"))
        for part in x.split(8192):
            h = _rms(part, eps) * gain
            part += (_silu(h @ gate.T) * (h @ up.T)) @ down.T
    return [(_rms(r, eps) * w["model.norm.weight"]) for r in x.split(counts)]


def _bozevik(cfg, w, x):
    eps, cached, results = cfg["norm"]["eps"], {}, [x]
    for i, layer in enumerate(cfg["layers"]):
        l, m, T = w.under(f"l{i}."), layer["mixer"], x.shape[0]
        mix, H, dk, R = l.under("mix."), m["heads"], m["dim"], m["kv_rank"]
        h = x + (torch.cat([torch.zeros_like(x[:1]), x[:-1]]) - x) * l["shift"]
        if "kv_from" not in m:
            d = mix.linear(h, "dkv")
            cached[i] = _rms(d[:, :R], eps) * mix["dkv.norm"], _rotate(d[:, None, R:], m["rot"], interleaved=True)
        c, r = cached[m.get("kv_from", i)]
        q = mix.linear(_rms(mix.linear(h, "dq"), eps) * mix["dq.norm"], "uq").view(T, H, -1)
        q = torch.cat([q[..., :dk], _rotate(q[..., dk:], m["rot"], interleaved=True)], dim=-1)
        k = torch.cat([mix.linear(c, "uk").view(T, H, dk), r.expand(T, H, -1)], dim=-1)
        o = _attention(q, k, mix.linear(c, "uv").view(T, H, -1), m["scale"])
        x = x + _layer_norm(mix.linear(o.reshape(T, -1), "o"), l["norm1"], eps)
        f, limit = l.under("mlp."), layer["mlp"]["limit"]
        g, u = f.linear(x, "gate").clamp(max=limit), f.linear(x, "up").clamp(-limit, limit)
        x = x + _layer_norm(f.linear(g * torch.sigmoid(1.702 * g) * (u + 1), "down"), l["norm2"], eps)
        results.append(x)
        x = sum(share * row for share, row in zip(l["dwa"], results))
    return _layer_norm(x, w["final.norm"], eps)


def _movivik(cfg, w, x):
    eps = cfg["norm"]["eps"]

    def grouped(w, h, m, bias, interleaved, unit):
        q, k, v = _qkv(w, h, m, bias=bias)
        q, k = (_rotate(y, m["rot"], interleaved) for y in (q, k))
        if unit:
            q, k = _rms(q, eps), _rms(k, eps)
        o = _attention(q, k, v, m["scale"], chunk=m.get("mask", {}).get("size", 0)) * torch.sigmoid(w.linear(h, "g"))[:, :, None]
        return w.linear(o.reshape(len(h), -1), "o")

    for i, layer in enumerate(cfg["layers"]):
        l, m = w.under(f"l{i}."), layer["mixer"]
        mix, h = l.under("mix."), _rms(x, eps) * l["norm1"]
        if layer["type"] == "attention":
            y = grouped(mix, h, m, True, True, False)
        else:
            left, right = grouped(mix.under("left."), h, m["left"], False, False, True), _linear_attention(mix.under("right."), h, m["right"], eps)
            y = 0.5 * (_rms(left, eps) * mix["left.out"] + _rms(right, eps) * mix["right.out"])
        x = x + _rms(y, eps) * l["norm1b"]
        h, f = _rms(x, eps) * l["norm2"], l.under("mlp.")
        y = f.linear(torch.nn.functional.gelu(f.linear(h, "gate"), approximate="tanh") * f.linear(h, "up"), "down")
        x = x + _rms(y, eps) * l["norm2b"]
    return _rms(x, eps) * w["final.norm"]


def _guvolix(cfg, w, x):
    eps = cfg["norm"]["eps"]
    x = x * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        l, m = w.under(f"l{i}."), layer["mixer"]
        mix, h, a = l.under("mix."), _rms(x, eps) * l["norm1"], m["left"]
        wl, (q, k, v) = mix.under("left."), _qkv(mix.under("left."), h, a)
        o = _attention(_rotate(q, a["rot"]), _rotate(k, a["rot"]), v, a["scale"], window=a["mask"]["size"],
                       keep=a["mask"].get("keep_first", 0), sink=wl["sink"])
        left = wl.linear(o.reshape(len(x), -1) * torch.sigmoid(wl.linear(h, "g")), "o")
        if layer["type"] == "parallel":
            right = _state_space(mix.under("right."), h, m["right"], eps)
            y = 0.5 * (_rms(left, eps) * mix["left.out"] + _rms(right, eps) * mix["right.out"])
        else:
            y = m["left_scale"] * left + m["right_scale"] * _matrix_memory(mix.under("right."), h, m["right"], eps)
        f = l.under("mlp.")
        x = x + y + f.linear(torch.nn.functional.gelu(f.linear(h, "up")), "down")
    return _rms(x, eps) * w["final.norm"]


def _fusazen(cfg, w, x):
    eps, taps, kept = cfg["norm"]["eps"], cfg["canon"]["taps"], {}
    x = x * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        l, m, T = w.under(f"l{i}."), layer["mixer"], x.shape[0]
        mix, h, conv = l.under("mix."), _rms(x, eps) * l["norm1"], l["canon1"]
        padded = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=torch.float64, device=DEVICE), h])
        h = h + sum(conv[:, j] * padded[j:j + T] for j in range(taps))
        if layer["type"] == "general_delta":
            y = _delta(mix, h, m, eps)
        elif layer["type"] == "attention_2":
            T, H, G = len(h), m["heads"], m["kv_heads"]
            q, k = (_rms(mix.linear(h, n), eps) * mix[n + ".norm"] for n in ("q", "k"))
            o = _attention(q.view(T, H, -1), k.view(T, G, -1), mix.linear(h, "v").view(T, G, -1), m["scale"] * mix["temp"],
                           chunk=m["mask"]["size"])
            y = mix.linear(o.reshape(T, -1), "o")
        else:
            H, G, dk, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
            if "kv_from" not in m:
                k = mix.linear(h, "k").view(T, G, 2, dk)
                kept[i] = [_rotate(k[:, :, a], rot) for a in (0, 1)], mix.linear(h, "v").view(T, G, -1)
            keys, v = kept[m.get("kv_from", i)]
            q = mix.linear(h, "q").view(T, H, 2, dk)
            a1, a2 = (_attention(_rotate(q[:, :, a], rot), keys[a], v, m["scale"], chunk=m["mask"]["size"]) for a in (0, 1))
            share = torch.exp((mix["lq1"] * mix["lk1"]).sum()) - torch.exp((mix["lq2"] * mix["lk2"]).sum()) + m["diff"]
            y = mix.linear((_rms(a1 - share * a2, eps) * (1 - m["diff"])).reshape(T, -1), "o")
        x = x + y
        f = l.under("mlp.")
        x = x + f.linear(torch.relu(f.linear(_rms(x, eps) * l["norm2"], "up") + f["up.b"]) ** 2, "down") + f["down.b"]
    return _rms(x, eps) * w["final.norm"]


def exact(case, seed):
    cfg, tokens = config(case), _tokens(case, seed)
    w = _Weights(cfg, seed)
    qwen = case["model"] == "qwen3"
    if case["kind"] == "prompt":
        places = [[n - 1 for n in _prompt_lengths(case)]] + ([[-1] * len(tokens)] if case["tail"] else [])
    else:
        tokens = tokens[:case["requests"]]        # (the long prompt's portion of a mixed step asks for no logits)
        places = [[-1] * len(tokens)]
    embed = w["model.embed_tokens.weight" if qwen else "embed"]
    rows = [embed[torch.tensor(t, device=DEVICE)] for t in tokens]
    if qwen:
        rows = _qwen3(cfg, w, rows)
    else:
        layers = {"movivik": _movivik, "guvolix": _guvolix, "bozevik": _bozevik, "fusazen": _fusazen}[case["model"]]
        rows = [layers(cfg, w, r) for r in rows]
    head = w["lm_head.weight"] if qwen else embed if case["model"] == "bozevik" else w["head"]
    return [torch.stack([r[at] for r, at in zip(rows, ats)]) @ head.T for ats in places]
