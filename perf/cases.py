"""What a user has this framework do, as cases that can be timed and compared.

Three designs are served: the integer-only W8A8 Qwen3 form, Sefevik (gated recurrences and latent attention) and Derelorn
(matrix memories, and windowed attention beside a state-space memory).  A user either feeds prompts or decodes one token for
every running request, so a case is one step of one of these on one batch:

    design   "integer": ``Qwen3ForCausalLMInteger`` over the int8 page pool; decode steps in a CUDA graph with ``DecodeBatch``
             "sefevik", "derelorn": ``Engine.open / step / close`` with token ids from the host, then the greedy arg-max
    size     layer shapes of the benchmark's models; the integer ones at full depth, the others as two repetitions of their pattern
             of layers: what 16-bit rounding does to random layers grows with depth until outputs cannot be compared
    dtype    "int8", "bfloat16" or "float32"
    phase    "prefill": ``requests`` new prompts in one step;  "decode": one token for each of ``requests`` requests
    low, high   prompt lengths, or tokens that the requests hold already; spread evenly over the range in a shuffled order

Weights, caches and states are random and made from the seed; the lengths follow from the case alone.  What is compared are the
logits and what the step leaves behind (keys and values, states); the integer design's logits and tokens are the same bit for
bit.  The floating-point designs' arg-max is taken, but not compared: two logits that lie close together may change places.
"""
from __future__ import annotations

import math
import random

import torch

import mini_sgl_integer_b200  # noqa: F401  (fails here, and not in the middle of a measurement, if the package is missing)

DEV = "cuda"
PAGE = 16

INTEGER = {      # layers, hidden, query heads, KV heads, intermediate, vocabulary
    "8B": dict(layers=36, hidden=4096, heads=32, kv=8, inter=12288, vocab=151936),
    "1.4B": dict(layers=24, hidden=2048, heads=16, kv=4, inter=6400, vocab=32768),
}
SEFEVIK = {      # (gru, gru, attention, gru, gru, attention on the cache of the one before) repeated
    "0.3B": dict(width=1024, depth=12, gru=1536, ff=4096, heads=16, dim=64, rot=32, vdim=64, rank=256, window=512, vocab=32768),
    "1.4B": dict(width=2048, depth=12, gru=3072, ff=8192, heads=16, dim=128, rot=64, vdim=128, rank=512, window=1024, vocab=32768),
    "4B": dict(width=4096, depth=12, gru=6144, ff=16384, heads=32, dim=128, rot=64, vdim=128, rank=512, window=1024, vocab=65536),
}
DERELORN = {     # (mlstm, parallel, mlstm, delta) repeated; heads and sizes of each mixer
    "0.3B": dict(width=1024, depth=8, ff=2816, vocab=32768, mlstm=(4, 128, 256), attn=(16, 4, 64, 512), mamba=(32, 64, 64, 1), delta=(8, 4, 128, 128)),
    "1.4B": dict(width=2048, depth=8, ff=5632, vocab=32768, mlstm=(8, 128, 256), attn=(16, 4, 128, 1024), mamba=(64, 64, 128, 1), delta=(16, 8, 128, 128)),
    "4B": dict(width=4096, depth=8, ff=11264, vocab=65536, mlstm=(16, 128, 256), attn=(32, 8, 128, 1024), mamba=(128, 64, 128, 1), delta=(32, 16, 128, 128)),
}
TAPS = 4         # of the short convolutions


def _case(name, design, size, dtype, phase, requests, low, high):
    c = dict(design=design, size=size, dtype=dtype, phase=phase, requests=requests, low=low, high=high)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user talking to the model: nothing but latency, every launch counts
        _case("integer-8b-decode-1", "integer", "8B", "int8", "decode", 1, 777, 777),
        # a small model under light load, odd batch
        _case("integer-1.4b-decode-37", "integer", "1.4B", "int8", "decode", 37, 50, 900),
        # the benchmark's headline: a full decode batch with contexts U[100, 2048]
        _case("integer-8b-decode-256", "integer", "8B", "int8", "decode", 256, 100, 2048),
        # the first token of a short question
        _case("integer-8b-prompt-1", "integer", "8B", "int8", "prefill", 1, 333, 333),
        # a server's prefill step: prompts of unequal length, about 8 k tokens together
        _case("integer-8b-prefill-15", "integer", "8B", "int8", "prefill", 15, 100, 1000),
        _case("sefevik-0.3b-decode-1", "sefevik", "0.3B", "bfloat16", "decode", 1, 450, 450),
        _case("sefevik-1.4b-decode-256", "sefevik", "1.4B", "bfloat16", "decode", 256, 100, 2048),
        _case("sefevik-1.4b-prefill-13", "sefevik", "1.4B", "bfloat16", "prefill", 13, 200, 1060),
        # the 32-bit form, which users hold the bf16 one against
        _case("sefevik-0.3b-f32-prefill-5", "sefevik", "0.3B", "float32", "prefill", 5, 60, 500),
        _case("derelorn-1.4b-decode-64", "derelorn", "1.4B", "bfloat16", "decode", 64, 100, 2048),
        # few long documents: longer than the attention window, little parallelism over requests
        _case("derelorn-1.4b-prefill-3", "derelorn", "1.4B", "bfloat16", "prefill", 3, 1500, 3500),
        _case("derelorn-0.3b-prompt-1", "derelorn", "0.3B", "bfloat16", "prefill", 1, 210, 210),
    ]


def draw(rng):
    """Another case of the same ranges: any design, 1 to 256 decoding requests with up to 2048 tokens, prompts of 8 to 3500
    tokens and at most 8192 together."""
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    design = rng.choice(["integer", "integer", "sefevik", "derelorn"])
    dtype = "int8" if design == "integer" else rng.choice(["bfloat16"] * 5 + ["float32"])
    size = rng.choice(["8B", "1.4B"] if design == "integer" else ["0.3B"] if dtype == "float32" else ["0.3B", "1.4B", "4B"])
    if rng.random() < 0.5:
        requests = log(1, 256)
        low = rng.randint(20, 1000)
        return _case(None, design, size, dtype, "decode", requests, low, rng.randint(low, 2048))
    total = log(32, 8192 if dtype != "float32" else 2048)
    requests = min(log(1, 24), total // 8)
    mean = total // requests
    if mean > 2300:
        requests, mean = 3, min(mean, total // 3)
    low = max(8, int(mean * rng.uniform(0.3, 1.0)))
    return _case(None, design, size, dtype, "prefill", requests, low, max(low, min(3500, 2 * mean - low)))


def lengths(case):
    """Of the prompts, or of what the requests hold already."""
    n, low, high = case["requests"], case["low"], case["high"]
    got = [low + (high - low) * i // max(1, n - 1) for i in range(n)] if n > 1 else [(low + high) // 2]
    random.Random(1000003 * n + high).shuffle(got)
    return got


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


# ----------------------------------------------------------------------------- configurations
def sefevik_config(s):
    layers = []
    for i in range(s["depth"]):
        mlp = {"kind": "dense", "ff": s["ff"]}
        if i % 3 != 2:
            layers.append({"type": "mingru", "mixer": {"width": s["gru"]}, "mlp": mlp})
            continue
        m = {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot"], "vdim": s["vdim"], "kv_rank": s["rank"],
             "scale": (s["dim"] + s["rot"]) ** -0.5, "mask": {"size": s["window"]},
             "rot": {"dims": s["rot"], "base": 1e6, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        if i % 6 == 5:
            m["kv_from"] = i - 3
        layers.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
    return {"architecture": "Sefevik", "vocab": s["vocab"], "width": s["width"], "norm": {"eps": 1e-6}, "layers": layers,
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 1_000_003, "mul_cur": 8191}}}


def derelorn_config(s):
    layers = []
    for i in range(s["depth"]):
        kind = ("mlstm", "parallel", "mlstm", "delta")[i % 4]
        if kind == "mlstm":
            m = dict(zip(("heads", "dim", "vdim"), s["mlstm"]), gate_cap=15.0)
        elif kind == "delta":
            m = dict(zip(("heads", "kv_heads", "dim", "vdim"), s["delta"]), conv=TAPS)
        else:
            h, g, d, w = s["attn"]
            mh, v, n, groups = s["mamba"]
            m = {"left": {"heads": h, "kv_heads": g, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": w}},
                 "right": {"heads": mh, "vdim": v, "state": n, "groups": groups, "conv": TAPS, "norm_groups": 1}}
        layers.append({"type": kind, "mixer": m, "mlp": {"kind": "dense", "ff": s["ff"]}})
    return {"architecture": "Derelorn", "vocab": s["vocab"], "width": s["width"], "norm": {"eps": 1e-6}, "layers": layers}


def _size(case):
    return {"integer": INTEGER, "sefevik": SEFEVIK, "derelorn": DERELORN}[case["design"]][case["size"]]


def _config(case):
    return sefevik_config(_size(case)) if case["design"] == "sefevik" else derelorn_config(_size(case))


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _weights(case, config, seed):
    """A random checkpoint under the names that the loader expects."""
    if case["design"] == "sefevik":
        from mini_sgl_integer_b200.models.config import SefevikConfig as Config
        from mini_sgl_integer_b200.models.sefevik import random_weights
    else:
        from mini_sgl_integer_b200.models.config import DerelornConfig as Config
        from mini_sgl_integer_b200.models.derelorn import random_weights
    return random_weights(Config.from_dict(config), seed, device=DEV, dtype=_dtype(case))


def _window(case):
    s = _size(case)
    return s["window"] if case["design"] == "sefevik" else s["attn"][3]


# ----------------------------------------------------------------------------- what requests hold when a decode step begins
def _held(case):
    """(first position whose keys are still kept, tokens held) of every request."""
    return [(max(0, n - _window(case)), n) for n in lengths(case)]


def _max_tokens(case):
    """That an engine has to hold: requests keep what lies in the window, in pages that may be partly empty."""
    if case["phase"] == "prefill":
        return sum(lengths(case))
    return max(max(lengths(case)) + 32, sum(b - a + 2 * PAGE for a, b in _held(case)))


def _token_ids(case, seed):
    """Prompts, or the next token of every request."""
    vocab = _size(case)["vocab"]
    counts = lengths(case) if case["phase"] == "prefill" else [1] * case["requests"]
    return torch.randint(0, vocab, (sum(counts),), device=DEV, generator=_generator(seed + 1)).split(counts)


def _memories(config):
    """(layer, planes [widths of the rows that it keeps per token], states [(name, shape)]) in the layers' order."""
    for i, l in enumerate(config["layers"]):
        m = l["mixer"]
        if l["type"] == "mingru":
            yield i, [], [("s", (m["width"],))]
        elif l["type"] == "latent_attention":
            yield i, [] if "kv_from" in m else [m["kv_rank"] + m["rot_dim"]], []
        elif l["type"] == "mlstm":
            yield i, [], [("S", (m["heads"], m["dim"], m["vdim"])), ("n", (m["heads"], m["dim"] + 1))]
        elif l["type"] == "delta":
            yield i, [], [("S", (m["heads"], m["dim"], m["vdim"])), ("conv", (TAPS - 1, 2 * m["kv_heads"] * m["dim"] + m["heads"] * m["vdim"]))]
        else:
            a, b = m["left"], m["right"]
            inner = b["heads"] * b["vdim"]
            yield i, [a["kv_heads"] * a["dim"], a["kv_heads"] * a["vdim"]], \
                [("S", (b["heads"], b["state"], b["vdim"])), ("conv", (TAPS - 1, inner + 2 * b["groups"] * b["state"]))]


def _memory(case, config, seed):
    """({layer: rows kept per token, of all requests one after the other}, {(layer, name): state}, last tokens) at the start
    of a decode step."""
    g, dtype = _generator(seed + 2), _dtype(case)
    count, kept = case["requests"], sum(n - first for first, n in _held(case))
    rows, states, kinds = {}, {}, [l["type"] for l in config["layers"]]
    for i, planes, state in _memories(config):
        if planes:
            rows[i] = [torch.randn((kept, w), device=DEV, generator=g, dtype=dtype) for w in planes]
        for name, shape in state:
            v = torch.randn((count, *shape), device=DEV, generator=g)
            if name == "n":
                v[..., -1].abs_()                      # the running maximum of the exponents starts at 0
            # what some tens of written tokens leave behind
            states[i, name] = v.mul_({"mlstm": 2.0, "delta": 0.5, "parallel": 0.2}[kinds[i]]) if name in ("S", "n") else v
    last = torch.randint(0, config["vocab"], (count,), device=DEV, generator=g).to(torch.int32)
    return rows, states, last


# ----------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    return _prepare_integer(case, seed) if case["design"] == "integer" else _prepare_engine(case, seed)


def run(state):
    return state["run"]()


def _prepare_engine(case, seed):
    from mini_sgl_integer_b200.engine import Engine
    from mini_sgl_integer_b200.engine.sample import greedy
    config = _config(case)
    n = lengths(case)
    decode = case["phase"] == "decode"
    tokens = [t.tolist() for t in _token_ids(case, seed)]
    engine = Engine(config=config, weights=_weights(case, config, seed), dtype=case["dtype"], max_tokens=_max_tokens(case), max_reqs=len(n),
                    max_len=max(n) + 32, max_portion=8192)
    # (the last page and the last state are the engine's own, for the padding of decode batches)
    planes = [plane(i)[:-1] for i, p, _ in _memories(config) for plane in (engine.cache.k_cache, engine.cache.v_cache)[:len(p)]]
    states = [engine.cache.state(i, name)[:len(n)] for i, _, s in _memories(config) for name, _ in s]
    if not decode:
        def prompts():
            reqs = [engine.open() for _ in tokens]
            logits = engine.step(reqs, tokens)
            greedy(logits)
            for r in reversed(reqs):
                engine.close(r)
            return {"logits": logits, "planes": planes, "states": states}
        return {"run": prompts}

    reqs = [engine.open() for _ in tokens]
    for r, (first, last) in zip(reqs, _held(case)):
        engine.manager.extend(r.table_idx, first, last + 1)

    def step():
        for r, k in zip(reqs, n):                      # the same step each time: contexts keep their length
            r.cached_len = r.device_len = k
        logits = engine.step(reqs, tokens)
        greedy(logits)
        return {"logits": logits, "planes": planes, "states": states}

    def fill():
        rows, values, last = _memory(case, config, seed)
        at = [engine.manager.locations(torch.full((b - a,), r.table_idx), torch.arange(a, b)) for r, (a, b) in zip(reqs, _held(case))]
        at = torch.cat(at).to(DEV)
        for i, p in rows.items():
            engine.cache.store_kv(p[0], p[-1], at, i)
        for (i, name), v in values.items():
            engine.cache.state(i, name)[:len(n)].copy_(v)
        engine.cache.prev_tokens[:len(n)].copy_(last)
    step()                                             # a program that decodes has captured its step
    fill()
    return {"run": step}


def _prepare_integer(case, seed):
    from mini_sgl_integer_b200.attention import Int8PagedKVCache
    from mini_sgl_integer_b200.engine.sample import greedy
    from mini_sgl_integer_b200.layers.decoder_layer import AttnBatch
    from mini_sgl_integer_b200.models import DecodeBatch, Qwen3ForCausalLMInteger, Qwen3IntegerConfig, random_weights
    s, n = _size(case), lengths(case)
    decode = case["phase"] == "decode"
    ids = torch.cat(_token_ids(case, seed)).to(torch.int32)
    cfg = Qwen3IntegerConfig(s["layers"], s["hidden"], s["heads"], s["kv"], s["inter"], s["vocab"], max_pos=4096)
    pages = [(k + int(decode) + PAGE - 1) // PAGE for k in n]
    pool = Int8PagedKVCache(s["kv"], s["layers"], 128, sum(pages), DEV)
    order = torch.randperm(sum(pages), device=DEV, generator=_generator(seed + 3)).to(torch.int32)
    table = torch.zeros((len(n), max(pages)), dtype=torch.int32, device=DEV)
    for row, p in zip(table, order.split(pages)):
        row[:len(p)] = p
    model = Qwen3ForCausalLMInteger(cfg, random_weights(cfg, seed, device=DEV, generate_on_device=True), pool)
    lens = torch.tensor(n, dtype=torch.int32, device=DEV)
    if not decode:
        seq = torch.repeat_interleave(torch.arange(len(n)), torch.tensor(n)).to(DEV)
        pos = torch.cat([torch.arange(k) for k in n]).to(DEV)
        loc = table[seq, pos // PAGE] * PAGE + pos % PAGE
        batch = AttnBatch(pos.to(torch.int32), loc.to(torch.int32), table, lens, lens, max(n))
        last = lens.cumsum(0) - 1

        def prompts():
            logits = model.forward(ids, batch, last)
            return {"logits": logits, "tokens": greedy(logits)}
        return {"run": prompts}

    g = _generator(seed + 2)
    for i in range(s["layers"]):                       # keys and values that earlier steps have left
        for codes in (pool.k_cache(i), pool.v_cache(i)):
            codes.copy_(torch.randint(-127, 128, codes.shape, dtype=torch.int8, device=DEV, generator=g))
        meta = pool.meta(i)
        scales = lambda lo, hi: torch.randint(lo, hi, (*meta.shape[:2], 16), dtype=torch.int8, device=DEV, generator=g).view(torch.int32)
        meta[:, :, :32] = torch.randint(2**30, 2**31 - 1, (*meta.shape[:2], 32), dtype=torch.int32, device=DEV, generator=g)
        meta[:, :, 32:36], meta[:, :, 36:40] = scales(35, 39), scales(36, 40)
    batch = DecodeBatch(table, lens, -(-(max(n) + 1) // PAGE) * PAGE, first_wave_rows=max(1, 296 // s["kv"]))

    def step():
        batch.seq_lens.copy_(lens)                     # the same step each time: contexts keep their length
        logits = model.forward(ids, batch.advance())
        return {"logits": logits, "tokens": greedy(logits)}
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()

    def replay():
        graph.replay()
        return out
    return {"run": replay, "keep": (model, batch, ids, lens)}


# ----------------------------------------------------------------------------- what a step cannot do without
def work(case):
    """Weights, states and the keys in reach read once; states, new keys and logits written; products counted as two."""
    s, n = _size(case), lengths(case)
    decode = case["phase"] == "decode"
    T = len(n) if decode else sum(n)
    pairs = lambda w: sum(min(k + 1, w) for k in n) if decode else sum(min(k, w) * (min(k, w) + 1) / 2 + max(0, k - w) * w for k in n)
    if case["design"] == "integer":
        h, kv, W = s["heads"] * 128, s["kv"] * 128, s["hidden"]
        per = W * (h + 2 * kv) + h * W + 3 * W * s["inter"]
        keys = (sum(n) + T if decode else T) * s["kv"] * 266 * s["layers"]
        return {"bytes": s["layers"] * per + s["vocab"] * W + keys + T * 2 * W + 4 * len(n) * s["vocab"],
                "flops": 2 * T * s["layers"] * per + 2 * len(n) * s["vocab"] * W + 4 * pairs(1 << 30) * h * s["layers"]}
    size, W = 4 if case["dtype"] == "float32" else 2, s["width"]
    rows = sum(min(k, _window(case)) for k in n) + T if decode else T
    weights = flops = moved = 0
    for i, planes, states in _memories(_config(case)):
        moved += rows * sum(planes) * size + (2 if decode else 1) * len(n) * 4 * sum(math.prod(shape) for _, shape in states)
    for l in _config(case)["layers"]:
        m = l["mixer"]
        weights += (2 if case["design"] == "sefevik" else 3) * W * l["mlp"]["ff"]
        if l["type"] == "mingru":
            weights += 4 * W * m["width"]
        elif l["type"] == "latent_attention":
            lat = m["kv_rank"] + m["rot_dim"]
            weights += W * m["heads"] * (m["dim"] + m["rot_dim"]) + (0 if "kv_from" in m else W * lat)
            weights += m["heads"] * (m["dim"] + m["vdim"]) * m["kv_rank"] + m["heads"] * m["vdim"] * W
            flops += 2 * pairs(s["window"]) * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif l["type"] == "parallel":
            a, b = m["left"], m["right"]
            weights += W * a["dim"] * (a["heads"] + 2 * a["kv_heads"]) + a["heads"] * a["vdim"] * W
            inner = b["heads"] * b["vdim"]
            weights += W * (2 * inner + 2 * b["groups"] * b["state"] + b["heads"]) + inner * W
            flops += 4 * pairs(s["attn"][3]) * a["heads"] * a["dim"] + 4 * T * b["heads"] * b["state"] * b["vdim"]
        else:
            qk, v = m.get("kv_heads", m["heads"]) * m["dim"], m["heads"] * m["vdim"]
            weights += W * (2 * qk + 2 * v + 2 * m["heads"]) + v * W
            flops += (4 if l["type"] == "mlstm" else 6) * T * m["heads"] * m["dim"] * m["vdim"]
    head = s["vocab"] * W
    return {"bytes": size * (weights + head + T * W) + moved + 4 * len(n) * s["vocab"], "flops": 2 * T * weights + 2 * len(n) * head + flops}


def tolerance(case):
    """Integers are exact.  Floating point: what another order of the sums, followed by the rounding of every intermediate
    result to the model's dtype over all its layers, was seen to change, times four."""
    if case["design"] == "integer":
        return "exact"
    return {"rel": 4e-5, "max": 2e-3, "differ": 0.0} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.9, "differ": 0.01}


# ----------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """The outputs of ``run`` from plain 64-bit arithmetic; the integer design's are whole numbers and have no such form."""
    if case["design"] == "integer":
        return None
    config = _config(case)
    return _Exact(case, config, _weights(case, config, seed), seed).outputs()


def _norm(x, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


class _Exact:
    def __init__(self, case, config, weights, seed):
        self.w, self.config, self.case = weights, config, case
        self.decode = case["phase"] == "decode"
        n = lengths(case)
        self.new = [1] * len(n) if self.decode else n
        self.old = n if self.decode else [0] * len(n)
        self.kept = [b - a for a, b in _held(case)] if self.decode else [0] * len(n)
        self.ids = _token_ids(case, seed)
        self.rows, self.states, self.last = _memory(case, config, seed) if self.decode else ({}, {}, None)
        self.pos = torch.cat([torch.arange(o, o + k, device=DEV) for o, k in zip(self.old, self.new)])
        # tokens as [request, step], longest request first, so that those still running are the first ones
        self.order = sorted(range(len(n)), key=lambda i: -self.new[i])
        self.keys = {}

    def W(self, name):
        return self.w[name].double()

    def linear(self, x, name):
        return x @ self.W(name).T

    def outputs(self):
        x = torch.cat([self.w["embed"][t] for t in self.ids]).double()
        x = self.sefevik(x) if self.case["design"] == "sefevik" else self.derelorn(x)
        ends = torch.tensor(self.new, device=DEV).cumsum(0) - 1
        logits = self.linear(_norm(x[ends]) * self.W("final.norm"), "head")
        planes, states = [], []
        for i, p, s in _memories(self.config):
            planes += [self.paged(i, k) for k in range(len(p))]
            states += [self.states[i, name] for name, _ in s]
        return {"logits": logits, "planes": planes, "states": states}

    # ---- rows per token, as the engine pages them: requests one after the other, each from the page of its first kept row on
    def paged(self, i, k):
        firsts = [a for a, _ in _held(self.case)] if self.decode else [0] * len(self.new)
        counts = [(o + n - 1) // PAGE - f // PAGE + 1 for f, o, n in zip(firsts, self.old, self.new)]
        held = sum(b - a + 2 * PAGE for a, b in _held(self.case)) if self.decode else sum(self.new)
        out = torch.zeros((-(-held // PAGE) + len(self.new)) * PAGE, self.keys[i][k].shape[1], device=DEV, dtype=torch.float64)
        base = 0
        for f, c, rows in zip(firsts, counts, self.keys[i][k].split([a + b for a, b in zip(self.kept, self.new)])):
            out[base * PAGE + f % PAGE:][:len(rows)] = rows
            base += c
        return out.view(-1, PAGE, out.shape[1])

    def with_kept(self, i, k, new):
        """Rows kept from earlier steps and the new ones, request by request."""
        if not self.decode:
            return new
        old = self.rows[i][k].double().split(self.kept)
        return torch.cat([t for pair in zip(old, new.split(self.new)) for t in pair])

    def attend(self, q, k, v, window, scale, sink=None):
        """q [T, H, d]; k [rows, G, d], v [rows, G, e] of all requests; [T, H, e]."""
        H, G, out = q.shape[1], k.shape[1], []
        counts = [a + b for a, b in zip(self.kept, self.new)]
        for qs, ks, vs, n in zip(q.split(self.new), k.split(counts), v.split(counts), self.new):
            m = len(ks)
            s = torch.einsum("tghd,sgd->ghts", qs.view(n, G, H // G, -1), ks) * scale
            at, key = torch.arange(m - n, m, device=DEV)[:, None], torch.arange(m, device=DEV)[None, :]
            s = s.masked_fill((key > at) | (at - key >= window), -math.inf)
            if sink is not None:
                s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(-1, -1, n, 1)], dim=-1)
            p = torch.softmax(s, -1)[..., :m]
            out.append(torch.einsum("ghts,sge->tghe", p, vs).reshape(n, H, -1))
        return torch.cat(out)

    # ---- steps of all requests at once
    def padded(self, x):
        parts = x.split(self.new)
        return torch.nn.utils.rnn.pad_sequence([parts[i] for i in self.order], batch_first=True)

    def unpadded(self, y):
        back = {i: y[k, :self.new[i]] for k, i in enumerate(self.order)}
        return torch.cat([back[i] for i in range(len(self.new))])

    def running(self):
        for t in range(max(self.new)):
            yield t, sum(n > t for n in self.new)

    def state(self, i, name, shape):
        if self.decode:
            return self.states[i, name].double()[self.order]
        return torch.zeros((len(self.new), *shape), device=DEV, dtype=torch.float64)

    def keep(self, i, name, value):
        out = torch.empty_like(value)
        out[self.order] = value
        self.states[i, name] = out

    # ---- Sefevik
    def sefevik(self, x):
        big, dt = self.config["embedding"]["bigram"], self.w["embed"].dtype
        rows = []
        for k, t in enumerate(self.ids):
            prev = torch.cat([self.last[k:k + 1].long() if self.decode else t[:1], t[:-1]])
            r = (prev * big["mul_prev"] + t * big["mul_cur"]) % big["buckets"]
            if not self.decode:
                r[0] = big["buckets"]
            rows.append(r)
        x = x + self.w["bigram"][torch.cat(rows)].double()
        history = [x]
        for i, layer in enumerate(self.config["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            y = self.mingru(x, i, m, p + "mix.") if layer["type"] == "mingru" else self.latent(x, i, m, p + "mix.")
            x = x + _norm(y) * self.W(p + "norm1")
            a, b = torch.nn.functional.softplus(self.W(p + "mlp.act")).tolist()
            z = self.linear(x, p + "mlp.up")
            low = z.clamp(max=0)
            z = torch.where(z > 0, a * z * z + 0.5 * z, (0.5 + b) * (torch.expm1(low) - low) + 0.5 * z)
            x = x + _norm(self.linear(z, p + "mlp.down")) * self.W(p + "norm2")
            history.append(x)
            x = sum(c * h for c, h in zip(self.W(p + "dwa").tolist(), history))
        return x

    def mingru(self, x, i, m, p):
        z = torch.sigmoid(self.linear(x, p + "z") + self.W(p + "z.b"))
        u = self.linear(x, p + "x") + self.W(p + "x.b")
        write, keep = self.padded(z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))), self.padded(1 - z)
        s, out = self.state(i, "s", (m["width"],)), torch.empty_like(write)
        for t, on in self.running():
            s[:on] = keep[:on, t] * s[:on] + write[:on, t]
            out[:on, t] = s[:on]
        self.keep(i, "s", s)
        return self.linear(self.unpadded(out) * _silu(self.linear(x, p + "g")), p + "o")

    def rotate(self, x, rot):
        dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
        f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)
        pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f = f / sc["factor"] * ramp + f * (1 - ramp)
        ang = (self.pos[:, None] * f.to(DEV)).view(len(self.pos), *[1] * (x.ndim - 2), -1)
        c, s = ang.cos() * (0.1 * math.log(sc["factor"]) + 1), ang.sin() * (0.1 * math.log(sc["factor"]) + 1)
        u, v = x.chunk(2, -1)
        return torch.cat([u * c - v * s, v * c + u * s], -1)

    def latent(self, x, i, m, p):
        H, d, r = m["heads"], m["dim"], m["kv_rank"]
        q = self.linear(x, p + "q").view(len(x), H, -1)
        if "kv_from" not in m:
            y = self.linear(x, p + "dkv")
            own = torch.cat([_norm(y[:, :r]) * self.W(p + "dkv.norm"), self.rotate(y[:, r:], m["rot"])], -1)
            self.keys[i] = [self.with_kept(i, 0, own)]
        rows = self.keys[m.get("kv_from", i)][0]
        # queries taken into the space of the cached rows: the keys of all heads are then the rows themselves
        ql = torch.einsum("thd,hdr->thr", q[..., :d], self.W(p + "uk").view(H, d, r))
        ql = torch.cat([ql, self.rotate(q[..., d:], m["rot"])], -1)
        o = self.attend(ql, rows[:, None], rows[:, None, :r], m["mask"]["size"], m["scale"], self.W(p + "sink"))
        o = torch.einsum("thr,hvr->thv", o, self.W(p + "uv").view(H, m["vdim"], r))
        return self.linear(o.flatten(1), p + "o")

    # ---- Derelorn
    def derelorn(self, x):
        x = _norm(x) * self.W("embed.norm")
        mixers = {"mlstm": self.mlstm, "delta": self.delta, "parallel": self.parallel}
        for i, layer in enumerate(self.config["layers"]):
            p = f"l{i}."
            y = mixers[layer["type"]](_norm(x) * self.W(p + "norm1"), i, layer["mixer"], p + "mix.")
            x = x + _norm(y) * self.W(p + "norm1b")
            h = _norm(x) * self.W(p + "norm2")
            y = self.linear(_silu(self.linear(h, p + "mlp.gate")) * self.linear(h, p + "mlp.up"), p + "mlp.down")
            x = x + _norm(y) * self.W(p + "norm2b")
        return x

    def mlstm(self, x, i, m, p):
        H, d, e, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        heads = lambda name, n: self.padded(self.linear(x, p + name).view(-1, H, n))
        gate = lambda name: cap * torch.tanh((self.linear(x, p + name) + self.W(p + name + ".b")) / cap)
        q, k, v = heads("q", d) * d ** -0.5, heads("k", d), heads("v", e)
        gi, gf = self.padded(gate("i")), self.padded(torch.nn.functional.logsigmoid(gate("f")))
        S, nm, out = self.state(i, "S", (H, d, e)), self.state(i, "n", (H, d + 1)), torch.zeros_like(v)
        for t, on in self.running():
            n, mx = nm[:on, :, :d], nm[:on, :, d]
            new = torch.maximum(gf[:on, t] + mx, gi[:on, t])
            keep, write = torch.exp(gf[:on, t] + mx - new)[..., None], torch.exp(gi[:on, t] - new)[..., None] * k[:on, t]
            S[:on] = keep[..., None] * S[:on] + write[..., None] * v[:on, t, :, None]
            nm[:on, :, :d], nm[:on, :, d] = keep * n + write, new
            den = torch.maximum((nm[:on, :, :d] * q[:on, t]).sum(-1).abs(), torch.exp(-new)) + 1e-6
            out[:on, t] = torch.einsum("bhdv,bhd->bhv", S[:on], q[:on, t]) / den[..., None]
        self.keep(i, "S", S)
        self.keep(i, "n", nm)
        o = _norm(self.unpadded(out)).flatten(1) * self.W(p + "norm") * torch.sigmoid(self.linear(x, p + "g"))
        return self.linear(o, p + "o")

    def conv(self, x, i, w, bias):
        """Causal, per channel, behind the inputs that the request has left."""
        x = self.padded(x)
        x = torch.cat([self.state(i, "conv", (TAPS - 1, x.shape[-1])), x], 1)
        counts = torch.tensor([self.new[k] for k in self.order], device=DEV)
        at = counts[:, None] + torch.arange(TAPS - 1, device=DEV)
        self.keep(i, "conv", x.gather(1, at[..., None].expand(-1, -1, x.shape[-1])))
        y = sum(x[:, j:x.shape[1] - TAPS + 1 + j] * w[:, j] for j in range(TAPS))
        return _silu(y if bias is None else y + bias)

    def delta(self, x, i, m, p):
        H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        y = self.conv(torch.cat([self.linear(x, p + c) for c in "qkv"], 1), i, torch.cat([self.W(f"{p}{c}.conv") for c in "qkv"]), None)
        unit = lambda z: (z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)
        q, k = (unit(z.unflatten(-1, (G, d))) for z in y[..., :2 * G * d].chunk(2, -1))
        q, v = q * d ** -0.5, y[..., 2 * G * d:].unflatten(-1, (H, e))
        beta = self.padded(torch.sigmoid(self.linear(x, p + "b")))
        g = torch.exp(-torch.exp(self.W(p + "A_log")) * torch.nn.functional.softplus(self.linear(x, p + "a") + self.W(p + "dt_bias")))
        g = self.padded(g)
        S, out = self.state(i, "S", (H, d, e)), torch.zeros_like(v)
        for t, on in self.running():
            s = g[:on, t, :, None, None] * S[:on]
            u = beta[:on, t, :, None] * (v[:on, t] - torch.einsum("bhdv,bhd->bhv", s, k[:on, t]))
            S[:on] = s + k[:on, t, ..., None] * u[..., None, :]
            out[:on, t] = torch.einsum("bhdv,bhd->bhv", S[:on], q[:on, t])
        self.keep(i, "S", S)
        o = (_norm(self.unpadded(out)) * self.W(p + "norm")).flatten(1) * _silu(self.linear(x, p + "g"))
        return self.linear(o, p + "o")

    def parallel(self, x, i, m, p):
        a, left = m["left"], p + "left."
        heads = lambda z, n: z.view(len(x), n, -1)
        q = _norm(self.linear(x, left + "q")) * self.W(left + "q.norm")
        k = self.with_kept(i, 0, _norm(self.linear(x, left + "k")) * self.W(left + "k.norm"))
        v = self.with_kept(i, 1, self.linear(x, left + "v"))
        self.keys[i] = [k, v]
        split = lambda z: z.view(len(z), a["kv_heads"], -1)
        o = self.attend(heads(q, a["heads"]), split(k), split(v), a["mask"]["size"], a["scale"])
        o = self.linear(o.flatten(1), left + "o")
        return 0.5 * (_norm(o) * self.W(left + "out") + _norm(self.mamba(x, i, m["right"], p + "right.")) * self.W(p + "right.out"))

    def mamba(self, x, i, m, p):
        H, e, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * e
        z, xbc, dt = self.linear(x, p + "in").split([inner, inner + 2 * G * N, H], 1)
        y = self.conv(xbc, i, self.W(p + "conv"), self.W(p + "conv.b"))
        v = y[..., :inner].unflatten(-1, (H, e))
        B, C = (c.unflatten(-1, (G, N)).repeat_interleave(H // G, 2) for c in y[..., inner:].chunk(2, -1))
        dt = torch.nn.functional.softplus(dt + self.W(p + "dt_bias"))
        decay, dt = self.padded(torch.exp(-torch.exp(self.W(p + "A_log")) * dt)), self.padded(dt)
        S, out = self.state(i, "S", (H, N, e)), torch.zeros_like(v)
        for t, on in self.running():
            S[:on] = decay[:on, t, :, None, None] * S[:on] + (dt[:on, t, :, None] * B[:on, t])[..., None] * v[:on, t, :, None]
            out[:on, t] = torch.einsum("bhnv,bhn->bhv", S[:on], C[:on, t]) + self.W(p + "D")[:, None] * v[:on, t]
        self.keep(i, "S", S)
        y = _norm((self.unpadded(out).flatten(1) * _silu(z)).view(len(x), m["norm_groups"], -1)).flatten(1)
        return self.linear(y * self.W(p + "norm"), p + "o")
