"""What this framework is asked to do in use, as cases that can be timed and checked: the attention path of a serving engine in
both directions, the steps around it, whole requests through the engine, and the kernels that carry the other model families.

A case fixes sizes, types and (through `ragged`) the lengths of its sequences; the values come from the seed.  `run` is one
pass through the public entry points as the engine's modules or a user's program call them; `exact` is the same result in 64
bits, written with plain torch.
"""
import math
import random

import torch

from minivllm_b200.engine.llm_engine import LLMEngine
from minivllm_b200.layers import attention, gla, mlstm, moe, sampler, window_attention

DEV = "cuda"
EPS = 1e-6
VOCAB = 32768
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

LISTED = [
    # A small decode step: a handful of conversations, where the launch and the host's call count.
    dict(name="decode_b16", kind="decode", batch=16, lo=64, hi=1024, heads=16, kv_heads=8, dtype="fp16", cache="same", ragged=1),
    # One layer of a full decode step of an 8B-sized model, 512 requests behind 512 to 2048 tokens.
    dict(name="decode_b512", kind="decode", batch=512, lo=512, hi=2048, heads=32, kv_heads=8, dtype="bf16", cache="same", ragged=2),
    # Decode from an 8-bit cache, the option for more requests in the same memory.
    dict(name="decode_int8_b64", kind="decode", batch=64, lo=1024, hi=4096, heads=32, kv_heads=8, dtype="fp16", cache="int8", ragged=3),
    # A prefill wave of whole prompts of mixed lengths.
    dict(name="prefill_32seq", kind="prefill", seqs=32, lo=128, hi=2048, heads=32, kv_heads=8, dtype="bf16", ragged=4),
    # Portions of prompts whose first half is in the cache already: chunked prefill, prefix hits, a second turn.
    dict(name="prefill_cached_16seq", kind="prefill_cached", seqs=16, lo=128, hi=2048, cached=0.5, heads=32, kv_heads=8, dtype="bf16", ragged=5),
    # Norm, rotary embedding and cache store in front of the attention of one prefill wave.
    dict(name="pre_attention_16384", kind="pre_attention", tokens=16384, heads=32, kv_heads=8, dtype="bf16", cache="same"),
    # Sampling with temperatures for a full batch at a large vocabulary.
    dict(name="sample_512", kind="sample", rows=512, vocab=151936, dtype="bf16", greedy_every=16),
    # Requests through the engine: one step for the prompts, then decoded tokens; scheduling, metadata and graphs included.
    dict(name="engine_16req", kind="engine", requests=16, lo=64, hi=256, steps=8, width=1024, layers=8, heads=16, kv_heads=8, ff=3072, ragged=6),
    # The feed-forward of the families with experts (a wave of prompts): routing, sort, grouped products, sum into the stream.
    dict(name="moe_16384", kind="moe", tokens=16384, width=2048, ff=1024, experts=64, top=6, shared=2048),
    # Windowed attention with distance biases and sinks (the attention of one family, and the kernel of three), whole prompts.
    dict(name="window_32seq", kind="window", seqs=32, lo=128, hi=2048, heads=16, kv_heads=4, window=1024, ragged=7),
    # Gated linear attention of one long prompt: few recurrences, each of them long.
    dict(name="gla_long", kind="gla", seqs=1, lo=16384, hi=16384, heads=8, dim=128, vdim=256, ragged=8),
    # Matrix memory of a wave of prompts: gates, running maxima and the recurrence.
    dict(name="mlstm_16seq", kind="mlstm", seqs=16, lo=512, hi=1536, heads=8, dim=128, vdim=256, ragged=9),
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    """Whole numbers spread over the logarithm of lo .. hi, odd ones as often as even ones."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice([c["kind"] for c in LISTED])
    c = {"kind": kind}
    heads, kv = rng.choice([(16, 8), (32, 8), (16, 4), (8, 2), (4, 1)])
    if kind == "decode":
        c["batch"] = _log_int(rng, 1, 512)
        c["hi"] = _log_int(rng, 64, min(8192, 1000000 // c["batch"]))
        c["lo"] = rng.randint(1, c["hi"])
        c.update(heads=heads, kv_heads=kv, dtype=rng.choice(["bf16", "fp16"]), cache=rng.choice(["same", "same", "int8"]))
    elif kind in ("prefill", "prefill_cached", "window"):
        c["seqs"] = _log_int(rng, 1, 48)
        c["hi"] = _log_int(rng, 32, min(8192 if kind == "prefill" else 4096, 36000 // c["seqs"]))
        c["lo"] = rng.randint(1, c["hi"])
        c.update(heads=heads, kv_heads=kv)
        if kind == "window":
            c["window"] = _log_int(rng, 128, 4096)
            c["heads"], c["kv_heads"] = min(heads, 16), min(kv, 4)
        else:
            c["dtype"] = rng.choice(["bf16", "fp16"])
        if kind == "prefill_cached":
            c["cached"] = round(rng.uniform(0.1, 0.9), 2)
    elif kind == "pre_attention":
        c.update(tokens=_log_int(rng, 1, 16384), heads=heads, kv_heads=kv, dtype=rng.choice(["bf16", "fp16"]),
                 cache=rng.choice(["same", "int8"]))
    elif kind == "sample":
        c.update(rows=_log_int(rng, 1, 512), vocab=rng.choice([32768, 50257, 100277, 151936]), dtype=rng.choice(["bf16", "fp16", "fp32"]),
                 greedy_every=rng.choice([0, 4, 16]))
    elif kind == "engine":
        c["hi"] = _log_int(rng, 16, 256)
        c.update(requests=_log_int(rng, 1, 16), lo=rng.randint(8, c["hi"]), steps=rng.randint(1, 8), width=1024, layers=8, heads=16,
                 kv_heads=8, ff=3072)
    elif kind == "moe":
        width, ff, experts, top, shared = rng.choice([(1024, 512, 32, 4, 1024), (2048, 1024, 64, 6, 2048), (2048, 1024, 64, 6, 0)])
        c.update(tokens=_log_int(rng, 1, 16384), width=width, ff=ff, experts=experts, top=top, shared=shared)
    else:
        c["seqs"] = _log_int(rng, 1, 24)
        c["hi"] = _log_int(rng, 24, 16384 // c["seqs"])
        c["lo"] = rng.randint(17, c["hi"])
        c["dim"], c["vdim"] = rng.choice([(128, 256), (128, 128), (64, 128)])
        c["heads"] = rng.choice([4, 8, 16]) if c["vdim"] < 256 else 8
    if "lo" in c:
        c["ragged"] = rng.randint(0, 1 << 20)
    return c


# ------------------------------------------------------------------------------------------------------------- inputs
def _lengths(case, count):
    r = random.Random(case["ragged"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(count)]


def _split(case):
    """Per sequence of a `prefill_cached` case: (tokens in the cache, new tokens)."""
    total = _lengths(case, case["seqs"])
    behind = [min(n - 1, int(n * case["cached"])) for n in total]
    return [(b, n - b) for b, n in zip(behind, total)]


class _Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16, scale=1.0, mean=0.0):
        """N(mean, scale), made in pieces so that large tensors need little memory beside themselves."""
        out = torch.empty(shape, dtype=dtype, device=DEV)
        flat = out.view(-1)
        for i in range(0, flat.numel(), 1 << 27):
            part = flat[i:i + (1 << 27)]
            part.copy_(torch.randn(part.numel(), generator=self.g, device=DEV).mul_(scale).add_(mean))
        return out

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.g, device=DEV) * (hi - lo) + lo

    def integers(self, lo, hi, *shape, dtype=torch.int64):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEV, dtype=dtype)

    def permutation(self, n):
        return torch.randperm(n, generator=self.g, device=DEV)


def _prefix(lens):
    return torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)


def _block_tables(d, lens, block):
    """(sequences, widest) int32 with -1 past a sequence's blocks, physical blocks in random order; and their number."""
    counts = [-(-n // block) for n in lens]
    ids, at = d.permutation(sum(counts)).to(torch.int32), 0
    tables = torch.full((len(lens), max(counts)), -1, dtype=torch.int32, device=DEV)
    for i, n in enumerate(counts):
        tables[i, :n] = ids[at:at + n]
        at += n
    return tables, at


BLOCK = 256


def prepare(case, seed):
    d, kind = _Draws(seed), case["kind"]
    s = {"kind": kind, "case": case}
    heads, kv, D = case.get("heads"), case.get("kv_heads"), 128
    dt = DTYPES[case.get("dtype", "bf16")]
    if kind == "decode":
        lens = _lengths(case, case["batch"])
        s["tables"], blocks = _block_tables(d, lens, BLOCK)
        s["ctx"] = torch.tensor(lens, dtype=torch.int32, device=DEV)
        s["q"] = d.normal(case["batch"], heads, D, dtype=dt)
        shape = (blocks, BLOCK, kv, D)
        if case["cache"] == "int8":
            s["k"], s["v"] = (d.integers(-127, 128, *shape, dtype=torch.int8) for _ in range(2))
            s["scales"] = {n: d.uniform(*shape[:3], lo=0.01, hi=0.02).half() for n in ("k_scale", "v_scale")}
        else:
            s["k"], s["v"], s["scales"] = d.normal(*shape, dtype=dt), d.normal(*shape, dtype=dt), {}
    elif kind == "prefill":
        lens = _lengths(case, case["seqs"])
        s["cu"], T = _prefix(lens), sum(lens)
        s["q"], s["k"], s["v"] = (d.normal(T, h, D, dtype=dt) for h in (heads, kv, kv))
    elif kind == "prefill_cached":
        spans = _split(case)
        s["cu_q"], s["cu_k"] = _prefix([n for _, n in spans]), _prefix([b + n for b, n in spans])
        s["tables"], blocks = _block_tables(d, [b + n for b, n in spans], BLOCK)
        s["q"] = d.normal(sum(n for _, n in spans), heads, D, dtype=dt)
        s["k"], s["v"] = (d.normal(blocks, BLOCK, kv, D, dtype=dt) for _ in range(2))
    elif kind == "pre_attention":
        T = case["tokens"]
        blocks = -(-T // BLOCK) + 1
        s["qkv"] = d.normal(T, (heads + 2 * kv) * D, dtype=dt)
        s["positions"] = d.integers(0, 2048, T)
        s["gq"], s["gk"] = (d.normal(D, dtype=dt, scale=0.1, mean=1.0) for _ in range(2))
        angle = torch.arange(2048, device=DEV).double()[:, None] * 1e6 ** (-torch.arange(0, D, 2, device=DEV).double() / D)
        s["cos"], s["sin"] = angle.cos().float(), angle.sin().float()
        s["slots"] = d.permutation(blocks * BLOCK)[:T].contiguous()
        store = torch.int8 if case["cache"] == "int8" else dt
        s["k_cache"], s["v_cache"] = (torch.zeros(blocks, BLOCK, kv, D, dtype=store, device=DEV) for _ in range(2))
        s["scales"] = {}
        if case["cache"] == "int8":
            s["scales"] = {n: torch.zeros(blocks, BLOCK, kv, dtype=torch.float16, device=DEV) for n in ("k_scale", "v_scale")}
    elif kind == "sample":
        rows = case["rows"]
        s["logits"] = d.normal(rows, case["vocab"], dtype=dt, scale=2.0)
        s["temps"] = d.uniform(rows, lo=0.4, hi=1.2)
        if case["greedy_every"]:
            s["temps"][::case["greedy_every"]] = 0.0
        s["step"], s["seed"] = torch.zeros(1, dtype=torch.int64, device=DEV), seed
    elif kind == "engine":
        s["engine"] = _engine(case, seed)
        g = random.Random(seed)
        s["prompts"] = [[g.randrange(VOCAB) for _ in range(n)] for n in _lengths(case, case["requests"])]
        s["next"] = [[g.randrange(VOCAB) for _ in range(case["requests"])] for _ in range(case["steps"])]
    elif kind == "moe":
        _, s["layer"], s["tail"] = _moe(case, seed)
        T, W = case["tokens"], case["width"]
        s["h"], s["x"] = d.normal(T, W), d.normal(T, W, dtype=torch.float32)
    elif kind == "window":
        lens = _lengths(case, case["seqs"])
        s["cu"], T = _prefix(lens), sum(lens)
        s["q"], s["kv"] = d.normal(T, heads * D), d.normal(T, kv * 2 * D)
        s["rel"], s["sink"] = d.normal(32, heads), d.normal(heads)
        s["bias"] = window_attention.distance_bias(s["rel"], 128, case["window"])
    else:
        lens = _lengths(case, case["seqs"])
        n, T, K, V = len(lens), sum(lens), case["dim"], case["vdim"]
        s["cu"] = _prefix(lens)
        p = d.normal(T, 2 * heads * K + heads * V)       # one product, as the layer's stacked projection leaves it
        s["q"], s["k"], s["v"] = p.split([heads * K, heads * K, heads * V], 1)
        s["slots"], s["starts"] = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
        s["S"] = torch.zeros(n, heads, K, V, device=DEV)
        if kind == "gla":
            s["z"] = d.normal(T, heads * K, mean=3.0)
        else:
            s["z"] = d.normal(T, 2 * heads, dtype=torch.float32)
            s["ib"], s["fb"] = d.normal(heads, scale=0.5, mean=-1.0), d.normal(heads, scale=0.5, mean=4.0)
            s["n"], s["m"] = torch.zeros(n, heads, K, device=DEV), torch.zeros(n, heads, device=DEV)
    return s


def _weights(case, seed):
    """The decoder's matrices by the model's parameter names."""
    d, c = _Draws(seed + 1), case
    rows = (c["heads"] + 2 * c["kv_heads"]) * 128
    mat = lambda o, i: d.normal(o, i, scale=i ** -0.5)
    w = {"embed": d.normal(VOCAB, c["width"]), "lm_head": mat(VOCAB, c["width"])}
    for i in range(c["layers"]):
        w.update({f"layers.{i}.qkv_w": mat(rows, c["width"]), f"layers.{i}.o_w": mat(c["width"], c["heads"] * 128),
                  f"layers.{i}.gate_up_w": mat(2 * c["ff"], c["width"]), f"layers.{i}.down_w": mat(c["width"], c["ff"])})
    return w


def _engine(case, seed):
    c = case
    e = LLMEngine(dict(vocab_size=VOCAB, hidden_size=c["width"], num_layers=c["layers"], num_heads=c["heads"], num_kv_heads=c["kv_heads"],
                       head_dim=128, intermediate_size=c["ff"], base=1e6, max_model_length=512, tie_word_embeddings=False,
                       block_size=BLOCK, max_num_seqs=c["requests"], num_kv_blocks=2 * c["requests"], max_num_batched_tokens=4096,
                       chunked_prefill=True, greedy=True, keep_logits=True, dtype=torch.bfloat16))
    w = _weights(case, seed)
    with torch.no_grad():
        for name, p in e.model_runner.model.named_parameters():
            if name in w:
                p.copy_(w[name])
    return e


def _moe(case, seed):
    """(weights by name, the layer, the rest of its arguments behind h and x)."""
    d, W, ff, E = _Draws(seed + 1), case["width"], case["ff"], case["experts"]
    w = {"router": d.normal(E, W, scale=W ** -0.5), "router.b": d.normal(E, scale=0.1)}
    gate, up, down = d.normal(E, ff, W, scale=W ** -0.5), d.normal(E, ff, W, scale=W ** -0.5), d.normal(E, W, ff, scale=ff ** -0.5)
    for e in range(E):
        w.update({f"e{e}.gate": gate[e], f"e{e}.up": up[e], f"e{e}.down": down[e]})
    spec = {"router": {"experts": E, "top": case["top"]}, "expert": {"ff": ff}}
    if case["shared"]:
        n = case["shared"]
        w.update({"shared.gate": d.normal(n, W, scale=W ** -0.5), "shared.up": d.normal(n, W, scale=W ** -0.5),
                  "shared.down": d.normal(W, n, scale=n ** -0.5), "shared.sg": d.normal(1, W, scale=W ** -0.5)})
        spec["shared"] = {"ff": n}
    w["gate"], w["gate.b"] = d.normal(W, W, scale=W ** -0.5), d.normal(W, scale=0.1)
    w["post"], w["next"] = d.normal(W, scale=0.1, mean=1.0), d.normal(W, scale=0.1, mean=1.0)
    layer = moe.MixtureOfExperts(spec, W, lambda name, shape: w[name], extra={"residual_gate": w["gate"]})
    return w, layer, (w["gate.b"], w["post"], w["next"], 0.5, 4, EPS)


# --------------------------------------------------------------------------------------------------------------- run
def run(s):
    with torch.inference_mode():
        return _RUN[s["kind"]](s, s["case"])


def _run_decode(s, c):
    return attention.paged_attention_decode(s["q"], s["k"], s["v"], s["tables"], s["ctx"], 128 ** -0.5, c["heads"], c["kv_heads"], 128, BLOCK,
                                            **s["scales"])


def _run_prefill(s, c):
    return attention.flash_attention_prefill(s["q"], s["k"], s["v"], s["cu"], 128 ** -0.5, c["heads"], c["kv_heads"], 128)


def _run_prefill_cached(s, c):
    return attention.flash_attention_prefill_paged(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], s["tables"], 128 ** -0.5, c["heads"],
                                                   c["kv_heads"], 128)


def _run_pre_attention(s, c):
    q, k = attention.qk_norm_rope_store(s["qkv"], s["positions"], s["cos"], s["sin"], s["gq"], s["gk"], EPS, c["heads"], c["kv_heads"], 128,
                                        s["k_cache"], s["v_cache"], s["slots"], **s["scales"])
    return {"q": q, "k": k, "k_cache": s["k_cache"], "v_cache": s["v_cache"], **s["scales"]}


def _run_sample(s, c):
    tokens = sampler.sampled_tokens(s["logits"], s["temps"], s["seed"], s["step"])
    s["step"].add_(1)
    return tokens


def _run_engine(s, c):
    e, ids = s["engine"], range(c["requests"])
    out = [e.score_step([(i, p, [len(p) - 1]) for i, p in enumerate(s["prompts"])])]
    for n, tokens in enumerate(s["next"]):
        out.append(e.score_step([(i, [tokens[i]], [0]) for i in ids], end=ids if n == c["steps"] - 1 else ()))
    return out


def _run_moe(s, c):
    return {"h": s["layer"](s["h"], s["x"], *s["tail"]), "x": s["x"]}


def _run_window(s, c):
    return window_attention.window_prefill(s["q"], s["kv"], s["cu"], s["cu"], c["kv_heads"], 128, 128, c["window"], 128 ** -0.5, s["bias"],
                                           s["sink"])


def _run_gla(s, c):
    out = gla.gla_scan(s["q"], s["k"], s["v"], s["z"], 16.0, s["cu"], s["slots"], s["starts"], s["S"], c["heads"], c["dim"], c["vdim"])
    return {"out": out, "S": s["S"]}


def _run_mlstm(s, c):
    chain = mlstm.mlstm_gates(s["z"], s["ib"], s["fb"], 15.0, s["cu"], s["slots"], s["starts"], s["m"], c["heads"])
    out, den = mlstm.mlstm_scan(s["q"], s["k"], s["v"], chain, s["cu"], s["slots"], s["starts"], s["S"], s["n"], c["heads"], c["dim"],
                                c["vdim"])
    return {"out": out, "den": den, "S": s["S"], "n": s["n"], "m": s["m"]}


_RUN = {"decode": _run_decode, "prefill": _run_prefill, "prefill_cached": _run_prefill_cached, "pre_attention": _run_pre_attention,
        "sample": _run_sample, "engine": _run_engine, "moe": _run_moe, "window": _run_window, "gla": _run_gla, "mlstm": _run_mlstm}


# -------------------------------------------------------------------------------------------------------------- work
def work(case):
    c, kind = case, case["kind"]
    H, G, D = c.get("heads"), c.get("kv_heads"), 128
    e = torch.empty((), dtype=DTYPES[c.get("dtype", "bf16")]).element_size()
    if kind == "decode":
        lens, B = _lengths(c, c["batch"]), c["batch"]
        row = D + 2 if c["cache"] == "int8" else D * e
        blocks = -(-max(lens) // BLOCK)
        return {"bytes": sum(lens) * G * 2 * row + 2 * B * H * D * e + B * (blocks + 1) * 4, "flops": 4 * H * D * sum(lens)}
    if kind in ("prefill", "prefill_cached"):
        spans = _split(c) if kind == "prefill_cached" else [(0, n) for n in _lengths(c, c["seqs"])]
        pairs = sum(n * b + n * (n + 1) // 2 for b, n in spans)
        return {"bytes": D * e * sum(2 * H * n + 2 * G * (b + n) for b, n in spans), "flops": 4 * H * D * pairs}
    if kind == "pre_attention":
        stored = 2 * G * (D + 2) if c["cache"] == "int8" else 2 * G * D * e
        row = (H + 2 * G) * D * e + (H + G) * D * e + stored + 16
        return {"bytes": c["tokens"] * row, "flops": c["tokens"] * (H + G) * D * 8}
    if kind == "sample":
        return {"bytes": c["rows"] * (c["vocab"] * e + 12), "flops": c["rows"] * c["vocab"] * 4}
    if kind == "engine":
        lens = _lengths(c, c["requests"])
        per = c["width"] * (H + 2 * G) * D + c["width"] * H * D + 3 * c["width"] * c["ff"]
        params, head, steps = c["layers"] * per, VOCAB * c["width"], c["steps"]
        kv = c["layers"] * 2 * G * D * 2
        seen = sum(n * (1 + steps) + steps * (steps + 1) // 2 for n in lens)
        return {"bytes": (1 + steps) * ((params + head) * 2 + len(lens) * VOCAB * 4) + kv * seen,
                "flops": 2 * params * (sum(lens) + steps * len(lens)) + 2 * head * (1 + steps) * len(lens)}
    if kind == "moe":
        T, W, ff = c["tokens"], c["width"], c["ff"]
        used = min(c["experts"], T * c["top"])
        dense = 3 * W * c["shared"] + W * W + W * c["experts"]
        return {"bytes": (used * 3 * W * ff + dense) * 2 + T * W * 12, "flops": 2 * T * (c["top"] * 3 * W * ff + dense)}
    if kind == "window":
        lens = _lengths(c, c["seqs"])
        full = lambda n: min(n, c["window"])
        pairs = sum(full(n) * (full(n) + 1) // 2 + (n - full(n)) * c["window"] for n in lens)
        return {"bytes": sum(lens) * 2 * D * (H + G) * 2, "flops": 4 * H * D * pairs}
    T, K, V = sum(_lengths(c, c["seqs"])), c["dim"], c["vdim"]
    state = c["seqs"] * H * K * V * 4
    if kind == "gla":
        return {"bytes": T * H * (3 * K + 2 * V) * 2 + state, "flops": T * H * 4 * K * V}
    return {"bytes": T * H * ((2 * K + 2 * V) * 2 + 12) + state + c["seqs"] * H * (K + 1) * 4, "flops": T * H * 4 * K * (V + 1)}


# About four times the error against 64 bits that the path showed, the rounding of its inputs between steps and of its results
# included: 2e-3 in bf16, 1e-3 and less in fp16, 1.1e-2 for the logits behind eight bf16 layers.
_TOLERANCE = {"bf16": 1e-2, "fp16": 4e-3, "engine": 3e-2}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    t = {"rel": _TOLERANCE["engine" if case["kind"] == "engine" else case.get("dtype", "bf16")]}
    if case["kind"] == "pre_attention" and case["cache"] == "int8":
        t["differ"] = 1e-3           # a code lies on a border between two where the row's maximum moves by a rounding step
    return t


# ------------------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] == "sample":
        return None                  # whole numbers
    if case["kind"] in ("engine", "moe"):
        return (_exact_engine if case["kind"] == "engine" else _exact_moe)(case, seed)
    return _EXACT[case["kind"]](prepare(case, seed), case)


def _attend(q, k, v, behind, scale=128 ** -0.5, bias_of=None, sink=None, window=None):
    """q (n, H, D) at positions behind .. behind + n - 1, k and v (m, G, D): causal attention in 64 bits."""
    n, H, _ = q.shape
    m, G, _ = k.shape
    out, step = torch.empty(n, H, v.shape[2], dtype=torch.float64, device=DEV), max(1, (1 << 27) // (H * m))
    k, v = (t.double().permute(1, 0, 2) for t in (k, v))
    for i in range(0, n, step):
        x = q[i:i + step].double().permute(1, 0, 2).reshape(G, H // G, -1, q.shape[2])
        sc = (x @ k[:, None].transpose(2, 3)) * scale                                    # G, H / G, rows, m
        dist = (behind + i + torch.arange(x.shape[2], device=DEV))[:, None] - torch.arange(m, device=DEV)[None]
        if bias_of is not None:
            sc += bias_of(dist.clamp(min=0)).view(G, H // G, *dist.shape)
        hide = dist < 0 if window is None else (dist < 0) | (dist >= window)
        sc.masked_fill_(hide, -math.inf)
        if sink is not None:
            sc = torch.cat([sc, sink.double().view(G, H // G, 1, 1).expand(-1, -1, x.shape[2], 1)], 3)
        p = sc.softmax(3)[..., :m]
        out[i:i + step] = (p @ v[:, None]).reshape(H, -1, v.shape[2]).permute(1, 0, 2)
    return out


def _rows_of(cache, table, n, scale=None):
    """The first n rows of a sequence in the paged cache."""
    blocks = table[:-(-n // BLOCK)].long()
    x = cache[blocks].flatten(0, 1)[:n].double()
    return x if scale is None else x * scale[blocks].flatten(0, 1)[:n].double()[..., None]


def _exact_decode(s, c):
    lens, sc = _lengths(c, c["batch"]), s["scales"]
    out = [_attend(s["q"][i:i + 1], _rows_of(s["k"], s["tables"][i], n, sc.get("k_scale")), _rows_of(s["v"], s["tables"][i], n, sc.get("v_scale")),
                   n - 1) for i, n in enumerate(lens)]
    return torch.cat(out)


def _exact_prefill(s, c):
    out, at = [], 0
    for n in _lengths(c, c["seqs"]):
        out.append(_attend(s["q"][at:at + n], s["k"][at:at + n], s["v"][at:at + n], 0))
        at += n
    return torch.cat(out)


def _exact_prefill_cached(s, c):
    out, at = [], 0
    for i, (b, n) in enumerate(_split(c)):
        out.append(_attend(s["q"][at:at + n], _rows_of(s["k"], s["tables"][i], b + n), _rows_of(s["v"], s["tables"][i], b + n), b))
        at += n
    return torch.cat(out)


def _rms(x, w):
    return x / (x.square().mean(-1, keepdim=True) + EPS).sqrt() * w.double()


def _rotate(x, cos, sin):
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _exact_pre_attention(s, c):
    H, G, T = c["heads"], c["kv_heads"], c["tokens"]
    q, k, v = s["qkv"].double().view(T, H + 2 * G, 128).split([H, G, G], 1)
    cos, sin = (s[n][s["positions"]].double()[:, None] for n in ("cos", "sin"))
    q, k = _rotate(_rms(q, s["gq"]), cos, sin), _rotate(_rms(k, s["gk"]), cos, sin)
    out = {"q": q, "k": k, "k_cache": None, "v_cache": None}
    if c["cache"] == "int8":
        return {**out, "k_scale": None, "v_scale": None}
    for name, x in (("k_cache", k), ("v_cache", v)):
        out[name] = torch.zeros(s[name].shape, dtype=torch.float64, device=DEV)
        out[name].view(-1, G, 128)[s["slots"]] = x
    return out


def _exact_engine(case, seed):
    c, w = case, _weights(case, seed)
    H, G, W = c["heads"], c["kv_heads"], c["width"]
    g = random.Random(seed)
    prompts = [[g.randrange(VOCAB) for _ in range(n)] for n in _lengths(c, c["requests"])]
    nxt = [[g.randrange(VOCAB) for _ in range(c["requests"])] for _ in range(c["steps"])]
    got = []
    layers = [{n: w[f"layers.{i}.{n}"].double() for n in ("qkv_w", "o_w", "gate_up_w", "down_w")} for i in range(c["layers"])]
    embed, head = w["embed"], w["lm_head"].double()
    norm = lambda x: x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt()
    for i, p in enumerate(prompts):
        ids = torch.tensor(p + [t[i] for t in nxt], device=DEV)
        angle = torch.arange(len(ids), device=DEV).double()[:, None] * 1e6 ** (-torch.arange(0, 128, 2, device=DEV).double() / 128)
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]
        h = norm(embed[ids].double())
        x = h
        for l in layers:
            q, k, v = (h @ l["qkv_w"].T).view(-1, H + 2 * G, 128).split([H, G, G], 1)
            o = _attend(_rotate(norm(q), cos, sin), _rotate(norm(k), cos, sin), v, 0)
            x = x + o.reshape(-1, H * 128) @ l["o_w"].T
            gate, up = (norm(x) @ l["gate_up_w"].T).chunk(2, 1)
            x = x + (torch.nn.functional.silu(gate) * up) @ l["down_w"].T
            h = norm(x)
        got.append((h[len(p) - 1:] @ head.T).cpu())
    return [torch.stack([x[t] for x in got]) for t in range(c["steps"] + 1)]


def _exact_moe(case, seed):
    c, (w, _, _), d = case, _moe(case, seed), _Draws(seed)
    T, W = c["tokens"], c["width"]
    h, x = d.normal(T, W).double(), d.normal(T, W, dtype=torch.float32).double()
    w = {n: t.double() if not n.startswith("e") else t for n, t in w.items()}
    mlp = lambda y, n: (torch.nn.functional.silu(y @ w[n + "gate"].double().T) * (y @ w[n + "up"].double().T)) @ w[n + "down"].double().T
    best, idx = (h @ w["router"].T + w["router.b"]).topk(c["top"])
    best, y = best.softmax(1), torch.zeros_like(h)
    for e in range(c["experts"]):
        rows, k = (idx == e).nonzero(as_tuple=True)
        y.index_add_(0, rows, mlp(h[rows], f"e{e}.") * best[rows, k][:, None])
    if c["shared"]:
        y += (h @ w["shared.sg"].T).sigmoid() * mlp(h, "shared.")
    y *= (h @ w["gate"].T + w["gate.b"]).sigmoid()
    norm = lambda t, g: (t.view(T, 4, -1) / (t.view(T, 4, -1).square().mean(-1, keepdim=True) + EPS).sqrt()).view(T, W) * w[g]
    x = x + 0.5 * norm(y, "post")
    return {"h": norm(x, "next"), "x": x}


def _exact_window(s, c):
    out, at, H = [], 0, c["heads"]
    far = lambda n: 16 + math.floor(math.log(n / 16) / math.log(128 / 16) * 16)     # half the 32 buckets, up to distance 128
    idx = torch.tensor([n if n < 16 else min(31, far(n)) for n in range(max(_lengths(c, c["seqs"])))], device=DEV)
    bias = s["rel"].double()[idx].T
    for n in _lengths(c, c["seqs"]):
        q, kv = s["q"][at:at + n].view(n, H, 128), s["kv"][at:at + n].view(n, 2, c["kv_heads"], 128)
        out.append(_attend(q, kv[:, 0], kv[:, 1], 0, bias_of=lambda dist: bias[:, dist], sink=s["sink"], window=c["window"]))
        at += n
    return torch.cat(out).view(-1, H * 128)


def _padded(s, x, width):
    """(tokens, heads * width) -> (longest, sequences, heads, width) in 64 bits, zeros past a sequence's end."""
    c = s["case"]
    lens = _lengths(c, c["seqs"])
    out, at = torch.zeros(max(lens), len(lens), c["heads"], width, dtype=torch.float64, device=DEV), 0
    for i, n in enumerate(lens):
        out[:n, i] = x[at:at + n].double().view(n, c["heads"], width)
        at += n
    return out


def _packed(s, x):
    lens = _lengths(s["case"], s["case"]["seqs"])
    return torch.cat([x[:n, i].flatten(1) for i, n in enumerate(lens)])


def _exact_gla(s, c):
    K, V = c["dim"], c["vdim"]
    q, k, v = _padded(s, s["q"], K) * K ** -0.5, _padded(s, s["k"], K), _padded(s, s["v"], V)
    alpha = (torch.nn.functional.logsigmoid(_padded(s, s["z"], K)) / 16.0).exp()
    S, out = torch.zeros(q.shape[1], c["heads"], K, V, dtype=torch.float64, device=DEV), torch.empty_like(v)
    alive = [torch.tensor(_lengths(c, c["seqs"]), device=DEV)[:, None, None] > t for t in range(q.shape[0])] if c["seqs"] > 1 else None
    for t in range(q.shape[0]):
        a = alpha[t] if alive is None else torch.where(alive[t], alpha[t], 1.0)
        S.mul_(a[..., None]).addcmul_(k[t][..., None], v[t][..., None, :])
        torch.matmul(q[t][..., None, :], S, out=out[t][..., None, :])
    return {"out": _packed(s, out), "S": S}


def _exact_mlstm(s, c):
    K, V, H = c["dim"], c["vdim"], c["heads"]
    q, k, v = _padded(s, s["q"], K) * K ** -0.5, _padded(s, s["k"], K), _padded(s, s["v"], V)
    cap = lambda x: 15.0 * torch.tanh(x / 15.0)
    i = cap(_padded(s, s["z"][:, :H], 1)[..., 0] + s["ib"].double())
    f = torch.nn.functional.logsigmoid(cap(_padded(s, s["z"][:, H:], 1)[..., 0] + s["fb"].double()))
    n_seq = q.shape[1]
    lens = torch.tensor(_lengths(c, c["seqs"]), device=DEV)[:, None]
    zeros = lambda *shape: torch.zeros(n_seq, H, *shape, dtype=torch.float64, device=DEV)
    S, n, m, out, den = zeros(K, V), zeros(K), zeros(), torch.empty_like(v), torch.empty_like(i)
    for t in range(q.shape[0]):
        on = lens > t
        new = torch.where(on, torch.maximum(f[t] + m, i[t]), m)
        keep = torch.where(on, (f[t] + m - new).exp(), 1.0)
        kw = k[t] * torch.where(on, (i[t] - new).exp(), 0.0)[..., None]
        S.mul_(keep[..., None, None]).addcmul_(kw[..., None], v[t][..., None, :])
        n, m = n * keep[..., None] + kw, new
        torch.matmul(q[t][..., None, :], S, out=out[t][..., None, :])
        den[t] = torch.maximum((n * q[t]).sum(-1).abs(), (-m).exp()) + 1e-6
    return {"out": _packed(s, out), "den": _packed(s, den[..., None]), "S": S, "n": n, "m": m}


_EXACT = {"decode": _exact_decode, "prefill": _exact_prefill, "prefill_cached": _exact_prefill_cached, "pre_attention": _exact_pre_attention,
          "window": _exact_window, "gla": _exact_gla, "mlstm": _exact_mlstm}
