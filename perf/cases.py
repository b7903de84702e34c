"""The work that this engine is timed on: whole steps of the engine, single layers and the sampler, over the sizes they
are used at.  Layer sizes are those of `bench.py` (the dense shapes "0.6b", "8b" and the sizes "1b" and "8b" of its designs);
weights, tokens and cached rows are seeded random numbers.

Kinds of cases and what they stand for:
  step        one call of the step function on a cut of a dense model (a few of its layers, the whole vocabulary): decoded
              tokens of several requests, possibly beside a portion of a prompt, as the scheduler puts them together
  attention   one grouped-query attention layer of a step: decoded tokens over long contexts, prompts, portions of prompts
  mlp         one gated feed-forward of a step
  experts     one routed feed-forward (4 of 32 experts)
  latent      one latent-attention layer (a window of 1,024, gated heads)
  recurrence  one gated linear attention or retention with its state
  sample      tokens chosen from a step's logits, the rows with different sampling parameters
A layer's pass is one layer of a running step: what the layers of one step share stands in the step's context."""
import math

import torch

from mini_rsglang_b200 import RuntimeConfig, SamplingParams
from mini_rsglang_b200.cache.storage import CacheEntry
from mini_rsglang_b200.engine import ModelRunner, SequenceStep
from mini_rsglang_b200.engine.context import StepContext
from mini_rsglang_b200.models import config_from_dict
from mini_rsglang_b200.parts import FEED_FORWARDS, MIXERS, PartSpec, Runtime
from mini_rsglang_b200.parts.linear import configure_library_products
from mini_rsglang_b200.sampling.sampler import Sampler

DEVICE = torch.device("cuda:0")
PAGE = 16
VOCAB = 151936
DENSE = {"0.6b": dict(width=1024, ff=3072, heads=16, kv_heads=8, tied=True), "8b": dict(width=4096, ff=12288, heads=32, kv_heads=8, tied=False)}
DESIGN = {"1b": dict(width=2048, ff=8192, heads=16), "8b": dict(width=4096, ff=12288, heads=32)}
HEAD, THETA, EPS = 128, 1000000.0, 1e-6
EXPERTS, TOP = 32, 4
LATENT = dict(dim=64, rot=32, vdim=64, rank=256, window=1024, factor=4.0, original=4096, fast=32.0, slow=1.0)
LINEAR = dict(dim=128, vdim=256, tau=16.0, rank=16, base=10000.0)
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    return [
        # one user's chat at the smallest shape: a single decoded token, bound by launches and latency
        {"name": "step_one_token", "kind": "step", "shape": "0.6b", "layers": 4, "decodes": 1, "context": 200, "portion": 0, "behind": 0},
        # the headline workload: 8 requests at a context of 4,096
        {"name": "step_decode_8", "kind": "step", "shape": "8b", "layers": 4, "decodes": 8, "context": 4096, "portion": 0, "behind": 0},
        # continuous batching: decoded tokens beside a portion of a prompt that fills the step's budget
        {"name": "step_mixed", "kind": "step", "shape": "8b", "layers": 4, "decodes": 27, "context": 1100, "portion": 485, "behind": 512},
        # many users with long contexts: reading the cache is everything
        {"name": "attention_decode_64", "kind": "attention", "shape": "8b", "dtype": "bfloat16", "requests": 64, "tokens": 1, "context": 4096},
        # a long prompt of odd length in one piece
        {"name": "attention_prompt", "kind": "attention", "shape": "8b", "dtype": "bfloat16", "requests": 1, "tokens": 3989, "context": 3989},
        # the 32-bit path: a prompt through an attention layer in float32
        {"name": "attention_float32", "kind": "attention", "shape": "0.6b", "dtype": "float32", "requests": 1, "tokens": 777, "context": 777},
        # a prompt through a dense feed-forward
        {"name": "mlp_prompt", "kind": "mlp", "shape": "8b", "dtype": "bfloat16", "rows": 1333},
        # decoded tokens through routed experts: every chosen expert's weights are read for a few rows
        {"name": "experts_decode_16", "kind": "experts", "size": "8b", "rows": 16},
        # a prompt through routed experts
        {"name": "experts_prompt", "kind": "experts", "size": "1b", "rows": 1777},
        # a prompt through a windowed latent attention
        {"name": "latent_prompt", "kind": "latent", "size": "1b", "requests": 1, "tokens": 2048, "context": 2048},
        # a prompt through a recurrence with one decay a key channel
        {"name": "recurrence_prompt", "kind": "recurrence", "form": "gated_linear_attention", "size": "1b", "requests": 1, "tokens": 2000, "context": 2000},
        # a step's logits to tokens: temperature, top-k and top-p over the whole vocabulary
        {"name": "sample_24", "kind": "sample", "rows": 24, "vocab": VOCAB},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, even over the logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "attention", "attention", "attention", "mlp", "mlp", "experts", "experts", "latent", "recurrence", "recurrence", "sample"])
    if kind == "step":
        context = _spread(rng, 64, 4096)
        portion = rng.choice([0, _spread(rng, 17, 480)])
        decodes = _spread(rng, 1, min(24 if portion else 64, 32768 // context))
        return {"kind": kind, "shape": rng.choice(["0.6b", "8b"]), "layers": 4, "decodes": decodes, "context": context, "portion": portion,
                "behind": rng.choice([0, _spread(rng, 64, 1024)]) if portion else 0}
    if kind == "attention":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        most = 262144 if dtype == "bfloat16" else 16384          # cached tokens of all requests
        shape = rng.choice(["0.6b", "8b"]) if dtype == "bfloat16" else "0.6b"
        if rng.random() < 0.5:
            context = _spread(rng, 64, 8192)
            requests = _spread(rng, 1, min(64, most // context))
            tokens = 1
        else:
            requests = rng.choice([1, 1, 2, 3])
            tokens = _spread(rng, 2, (4000 if dtype == "bfloat16" else 900) // requests)
            context = tokens + rng.choice([0, _spread(rng, 1, 1500 if tokens * requests < 2500 else 64)])
        return {"kind": kind, "shape": shape, "dtype": dtype, "requests": requests, "tokens": tokens, "context": context}
    if kind == "mlp":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        return {"kind": kind, "shape": rng.choice(["0.6b", "8b"]) if dtype == "bfloat16" else "0.6b", "dtype": dtype,
                "rows": _spread(rng, 1, 1400 if dtype == "bfloat16" else 700)}
    if kind == "experts":
        return {"kind": kind, "size": rng.choice(["1b", "8b"]), "rows": _spread(rng, 1, 2048)}
    if kind in ("latent", "recurrence"):
        case = {"kind": kind, "size": rng.choice(["1b", "8b"])}
        if kind == "recurrence":
            case["form"] = rng.choice(["gated_linear_attention", "retention"])
        if rng.random() < 0.4:
            return dict(case, requests=_spread(rng, 1, 64), tokens=1, context=_spread(rng, 16, 4096))
        requests = rng.choice([1, 1, 2, 5])
        tokens = _spread(rng, 2, 2048 // requests)
        return dict(case, requests=requests, tokens=tokens, context=tokens + rng.choice([0, _spread(rng, 1, 1500)]))
    return {"kind": kind, "rows": _spread(rng, 1, 64), "vocab": rng.choice([VOCAB, 32768])}


# ---------------------------------------------------------------------------------------------- inputs from a seed
class _Draws:
    """Seeded tensors on the device, in the order they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(int(seed) * 7919 + 13)

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=self.gen)

    def whole(self, low, high, shape):
        return torch.randint(low, high, shape, generator=self.gen, device=DEVICE)

    def weights(self, shapes, dtype):
        """name -> (shape, role): matrices N(0, 0.02), norm scales 1 + N(0, 0.05), biases N(0, 0.5)."""
        out = {}
        for name, (shape, role) in shapes.items():
            if role == "matrix":
                out[name] = self.normal(shape, 0.02, 0.0, dtype)
            elif role == "vector":
                out[name] = self.normal(shape, 0.05, 1.0)
            else:
                out[name] = self.normal(shape, 0.5)
        return out


def _dense_shapes(s, prefix):
    w, q, kv = s["width"], s["heads"] * HEAD, s["kv_heads"] * HEAD
    a, m = f"{prefix}.self_attn", f"{prefix}.mlp"
    attention = {f"{a}.q_proj.weight": ((q, w), "matrix"), f"{a}.k_proj.weight": ((kv, w), "matrix"), f"{a}.v_proj.weight": ((kv, w), "matrix"),
                 f"{a}.o_proj.weight": ((w, q), "matrix"), f"{a}.q_norm.weight": ((HEAD,), "vector"), f"{a}.k_norm.weight": ((HEAD,), "vector")}
    mlp = {f"{m}.gate_proj.weight": ((s["ff"], w), "matrix"), f"{m}.up_proj.weight": ((s["ff"], w), "matrix"),
           f"{m}.down_proj.weight": ((w, s["ff"]), "matrix")}
    return attention, mlp


def _model_shapes(case):
    s = DENSE[case["shape"]]
    shapes = {"model.embed_tokens.weight": ((VOCAB, s["width"]), "matrix"), "model.norm.weight": ((s["width"],), "vector")}
    if not s["tied"]:
        shapes["lm_head.weight"] = ((VOCAB, s["width"]), "matrix")
    for i in range(case["layers"]):
        p = f"model.layers.{i}"
        shapes.update({f"{p}.input_layernorm.weight": ((s["width"],), "vector"), f"{p}.post_attention_layernorm.weight": ((s["width"],), "vector")})
        for part in _dense_shapes(s, p):
            shapes.update(part)
    return shapes


def _expert_shapes(case):
    s = DESIGN[case["size"]]
    w, inner = s["width"], s["ff"] // 8
    shapes = {"x.router.weight": ((EXPERTS, w), "matrix"), "x.router.bias": ((EXPERTS,), "bias")}
    for e in range(EXPERTS):
        shapes.update({f"x.experts.{e}.gate_proj.weight": ((inner, w), "matrix"), f"x.experts.{e}.up_proj.weight": ((inner, w), "matrix"),
                       f"x.experts.{e}.down_proj.weight": ((w, inner), "matrix")})
    return shapes


def _latent_shapes(case):
    s, m = DESIGN[case["size"]], LATENT
    w, H = s["width"], s["heads"]
    return {"x.q_proj.weight": ((H * (m["dim"] + m["rot"]), w), "matrix"), "x.kv_down_proj.weight": ((m["rank"] + m["rot"], w), "matrix"),
            "x.kv_norm.weight": ((m["rank"],), "vector"), "x.k_up_proj.weight": ((H * m["dim"], m["rank"]), "matrix"),
            "x.v_up_proj.weight": ((H * m["vdim"], m["rank"]), "matrix"), "x.gate_proj.weight": ((H, w), "matrix"),
            "x.o_proj.weight": ((w, H * m["vdim"]), "matrix")}


def _recurrence_shapes(case):
    w = DESIGN[case["size"]]["width"]
    H, d, e = w // 128, LINEAR["dim"], LINEAR["vdim"]
    shapes = {"x.q_proj.weight": ((H * d, w), "matrix"), "x.k_proj.weight": ((H * d, w), "matrix"), "x.v_proj.weight": ((H * e, w), "matrix"),
              "x.g_proj.weight": ((H * e, w), "matrix"), "x.o_proj.weight": ((w, H * e), "matrix")}
    if case["form"] == "gated_linear_attention":
        shapes.update({"x.norm.weight": ((e,), "vector"), "x.a_down.weight": ((LINEAR["rank"], w), "matrix"),
                       "x.a_up.weight": ((H * d, LINEAR["rank"]), "matrix"), "x.a_up.bias": ((H * d,), "bias")})
    return shapes


def _retention_decays(heads):
    return [1.0 - 2.0 ** (-5.0 - 7.0 * i / heads) for i in range(heads)]


def _contexts(case):
    """Tokens in the cache after the step, request by request: the first request has all of `context`, later ones up to a quarter
    less (requests that came later); a prompt's requests bring `tokens` each."""
    n, context, tokens = case["requests"], case["context"], case["tokens"]
    return [max(tokens, context - (i * context) // (4 * n)) for i in range(n)]


class _Step:
    """One step's facts: `tokens` of each request, contexts of `lengths` after it, pages scattered over the pool."""

    def __init__(self, draws, lengths, tokens):
        n = len(lengths)
        pages = [-(-length // PAGE) for length in lengths]
        self.pages = sum(pages) + 3
        order = torch.randperm(self.pages, generator=draws.gen, device=DEVICE)
        table = torch.full((n, max(pages)), -1, dtype=torch.int64, device=DEVICE)
        at = 0
        for i, count in enumerate(pages):
            table[i, :count] = order[at:at + count]
            at += count
        self.lengths, self.starts, self.tokens, self.table = lengths, [length - tokens for length in lengths], tokens, table
        self.positions = torch.cat([torch.arange(s, s + tokens, device=DEVICE) for s in self.starts])
        self.seq = torch.arange(n, device=DEVICE).repeat_interleave(tokens)
        self.slots = table[self.seq, self.positions // PAGE] * PAGE + self.positions % PAGE

    def context(self):
        n, t = len(self.lengths), self.tokens
        i32 = lambda x: torch.as_tensor(x, device=DEVICE).to(torch.int32)      # noqa: E731
        tiles = i32([[i, i, 1, 0] for i in range(n)]) if t == 1 else None
        return StepContext(num_tokens=n * t, num_sequences=n, token_ids=i32([0] * (n * t)), positions=i32(self.positions), seq_of_token=i32(self.seq),
                           q_start=i32([i * t for i in range(n + 1)]), context_len=i32(self.lengths), state_slots=i32(list(range(n))), want_rows=None,
                           block_tables=[i32(self.table)], slots=[i32(self.slots)], host_q_start=[i * t for i in range(n + 1)],
                           host_start_pos=list(self.starts), host_state_slots=list(range(n)), max_query_len=t, max_context_len=max(self.lengths),
                           fresh=[s == 0 for s in self.starts], decode_tiles=tiles, real_sequences=n)

    def rows_of(self, cache, i):
        """Request i's cached rows in order: [its length, heads, d]."""
        at = torch.arange(self.lengths[i], device=DEVICE)
        return cache[self.table[i, at // PAGE], :, at % PAGE]


def _tokens_of(case, seed):
    """Token ids of every request of a step: (prompt so far and the step's tokens, how many of them the step brings)."""
    draws = _Draws(seed + 1)
    lengths = [(max(1, case["context"] - (i * case["context"]) // (4 * case["decodes"])), 1) for i in range(case["decodes"])]
    if case["portion"]:
        lengths.append((case["behind"] + case["portion"], case["portion"]))
    return [(draws.whole(0, VOCAB, (length,)).tolist(), new) for length, new in lengths]


def _layer_inputs(case, seed):
    """Weights, hidden rows, step and cache of a layer case, from the seed alone."""
    kind, draws = case["kind"], _Draws(seed)
    dtype = TYPES[case.get("dtype", "bfloat16")]
    got = {"step": None}
    if kind == "attention":
        s = DENSE[case["shape"]]
        got["weights"] = draws.weights(_dense_shapes(s, "x")[0], dtype)
        got["step"] = step = _Step(draws, _contexts(case), case["tokens"])
        rows, width = case["requests"] * case["tokens"], s["width"]
        got["k"] = draws.normal((step.pages, s["kv_heads"], PAGE, HEAD), dtype=dtype)
        got["v"] = draws.normal((step.pages, s["kv_heads"], PAGE, HEAD), dtype=dtype)
    elif kind == "mlp":
        s = DENSE[case["shape"]]
        got["weights"] = draws.weights(_dense_shapes(s, "x")[1], dtype)
        rows, width = case["rows"], s["width"]
    elif kind == "experts":
        got["weights"] = draws.weights(_expert_shapes(case), dtype)
        rows, width = case["rows"], DESIGN[case["size"]]["width"]
    elif kind == "latent":
        got["weights"] = draws.weights(_latent_shapes(case), dtype)
        got["step"] = step = _Step(draws, _contexts(case), case["tokens"])
        rows, width = case["requests"] * case["tokens"], DESIGN[case["size"]]["width"]
        got["k"] = draws.normal((step.pages, 1, PAGE, LATENT["rank"] + LATENT["rot"]), dtype=dtype)
    else:
        got["weights"] = draws.weights(_recurrence_shapes(case), dtype)
        got["step"] = _Step(draws, _contexts(case), case["tokens"])
        rows, width = case["requests"] * case["tokens"], DESIGN[case["size"]]["width"]
        H = width // 128
        got["state"] = draws.normal((case["requests"], H * LINEAR["dim"] * LINEAR["vdim"]), 0.5)
    got["h"] = draws.normal((rows, width), dtype=dtype)       # a normed row: unit mean square
    return got


def _part(case):
    kind = case["kind"]
    if kind == "attention":
        s = DENSE[case["shape"]]
        norm = PartSpec("rmsnorm", {"width": HEAD, "eps": EPS})
        return MIXERS.build(PartSpec("gqa_attention", {"width": s["width"], "num_heads": s["heads"], "num_kv_heads": s["kv_heads"], "head_dim": HEAD,
                                                       "q_norm": norm, "k_norm": norm,
                                                       "position": PartSpec("rope", {"head_dim": HEAD, "theta": THETA})}), "x.self_attn")
    if kind == "mlp":
        s = DENSE[case["shape"]]
        return FEED_FORWARDS.build(PartSpec("swiglu", {"width": s["width"], "inner": s["ff"]}), "x.mlp")
    s = DESIGN[case["size"]]
    if kind == "experts":
        return FEED_FORWARDS.build(PartSpec("routed_experts", {"width": s["width"], "experts": EXPERTS, "top": TOP, "inner": s["ff"] // 8,
                                                               "router_bias": True, "float32_out": True}), "x")
    if kind == "latent":
        m = LATENT
        position = PartSpec("yarn_rope", {"rotary_dim": m["rot"], "theta": THETA, "factor": m["factor"], "original": m["original"], "fast": m["fast"],
                                          "slow": m["slow"]})
        return MIXERS.build(PartSpec("latent_attention", {"width": s["width"], "num_heads": s["heads"], "head_dim": m["dim"], "rotary_head_dim": m["rot"],
                                                          "value_dim": m["vdim"], "latent_dim": m["rank"], "scale": (m["dim"] + m["rot"]) ** -0.5,
                                                          "eps": EPS, "position": position, "window": m["window"], "output_gate": True}), "x")
    H = s["width"] // 128
    common = {"width": s["width"], "heads": H, "head_dim": LINEAR["dim"], "value_dim": LINEAR["vdim"], "eps": EPS}
    if case["form"] == "retention":
        return MIXERS.build(PartSpec("retention", dict(common, decay=_retention_decays(H),
                                                       position=PartSpec("rope", {"head_dim": LINEAR["dim"], "theta": LINEAR["base"]}))), "x")
    return MIXERS.build(PartSpec("gated_linear_attention", dict(common, tau=LINEAR["tau"], decay_rank=LINEAR["rank"])), "x")


def _sampling(case, seed):
    """Logits and every row's parameters: most rows with a temperature and top-p, some with top-k, some greedy."""
    draws = _Draws(seed)
    rows = case["rows"]
    logits = draws.normal((rows, case["vocab"]), 2.5)
    params = []
    for i in range(rows):
        kw = [dict(temperature=0.8, top_p=0.95), dict(temperature=0.7, top_k=50, top_p=0.9), dict(temperature=1.0), dict(temperature=0.6, top_k=20),
              dict(temperature=1.0, top_p=0.9), dict(temperature=0.0)][i % 6]
        params.append(SamplingParams(seed=int(seed) * 1009 + i, **kw))
    return logits, params, [(i * 37) % 200 for i in range(rows)]


# ---------------------------------------------------------------------------------------------- before, during
def prepare(case, seed):
    configure_library_products()
    kind = case["kind"]
    if kind == "sample":
        logits, params, draws = _sampling(case, seed)
        return {"kind": kind, "sampler": Sampler(DEVICE), "logits": logits, "params": params, "draws": draws}
    if kind == "step":
        s = DENSE[case["shape"]]
        config = config_from_dict(dict(model_type="qwen3", architectures=["Qwen3ForCausalLM"], hidden_size=s["width"], intermediate_size=s["ff"],
                                       num_hidden_layers=case["layers"], num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"],
                                       head_dim=HEAD, vocab_size=VOCAB, max_position_embeddings=40960, rms_norm_eps=EPS, rope_theta=THETA,
                                       tie_word_embeddings=s["tied"], hidden_act="silu", eos_token_id=VOCAB - 1))
        tensors = _Draws(seed).weights(_model_shapes(case), torch.bfloat16)
        requests = _tokens_of(case, seed)
        pages = sum(-(-len(tokens) // PAGE) for tokens, _ in requests) + 8
        limits = RuntimeConfig(max_seq_len=8192, page_size=PAGE, prefill_budget=8192, max_running=len(requests))
        runner = ModelRunner(config, tensors, Runtime(DEVICE, torch.bfloat16, PAGE), limits, num_pages=pages)
        # the requests' earlier tokens, a few thousand rows a step; no logits are wanted
        earlier, rows, work = [], 0, []
        for r, (tokens, new) in enumerate(requests):
            runner.cache.open(r)
            runner.cache.extend(r, len(tokens))
            if len(tokens) > new:
                earlier.append(SequenceStep(r, tokens[:-new], 0, []))
                rows += len(tokens) - new
            if rows > 8192 or (r + 1 == len(requests) and rows):
                runner.forward(earlier)
                earlier, rows = [], 0
            work.append(SequenceStep(r, tokens[-new:], len(tokens) - new, [new - 1]))
        torch.cuda.synchronize()
        return {"kind": kind, "runner": runner, "work": work}
    got = _layer_inputs(case, seed)
    part = _part(case)
    part.bind(got["weights"], Runtime(DEVICE, TYPES[case.get("dtype", "bfloat16")], PAGE))
    state = {"kind": kind, "part": part, "h": got["h"], "ctx": None, "cache": None}
    if got["step"] is not None:
        state["ctx"] = got["step"].context()
        state["cache"] = CacheEntry(group=0, k=got.get("k"), v=got.get("v"), state=got.get("state"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "sample":
        return state["sampler"].launch(state["logits"], state["params"], state["draws"]).tokens
    with torch.no_grad():
        if kind == "step":
            return state["runner"].forward(state["work"])
        if kind in ("mlp", "experts"):
            return state["part"].forward(state["h"], state["ctx"])
        cache = state["cache"]
        y = state["part"].forward(state["h"], state["ctx"], cache)
        if kind == "recurrence":
            return y, cache.state
        return (y, cache.k, cache.v) if kind == "attention" else (y, cache.k)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(case, window=0):
    """(query, key) pairs of a step's attention."""
    total = 0
    for length in _contexts(case):
        for p in range(length - case["tokens"], length):
            total += min(p + 1, window) if window else p + 1
    return total


def _cached(case, window=0):
    """Cached tokens that the step reads."""
    return sum(min(length, case["tokens"] + window - 1) if window else length for length in _contexts(case))


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 4 * case["rows"] * case["vocab"]}
    if kind == "step":
        s = DENSE[case["shape"]]
        q, kv = s["heads"] * HEAD, s["kv_heads"] * HEAD
        per_layer = (q + 2 * kv) * s["width"] + s["width"] * q + 3 * s["ff"] * s["width"]
        requests = [(max(1, case["context"] - (i * case["context"]) // (4 * case["decodes"])), 1) for i in range(case["decodes"])]
        if case["portion"]:
            requests.append((case["behind"] + case["portion"], case["portion"]))
        rows, cached = sum(n for _, n in requests), sum(length for length, _ in requests)
        pairs = sum(sum(range(length - n + 1, length + 1)) for length, n in requests)
        return {"bytes": 2 * (case["layers"] * per_layer + VOCAB * s["width"]) + 2 * 2 * kv * case["layers"] * cached + 4 * VOCAB * len(requests),
                "flops": 2 * rows * case["layers"] * per_layer + 2 * len(requests) * VOCAB * s["width"] + 4 * q * case["layers"] * pairs}
    if kind == "experts":
        s = DESIGN[case["size"]]
        w, inner, rows = s["width"], s["ff"] // 8, case["rows"]
        hit = EXPERTS * (1 - (1 - TOP / EXPERTS) ** rows)               # experts that some row chooses
        return {"bytes": 2 * (hit * 3 * w * inner + EXPERTS * w + rows * w) + 4 * rows * w, "flops": 2 * rows * (TOP * 3 * w * inner + EXPERTS * w)}
    if kind == "mlp":
        s = DENSE[case["shape"]]
        element, params = (2 if case["dtype"] == "bfloat16" else 4), 3 * s["ff"] * s["width"]
        return {"bytes": element * (params + 2 * case["rows"] * s["width"]), "flops": 2 * case["rows"] * params}
    rows = case["requests"] * case["tokens"]
    if kind == "attention":
        s = DENSE[case["shape"]]
        element, q, kv = (2 if case["dtype"] == "bfloat16" else 4), s["heads"] * HEAD, s["kv_heads"] * HEAD
        params = (2 * q + 2 * kv) * s["width"]
        return {"bytes": element * (params + 2 * rows * s["width"] + 2 * kv * _cached(case)), "flops": 2 * rows * params + 4 * q * _pairs(case)}
    s = DESIGN[case["size"]]
    if kind == "latent":
        m, w, H = LATENT, s["width"], s["heads"]
        params = (H * (m["dim"] + m["rot"]) + m["rank"] + m["rot"] + H + H * m["vdim"]) * w + H * (m["dim"] + m["vdim"]) * m["rank"]
        pair = min(2 * (m["dim"] + m["rot"] + m["vdim"]), 2 * (2 * m["rank"] + m["rot"])) * H      # keys and values made, or in the latent space
        return {"bytes": 2 * (params + 2 * rows * w + (m["rank"] + m["rot"]) * _cached(case, m["window"])),
                "flops": 2 * rows * params + pair * _pairs(case, m["window"])}
    w = s["width"]
    H, d, e = w // 128, LINEAR["dim"], LINEAR["vdim"]
    params = w * H * (2 * d + 3 * e) + (LINEAR["rank"] * (w + H * d) if case["form"] == "gated_linear_attention" else 0)
    return {"bytes": 2 * (params + rows * w) + 4 * rows * w + 8 * case["requests"] * H * d * e, "flops": 2 * rows * params + 5 * rows * H * d * e}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return {"differ": 0.1}                         # a draw that falls on the edge of two tokens
    if case.get("dtype") == "float32":
        # about four times the error against 64 bits: 1.7e-6 with hundreds of keys, 1.2e-5 for a token behind 4,000 keys
        return {"rel": 5e-5, "max": 1e-3} if kind == "attention" else {"rel": 1e-5, "max": 2e-4}
    if kind == "step":
        return {"rel": 5e-2, "max": 0.4}               # 1.5e-2 against 64 bits: a rounding travels through four layers
    return {"rel": 1.5e-2, "max": 0.1}                 # 3.5e-3 to 4.1e-3 against 64 bits


# ---------------------------------------------------------------------------------------------- in 64 bits, without the engine
def _rms(x, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight.double()


def _mm(x, weight):
    return x @ weight.double().t()


def _turn(x, angles, magnitude=1.0):
    """Split halves of the last axis turned by angles [rows, half]; x [rows, heads, dims]."""
    half = x.shape[-1] // 2
    c, s = (torch.cos(angles) * magnitude)[:, None], (torch.sin(angles) * magnitude)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _angles(positions, dims, base):
    j = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    frequencies = (1.0 / torch.pow(torch.tensor(base, dtype=torch.float64, device=DEVICE), 2.0 * j / dims).float()).double()
    return positions.double()[:, None] * frequencies[None]


def _stretched_angles(positions):
    m, half = LATENT, LATENT["rot"] // 2

    def pair_of(turns):
        return m["rot"] * math.log(m["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(THETA))

    lo, hi = max(math.floor(pair_of(m["fast"])), 0), min(math.ceil(pair_of(m["slow"])), m["rot"] - 1)
    out = []
    for i in range(half):
        f, ramp = THETA ** (-2.0 * i / m["rot"]), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        out.append(f / m["factor"] * ramp + f * (1.0 - ramp))
    frequencies = torch.tensor(out, dtype=torch.float64, device=DEVICE).float().double()
    return positions.double()[:, None] * frequencies[None], 0.1 * math.log(m["factor"]) + 1.0


def _attend(q, k, v, start, scale, window=0):
    """q [t, d], k [n, d], v [n, e]: the rows' positions are start, start + 1, ..."""
    scores = q @ k.t() * scale
    at = torch.arange(start, start + q.shape[0], device=DEVICE)[:, None]
    key = torch.arange(k.shape[0], device=DEVICE)[None]
    seen = key <= at
    if window:
        seen &= key > at - window
    return torch.softmax(scores.masked_fill_(~seen, -math.inf), dim=-1) @ v


def _dense_heads(h, w, a, s, positions):
    rows, heads, kv = h.shape[0], s["heads"], s["kv_heads"]
    angles = _angles(positions, HEAD, THETA)
    q = _turn(_rms(_mm(h, w[f"{a}.q_proj.weight"]).view(rows, heads, HEAD), w[f"{a}.q_norm.weight"]), angles)
    k = _turn(_rms(_mm(h, w[f"{a}.k_proj.weight"]).view(rows, kv, HEAD), w[f"{a}.k_norm.weight"]), angles)
    return q, k, _mm(h, w[f"{a}.v_proj.weight"]).view(rows, kv, HEAD)


def _dense_mlp(h, w, m):
    z = _mm(h, w[f"{m}.gate_proj.weight"])
    return _mm(z * torch.sigmoid(z) * _mm(h, w[f"{m}.up_proj.weight"]), w[f"{m}.down_proj.weight"])


def _exact_step(case, seed):
    s, w = DENSE[case["shape"]], _Draws(seed).weights(_model_shapes(case), torch.bfloat16)
    logits = []
    for tokens, _ in _tokens_of(case, seed):
        x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)].double()
        positions = torch.arange(len(tokens), device=DEVICE)
        for i in range(case["layers"]):
            p = f"model.layers.{i}"
            q, k, v = _dense_heads(_rms(x, w[f"{p}.input_layernorm.weight"]), w, f"{p}.self_attn", s, positions)
            group = s["heads"] // s["kv_heads"]
            if i + 1 == case["layers"]:          # only the last row's logits are wanted
                x, q = x[-1:], q[-1:]
            start = len(tokens) - q.shape[0]
            out = torch.stack([_attend(q[:, j], k[:, j // group], v[:, j // group], start, HEAD ** -0.5) for j in range(s["heads"])], dim=1)
            x = x + _mm(out.reshape(len(x), -1), w[f"{p}.self_attn.o_proj.weight"])
            x = x + _dense_mlp(_rms(x, w[f"{p}.post_attention_layernorm.weight"]), w, f"{p}.mlp")
        head = w["model.embed_tokens.weight" if s["tied"] else "lm_head.weight"]
        last = _rms(x[-1:], w["model.norm.weight"])
        logits.append(torch.cat([_mm(last, part) for part in head.split(16384)], dim=1))
    return torch.cat(logits)


def _exact_attention(case, got):
    s, w, step, n = DENSE[case["shape"]], got["weights"], got["step"], case["tokens"]
    group = s["heads"] // s["kv_heads"]
    q, k, v = _dense_heads(got["h"].double(), w, "x.self_attn", s, step.positions)
    k_cache, v_cache = got["k"].double(), got["v"].double()
    page, offset = step.slots // PAGE, step.slots % PAGE
    k_cache[page, :, offset] = k
    v_cache[page, :, offset] = v
    out = torch.empty_like(q)
    for i, start in enumerate(step.starts):
        keys, values = step.rows_of(k_cache, i), step.rows_of(v_cache, i)
        for j in range(s["heads"]):
            out[i * n:(i + 1) * n, j] = _attend(q[i * n:(i + 1) * n, j], keys[:, j // group], values[:, j // group], start, HEAD ** -0.5)
    return _mm(out.reshape(len(out), -1), w["x.self_attn.o_proj.weight"]), k_cache, v_cache


def _exact_experts(case, got):
    w, h = got["weights"], got["h"].double()
    z = _mm(h, w["x.router.weight"]) + w["x.router.bias"].double()
    chosen = torch.topk(z, TOP, dim=1).indices
    share = torch.softmax(torch.gather(z, 1, chosen), dim=1)
    out = torch.zeros_like(h)
    for e in range(EXPERTS):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            out[rows] += _dense_mlp(h[rows], w, f"x.experts.{e}") * share[rows, place][:, None]
    return out


def _exact_latent(case, got):
    s, m, w, step, n = DESIGN[case["size"]], LATENT, got["weights"], got["step"], case["tokens"]
    H, h = s["heads"], got["h"].double()
    angles, magnitude = _stretched_angles(step.positions)
    q = _mm(h, w["x.q_proj.weight"]).view(len(h), H, m["dim"] + m["rot"])
    q_rot = _turn(q[..., m["dim"]:], angles, magnitude)
    down = _mm(h, w["x.kv_down_proj.weight"])
    latent = _rms(down[:, :m["rank"]], w["x.kv_norm.weight"])
    k_rot = _turn(down[:, None, m["rank"]:], angles, magnitude)[:, 0]
    cache = got["k"].double()
    cache[step.slots // PAGE, 0, step.slots % PAGE] = torch.cat([latent, k_rot], dim=1)
    up_k, up_v = w["x.k_up_proj.weight"].double().view(H, m["dim"], -1), w["x.v_up_proj.weight"].double().view(H, m["vdim"], -1)
    out = torch.empty((len(h), H, m["vdim"]), dtype=torch.float64, device=DEVICE)
    for i, start in enumerate(step.starts):
        rows = step.rows_of(cache, i)[:, 0]
        c, turned = rows[:, :m["rank"]], rows[:, m["rank"]:]
        part = slice(i * n, (i + 1) * n)
        for j in range(H):
            out[part, j] = _attend(torch.cat([q[part, j, :m["dim"]], q_rot[part, j]], dim=1), torch.cat([c @ up_k[j].t(), turned], dim=1),
                                   c @ up_v[j].t(), start, (m["dim"] + m["rot"]) ** -0.5, m["window"])
    out = out * torch.sigmoid(_mm(h, w["x.gate_proj.weight"]))[..., None]
    return _mm(out.reshape(len(h), -1), w["x.o_proj.weight"]), cache


def _exact_recurrence(case, got):
    w, step, n, h = got["weights"], got["step"], case["tokens"], got["h"].double()
    H, d, e, rows = DESIGN[case["size"]]["width"] // 128, LINEAR["dim"], LINEAR["vdim"], got["h"].shape[0]
    q, k, v = (_mm(h, w[f"x.{name}_proj.weight"]).view(rows, H, size) for name, size in (("q", d), ("k", d), ("v", e)))
    if case["form"] == "retention":
        angles = _angles(step.positions, d, LINEAR["base"])
        q, k = _turn(q, angles), _turn(k, angles)
        decay = torch.tensor(_retention_decays(H), dtype=torch.float32, device=DEVICE).double()[None, :, None].expand(rows, H, d)
        norm = None
    else:
        low = _mm(_mm(h, w["x.a_down.weight"]), w["x.a_up.weight"]) + w["x.a_up.bias"].double()
        decay = torch.exp(torch.nn.functional.logsigmoid(low) / LINEAR["tau"]).view(rows, H, d)
        norm = w["x.norm.weight"]
    state = got["state"].double().view(-1, H, d, e)
    o = torch.empty((rows, H, e), dtype=torch.float64, device=DEVICE)
    # the requests walk side by side: [requests, H, d, e]
    S = torch.stack([state[i] if start else torch.zeros_like(state[i]) for i, start in enumerate(step.starts)])
    rows_at = torch.arange(case["requests"], device=DEVICE) * n
    for t in range(n):
        at = rows_at + t
        S = S * decay[at][..., None] + k[at][..., None] * v[at][:, :, None, :]
        o[at] = (S * q[at][..., None]).sum(2)
    g = _mm(h, w["x.g_proj.weight"])
    y = _rms(o * d ** -0.5, norm).reshape(rows, -1) * g * torch.sigmoid(g)
    return _mm(y, w["x.o_proj.weight"]), S.reshape(case["requests"], -1)


def _draw_u(seed, index):
    """u in [0, 1) of a request's draw: the splitmix64 finaliser over (seed, draw index)."""
    mask = (1 << 64) - 1
    z = (seed + 0x9E3779B97F4A7C15 * (index + 1)) & mask
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
    return ((z ^ (z >> 31)) >> 40) / 16777216.0


def _exact_sample(case, seed):
    logits, params, draws = _sampling(case, seed)
    tokens = []
    for row, p, index in zip(logits.double(), params, draws):
        if p.temperature == 0.0 or p.top_k == 1:
            tokens.append(int(torch.argmax(row)))
            continue
        order = torch.sort(row, descending=True, stable=True).indices
        if p.top_k:
            order = order[:p.top_k]
        weight = torch.exp((row[order] - row[order[0]]) / p.temperature)
        if p.top_p < 1.0:
            reached = torch.cumsum(weight, 0) >= p.top_p * weight.sum()
            order = order[:int(torch.argmax(reached.int())) + 1]
        kept = torch.sort(order).values
        running = torch.cumsum(torch.exp((row[kept] - row.max()) / p.temperature), 0)
        at = int(torch.searchsorted(running, _draw_u(p.seed, index) * running[-1], right=True))
        tokens.append(int(kept[min(at, len(kept) - 1)]))
    return torch.tensor(tokens, dtype=torch.int32, device=DEVICE)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "sample":
            return _exact_sample(case, seed)
        if kind == "step":
            return _exact_step(case, seed)
        got = _layer_inputs(case, seed)
        if kind == "mlp":
            return _dense_mlp(got["h"].double(), got["weights"], "x.mlp")
        return {"attention": _exact_attention, "experts": _exact_experts, "latent": _exact_latent, "recurrence": _exact_recurrence}[kind](case, got)
