"""The work this framework is used for, as cases whose time and outputs can be measured.

Three families, each through the entry points that a program calls:

* "llama": steps of the Llama decoder at the layer sizes of the 1B, 8B and 13B shapes that the repository's
  configurations and benchmark use: captured decode steps (`ModelRunner.decode_step`), whole prompts
  (`ModelRunner.step`), and a prompt's portion beside single tokens (`ModelRunner.prepare` and `Model.forward`, which
  is what `ModelRunner.step` does before it moves the lengths on). bfloat16, and the float32 engine.
* "delta": the recurrent mixers of the Bunosun ("channel") and Rerilorn ("general") decoders, over prompt portions of
  one or several requests, and over single tokens inside a CUDA graph, as the engine runs decode steps.
* "experts": the routed feed-forward of the Bunosun, Puvirax, Pakarax and Zemarax decoders, over prompts and over
  single tokens inside a CUDA graph.

The decoders whose layers a case runs are deeper in real use; a few layers (and the 13B shape's vocabulary) are enough
to keep the device busy and let three copies of the weights stay on the card.
"""

from __future__ import annotations

import math

import torch

from pulsarlm_b200.cache.manager import CacheManager, StateBinding
from pulsarlm_b200.config.registry import read_model_config
from pulsarlm_b200 import models as _models  # noqa: F401  (registers the architectures)
from pulsarlm_b200.engine.runner import ModelRunner, StepEntry
from pulsarlm_b200.models.model import HostStep, Model, StepBatch
from pulsarlm_b200.parts.registry import BuildContext, build_part
from pulsarlm_b200.parts.spec import PartSpec
from pulsarlm_b200.sampling.params import SamplingParams

DEV = "cuda:0"
PAGE = 16
VOCAB = 32000
EPS = 1e-5
UNIT_EPS = 1e-6
TAPS = 4
DECAY_SCALE = math.exp(-0.5)

SHAPES = {
    "1b": {"hidden": 2048, "heads": 32, "kv": 8, "dim": 64, "ff": 8192, "theta": 500000.0, "factor": 32.0, "tied": True},
    "8b": {"hidden": 4096, "heads": 32, "kv": 8, "dim": 128, "ff": 14336, "theta": 500000.0, "factor": 8.0, "tied": False},
    "13b": {"hidden": 5120, "heads": 40, "kv": 40, "dim": 128, "ff": 13824, "theta": 10000.0, "factor": None, "tied": False},
}


# ------------------------------------------------------------------------------------------------ the cases

def _llama(name, shape, layers, mode, dtype="bfloat16", **sizes):
    return {"name": name, "family": "llama", "shape": shape, "layers": layers, "mode": mode, "dtype": dtype, **sizes}


def listed():
    return [
        # One user's chat on the small model, one token a step: launches and latency count.
        _llama("decode_1b_b1", "1b", 8, "decode", batch=1, context=1000, uneven=False),
        # The headline decode step: eight users of the 8B shape in the middle of their answers.
        _llama("decode_8b_b8", "8b", 4, "decode", batch=8, context=2048, uneven=False),
        # A full batch on the small model with histories of all lengths, as a server's requests have.
        _llama("decode_1b_b64", "1b", 4, "decode", batch=64, context=2048, uneven=True),
        # A whole prompt of 2,048 tokens in one step on the 8B shape: the time to the first token.
        _llama("prefill_8b_2048", "8b", 2, "prefill", tokens=2048, history=0),
        # A serving step: a portion of a longer prompt beside the single tokens of the requests that are being answered.
        _llama("mixed_1b_512", "1b", 4, "mixed", batch=40, context=1500, uneven=True, tokens=512, history=700),
        # The float32 engine, which answers are checked against: a prompt of odd length, and single tokens.
        _llama("float32_prefill", "1b", 2, "prefill", "float32", tokens=509, history=0),
        _llama("float32_decode_b8", "1b", 2, "decode", "float32", batch=8, context=600, uneven=False),
        # Recurrent layers over a whole prompt, over the portions of several requests, and over a full batch's tokens.
        {"name": "channel_delta_prompt", "family": "delta", "kind": "channel", "width": 2048, "dim": 64, "vdim": 64,
         "entries": 1, "tokens": 2048, "graph": False},
        {"name": "general_delta_portions", "family": "delta", "kind": "general", "width": 2048, "dim": 64, "vdim": 64,
         "entries": 5, "tokens": 1283, "graph": False},
        {"name": "channel_delta_decode", "family": "delta", "kind": "channel", "width": 2048, "dim": 64, "vdim": 64,
         "entries": 64, "tokens": 64, "graph": True},
        # Routed experts over a prompt's portion and over eight users' tokens.
        {"name": "experts_prompt", "family": "experts", "width": 2048, "experts": 32, "top": 4, "groups": 4, "keep": 2,
         "ff": 1024, "shared": 1024, "unit": "gated_silu", "tokens": 2048, "graph": False},
        {"name": "experts_decode", "family": "experts", "width": 2048, "experts": 32, "top": 4, "groups": 4, "keep": 2,
         "ff": 1024, "shared": 1024, "unit": "gated_silu", "tokens": 8, "graph": True},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    what = rng.choice(["decode", "decode", "prefill", "mixed", "float32", "delta", "delta", "delta_decode", "experts",
                       "experts_decode"])
    if what == "decode":
        shape = rng.choice(["1b", "8b", "13b"])
        batch = _log(rng, 1, 64)
        most = {"1b": 6000, "8b": 4000, "13b": 1500}[shape]
        return _llama_drawn(shape, {"1b": rng.randint(2, 8), "8b": 2, "13b": 2}[shape], "decode", batch=batch,
                            context=_log(rng, 64, most), uneven=rng.random() < 0.5)
    if what == "prefill":
        shape = rng.choice(["1b", "8b", "13b"])
        return _llama_drawn(shape, {"1b": 3, "8b": 2, "13b": 2}[shape], "prefill", tokens=_log(rng, 17, 2000),
                            history=rng.choice([0, 0, rng.randint(1, 2000)]))
    if what == "mixed":
        return _llama_drawn("1b", rng.randint(2, 4), "mixed", batch=_log(rng, 1, 63), context=_log(rng, 64, 3000),
                            uneven=True, tokens=_log(rng, 16, 512), history=rng.randint(0, 3000))
    if what == "float32":
        if rng.random() < 0.5:
            return _llama_drawn("1b", 1, "prefill", "float32", tokens=_log(rng, 9, 500), history=0)
        return _llama_drawn("1b", 1, "decode", "float32", batch=_log(rng, 1, 32), context=_log(rng, 30, 1000), uneven=True)
    if what in ("delta", "delta_decode"):
        kind = rng.choice(["channel", "general"])
        dim = rng.choice([64, 64, 64, 128, 32])
        vdim = dim if kind == "general" else rng.choice([dim, 64, 128])
        case = {"family": "delta", "kind": kind, "width": 128 * rng.randint(4, 24), "dim": dim, "vdim": vdim}
        if what == "delta":
            entries = rng.choice([1, 1, 2, 3, rng.randint(4, 12)])
            return {**case, "entries": entries, "tokens": entries * 2 + _log(rng, 20, 2000), "graph": False}
        entries = _log(rng, 1, 64)
        return {**case, "entries": entries, "tokens": entries, "graph": True}
    experts = rng.choice([8, 16, 32, 64])
    groups = rng.choice([1, 4])
    case = {"family": "experts", "width": 128 * rng.randint(4, 24), "experts": experts, "top": rng.choice([1, 2, 4]),
            "groups": groups, "keep": groups // 2 or 1, "ff": 64 * rng.randint(4, 20), "shared": rng.choice([0, 1024]),
            "unit": rng.choice(["gated_silu", "gated_silu", "relu2", "gelu"])}
    if what == "experts":
        return {**case, "tokens": _log(rng, 48, 2048), "graph": False}
    return {**case, "tokens": _log(rng, 1, 64), "graph": True}


def _llama_drawn(*a, **k):
    case = _llama(None, *a, **k)
    del case["name"]
    return case


# ------------------------------------------------------------------------------------------------ inputs

def _generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _normal(gen, shape, std, dtype, mean=0.0):
    x = torch.empty(shape, dtype=dtype, device=DEV)
    return x.normal_(mean, std, generator=gen)


def _spread(total, count):
    """`count` lengths of all sizes, from one token up, that sum to `total`."""
    weights = [(i + 1) ** 2 for i in range(count)]
    lengths = [1 + (total - count) * w // sum(weights) for w in weights]
    lengths[-1] += total - sum(lengths)
    return lengths


def _contexts(case):
    """Tokens that each single-token request of a step holds before it."""
    b, c = case.get("batch", 0), case.get("context", 0)
    if not case.get("uneven"):
        return [c] * b
    return [max(1, int(c * (0.15 + 1.7 * ((7 * i + 3) % b) / max(1, b - 1)))) if b > 1 else c for i in range(b)]


def _llama_config(case):
    s = SHAPES[case["shape"]]
    rope = None if s["factor"] is None else {"rope_type": "llama3", "factor": s["factor"], "low_freq_factor": 1.0,
                                             "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": case["layers"], "hidden_size": s["hidden"],
            "num_attention_heads": s["heads"], "num_key_value_heads": s["kv"], "head_dim": s["dim"],
            "intermediate_size": s["ff"], "vocab_size": VOCAB, "rms_norm_eps": EPS, "rope_theta": s["theta"],
            "rope_scaling": rope, "tie_word_embeddings": s["tied"], "max_position_embeddings": 131072}


def _llama_weights(case, seed):
    """Every tensor by its checkpoint name, N(0, 0.02) and norms around one, as the benchmark's random models."""
    s, dtype = SHAPES[case["shape"]], getattr(torch, case["dtype"])
    h, q, kv, ff = s["hidden"], s["heads"] * s["dim"], s["kv"] * s["dim"], s["ff"]
    gen = _generator(seed, 1)
    out = {"model.embed_tokens.weight": _normal(gen, (VOCAB, h), 0.02, dtype)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (q, h)), ("self_attn.k_proj", (kv, h)), ("self_attn.v_proj", (kv, h)),
                            ("self_attn.o_proj", (h, q)), ("mlp.gate_proj", (ff, h)), ("mlp.up_proj", (ff, h)),
                            ("mlp.down_proj", (h, ff))):
            out[p + name + ".weight"] = _normal(gen, shape, 0.02, dtype)
        out[p + "input_layernorm.weight"] = _normal(gen, (h,), 0.02, dtype, 1.0)
        out[p + "post_attention_layernorm.weight"] = _normal(gen, (h,), 0.02, dtype, 1.0)
    out["model.norm.weight"] = _normal(gen, (h,), 0.02, dtype, 1.0)
    if not s["tied"]:
        out["lm_head.weight"] = _normal(gen, (VOCAB, h), 0.02, dtype)
    return out


def _llama_entries(case):
    """(tokens held before the step, tokens of the step) of every request, singles first."""
    out = [(c, 1) for c in _contexts(case)] if case["mode"] != "prefill" else []
    return out + ([(case["history"], case["tokens"])] if case["mode"] != "decode" else [])


def _llama_tokens(case, seed):
    gen = torch.Generator().manual_seed(int(seed) + 17)
    return [torch.randint(0, VOCAB, (n,), generator=gen).tolist() for _, n in _llama_entries(case)]


def _llama_history(case, seed):
    """Keys (rotated, as the cache keeps them) and values [held, kv heads, dim] of every layer and request."""
    s, dtype = SHAPES[case["shape"]], getattr(torch, case["dtype"])
    gen = _generator(seed, 2)
    return [[(_normal(gen, (held, s["kv"], s["dim"]), 1.0, dtype), _normal(gen, (held, s["kv"], s["dim"]), 1.0, dtype))
             for held, _ in _llama_entries(case)] for _ in range(case["layers"])]


def _prepare_llama(case, seed):
    dtype = getattr(torch, case["dtype"])
    arch, cfg = read_model_config(_llama_config(case))
    model = Model(arch.describe(cfg), dtype, torch.device(DEV))
    model.load(_llama_weights(case, seed))
    entries = _llama_entries(case)
    pages = sum(-(-(held + n + 1) // PAGE) for held, n in entries) + 8
    cache = CacheManager(model.cache_needs(), PAGE, pages, max(4, len(entries)), dtype, DEV)
    runner = ModelRunner(model, cache)
    history = _llama_history(case, seed)
    for r, (held, _) in enumerate(entries):
        if not held:
            continue
        cache.open(r)
        cache.reserve(r, held)
        cache.commit(r, held)
        pages_of = torch.tensor(cache.held_pages(r, 0), dtype=torch.long, device=DEV)
        at = torch.arange(held, device=DEV)
        for layer, binding in enumerate(cache.bindings()):
            k, v = history[layer][r]
            binding.k_pool[pages_of[at // PAGE], :, at % PAGE] = k
            binding.v_pool[pages_of[at // PAGE], :, at % PAGE] = v
    del history
    tokens = _llama_tokens(case, seed)
    state = {"family": "llama", "mode": case["mode"], "runner": runner, "model": model, "held": entries[-1][0],
             "entries": [StepEntry(r, t, [len(t) - 1]) for r, t in enumerate(tokens)]}
    if case["mode"] == "decode" and runner.graphs_allowed:
        n = len(tokens)
        runner.decode_step(state["entries"], [SamplingParams()] * n, [0] * n, [0] * n)
        state["graph"], state["n"] = runner.last_graph, n
    return state


def _run_llama(state):
    runner = state["runner"]
    if state["mode"] == "decode":
        # The step that `decode_step` captured, replayed: the batch's arrays go to the device and the graph is launched.
        graph = state["graph"]
        graph.replay()
        return {"logits": graph.logits[: state["n"]]}
    if state["mode"] == "prefill" and not state["held"]:
        logits = runner.step(state["entries"])
        runner.end(0)
        return {"logits": logits}
    batch, _ = runner.prepare(state["entries"])  # (the lengths stay, so the next pass is the same step)
    return {"logits": state["model"].forward(batch)}


# --- recurrent mixers

def _delta_sizes(case):
    heads = max(1, case["width"] // case["vdim"])
    return heads, case["dim"], case["vdim"]


def _delta_weights(case, seed):
    """Projections that keep the scale of what they read, decays from nearly none to a few tokens' memory."""
    w = case["width"]
    heads, d, vd = _delta_sizes(case)
    gen, bf = _generator(seed, 3), torch.bfloat16
    inner = 64
    std = w ** -0.5
    if case["kind"] == "channel":
        t = {"q": (heads * d, w), "k": (heads * d, w), "v": (heads * vd, w), "b": (heads, w), "a1": (inner, w), "g1": (inner, w)}
        out = {n: _normal(gen, s, std, bf) for n, s in t.items()}
        out |= {"a2": _normal(gen, (heads * d, inner), 0.5 * inner ** -0.5, bf), "g2": _normal(gen, (heads * vd, inner), inner ** -0.5, bf),
                "q_conv": _normal(gen, (heads * d, TAPS), 0.5, bf), "k_conv": _normal(gen, (heads * d, TAPS), 0.5, bf),
                "v_conv": _normal(gen, (heads * vd, TAPS), 0.5, bf), "o": _normal(gen, (w, heads * vd), (heads * vd) ** -0.5, bf),
                "A_log": _normal(gen, (heads,), 0.5, torch.float32, 0.5),
                "dt_bias": _normal(gen, (heads * d,), 1.0, torch.float32, -3.0), "norm": _normal(gen, (vd,), 0.02, torch.float32, 1.0)}
        return out
    out = {n: _normal(gen, (heads * d, w), std, bf) for n in ("r", "k", "v", "g", "a")}
    out |= {"w1": _normal(gen, (inner, w), std, bf), "w2": _normal(gen, (heads * d, inner), 0.5 * inner ** -0.5, bf),
            "o": _normal(gen, (w, heads * d), (heads * d) ** -0.5, bf), "a_bias": _normal(gen, (heads * d,), 1.0, torch.float32),
            "w0": _normal(gen, (heads * d,), 1.5, torch.float32, -3.0), "norm": _normal(gen, (heads * d,), 0.02, torch.float32, 1.0)}
    return out


def _delta_inputs(case, seed):
    """What the layer reads, the states that earlier portions left, and the convolutions' last inputs."""
    heads, d, vd = _delta_sizes(case)
    gen = _generator(seed, 4)
    h = _normal(gen, (case["tokens"], case["width"]), 1.0, torch.bfloat16)
    states = _normal(gen, (case["entries"] + 1, heads, d, vd), 0.1, torch.float32)
    conv = _normal(gen, (case["entries"] + 1, TAPS - 1, heads * (2 * d + vd)), 1.0, torch.bfloat16) if case["kind"] == "channel" else None
    return h, states, conv


def _batch(lengths, part, graph):
    """A step's batch of requests that bring `lengths` tokens, request i in state slot i."""
    n, total = len(lengths), sum(lengths)
    first = [sum(lengths[:i]) for i in range(n)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    singles = sum(1 for v in lengths if v == 1)
    step = HostStep(n, total, singles, list(lengths), list(lengths), first, PAGE)
    plans = {}
    if part.plan_key() is not None:
        plans[part.plan_key()] = {k: torch.from_numpy(v).to(DEV) for k, v in part.plan_step(step).items()}
    return StepBatch(tokens=ints([0] * total), pos=ints([p for v in lengths for p in range(v)]),
                     entry=ints([i for i, v in enumerate(lengths) for _ in range(v)]), tables={}, slots=ints(list(range(n))),
                     want_rows=None, status=ints([0]), n_tokens=total, n_entries=n, n_decode=singles,
                     host_query_lens=list(lengths), host_context_lens=list(lengths), extras={"graph": True} if graph else {},
                     plans=plans)


def _captured(call):
    """The call inside a CUDA graph, as the engine captures its steps of single tokens: (graph, its result)."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = call()
    return graph, out


def _prepare_part(case, seed):
    ctx = BuildContext(torch.bfloat16, torch.device(DEV))
    kept = {}
    if case["family"] == "delta":
        heads, d, vd = _delta_sizes(case)
        weights = _delta_weights(case, seed)
        params = {"hidden_size": case["width"], "n_heads": heads, "head_dim": d, "eps": 1e-6}
        if case["kind"] == "channel":
            params |= {"value_dim": vd, "taps": TAPS}
        part = build_part("mixer", PartSpec("channel_delta" if case["kind"] == "channel" else "general_delta", params,
                                            {n: n for n in weights}), ctx)
        h, states, conv = _delta_inputs(case, seed)
        part.bind_cache(StateBinding(states))
        kept["state"] = states
        if conv is not None:
            part.state_holders()[0].bind_cache(StateBinding(conv))
            kept["filter"] = conv
        lengths = _spread(case["tokens"], case["entries"])
    else:
        weights = _expert_weights(case, seed)
        params = {"hidden_size": case["width"], "expert_size": case["ff"], "n_experts": case["experts"], "top": case["top"],
                  "groups": case["groups"], "keep_groups": case["keep"], "shared_size": case["shared"] or None, "expert": case["unit"]}
        names = {"router": "router", "correction": "correction", "expert_gate": "e{e}.gate", "expert_up": "e{e}.up",
                 "expert_down": "e{e}.down", "shared_gate": "shared.gate", "shared_up": "shared.up", "shared_down": "shared.down"}
        part = build_part("feed_forward", PartSpec("moe", params, names), ctx)
        h = _normal(_generator(seed, 6), (case["tokens"], case["width"]), 1.0, torch.bfloat16)
        lengths = [1] * case["tokens"] if case["graph"] else [case["tokens"]]
    part.load(weights)
    batch = _batch(lengths, part, case["graph"])
    state = {"family": case["family"], "part": part, "h": h, "batch": batch, "kept": kept, "entries": case.get("entries", 0)}
    if case["graph"]:
        before = {n: t.clone() for n, t in kept.items()}
        state["graph"], state["out"] = _captured(lambda: part.forward(h, batch))
        for n, t in before.items():
            kept[n].copy_(t)
    return state


def _run_part(state):
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = state["part"].forward(state["h"], state["batch"])
    return {"out": out, **{n: t[: state["entries"]] for n, t in state["kept"].items()}}


# --- routed experts

def _expert_weights(case, seed):
    w, f, fs = case["width"], case["ff"], case["shared"]
    gated = case["unit"] == "gated_silu"
    gen, bf = _generator(seed, 5), torch.bfloat16
    out = {"router": _normal(gen, (case["experts"], w), w ** -0.5, torch.float32),
           "correction": _normal(gen, (case["experts"],), 0.01, torch.float32)}
    for e in range(case["experts"]):
        if gated:
            out[f"e{e}.gate"] = _normal(gen, (f, w), w ** -0.5, bf)
        out[f"e{e}.up"] = _normal(gen, (f, w), w ** -0.5, bf)
        out[f"e{e}.down"] = _normal(gen, (w, f), f ** -0.5, bf)
    if fs:
        if gated:
            out["shared.gate"] = _normal(gen, (fs, w), w ** -0.5, bf)
        out["shared.up"] = _normal(gen, (fs, w), w ** -0.5, bf)
        out["shared.down"] = _normal(gen, (w, fs), fs ** -0.5, bf)
    return out


def prepare(case, seed):
    return _prepare_llama(case, seed) if case["family"] == "llama" else _prepare_part(case, seed)


def run(state):
    return _run_llama(state) if state["family"] == "llama" else _run_part(state)


# ------------------------------------------------------------------------------------------------ what a pass needs

def work(case):
    if case["family"] == "llama":
        s = SHAPES[case["shape"]]
        size = 2 if case["dtype"] == "bfloat16" else 4
        h, q, kv, ff = s["hidden"], s["heads"] * s["dim"], s["kv"] * s["dim"], s["ff"]
        layer = (q + 2 * kv) * h + h * q + 3 * ff * h
        entries = _llama_entries(case)
        tokens = sum(n for _, n in entries)
        keys = sum(held + n for held, n in entries)                                # read once per request
        pairs = sum(n * held + n * (n + 1) // 2 for held, n in entries)
        nbytes = (case["layers"] * layer + VOCAB * h) * size + case["layers"] * keys * 2 * kv * size \
            + tokens * (h * size + 4) + len(entries) * VOCAB * 4
        flops = case["layers"] * (2.0 * layer * tokens + 4.0 * s["heads"] * s["dim"] * pairs) + 2.0 * VOCAB * h * len(entries)
        return {"bytes": nbytes, "flops": flops}
    w, t = case["width"], case["tokens"]
    if case["family"] == "delta":
        heads, d, vd = _delta_sizes(case)
        inner = 64
        if case["kind"] == "channel":
            rows = heads * (2 * d + vd) + heads + 2 * inner
            params = rows * w + heads * (d + vd) * inner + w * heads * vd
            extra = case["entries"] * heads * (2 * d + vd) * (TAPS - 1) * 2 * 2
        else:
            params = (5 * heads * d + inner) * w + heads * d * inner + w * heads * d
            extra = 0
        state = 2 * case["entries"] * heads * d * vd * 4
        return {"bytes": params * 2 + t * w * 2 * 2 + state + extra, "flops": 2.0 * params * t + 8.0 * t * heads * d * vd}
    mats = 3 if case["unit"] == "gated_silu" else 2
    used = min(case["experts"], case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** t))
    params = mats * w * (case["ff"] * used + case["shared"])
    return {"bytes": params * 2 + case["experts"] * w * 4 + t * w * 4,
            "flops": 2.0 * t * (mats * w * (case["ff"] * case["top"] + case["shared"]) + case["experts"] * w)}


def tolerance(case):
    """About four times what the path is off 64 bits by: 4e-6 in float32; 0.004 for a mixer or the experts in bfloat16
    (one rounding of every product's result); 0.011 to 0.015 for a few whole layers and the head in bfloat16."""
    if case["family"] != "llama":
        return {"rel": 0.015, "max": 0.2}
    if case["dtype"] == "float32":
        return {"rel": 1.6e-5}
    return {"rel": 0.03, "max": 0.4}


# ------------------------------------------------------------------------------------------------ 64-bit results

def exact(case, seed):
    with torch.no_grad():
        return {"llama": _exact_llama, "delta": _exact_delta, "experts": _exact_experts}[case["family"]](case, seed)


def _norm64(x, weight, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * weight.double()


def _frequencies(s):
    f = s["theta"] ** (-torch.arange(0, s["dim"], 2, dtype=torch.float64) / s["dim"])
    if s["factor"] is None:
        return f.to(DEV)
    wave = 2 * math.pi / f
    blend = (8192.0 / wave - 1.0) / (4.0 - 1.0)
    mid = (1 - blend) * f / s["factor"] + blend * f
    return torch.where(wave < 8192.0 / 4.0, f, torch.where(wave > 8192.0 / 1.0, f / s["factor"], mid)).to(DEV)


def _rotate(x, pos, freq):
    angle = pos.double()[:, None] * freq[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _exact_llama(case, seed):
    s = SHAPES[case["shape"]]
    w = _llama_weights(case, seed)
    history = _llama_history(case, seed)
    entries, tokens = _llama_entries(case), _llama_tokens(case, seed)
    freq = _frequencies(s)
    flat = torch.tensor([t for ts in tokens for t in ts], device=DEV)
    pos = torch.cat([torch.arange(held, held + n, device=DEV) for held, n in entries])
    x = w["model.embed_tokens.weight"][flat].double()
    group = s["heads"] // s["kv"]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        product = lambda a, n: a @ w[p + n + ".weight"].double().t()  # noqa: E731,B023
        h = _norm64(x, w[p + "input_layernorm.weight"], EPS)
        q = _rotate(product(h, "self_attn.q_proj").view(-1, s["heads"], s["dim"]), pos, freq)
        k = _rotate(product(h, "self_attn.k_proj").view(-1, s["kv"], s["dim"]), pos, freq)
        v = product(h, "self_attn.v_proj").view(-1, s["kv"], s["dim"])
        outs, at = [], 0
        for r, (held, n) in enumerate(entries):
            keys = torch.cat([history[i][r][0].double(), k[at:at + n]]).transpose(0, 1)      # [kv, held + n, dim]
            values = torch.cat([history[i][r][1].double(), v[at:at + n]]).transpose(0, 1)
            mine = q[at:at + n].view(n, s["kv"], group, s["dim"]).permute(1, 2, 0, 3)          # [kv, group, n, dim]
            scores = mine @ keys[:, None].transpose(-1, -2) * s["dim"] ** -0.5
            late = torch.arange(held + n, device=DEV)[None] > (held + torch.arange(n, device=DEV))[:, None]
            scores.masked_fill_(late, -math.inf)
            outs.append((torch.softmax(scores, -1) @ values[:, None]).permute(2, 0, 1, 3).reshape(n, -1))
            at += n
        x = x + product(torch.cat(outs), "self_attn.o_proj")
        h = _norm64(x, w[p + "post_attention_layernorm.weight"], EPS)
        x = x + product(torch.nn.functional.silu(product(h, "mlp.gate_proj")) * product(h, "mlp.up_proj"), "mlp.down_proj")
    last = torch.tensor([sum(n for _, n in entries[: r + 1]) - 1 for r in range(len(entries))], device=DEV)
    h = _norm64(x[last], w["model.norm.weight"], EPS)
    return {"logits": h @ w["model.embed_tokens.weight" if s["tied"] else "lm_head.weight"].double().t()}


def _exact_delta(case, seed):
    w = {n: t.double() for n, t in _delta_weights(case, seed).items()}
    h, states, conv = _delta_inputs(case, seed)
    h, states = h.double(), states.double()[: case["entries"]].clone()
    heads, d, vd = _delta_sizes(case)
    lengths = _spread(case["tokens"], case["entries"])
    out = {"state": states}
    if case["kind"] == "channel":
        conv = conv.double()
        raw = torch.cat([h @ w[n].t() for n in ("q", "k", "v")], dim=1)
        taps = torch.cat([w[n + "_conv"] for n in ("q", "k", "v")])                            # [channels, taps]
        filtered, left, at = [], [], 0
        for e, n in enumerate(lengths):
            seen = torch.cat([conv[e], raw[at:at + n]])                                       # [taps - 1 + n, channels]
            filtered.append(sum(seen[j:j + n] * taps[:, j] for j in range(TAPS)))
            left.append(seen[-(TAPS - 1):])
            at += n
        out["filter"] = torch.stack(left)
        filtered = torch.nn.functional.silu(torch.cat(filtered))
        q, k, v = filtered.split([heads * d, heads * d, heads * vd], dim=1)
        q, k, v = q.view(-1, heads, d), k.view(-1, heads, d), v.view(-1, heads, vd)
        unit = lambda z: z * torch.rsqrt(z.pow(2).sum(-1, keepdim=True) + UNIT_EPS)  # noqa: E731
        q, k = unit(q) * d ** -0.5, unit(k)
        b = torch.sigmoid(h @ w["b"].t())
        g = torch.exp(-torch.exp(w["A_log"])[None, :, None]
                      * torch.nn.functional.softplus((h @ w["a1"].t()) @ w["a2"].t() + w["dt_bias"]).view(-1, heads, d))
        gate = torch.sigmoid((h @ w["g1"].t()) @ w["g2"].t())
        norm = w["norm"].repeat(heads)
    else:
        r, k, v, a = ((h @ w[n].t()).view(-1, heads, d) for n in ("r", "k", "v", "a"))
        a = torch.sigmoid(a + w["a_bias"].view(heads, d))
        decay = torch.exp(-DECAY_SCALE * torch.sigmoid(torch.tanh(h @ w["w1"].t()) @ w["w2"].t() + w["w0"])).view(-1, heads, d)
        u = k * torch.rsqrt(k.pow(2).sum(-1, keepdim=True) + UNIT_EPS)
        gate = torch.sigmoid(h @ w["g"].t())
        norm = w["norm"]
    # Requests side by side: step j advances every request that has a token j.
    o = torch.empty((case["tokens"], heads, vd), dtype=torch.float64, device=DEV)
    first = [sum(lengths[:i]) for i in range(len(lengths))]
    for j in range(max(lengths)):
        alive = [e for e, n in enumerate(lengths) if n > j]
        rows, who = torch.tensor([first[e] + j for e in alive], device=DEV), torch.tensor(alive, device=DEV)
        S = states[who]
        if case["kind"] == "channel":
            S = S * g[rows][..., None]
            kj = k[rows]
            uj = b[rows][..., None] * (v[rows] - torch.einsum("ehij,ehi->ehj", S, kj))
            S = S + kj[..., None] * uj[:, :, None]
            o[rows] = torch.einsum("ehij,ehi->ehj", S, q[rows])
        else:
            uj = u[rows]
            read = torch.einsum("ehij,ehi->ehj", S, uj)
            S = decay[rows][..., None] * S - (a[rows] * uj)[..., None] * read[:, :, None] + k[rows][..., None] * v[rows][:, :, None]
            o[rows] = torch.einsum("ehij,ehi->ehj", S, r[rows])
        states[who] = S
    o = (o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6)).reshape(case["tokens"], heads * vd) * norm * gate
    return {"out": o @ w["o"].t(), **out}


def _exact_experts(case, seed):
    w = {n: t.double() for n, t in _expert_weights(case, seed).items()}
    h = _normal(_generator(seed, 6), (case["tokens"], case["width"]), 1.0, torch.bfloat16).double()
    s = torch.softmax(h @ w["router"].t(), dim=-1)
    choice = s + w["correction"]
    per = case["experts"] // case["groups"]
    if case["groups"] > 1:
        best = choice.view(-1, case["groups"], per).max(-1).values.topk(case["keep"], dim=-1).indices
        stays = torch.zeros((h.shape[0], case["groups"]), dtype=torch.bool, device=DEV).scatter_(1, best, True)
        choice = choice.masked_fill(~stays.repeat_interleave(per, dim=1), -math.inf)
    ids = choice.topk(case["top"], dim=-1).indices
    weights = s.gather(1, ids)
    weights = weights / (weights.sum(-1, keepdim=True) + 1e-20)

    def feed(x, p):
        if case["unit"] == "gated_silu":
            z = torch.nn.functional.silu(x @ w[p + ".gate"].t()) * (x @ w[p + ".up"].t())
        elif case["unit"] == "relu2":
            z = torch.relu(x @ w[p + ".up"].t()).pow(2)
        else:
            z = torch.nn.functional.gelu(x @ w[p + ".up"].t())
        return z @ w[p + ".down"].t()

    out = feed(h, "shared") if case["shared"] else torch.zeros_like(h)
    for e in range(case["experts"]):
        row, place = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            out.index_add_(0, row, weights[row, place][:, None] * feed(h[row], f"e{e}"))
    return {"out": out}
