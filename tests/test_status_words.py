"""Kernels whose waits are bounded get the step's status word from the parts that launch them (no GPU: the launches are
recorded instead of made)."""

from __future__ import annotations

import ast
import pathlib

import pytest
import torch

from pulsarlm_b200 import models as _models  # noqa: F401  (registers the parts)
from pulsarlm_b200.cache.manager import StateBinding
from pulsarlm_b200.kernels import ops
from pulsarlm_b200.models.model import HostStep, StepBatch
from pulsarlm_b200.parts import linear
from pulsarlm_b200.parts.registry import BuildContext, build_part, part_class
from pulsarlm_b200.parts.spec import PartSpec

BF = torch.bfloat16


@pytest.fixture
def launches(monkeypatch):
    """(name, arguments) of every entry point that is called; its last argument is the stream, the one before it the status word."""
    made = []
    monkeypatch.setattr(ops, "_call", lambda name, *args: made.append((name, args)))
    monkeypatch.setattr(ops, "_dev", lambda *tensors: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return made


def _part(kind, name, params, names):
    """With weights of zeros, ranks that a checkpoint decides being 16."""
    spec = PartSpec(name, params, names if isinstance(names, dict) else {n: n for n in names})
    part = build_part(kind, spec, BuildContext(BF, torch.device("cpu")))
    needs = part_class(kind, name).tensor_needs(spec)
    part.load({n: torch.zeros([d if d >= 0 else 16 for d in need.shape], dtype=BF) for n, need in needs.items()})
    return part


def _batch(part, lengths):
    n, total = len(lengths), sum(lengths)
    first = [sum(lengths[:i]) for i in range(n)]
    singles = sum(1 for v in lengths if v == 1)
    ints = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    step = HostStep(n, total, singles, lengths, lengths, first, 16)
    plans = {}
    if part.plan_key() is not None:
        plans[part.plan_key()] = {k: torch.from_numpy(v) for k, v in part.plan_step(step).items()}
    return StepBatch(ints([0] * total), ints(range(total)), ints([i for i, v in enumerate(lengths) for _ in range(v)]), {},
                     ints(range(n)), None, ints([0]), total, n, singles, lengths, lengths, plans=plans)


def _check(launches, name, batch, count):
    found = [args for called, args in launches if called == name]
    assert len(found) == count and all(args[-2] == batch.status.data_ptr() for args in found)


@pytest.mark.parametrize("lengths", [[40], [1, 1, 20]])
def test_delta_rules_in_chunks(launches, lengths):
    heads, dim, hidden, total = 2, 64, 128, sum(lengths)
    states = torch.zeros((len(lengths), heads, dim, dim))
    sizes = {"hidden_size": hidden, "n_heads": heads, "head_dim": dim, "eps": 1e-6}
    channel = _part("mixer", "channel_delta", {**sizes, "value_dim": dim, "taps": 4},
                    ("q", "k", "v", "b", "a1", "a2", "g1", "g2", "q_conv", "k_conv", "v_conv", "o", "A_log", "dt_bias", "norm"))
    channel.bind_cache(StateBinding(states))
    channel.state_holders()[0].bind_cache(StateBinding(torch.zeros((len(lengths), 3, heads * 3 * dim), dtype=BF)))
    general = _part("mixer", "general_delta", sizes,
                    ("r", "k", "v", "g", "a", "w1", "w2", "o", "a_bias", "w0", "norm"))
    general.bind_cache(StateBinding(states))
    for part, name in ((channel, "pl_gated_delta"), (general, "pl_delta_rule")):
        batch = _batch(part, lengths)
        part.forward(torch.zeros((total, hidden), dtype=BF), batch)
        _check(launches, name, batch, 1)


@pytest.mark.parametrize("expert,weigh_input", [("gated_silu", False), ("relu2", False), ("clamped", True)])
def test_grouped_products_of_experts(launches, expert, weigh_input):
    params = {"hidden_size": 64, "expert_size": 64, "n_experts": 4, "top": 2, "shared_size": None, "expert": expert,
              "weigh_input": weigh_input, "expert_limit": 7.0}
    part = _part("feed_forward", "moe", params, {"router": "router", "expert_gate": "e{e}.gate", "expert_up": "e{e}.up",
                                                 "expert_down": "e{e}.down"})
    batch = _batch(part, [64])
    part.forward(torch.zeros((64, 64), dtype=BF), batch)
    _check(launches, "pl_gemm_bf16_grouped", batch, 2)
    part.forward(torch.zeros((64, 64), dtype=BF), None)  # (no step, nowhere to report to)
    assert [args[-2] for called, args in launches if called == "pl_gemm_bf16_grouped"][2:] == [None, None]


@pytest.mark.parametrize("tokens", [1, 8, 40, 100])
def test_products_of_layers(launches, monkeypatch, tokens):
    monkeypatch.setattr(linear, "GEMM_ROUTE", "tcgen05")
    gated = _part("feed_forward", "gated_mlp", {"hidden_size": 64, "intermediate_size": 128}, ("gate", "up", "down"))
    plain = _part("feed_forward", "mlp", {"hidden_size": 64, "intermediate_size": 128}, ("up", "down"))
    head = _part("head", "linear", {"hidden_size": 64, "vocab_size": 96}, ("weight",))
    h, batch = torch.zeros((tokens, 64), dtype=BF), _batch(gated, [tokens])
    gated.forward(h, batch)
    plain.forward(h, batch)
    head.forward(h, batch.status)
    products = [args for name, args in launches if name.startswith("pl_gemm_bf16")]
    assert len(products) == 5 and all(args[-2] == batch.status.data_ptr() for args in products)


def test_no_part_leaves_the_status_word_out():
    """(the positional place of `status`, counted from 0, in each function of parts/linear.py)"""
    places = {"linear": 3, "gated_linear": 3, "gated_feed_forward": 5, "activated_linear": 4}
    for path in pathlib.Path(linear.__file__).parent.glob("*.py"):
        for node in ast.walk(ast.parse(path.read_text())):
            if isinstance(node, ast.Call) and isinstance(node.func, ast.Name) and node.func.id in places:
                given = len(node.args) > places[node.func.id] or any(k.arg == "status" for k in node.keywords)
                assert given, f"{path.name}:{node.lineno}"
