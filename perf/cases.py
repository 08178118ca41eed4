"""Performance cases of the compressed linear layers, through the package's public entry points.

Four kinds of work, as a program that serves a compressed model has them:

  linear   one ``CompressedLinear`` called eagerly: 1 to 8 activation rows take the fused decode + product, more rows
           (several sequences at once, prompts) decode and then multiply;
  step     the linear layers of decoder blocks for one token per sequence, captured into a CUDA graph and replayed,
           with the projections separate or stacked (``convert_all_linear(fuse_siblings=...)``);
  dense    ``weight.get_weight()``: a whole layer back to BF16 (export, merging, checks);
  convert  ``convert(linear, name)``: an ``nn.Linear`` compressed, on the host (a checkpoint as it is loaded) or on
           the device (a model that is already there).

Weights are N(0, s) with s between 0.012 and 0.04, the range of trained projection matrices; activations are N(0, 1).
"""
from __future__ import annotations

import math
import random

import torch
from torch import nn

from bf16_huffman_infer_b200 import (
    ANSWeight, CompressedLinear, HuffmanWeight, convert, convert_all_linear, set_ans_precision, set_huffman_tables,
)
from bf16_huffman_infer_b200.utils import chunk_count_for_k

# stored bytes per weight on N(0, s): sign + mantissa byte, and the exponent records of each coder
STORED = {"limit6": 1.45, "escape": 1.39, "reference": 1.39, "ans": 1.44, "smallest": 1.44}

LAYER = {"coder": "huffman", "tables": "limit6", "bits": 8}


def listed():
    return [
        # a key or value projection (1024 x 4096), one sequence, not graphed: the smallest call, where the host path and
        # the launch are most of the time
        {"name": "linear_kv_1row", "kind": "linear", **LAYER, "m": 1024, "k": 4096, "rows": 1, "bias": False},
        # stacked q/k/v of a 3584-wide model, with its bias, three sequences
        {"name": "linear_qkv_bias_3rows", "kind": "linear", **LAYER, "m": 4608, "k": 3584, "rows": 3, "bias": True},
        # an output head over 151936 tokens: the largest matrix of a model, four sequences
        {"name": "linear_head_4rows", "kind": "linear", **LAYER, "m": 151936, "k": 4096, "rows": 4, "bias": False},
        # gate or up projection, sixteen sequences decoded at once: past the fused product's eight rows
        {"name": "linear_gate_16rows", "kind": "linear", **LAYER, "m": 12288, "k": 4096, "rows": 16, "bias": False},
        # down projection over a prompt of 2048 tokens, the other coder: the most arithmetic
        {"name": "linear_down_prompt_ans", "kind": "linear", "coder": "ans", "tables": "", "bits": 8,
         "m": 4096, "k": 12288, "rows": 2048, "bias": False},
        # one decode step of an 8B model's blocks, stacked projections, one sequence, the default tables
        {"name": "step_8b_1row", "kind": "step", **LAYER, "hidden": 4096, "inter": 12288, "kv": 1024, "blocks": 2,
         "stacked": True, "rows": 1},
        # the same widths with eight sequences, separate projections and the smallest tables
        {"name": "step_8b_escape_8rows", "kind": "step", "coder": "huffman", "tables": "escape", "bits": 8,
         "hidden": 4096, "inter": 12288, "kv": 1024, "blocks": 1, "stacked": False, "rows": 8},
        # a 7B model's block with the rANS coder, two sequences; 18944 columns make four chunks of an odd width
        {"name": "step_7b_ans_2rows", "kind": "step", "coder": "ans", "tables": "", "bits": 8,
         "hidden": 3584, "inter": 18944, "kv": 512, "blocks": 1, "stacked": True, "rows": 2},
        # a 1.7B model's blocks with the tables of the reference's builder: many small launches
        {"name": "step_2b_reference_1row", "kind": "step", "coder": "huffman", "tables": "reference", "bits": 8,
         "hidden": 2048, "inter": 6144, "kv": 1024, "blocks": 4, "stacked": False, "rows": 1},
        # a vocabulary-sized layer with a ragged row count back to BF16
        {"name": "dense_ragged", "kind": "dense", **LAYER, "m": 32003, "k": 2560},
        # a layer of a checkpoint in host memory, compressed as it is loaded
        {"name": "convert_host", "kind": "convert", **LAYER, "m": 4096, "k": 4096, "host": True},
        # a layer of a model on the device, both coders tried and the smaller kept
        {"name": "convert_device_smallest", "kind": "convert", "coder": "smallest", "tables": "limit6", "bits": 8,
         "m": 12288, "k": 4096, "host": False},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng: random.Random, lo: int, hi: int) -> int:
    """A row length that the format can store: a multiple of 128 that splits into chunks."""
    while True:
        k = 128 * _log_int(rng, lo // 128, hi // 128)
        try:
            chunk_count_for_k(k)
        except RuntimeError:
            continue
        return k


def _coder(rng: random.Random) -> dict:
    pick = rng.random()
    if pick < 0.3:
        return {"coder": "ans", "tables": "", "bits": rng.choice([8, 8, 10, 12])}
    return {"coder": "huffman", "tables": rng.choice(["limit6", "limit6", "limit6", "escape", "reference"]), "bits": 8}


def draw(rng: random.Random) -> dict:
    kind = rng.choices(["linear", "step", "dense", "convert"], [9, 5, 2, 4])[0]
    case = {"kind": kind, **_coder(rng)}
    if kind == "step":
        hidden = _width(rng, 1024, 6144)
        case.update(hidden=hidden, inter=_width(rng, 5 * hidden // 2, 11 * hidden // 2), kv=128 * rng.randint(2, 8),
                    rows=rng.randint(1, 8), stacked=rng.random() < 0.5)
        per_block = hidden * (2 * hidden + 2 * case["kv"] + 3 * case["inter"])
        case["blocks"] = rng.randint(1, max(1, min(4, 380_000_000 // per_block)))
        return case
    k = _width(rng, 1024, 28672)
    most = {"linear": 300_000_000, "dense": 120_000_000, "convert": 50_000_000}[kind]
    m = _log_int(rng, 256, min(65536, most // k))
    case.update(m=m, k=k)
    if kind == "linear":
        rows = rng.randint(1, 8) if rng.random() < 0.6 else _log_int(rng, 9, min(2048, max(9, 100_000_000_000 // (m * k))))
        case.update(rows=rows, bias=rng.random() < 0.3)
    elif kind == "convert":
        case["host"] = rng.random() < 0.5
        if rng.random() < 0.3:
            case.update(coder="smallest", tables="limit6", bits=8)
    return case


# ---- what a program has in hand before the call --------------------------------------------------------------------
def _normal(gen: torch.Generator, *shape: int, scale: float = 1.0) -> torch.Tensor:
    """BF16 N(0, scale) on the device, made in slabs so that a large matrix needs no large FP32 copy."""
    out = torch.empty(shape, dtype=torch.bfloat16, device=gen.device)
    for slab in out.split(8192):
        slab.copy_(torch.randn(slab.shape, dtype=torch.float32, device=gen.device, generator=gen) * scale)
    return out


class _Options:
    """The table builder and the rANS precision that a case asks for, put back afterwards."""

    def __init__(self, case: dict):
        self.case = case

    def __enter__(self):
        self.tables = set_huffman_tables(self.case["tables"] or "limit6")
        self.bits = set_ans_precision(self.case["bits"])

    def __exit__(self, *exc):
        set_huffman_tables(self.tables)
        set_ans_precision(self.bits)


def _dense_layer(m: int, k: int, dev: torch.device) -> nn.Linear:
    return nn.Linear(k, m, bias=False, dtype=torch.bfloat16, device=dev).requires_grad_(False)


class _Block(nn.Module):
    """The linear layers of a decoder block.  Each reads an activation of its width that is there already: the residual
    stream, or what the layer before it made."""

    def __init__(self, case: dict, dev: torch.device):
        super().__init__()
        hidden, inter, kv = case["hidden"], case["inter"], case["kv"]
        self.q_proj, self.k_proj, self.v_proj = (_dense_layer(m, hidden, dev) for m in (hidden, kv, kv))
        self.o_proj = _dense_layer(hidden, hidden, dev)
        self.gate_proj, self.up_proj = _dense_layer(inter, hidden, dev), _dense_layer(inter, hidden, dev)
        self.down_proj = _dense_layer(hidden, inter, dev)

    def forward(self, x: torch.Tensor):
        q, k, v = self.q_proj(x), self.k_proj(x), self.v_proj(x)
        o = self.o_proj(q)
        gate, up = self.gate_proj(o), self.up_proj(o)
        return [q, k, v, o, gate, up, self.down_proj(gate)]


def _prepare_step(case: dict, gen: torch.Generator, scale: float) -> dict:
    dev = gen.device
    blocks = nn.ModuleList(_Block(case, dev) for _ in range(case["blocks"]))
    for p in blocks.parameters():
        p.copy_(_normal(gen, *p.shape, scale=scale))
    convert_all_linear(blocks, min_out_features=0, progress=False, algo=case["coder"], fuse_siblings=case["stacked"],
                       huffman_tables=case["tables"] or "limit6")
    blocks.to(dev)
    x = [_normal(gen, case["rows"], 1, case["hidden"]) for _ in blocks]

    def step():
        return [y for block, xb in zip(blocks, x) for y in block(xb)]

    side = torch.cuda.Stream(device=dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream(dev).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    return {"kind": "step", "graph": graph, "out": out, "keep": (blocks, x)}


@torch.no_grad()
def prepare(case: dict, seed: int) -> dict:
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    scale = random.Random(seed).uniform(0.012, 0.04)
    with _Options(case):
        if case["kind"] == "step":
            return _prepare_step(case, gen, scale)
        m, k = case["m"], case["k"]
        w = _normal(gen, m, k, scale=scale)
        if case["kind"] == "convert":
            linear = _dense_layer(m, k, torch.device("cpu") if case["host"] else dev)
            linear.weight.copy_(w)
            # the part of a checkpoint shard that takes the layer's records and tables: their sizes depend on the values,
            # and records that need more than 8 bits per weight are not kept
            home = linear.weight.device
            shard = {"exp": torch.zeros(m * k // 4, dtype=torch.int32, device=home),
                     "tables": torch.zeros(1 << 14, dtype=torch.uint8, device=home)}
            return {"kind": "convert", "linear": linear, "case": case, "shard": shard}
        weight = (ANSWeight if case["coder"] == "ans" else HuffmanWeight).compress(w, to_cpu=False)
        if case["kind"] == "dense":
            return {"kind": "dense", "weight": weight}
        bias = nn.Parameter(_normal(gen, m), requires_grad=False) if case["bias"] else None
        rows = case["rows"]
        # one token of each sequence while decoding, one sequence of many tokens for a prompt
        x = _normal(gen, rows, k).view((rows, 1, k) if rows <= 64 else (1, rows, k))
        return {"kind": "linear", "layer": CompressedLinear(weight, bias), "x": x}


@torch.no_grad()
def run(state: dict):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "step":
        state["graph"].replay()
        return state["out"]
    if kind == "dense":
        return state["weight"].get_weight()
    with _Options(state["case"]):
        module = convert(state["linear"], "linear", algo=state["case"]["coder"])
    shard, at = state["shard"], 0
    buffers = dict(module.weight.named_buffers())
    rem, exp, offsets = buffers.pop("rem"), buffers.pop("exp"), buffers.pop("offsets")
    shard["exp"][:exp.numel()].copy_(exp)
    for table in buffers.values():
        table = table.view(torch.uint8)
        shard["tables"][at:at + table.numel()].copy_(table)
        at += table.numel()
    return {"rem": rem, "offsets": offsets, **shard}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def work(case: dict) -> dict:
    stored = STORED[case["tables"] or case["coder"]] if case["coder"] != "smallest" else STORED["smallest"]
    if case["kind"] == "step":
        hidden, inter, kv, n, rows = case["hidden"], case["inter"], case["kv"], case["blocks"], case["rows"]
        weights = n * hidden * (2 * hidden + 2 * kv + 3 * inter)
        read = hidden + hidden + hidden + inter                    # x, q, o and gate are each read once
        written = hidden + 2 * kv + hidden + 2 * inter + hidden
        return {"bytes": weights * stored + 2 * n * rows * (read + written), "flops": 2 * rows * weights}
    weights = case["m"] * case["k"]
    if case["kind"] == "linear":
        return {"bytes": weights * stored + 2 * case["rows"] * (case["m"] + case["k"]), "flops": 2 * case["rows"] * weights}
    return {"bytes": weights * (stored + 2), "flops": 0}


def tolerance(case: dict):
    """Decoded weights and compressed buffers are exact.  Products are BF16 roundings of 32-bit sums: two orders of
    summation round some outputs to neighbouring values, and a step's later layers read such outputs."""
    if case["kind"] == "linear":
        return {"rel": 4e-3, "max": 2e-2}
    if case["kind"] == "step":
        return {"rel": 8e-3, "max": 4e-2}
    return "exact"
