"""The packed ternary path as a user's program drives it, from one decoded token to a long prompt.

Every case goes through the package's public entry points (``PackedLinear``, ``PackedEmbedding``,
``tq1_swiglu``, ``ChainPlan``, ``GraphedStep``, ``load_tiled``, ``encode_tq1_blocks``). Shapes are those
of the 27B-class decoder that the benchmark and ``layout.MODEL_LINEAR_SHAPES`` describe (hidden 5120,
feed-forward 17408, 151936-row vocabulary) and generic ragged ones; weights and activations have the
benchmark's distributions.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from ternel_b200.chain import ChainPlan, Link, blocks_to_panels
from ternel_b200.format import encode_tq1_blocks
from ternel_b200.graphs import GraphedStep
from ternel_b200.layout import PackedTensorLayout, pack_blocks
from ternel_b200.modules import PackedEmbedding, PackedLinear
from ternel_b200.ops import interleave_gate_up, tq1_swiglu
from ternel_b200.stack import random_blocks_device, swiglu_gain, unit_gain

GROUP, BLOCK = 128, 28
# the largest listed product (2048 tokens through gate_proj/up_proj); drawn ones stay below it
LARGEST_MACS = 2048 * 17408 * 5120


def listed() -> list[dict]:
    return [
        # k_proj / v_proj of one decoded token, called as a module: the smallest product of a model, where
        # the call itself counts
        {"name": "decode_kv", "path": "linear", "m": 1, "n": 1024, "k": 5120, "out": "f16"},
        # the tied output head of one decoded token, logits
        {"name": "decode_head", "path": "head", "m": 1, "n": 151936, "k": 5120, "out": "f16"},
        # eight decoder layers of one decoded token as one chain (q|k|v, o, gate|up with SiLU*up, down)
        {"name": "decode_chain", "path": "chain", "layers": 8, "hidden": 5120, "ffn": 17408, "kv": 1024},
        # one decoder layer for eight sequences decoding together, replayed as a CUDA graph
        {"name": "batch8_layer", "path": "layer", "m": 8, "hidden": 5120, "ffn": 17408, "kv": 1024},
        # down_proj in a server that decodes 48 sequences together
        {"name": "batch48_down", "path": "linear", "m": 48, "n": 5120, "k": 17408, "out": "f16"},
        # a layer of a model whose width is a multiple of the group alone, odd rows, few tokens, FP32 results
        {"name": "ragged_batch5", "path": "linear", "m": 5, "n": 4099, "k": 2176, "out": "f32"},
        # down_proj over an ordinary prompt
        {"name": "prefill_down", "path": "linear", "m": 512, "n": 5120, "k": 17408, "out": "f16"},
        # gate_proj / up_proj over a long prompt: the largest product
        {"name": "prefill_up_long", "path": "linear", "m": 2048, "n": 17408, "k": 5120, "out": "f16"},
        # fused gate|up with SiLU*up over a prompt of no particular length
        {"name": "prefill_swiglu", "path": "swiglu", "m": 777, "n": 34816, "k": 5120, "out": "f16"},
        # the prompt's token embeddings
        {"name": "embed_prompt", "path": "embed", "m": 2048, "n": 151936, "k": 5120, "out": "f16"},
        # one weight of a converted checkpoint (host arrays) into its module: byte scan, relayout, upload
        {"name": "load_o_proj", "path": "load", "n": 5120, "k": 5120},
        # packing one trained ternary weight for a checkpoint, on the host
        {"name": "encode_o_proj", "path": "encode", "n": 5120, "k": 5120},
    ]


def _log(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _shape(rng, m: int) -> tuple[int, int]:
    """Rows and columns of a weight: rows of any number, columns a multiple of the group (a third of them of
    the group alone), within the listed products' work."""
    while True:
        n = _log(rng, 48, 34816)
        n -= n % rng.choice((1, 16, 128))
        k = GROUP * _log(rng, 4, 136)
        if rng.random() < 0.67:
            k = max(512, k - k % 512)
        if n >= 16 and m * n * k <= LARGEST_MACS // 2 and n * k <= 34816 * 5120:
            return n, k


def draw(rng) -> dict:
    path = rng.choice(("linear1", "linear", "linear", "prefill", "swiglu", "chain", "layer", "embed", "host"))
    out = rng.choice(("f16", "f16", "f32"))
    if path == "linear1":
        n, k = _shape(rng, 1)
        return {"path": "linear", "m": 1, "n": n, "k": k, "out": out}
    if path in ("linear", "prefill"):
        m = _log(rng, 2, 128) if path == "linear" else _log(rng, 128, 2048)
        n, k = _shape(rng, m)
        return {"path": "linear", "m": m, "n": n, "k": k, "out": out}
    if path == "swiglu":
        m = _log(rng, 1, 1024)
        return {"path": "swiglu", "m": m, "n": 2 * rng.randint(256, 17408), "k": 512 * rng.randint(1, 10), "out": out}
    if path in ("chain", "layer"):
        sizes = {"hidden": 512 * rng.randint(2, 10), "ffn": 512 * rng.randint(4, 34), "kv": 128 * rng.randint(1, 8)}
        if path == "chain":
            return {"path": path, "layers": rng.randint(1, 8), **sizes}
        return {"path": path, "m": _log(rng, 2, 64), **sizes}
    if path == "embed":
        return {"path": "embed", "m": _log(rng, 1, 8192), "n": 16 * rng.randint(2000, 9496),
                "k": GROUP * rng.randint(4, 40), "out": out}
    return {"path": rng.choice(("load", "encode")), "n": 16 * _log(rng, 3, 640), "k": GROUP * _log(rng, 4, 48)}


def _weights(gen: torch.Generator, n: int, k: int) -> torch.Tensor:
    return random_blocks_device(n, k, gen, "cuda")


def _activations(gen: torch.Generator, m: int, k: int) -> torch.Tensor:
    return torch.randn((m, k), generator=gen, device="cuda").to(torch.float16)


def _linear(gen: torch.Generator, n: int, k: int, out: str = "f16") -> PackedLinear:
    module = PackedLinear(PackedTensorLayout.for_tensor(n, k), device="cuda",
                          out_dtype=torch.float32 if out == "f32" else None)
    module.load_blocks(_weights(gen, n, k))
    return module


def _chain(case: dict, gen: torch.Generator) -> dict:
    hidden, ffn, kv = case["hidden"], case["ffn"], case["kv"]
    shapes = ((hidden + 2 * kv, hidden), (hidden, hidden), (2 * ffn, hidden), (hidden, ffn))
    x = _activations(gen, 1, hidden)[0]
    links = []
    for layer in range(case["layers"]):
        for j, (n, k) in enumerate(shapes):
            swiglu = j == 2
            gain = swiglu_gain(1.0 / unit_gain(k)) if swiglu else unit_gain(k)
            y = torch.zeros(n // 2 if swiglu else n, dtype=torch.float16, device="cuda")
            # o reads the q rows of q|k|v, the first of its outputs
            source = {"x": x} if not links else {"source": len(links) - 1}
            links.append(Link(blocks=blocks_to_panels(_weights(gen, n, k)), panel_rows=n, y=y, swiglu=swiglu,
                              out_scale=gain, **source))
    return {"plan": ChainPlan(links), "outputs": [link.y for link in links]}


def _layer(case: dict, gen: torch.Generator) -> dict:
    hidden, ffn, kv = case["hidden"], case["ffn"], case["kv"]
    q, k, v = _linear(gen, hidden, hidden), _linear(gen, kv, hidden), _linear(gen, kv, hidden)
    o, down = _linear(gen, hidden, hidden), _linear(gen, hidden, ffn)
    gate_up = interleave_gate_up(_weights(gen, ffn, hidden), _weights(gen, ffn, hidden))

    def forward(x):
        query = q(x)
        attended = o(query)
        gated = tq1_swiglu(gate_up, attended)
        return query, k(x), v(x), attended, gated, down(gated)

    x = _activations(gen, case["m"], hidden)
    return {"step": GraphedStep(forward, [x]), "x": x, "keep": (q, k, v, o, down, gate_up)}


def prepare(case: dict, seed: int) -> dict:
    path = case["path"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if path == "chain":
        return {"path": path, **_chain(case, gen)}
    if path == "layer":
        return {"path": path, **_layer(case, gen)}
    n, k = case["n"], case["k"]
    if path == "encode":
        rng = np.random.default_rng(seed)
        codes = rng.choice(np.arange(3, dtype=np.uint8), size=(n * k // GROUP, GROUP), p=(0.3, 0.4, 0.3))
        scales = (np.abs(rng.standard_normal(n * k // GROUP)) * 0.02).astype(np.float16)
        return {"path": path, "codes": codes, "scales": scales.view(np.uint8).reshape(-1, 2)}
    layout = PackedTensorLayout.for_tensor(n, k)
    if path == "load":
        codes, scales = pack_blocks(_weights(gen, n, k).cpu().numpy(), layout=layout)
        return {"path": path, "module": PackedLinear(layout, device="cuda"), "codes": codes, "scales": scales}
    if path in ("embed", "head"):
        dtype = torch.float32 if case["out"] == "f32" else torch.float16
        table = PackedEmbedding(layout, dtype=dtype, device="cuda")
        table.load_blocks(_weights(gen, n, k))
        if path == "head":
            return {"path": path, "table": table, "x": _activations(gen, case["m"], k)}
        return {"path": path, "table": table, "ids": torch.randint(0, n, (case["m"],), generator=gen, device="cuda")}
    x = _activations(gen, case["m"], k)
    if path == "swiglu":
        return {"path": path, "blocks": interleave_gate_up(_weights(gen, n // 2, k), _weights(gen, n // 2, k)), "x": x,
                "dtype": torch.float32 if case["out"] == "f32" else torch.float16}
    return {"path": path, "module": _linear(gen, n, k, case["out"]), "x": x}


def run(state: dict):
    path = state["path"]
    if path == "linear":
        return state["module"](state["x"])
    if path == "head":
        return state["table"].as_linear(state["x"])
    if path == "swiglu":
        return tq1_swiglu(state["blocks"], state["x"], out_dtype=state["dtype"])
    if path == "embed":
        return state["table"](state["ids"])
    if path == "layer":
        return state["step"](state["x"])
    if path == "chain":
        state["plan"].run()
        return state["outputs"]
    if path == "load":
        state["module"].load_tiled(state["codes"], state["scales"])
        return state["module"].blocks
    return encode_tq1_blocks(state["scales"], state["codes"])


def work(case: dict) -> dict:
    path = case["path"]
    if path in ("chain", "layer"):
        hidden, ffn, kv = case["hidden"], case["ffn"], case["kv"]
        m, layers = case.get("m", 1), case.get("layers", 1)
        weights = layers * (2 * hidden * (hidden + kv) + 3 * hidden * ffn)
        # the layer's input once, every projection's output once
        values = hidden + layers * (3 * hidden + 2 * kv + ffn)
        return {"bytes": weights // GROUP * BLOCK + 2 * m * values, "flops": 2 * m * weights}
    packed = case["n"] * case["k"] // GROUP * BLOCK
    if path == "load":
        return {"bytes": 2 * packed, "flops": 0}
    if path == "encode":
        return {"bytes": case["n"] * case["k"] + packed, "flops": 0}
    m, n, k, size = case["m"], case["n"], case["k"], 4 if case["out"] == "f32" else 2
    if path == "embed":
        return {"bytes": m * (8 + k // GROUP * BLOCK + size * k), "flops": 0}
    outputs = n // 2 if path == "swiglu" else n
    return {"bytes": packed + 2 * m * k + size * m * outputs, "flops": 2 * m * n * k}


def tolerance(case: dict):
    path = case["path"]
    if path in ("embed", "load", "encode"):
        return "exact"          # one rounding of -s, 0 or +s, and byte copies
    if path == "chain":
        # a link reads its source rounded to FP16; SiLU*up spreads a last-place difference by about 1.4 per layer
        return {"rel": 1e-2}
    if path == "layer":
        return {"rel": 2e-3}    # four FP16 roundings in a row
    if case["out"] == "f16":
        return {"rel": 1e-3}    # one FP16 rounding of an FP32 sum
    return {"rel": 2e-5}        # FP32 sums of up to 17408 products of FP16 values
