"""What a user of dynquant_b200 has it do, as cases that can be timed and compared.

Every case is one pass through a public entry point, over synthetic tensors of the shapes this
repository's configurations, tests and benchmark use (or odd sizes around them).  Kinds:

* ``linear``     -- ``runtime.DynQuantLinear``: a packed module in a PyTorch model, from one decode
                    token over a batch of sequences to a prefill of thousands of tokens;
* ``fused``      -- ``plugin.DynQuantLinearMethod.apply``: a serving framework's fused layer (q/k/v
                    with bias, gate/up), every shard with its own width;
* ``step``       -- ``stack.StepRunner``: the packed linears of a decode step, captured once and
                    replayed per token, every stage's members writing side by side;
* ``moe``        -- ``plugin.DynQuantMoEMethod.apply``: an expert layer, decode batches to prefill;
* ``embedding``  -- ``runtime.DynQuantEmbedding``: token rows out of a packed vocabulary table;
* ``dequantize`` -- ``QuantTensor.dequantize``: packed to dense, bit-exact;
* ``encode``     -- ``runtime.DynQuantLinear.from_linear``: dense to packed, bit-exact.
"""

from __future__ import annotations

import math
import random

import torch

from dynquant_b200 import workloads
from dynquant_b200.format import row_geometry
from dynquant_b200.plugin import DynQuantLinearMethod, DynQuantMoEMethod, ShardSpec
from dynquant_b200.runtime import DynQuantEmbedding, DynQuantLinear
from dynquant_b200.stack import StepRunner

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
VOCAB = 248320  # rows of the benchmark's embedding / lm_head
MOST_FLOPS = 2.0 * 4096 * 14336 * 4096  # no drawn case costs more than the largest listed one


def listed() -> list[dict]:
    return [
        # one decode token through one small packed layer of an eager model: BASELINE's first configuration
        dict(name="linear decode m1", kind="linear", m=1, rows=6144, k=2048, bits=4, group=128, dtype="bf16", bias=False),
        # q/k/v of the 2B stack in a serving framework, four sequences, biases as Qwen models have them
        dict(name="fused qkv m4", kind="fused", m=4, sizes="2048,1024,1024", widths="3,2,4", k=2048, group=128,
             dtype="bf16", bias=True),
        # the captured decode step of a small dense model with its lm_head: single-sequence latency
        dict(name="step 2b m1", kind="step", stack="2b", layers=15, head=True, m=1),
        # the captured decode step of a 14B model's layers, four sequences
        dict(name="step 14b m4", kind="step", stack="14b", layers=15, head=False, m=4),
        # continuous batching: a few dozen sequences, fp16, an odd number of rows, 64-value groups
        dict(name="linear batch m24 odd", kind="linear", m=24, rows=4097, k=4096, bits=3, group=64, dtype="fp16", bias=False),
        # a short prompt's prefill through a down projection
        dict(name="linear prefill m333", kind="linear", m=333, rows=4096, k=14336, bits=3, group=128, dtype="bf16", bias=True),
        # a long prompt's prefill through an up projection: the largest case
        dict(name="linear prefill m4096", kind="linear", m=4096, rows=14336, k=4096, bits=4, group=128, dtype="bf16",
             bias=False),
        # an expert layer (Qwen3-30B-A3B shape) decoding four tokens
        dict(name="moe decode t4", kind="moe", tokens=4, experts=128, topk=8, hidden=2048, inter=768, bits_gate_up=3,
             bits_down=4, dtype="bf16"),
        # the same layer prefilling an odd number of tokens
        dict(name="moe prefill t1000", kind="moe", tokens=1000, experts=128, topk=8, hidden=2048, inter=768, bits_gate_up=3,
             bits_down=4, dtype="bf16"),
        # token rows of a prompt out of the packed table
        dict(name="embedding 512", kind="embedding", ids=512, rows=VOCAB, k=2048, bits=8, group=128),
        # a whole layer back to dense
        dict(name="dequantize 14336x4096", kind="dequantize", rows=14336, k=4096, bits=3, group=128, dtype="bf16"),
        # packing a dense layer
        dict(name="encode 2048x6144", kind="encode", rows=2048, k=6144, bits=4, group=128, dtype="bf16", symmetric=False),
    ]


# --------------------------------------------------------------------------
# more cases of the same ranges
# --------------------------------------------------------------------------


def _log(rng: random.Random, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _bits(rng: random.Random) -> int:
    return rng.choice((2, 3, 4, 8))


def _width(rng: random.Random, low: int, high: int) -> int:
    """A reduction axis: whole 128-value groups mostly, else a multiple of 32 (a tensor-parallel slice)."""
    unit = 128 if rng.random() < 0.8 else 32
    return max(unit, _log(rng, low, high) // unit * unit)


def _rows(rng: random.Random, low: int, high: int) -> int:
    """Output rows: multiples of 128 mostly, else any number."""
    n = _log(rng, low, high)
    return n if rng.random() < 0.3 else max(128, n // 128 * 128)


def _group(rng: random.Random) -> int:
    return 64 if rng.random() < 0.25 else 128


def _dtype(rng: random.Random) -> str:
    return "fp16" if rng.random() < 0.25 else "bf16"


def _tokens(rng: random.Random, high: int) -> int:
    """Activation rows: a third each of decode (1..8), batches (9..64) and prefill."""
    return _log(rng, *rng.choice(((1, 8), (9, 64), (65, high))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("linear",) * 4 + ("fused",) * 2 + ("step",) * 2 + ("moe",) * 2 + ("embedding", "dequantize", "encode"))
    if kind == "linear":
        rows, k = _rows(rng, 512, 28672), _width(rng, 512, 18944)
        m = max(1, min(_tokens(rng, 4096), int(MOST_FLOPS / (2.0 * rows * k))))
        return dict(kind=kind, m=m, rows=rows, k=k, bits=_bits(rng), group=_group(rng), dtype=_dtype(rng),
                    bias=rng.random() < 0.3)
    if kind == "fused":
        k = _width(rng, 1024, 8192)
        if rng.random() < 0.5:
            q = _rows(rng, 1024, 8192)
            kv = max(128, q // rng.choice((1, 2, 4, 8)))
            sizes = (q, kv, kv)
        else:
            sizes = (_rows(rng, 1024, 17408),) * 2
        m = max(1, min(_tokens(rng, 2048), int(MOST_FLOPS / (2.0 * sum(sizes) * k))))
        return dict(kind=kind, m=m, sizes=",".join(map(str, sizes)), widths=",".join(str(_bits(rng)) for _ in sizes), k=k,
                    group=_group(rng), dtype=_dtype(rng), bias=rng.random() < 0.5)
    if kind == "step":
        stack = rng.choice(("2b", "14b"))
        return dict(kind=kind, stack=stack, layers=rng.randint(2, 15), head=stack == "2b" and rng.random() < 0.5,
                    m=rng.choice((1, 1, 2, 3, 4, 6, 8)))
    if kind == "moe":
        dtype = _dtype(rng)
        widths = (2, 3, 4) if dtype == "fp16" else (2, 3, 4, 8)  # (8-bit codes at these scales overflow fp16)
        experts = rng.choice((8, 16, 60, 64, 128))
        return dict(kind=kind, tokens=_tokens(rng, 2048), experts=experts, topk=rng.choice((2, 4, 6, 8)),
                    hidden=rng.choice((1024, 2048, 2816, 4096)), inter=rng.choice((512, 768, 1024, 1408, 1536)),
                    bits_gate_up=rng.choice(widths), bits_down=rng.choice(widths), dtype=dtype)
    if kind == "embedding":
        return dict(kind=kind, ids=_log(rng, 1, 4096), rows=_rows(rng, 32000, VOCAB), k=_width(rng, 1024, 4096),
                    bits=rng.choice((4, 8, 8)), group=_group(rng))
    if kind == "dequantize":
        k = _width(rng, 512, 14336)
        return dict(kind=kind, rows=_rows(rng, 512, min(28672, 2 * 14336 * 4096 // k)), k=k, bits=_bits(rng),
                    group=_group(rng), dtype=_dtype(rng))
    k = _width(rng, 512, 6144)
    return dict(kind=kind, rows=_rows(rng, 256, 2048), k=k, bits=_bits(rng), group=_group(rng), dtype=_dtype(rng),
                symmetric=rng.random() < 0.3)


# --------------------------------------------------------------------------
# inputs, one pass
# --------------------------------------------------------------------------


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _packed(rows: int, k: int, bits: int, group: int, meta: torch.dtype, gen: torch.Generator):
    return workloads.random_quant_tensor(rows, k, bits, group_size=group, meta_dtype=meta, device="cuda", generator=gen)


def _normal(gen: torch.Generator, dtype: torch.dtype, *shape: int) -> torch.Tensor:
    return torch.randn(*shape, device="cuda", generator=gen).to(dtype)


def _ints(text: str) -> list[int]:
    return [int(v) for v in text.split(",")]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    gen = _generator(seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    state: dict = {"kind": kind}
    if kind == "linear":
        weight = _packed(case["rows"], case["k"], case["bits"], case["group"], torch.float16, gen)
        bias = _normal(gen, dtype, case["rows"]) if case["bias"] else None
        state["module"] = DynQuantLinear(weight, bias)
        state["x"] = _normal(gen, dtype, case["m"], case["k"])
    elif kind == "fused":
        sizes, widths, k = _ints(case["sizes"]), _ints(case["widths"]), case["k"]
        specs = [ShardSpec(f"shard{i}", b, case["group"], n) for i, (n, b) in enumerate(zip(sizes, widths))]
        method, layer = DynQuantLinearMethod(None, specs), torch.nn.Module()
        method.create_weights(layer, k, sizes, k, sum(sizes), dtype, device="cuda")
        for i, (n, b) in enumerate(zip(sizes, widths)):
            method.load_shard(layer, i, _packed(n, k, b, case["group"], dtype, gen))
        state["method"], state["layer"] = method, layer
        state["bias"] = _normal(gen, dtype, sum(sizes)) if case["bias"] else None
        state["x"] = _normal(gen, dtype, case["m"], k)
    elif kind == "step":
        if case["stack"] == "2b":
            stack = workloads.qwen2b_stack(seed=seed, layers=case["layers"], vocab=VOCAB if case["head"] else 0)
        else:
            stack = workloads.qwen14b_linear_set(seed=seed, layers=case["layers"])
        runner = StepRunner(stack, case["m"], stage_outputs=True)
        for x in runner.inputs.values():
            x.copy_(_normal(gen, x.dtype, *x.shape))
        runner.capture()
        state["runner"] = runner
    elif kind == "moe":
        experts, hidden, inter = case["experts"], case["hidden"], case["inter"]
        method = DynQuantMoEMethod(None, bits_gate_up=case["bits_gate_up"], bits_down=case["bits_down"])
        layer = torch.nn.Module()
        method.create_weights(layer, experts, hidden, inter, dtype, device="cuda")
        method.load_banks(layer, _packed(experts * 2 * inter, hidden, case["bits_gate_up"], 128, dtype, gen),
                          _packed(experts * hidden, inter, case["bits_down"], 128, dtype, gen))
        ids, weights = workloads.seeded_routing(case["tokens"], experts, case["topk"], seed, device="cuda")
        state.update(method=method, layer=layer, ids=ids, weights=weights, x=_normal(gen, dtype, case["tokens"], hidden))
    elif kind == "embedding":
        state["module"] = DynQuantEmbedding(_packed(case["rows"], case["k"], case["bits"], case["group"], torch.float16, gen))
        state["ids"] = torch.randint(case["rows"], (case["ids"],), device="cuda", generator=gen)
    elif kind == "dequantize":
        state["weight"] = _packed(case["rows"], case["k"], case["bits"], case["group"], dtype, gen)
    else:
        linear = torch.nn.Linear(case["k"], case["rows"], bias=False, device="meta")
        dense = _normal(gen, dtype, case["rows"], case["k"]) * 0.02
        linear.weight = torch.nn.Parameter(dense, requires_grad=False)
        state.update(linear=linear, bits=case["bits"], group=case["group"], symmetric=case["symmetric"])
    return state


def run(state: dict):
    kind = state["kind"]
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "fused":
        return state["method"].apply(state["layer"], state["x"], state["bias"])
    if kind == "step":
        state["runner"].replay()
        return state["runner"].stage_buffers
    if kind == "moe":
        return state["method"].apply(state["layer"], state["x"], state["weights"], state["ids"])
    if kind == "embedding":
        return state["module"](state["ids"])
    if kind == "dequantize":
        return state["weight"].dequantize()
    packed = DynQuantLinear.from_linear(state["linear"], state["bits"], group_size=state["group"], symmetric=state["symmetric"])
    return {"qweight": packed.qweight, "scales": packed.scales, "offsets": packed.offsets}


# --------------------------------------------------------------------------
# what a pass cannot do without, and how close another implementation comes
# --------------------------------------------------------------------------


def _packed_bytes(rows: float, k: int, bits: float, group: int) -> float:
    """Words, scales and offsets (16-bit) of a packed matrix."""
    groups = row_geometry(8, group, k).num_groups
    return rows * groups * (group * bits / 8 + 4)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["rows"], case["k"]
        return {"bytes": _packed_bytes(n, k, case["bits"], case["group"]) + 2 * m * (n + k) + 2 * n * case["bias"],
                "flops": 2.0 * m * n * k}
    if kind == "fused":
        m, k, sizes = case["m"], case["k"], _ints(case["sizes"])
        weights = sum(_packed_bytes(n, k, b, case["group"]) for n, b in zip(sizes, _ints(case["widths"])))
        return {"bytes": weights + 2 * m * (sum(sizes) + k) + 2 * sum(sizes) * case["bias"], "flops": 2.0 * m * sum(sizes) * k}
    if kind == "step":
        # the width maps are seeded: their mean is fixed, which module has which width is not
        small = case["stack"] == "2b"
        h, inter, q, kv, bits = (2048, 6144, 2048, 1024, 3.25) if small else (5120, 17408, 5120, 1024, 3.5)
        shapes = [(q + 2 * kv, h), (h, q), (2 * inter, h), (h, inter)]
        m, total = case["m"], sum(n * k for n, k in shapes)
        moved = sum(_packed_bytes(n, k, bits, 128) + 2 * m * (n + k) for n, k in shapes) * case["layers"]
        flops = 2.0 * m * total * case["layers"]
        if case["head"]:
            moved += _packed_bytes(VOCAB, h, 8, 128) + 2 * m * (VOCAB + h)
            flops += 2.0 * m * VOCAB * h
        return {"bytes": moved, "flops": flops}
    if kind == "moe":
        t, e, topk, h, inter = (case[key] for key in ("tokens", "experts", "topk", "hidden", "inter"))
        active = e * (1.0 - (1.0 - topk / e) ** t)  # experts that some token chose, expected
        expert = _packed_bytes(2 * inter, h, case["bits_gate_up"], 128) + _packed_bytes(h, inter, case["bits_down"], 128)
        return {"bytes": active * expert + 4 * t * h + 8 * t * topk, "flops": 2.0 * t * topk * 3 * h * inter}
    if kind == "embedding":
        n, k = case["ids"], case["k"]
        return {"bytes": _packed_bytes(n, k, case["bits"], case["group"]) + 2 * n * k + 8 * n, "flops": 2.0 * n * k}
    n, k = case["rows"], case["k"]  # dequantize, encode: packed on one side, dense on the other
    return {"bytes": _packed_bytes(n, k, case["bits"], case["group"]) + 2 * n * k, "flops": 2.0 * n * k}


def tolerance(case: dict):
    if case["kind"] in ("embedding", "dequantize", "encode"):
        return "exact"
    # 16-bit inputs and results, fp32 sums: where a weight is decoded to 16 bits on the way (prefill) and
    # where an expert's intermediate is rounded, two correct programs differ by a few roundings
    return {"rel": 1e-2 if case.get("dtype", "bf16") == "bf16" else 2e-3}
