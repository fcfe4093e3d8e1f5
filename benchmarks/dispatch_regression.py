"""The dispatch rules, each against the dispatch without it, over the shapes around its thresholds.

Needs a tuning build (``python -m dynquant_b200.build --tuning``): its environment switches take one
rule out of the dispatch at a time.  Every point is timed both ways -- CUDA events around one CUDA graph
over a ring of distinct weight tensors larger than twice the L2, so the packed bytes come from HBM --
and the two outputs are compared.  One JSON object per (rule, shape, width) whose kernel the rule
changes: ``m<M>`` = [us without, us with, kernel without, kernel with, largest relative difference];
a line per rule counts the points that kept their kernel, got faster, got slower.

Rules: ``models`` (both switches of the one-matrix kernels, the linear layers of real models),
``rows_96k`` and ``sliced_20m`` (one term each of ``rows_kernel_first`` and ``stream_sliced_first``),
``fused`` (``stream_sliced_fused_ctas``), ``gemm`` (``gemm_first`` up to 64 rows).

    python benchmarks/dispatch_regression.py [--rule NAME ...] [--bits 2,3,4,8] [--force]
"""

from __future__ import annotations

import argparse
import json
import os
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

from dynquant_b200 import ops  # noqa: E402
from dynquant_b200.workloads import random_quant_tensor  # noqa: E402


def one(shapes, m, group=128):
    """Calls of one matrix: (rows of each matrix, reduction axis, group, activation rows)."""
    return [((rows,), k, group, m) for rows, k in shapes]


# q/k/v, o, gate/up and down projections of hidden sizes 1536..8192
MODELS = [(4096, 4096), (11008, 4096), (4096, 11008), (1024, 4096), (3584, 3584), (512, 3584), (18944, 3584),
          (3584, 18944), (1536, 1536), (8960, 1536), (1536, 8960), (5120, 13824), (13824, 5120), (8192, 8192),
          (1024, 8192), (28672, 8192), (8192, 28672), (3072, 8192), (8192, 3072), (2048, 16384), (16384, 2048),
          (8192, 29568), (6144, 4096), (4608, 3584), (2560, 9728), (9728, 2560)]
RULES = {
    "models": (("DQ_B200_ROWS_SMALL_M", "DQ_B200_STREAM_SLICED"), one(MODELS, (1, 4, 8)) + one(MODELS, (1, 4, 8), 64)),
    # six to eight rows whose staged activation takes 96 to 144 KB, below 16 M values (and just outside)
    "rows_96k": (("DQ_B200_ROWS_96K",), one([
        (512, 6144), (1024, 6144), (1536, 6144), (2048, 6144), (2560, 6144), (1024, 7168), (2048, 7168), (512, 8192), (1024, 8192),
        (1536, 8192), (1920, 8192), (768, 9216), (1536, 9216), (1024, 10240), (1280, 12288), (1024, 3072), (2048, 3072), (5120, 3072),
        (1024, 3584), (4096, 3584), (1024, 4096), (2048, 4096), (3840, 4096)], (6, 7, 8))),
    # 20 M values and more, reduction axes that do not slice eight ways, about a CTA per SM
    "sliced_20m": (("DQ_B200_SLICED_20M",), one([
        (4096, 5120), (5120, 5120), (5632, 5120), (3072, 7168), (4096, 7168), (5120, 7168), (2560, 9216), (4096, 9216), (5632, 9216),
        (6144, 3584), (8192, 3584), (11264, 3584), (8192, 2560), (10240, 2560), (8192, 2816), (16384, 2816), (2048, 11008), (4096, 11008),
        (8192, 11008), (2560, 13824), (5120, 4608), (5632, 3840), (7168, 4608), (8704, 4608), (4608, 4608), (9472, 3584), (10240, 3584),
        (5632, 4352), (3840, 5632), (4096, 6656), (3328, 6144), (2816, 8704), (4608, 8704), (5120, 6656),
        (1536, 13824), (1536, 18944), (2304, 9728), (3072, 8960), (3328, 7936)], (1, 2, 4, 8))),
    "fused": (("DQ_B200_FUSED_SLICED",), [(rows, k, 128, (1, 2, 4, 8)) for rows, k in [
        ((12800, 12800), 4096), ((13312, 13312), 4096), ((16384, 16384), 4096), ((9216, 9216), 5120), ((7168, 7168), 8192),
        ((9472, 9472), 8192), ((5504, 5504), 8192), ((4096, 4096), 12288), ((8704, 8704), 6144), ((15360, 15360), 3072),
        ((5120, 5120), 10240), ((3584, 3584), 7168), ((5120, 512, 512), 5120), ((6144, 6144), 5120), ((4096, 4096), 7168),
        ((4096, 1024, 1024), 4096), ((6144, 1024, 1024), 4096), ((5120, 1024, 1024), 5120), ((8192, 1024, 1024), 8192),
        ((3072, 1024, 1024), 6144), ((2048, 512, 512), 8192), ((3584, 512, 512), 3584), ((8960, 8960), 1536), ((6144, 6144), 2048),
        ((9728, 9728), 2560), ((3072, 3072), 8192), ((5632, 5632), 4096), ((8192, 8192), 3072), ((8192, 8192), 4096), ((8192, 8192), 6144),
        ((11008, 11008), 4096), ((12288, 12288), 4096), ((6144, 6144), 8192), ((24576, 24576), 2048), ((14336, 14336), 4096),
        ((18944, 18944), 3584), ((13824, 13824), 5120), ((17408, 17408), 5120), ((28672, 28672), 8192)]]),
    "gemm": (("DQ_B200_GEMM_FIRST",), one([
        (1009, 1024), (2688, 512), (5760, 1024), (2816, 2048), (6144, 2048), (3584, 3584), (1024, 4096), (4096, 4096), (16384, 4096),
        (20480, 4096), (1536, 8960), (2048, 16384), (8192, 8192), (1024, 8192), (2048, 8192), (4096, 8192), (14336, 8192), (4096, 14336),
        (5120, 5120), (3072, 6144), (5120, 17408), (11008, 4096), (28672, 4096), (1024, 2048), (2048, 4096), (2560, 9216), (1536, 6144)], (9, 12, 16, 24, 32, 48)) + one([
        (512, 1152), (1024, 5760), (3072, 2880), (2048, 4224), (12288, 1920)], (1, 2, 4, 8), 64) + one([
        (256, 3584), (896, 3584), (1536, 3584), (1152, 7936), (1536, 8960), (512, 14336), (1536, 14336), (1024, 18944), (25390, 4736),
        (12288, 3712), (9216, 4480), (7407, 10624), (4096, 11136), (2048, 12672), (16384, 10368),
        (1024, 12672), (3072, 11136), (2048, 10624), (3072, 12672), (1152, 3584), (1280, 4608), (1536, 4608), (1152, 5632), (1408, 5632),
        (1152, 6656), (1280, 7936), (1408, 7936), (1536, 7936), (1152, 8960), (1280, 8960), (1152, 9728), (1536, 9728), (1024, 11008),
        (1536, 11008), (1152, 13824), (1536, 13824), (1536, 18944), (512, 18944), (256, 14336), (768, 14336), (1024, 14336), (512, 12288),
        (512, 16384), (1024, 16384), (512, 10240)], (1, 4, 6, 8))),
}


def timed(fn, ring, reps: int = 3) -> float:
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for q in ring[:2]:
            fn(q)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            for q in ring:
                fn(q)
    best = float("inf")
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(True), torch.cuda.Event(True)
        e0.record()
        graph.replay()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) * 1000 / len(ring))
    return best


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--rule", action="append", choices=sorted(RULES), help="repeatable (default: all)")
    ap.add_argument("--bits", default="2,3,4,8")
    ap.add_argument("--force", action="store_true", help="the kernel that the rule is about wherever it qualifies, against none")
    args = ap.parse_args()
    stamp = Path(__file__).resolve().parent.parent / "dynquant_b200" / "lib" / "obj" / "build_kind.txt"
    if not stamp.exists() or stamp.read_text().strip() != "tuning":
        print("note: not a tuning build -- the switches are ignored and both arms run the full dispatch "
              "(python -m dynquant_b200.build --tuning)", file=sys.stderr)

    def switch_to(env, switches):
        for s in switches:
            os.environ.pop(s, None)
        os.environ.update(env)

    for rule in args.rule or RULES:
        switches, points = RULES[rule]
        same = better = worse = 0
        for rows, k, group, rows_m in points:
            for bits in (int(b) for b in args.bits.split(",")):
                nbytes = sum(rows) * k * bits // 8
                n = max(2, min(24, (300 << 20) // nbytes + 1)) if nbytes < (150 << 20) else 3
                gen = torch.Generator(device="cuda").manual_seed(bits)
                ring = [[random_quant_tensor(r, k, bits, group_size=group, meta_dtype=torch.float16, device="cuda", generator=gen)
                         for r in rows] for _ in range(n)]
                rec = {}
                for m in rows_m:
                    x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)

                    def fn(q):
                        return ops.quantized_matmul(x, q[0]) if len(q) == 1 else ops.gemv_shards(x, q)

                    arms = []
                    for env in ({s: "0" for s in switches}, {s: "1" for s in switches} if args.force else {}):
                        switch_to(env, switches)
                        out = fn(ring[0])
                        torch.cuda.synchronize()
                        arms.append([env, out, ops.last_kernel(), 0.0])
                    if arms[0][2] == arms[1][2]:
                        same += 1
                        continue
                    for arm in arms:
                        switch_to(arm[0], switches)
                        arm[3] = timed(fn, ring)
                    (_, ref, old, t_old), (_, got, new, t_new) = arms
                    rec[f"m{m}"] = [round(t_old, 1), round(t_new, 1), old, new, f"{float((got - ref).abs().max() / ref.abs().max()):.0e}"]
                    if t_new > 1.03 * t_old:
                        worse += 1
                    else:
                        better += 1
                if rec:
                    print(json.dumps({"rule": rule, "shape": [*rows, k], "bits": bits, "group": group, **rec}), flush=True)
                del ring
        switch_to({}, switches)
        print(json.dumps({"rule": rule, "kept_their_kernel": same, "changed_not_slower": better, "changed_slower": worse}), flush=True)


if __name__ == "__main__":
    main()
