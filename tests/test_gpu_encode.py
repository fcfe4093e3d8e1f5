"""``dq_encode`` and ``dq_dequant_rows`` against the host encoder and the gathered dequant."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize(("rows", "k", "group", "symmetric", "dtype"), [
    (5, 256, 128, False, torch.bfloat16),
    (7, 328, 128, True, torch.float16),    # a last group of 72 values, padded with zeros
    (33, 1000, 64, False, torch.float32),  # ... of 40
    (3, 96, 32, True, torch.bfloat16),
    (2, 4096, 256, False, torch.float16),
])
def test_encode_is_bit_identical_to_the_host_encoder(bits, rows, k, group, symmetric, dtype):
    from dynquant_b200 import QuantTensor
    from dynquant_b200.runtime import DynQuantLinear

    gen = torch.Generator().manual_seed(bits * 1000 + k)
    w = (torch.randn(rows, k, generator=gen) * 0.05).to(dtype)
    w[0] = 0.25          # constant groups: scale 0
    w[1, :group] = 0.0   # ... of zeros
    w[-1, 3] = 1e-7 if dtype == torch.float16 else 1e-30  # a tiny range next to it
    meta = dtype if dtype != torch.float32 else torch.float16
    want = QuantTensor.from_dense(w, bits=bits, group_size=group, symmetric=symmetric, compute_dtype=meta)
    linear = torch.nn.Linear(k, rows, bias=False, device="meta")
    linear.weight = torch.nn.Parameter(w.cuda(), requires_grad=False)
    got = DynQuantLinear.from_linear(linear, bits, group_size=group, symmetric=symmetric)
    assert torch.equal(got.qweight.cpu(), want.packed)
    assert torch.equal(got.scales.cpu(), want.scales) and got.scales.dtype == meta
    assert torch.equal(got.offsets.cpu(), want.offsets)


@pytest.mark.parametrize("ids_dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize(("k", "group", "bits"), [(512, 128, 8), (328, 64, 3), (100, -1, 4), (2048, 128, 2)])
def test_embedding_rows_equal_the_rows_of_the_dense_table(k, group, bits, ids_dtype):
    from dynquant_b200 import QuantTensor
    from dynquant_b200.runtime import DynQuantEmbedding

    table = QuantTensor.from_dense(torch.randn(300, k), bits=bits, group_size=group, compute_dtype=torch.bfloat16).to("cuda")
    ids = torch.randint(300, (3, 41), device="cuda").to(ids_dtype)
    got = DynQuantEmbedding(table)(ids)
    assert got.shape == (3, 41, k)
    assert torch.equal(got, table.dequantize()[ids.long()])


@pytest.mark.parametrize("m", [1, 24, 100])
def test_a_call_right_behind_the_encoder_waits_for_its_words(m):
    """The multiplying kernels request weights before their programmatic dependency resolves: the
    edge that leaves the encoder must be an ordinary one."""
    from cuda.bindings import runtime as cudart

    from dynquant_b200.runtime import DynQuantLinear

    rows, k = 640, 1024
    linear = torch.nn.Linear(k, rows, bias=False, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    want = DynQuantLinear.from_linear(linear, 4)
    torch.cuda.synchronize()
    want = want(x)
    torch.cuda.synchronize()
    for _ in range(20):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            got = DynQuantLinear.from_linear(linear, 4)(x)
        stream.synchronize()
        assert torch.equal(got, want)

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        layer = DynQuantLinear.from_linear(linear, 4)
        got = layer(x)
    raw = cudart.cudaGraph_t(graph.raw_cuda_graph())
    err, _, _, _, count = cudart.cudaGraphGetEdges_v2(raw)
    assert err == cudart.cudaError_t.cudaSuccess and count >= 2
    err, sources, targets, _, _ = cudart.cudaGraphGetEdges_v2(raw, count)
    err, roots, _ = cudart.cudaGraphGetRootNodes(raw, 1)
    kind = lambda node: cudart.cudaGraphNodeGetType(node)[1]  # noqa: E731
    assert kind(roots[0]) == cudart.cudaGraphNodeType.cudaGraphNodeTypeKernel
    behind = [t for s, t in zip(sources, targets) if int(s) == int(roots[0])]
    # (a programmatic edge joins two kernels: none leaves the encoder)
    assert behind and all(kind(t) == cudart.cudaGraphNodeType.cudaGraphNodeTypeMemset for t in behind)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("bad", [300, -1, 2**40])
@pytest.mark.parametrize("k", [512, 100])
def test_an_id_outside_the_table_is_raised_by_the_next_call(k, bad):
    from dynquant_b200 import QuantTensor, ops
    from dynquant_b200.runtime import DynQuantEmbedding

    table = DynQuantEmbedding(QuantTensor.from_dense(torch.randn(300, k), bits=4, group_size=-1, compute_dtype=torch.bfloat16).to("cuda"))
    good = torch.tensor([0, 299, 7], device="cuda")
    want = table(good)
    ids = torch.tensor([0, bad, 7], device="cuda")
    rows = table(ids)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="id outside"):
        table(good)
    assert torch.equal(table(good), want)  # raised once
    assert torch.equal(rows[::2], want[::2]) and bool(rows[1].isnan().all())
    table(ids)
    with pytest.raises(RuntimeError, match="id outside"):
        ops.check_status()
    ops.check_status()
