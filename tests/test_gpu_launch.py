"""What a call launches, read from the kernel nodes of a captured graph: grids, arguments and launch attributes."""

from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def done(result):
    assert int(result[0]) == 0, result[0]
    return result[1] if len(result) == 2 else result[1:]


def kernel_nodes(call, stream=None):
    """``(kernel, grid, node)`` of every kernel that ``call`` launches, in launch order."""
    from cuda.bindings import driver

    call()  # per-kernel attributes are set outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = done(driver.cuGraphGetNodes(raw, 0))[1]
    out = []
    for node in done(driver.cuGraphGetNodes(raw, count))[0]:
        if done(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = done(driver.cuGraphKernelNodeGetParams(node))
            out.append((done(driver.cuFuncGetName(p.func)).decode(), (p.gridDimX, p.gridDimY, p.gridDimZ), node))
    return graph, out


@pytest.mark.parametrize("tokens", [2, 3, 4, 6])
@pytest.mark.parametrize("rank", [0, 5])
def test_a_rank_of_an_expert_layer_is_launched_for_its_share_of_the_assignments(tokens, rank):
    """16 of 128 experts: an eighth of the assignments come here, so the experts that have work are
    spread over more CTAs than if every assignment were theirs; the result is the same up to the order of sums."""
    from dynquant_b200 import ops
    from dynquant_b200.workloads import qwen3_moe_layer, seeded_routing

    layer = qwen3_moe_layer("cuda", seed=3, num_experts=16, hidden=2048, inter=768, topk=8)
    ids, w = seeded_routing(tokens, 128, 8, seed=tokens, device="cuda")
    x = torch.randn(tokens, 2048, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()

    def call(total):
        return ops.moe_gemv(x, ids, w, layer.gate_up, layer.down, num_experts=16, first_expert=16 * rank,
                            out_dtype=torch.float32, total_experts=total)

    share, whole = call(128), call(None)
    assert float((share - whole).norm()) <= 2e-3 * float(whole.norm())
    (_, of_share), (_, of_whole) = kernel_nodes(lambda: call(128)), kernel_nodes(lambda: call(None))
    assert "moe_grouped_kernel" in of_share[0][0] and of_share[0][1][1] == of_whole[0][1][1]
    if rank == 0:  # (without the total, the experts below the first are all that is known of the others)
        assert of_share[0][1][0] > of_whole[0][1][0]


def slices_of(call):
    """Slices of the reduction axis of every moe_grouped_kernel that ``call`` launches, from the kernel's argument: its
    integers after six pointers hold the steps of the axis, slices, row tiles and steps per slice, in this order."""
    from cuda.bindings import driver

    graph, nodes = kernel_nodes(call)
    out = []
    for name, _, node in nodes:
        if "moe_grouped_kernel" in name:
            arrays = done(driver.cuGraphKernelNodeGetParams(node)).kernelParams
            argument = ctypes.cast(arrays, ctypes.POINTER(ctypes.c_void_p))[0]
            numbers = (ctypes.c_int32 * 16).from_address(argument + 6 * 8)
            in_features, steps, slices, tiles, share = numbers[11:16]
            assert steps == -(-in_features // 128) and slices * share == steps and slices * tiles == 8
            out.append(slices)
    return out


def window_of(call, stream=None):
    """First and last address of the L2 access policy window of the ONE kernel that ``call`` launches; None without one."""
    from cuda.bindings import driver

    graph, nodes = kernel_nodes(call, stream)
    assert len(nodes) == 1, [name for name, *_ in nodes]
    window = done(driver.cuGraphKernelNodeGetAttribute(
        nodes[0][2], driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_ACCESS_POLICY_WINDOW)).accessPolicyWindow
    return (int(window.base_ptr), int(window.base_ptr) + int(window.num_bytes)) if int(window.num_bytes) else None


def side_by_side(sizes, k, gap):
    """4-bit matrices whose packed words lie in one buffer, ``gap`` bytes apart, and the bytes of the first gap."""
    from dynquant_b200.workloads import random_quant_tensor

    shards = [random_quant_tensor(n, k, 4, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)) for n in sizes]
    words = [q.packed.numel() for q in shards]
    buffer = torch.zeros(sum(words) + gap // 4 * len(sizes), dtype=torch.int32, device="cuda")
    at = 0
    for q, n in zip(shards, words):
        q.packed = buffer[at:at + n].copy_(q.packed.view(-1)).view(q.packed.shape)
        at += n + gap // 4
    return shards, buffer[words[0]:words[0] + gap // 4]


def extent(*tensors):
    return min(t.data_ptr() for t in tensors), max(t.data_ptr() + t.numel() * t.element_size() for t in tensors)


@pytest.mark.parametrize("between", [None, "x", "out", "bias"])
def test_the_window_covers_weights_only(between):
    """Two matrices close together: one window over both -- unless the launch's own activation, output or bias lies
    between them; then over the larger one."""
    from dynquant_b200 import ops

    shards, gap = side_by_side((1024, 2048), 2048, 1 << 16)
    x, out, bias = (torch.empty(n, dtype=torch.bfloat16, device="cuda") for n in (2048, 3072, 3072))
    inside = gap.view(torch.bfloat16)
    x, out, bias = (inside[:t.numel()] if name == between else t for name, t in (("x", x), ("out", out), ("bias", bias)))
    x.normal_(), bias.normal_()
    window = window_of(lambda: ops.gemv_shards(x.view(1, -1), shards, bias, out=out.view(1, -1)))
    assert ops.last_kernel() == "gemv_mma_tile_kernel"
    assert window == (extent(shards[1].packed) if between else extent(*(q.packed for q in shards)))


def test_matrices_far_apart_get_a_window_over_the_largest():
    from dynquant_b200 import ops

    shards, _ = side_by_side((1024, 2048), 2048, 8 << 20)
    x = torch.randn(1, 2048, device="cuda").to(torch.bfloat16)
    assert window_of(lambda: ops.gemv_shards(x, shards)) == extent(shards[1].packed)


def test_weights_that_a_call_reads_again_have_no_window():
    from dynquant_b200 import ops

    (qt,), _ = side_by_side((1024,), 512, 0)  # too short for the many-rows kernel: two chunks of rows in one launch
    x = torch.randn(12, 512, device="cuda").to(torch.bfloat16)
    assert window_of(lambda: ops.gemv_row_chunks(x, [qt])) is None
    assert ops.last_kernel() == "gemv_mma_tile_kernel"
    assert window_of(lambda: ops.gemv_shards(x[:1], [qt, qt])) is None  # the same matrix twice in one launch
    assert window_of(lambda: ops.gemv_row_chunks(x[:1], [qt])) == extent(qt.packed)


@pytest.mark.parametrize(("rows", "k", "kernel"), [
    (2048, 2048, "gemv_mma_tile_kernel"),
    (5120, 17408, "gemv_mma_stream_sliced_kernel"),
    (32768, 2048, "gemv_mma_stream_kernel"),
])
def test_a_window_of_the_stream_stays(rows, k, kernel):
    """A host that keeps its cache resident through its stream's own window keeps it under these launches."""
    from cuda.bindings import runtime

    from dynquant_b200 import ops

    (qt,), _ = side_by_side((rows,), k, 0)
    x = torch.randn(1, k, device="cuda").to(torch.bfloat16)
    cache = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()

    def call():
        return ops.gemv(x, qt.packed, qt.scales, qt.offsets, 4, 128, k)

    want = call()
    assert ops.last_kernel() == kernel
    assert window_of(call, stream) == extent(qt.packed)
    value = runtime.cudaStreamAttrValue()
    value.accessPolicyWindow.base_ptr, value.accessPolicyWindow.num_bytes = cache.data_ptr(), cache.numel()
    value.accessPolicyWindow.hitRatio = 1.0
    value.accessPolicyWindow.hitProp = runtime.cudaAccessProperty.cudaAccessPropertyNormal
    value.accessPolicyWindow.missProp = runtime.cudaAccessProperty.cudaAccessPropertyStreaming
    done((*runtime.cudaStreamSetAttribute(stream.cuda_stream, runtime.cudaStreamAttrID.cudaLaunchAttributeAccessPolicyWindow, value), None))
    assert window_of(call, stream) in (None, extent(cache))  # whether a capture records the stream's is CUDA's affair
    with torch.cuda.stream(stream):
        got = call()
    stream.synchronize()
    assert torch.equal(got, want)
