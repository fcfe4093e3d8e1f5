"""What a call launches, read from the kernel nodes of a captured graph: grids and launch attributes."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def kernel_nodes(call):
    """``(kernel, grid, node)`` of every kernel that ``call`` launches, in launch order."""
    from cuda.bindings import driver

    def done(result):
        assert int(result[0]) == 0, result[0]
        return result[1] if len(result) == 2 else result[1:]

    call()  # per-kernel attributes are set outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
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
