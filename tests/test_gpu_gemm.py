"""The tcgen05 kernel for many activation rows (``gemm_umma_kernel``) at the edges of its tiles."""

from __future__ import annotations

import pytest
import torch

from test_gpu_parity import oracle_gemv, within_one_ulp_16
from test_gpu_shapes import random_qt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize(("m", "rows", "k", "group", "act", "meta", "offsets"), [
    (9, 129, 640, 128, torch.bfloat16, torch.float16, True),     # one row past a tile, an odd number of chunks
    (64, 257, 1152, 64, torch.float16, torch.bfloat16, False),   # the last row count with split weights
    (65, 127, 128, 128, torch.bfloat16, torch.bfloat16, True),   # the first without, one chunk
    (256, 640, 2048, 128, torch.float16, torch.float16, True),   # a full token tile, sliced over a cluster
    (257, 1000, 416, 64, torch.bfloat16, torch.float16, True),   # one token past it, a ragged reduction axis
    (700, 20000, 256, 256, torch.bfloat16, torch.bfloat16, False),  # several tiles per block
    (206, 1536, 8192, 128, torch.bfloat16, torch.float16, True),    # the shortest rings: slots refilled at once
])
def test_many_rows_match_the_oracle(bits, m, rows, k, group, act, meta, offsets):
    import ctypes

    from dynquant_b200 import _lib, ops

    qt = random_qt(rows, k, bits, group=group, meta=meta, seed=m + bits, offsets=offsets)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(act).cuda()
    bias = torch.randn(rows, generator=torch.Generator().manual_seed(3)).to(act).cuda()
    lib, tag = _lib.load(), _lib.DQ_BF16 if act == torch.bfloat16 else _lib.DQ_F16
    w = ops.weight_descriptor("gemm", qt.packed, qt.scales, qt.offsets, bits, group, k)
    padded = torch.full((m + 2, rows), 7.0, dtype=act, device="cuda")
    out, stream = padded[1:-1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = lib.dq_gemm_shards(x.data_ptr(), tag, m, ctypes.byref(w), 1, bias.data_ptr(), out.data_ptr(), rows, tag, stream)
    if bits == 3 and group == 64 and -(-k // 64) % 2:
        assert rc == _lib.DQ_ERR_UNSUPPORTED  # rows that are not whole 16-byte pieces
        return
    assert rc == _lib.DQ_OK and ops.last_kernel() == "gemm_umma_kernel"
    assert lib.dq_gemm_status(stream) == _lib.DQ_OK
    assert bool((padded[0] == 7.0).all()) and bool((padded[-1] == 7.0).all())
    dense = ops.dequant(qt.packed, qt.scales, qt.offsets, bits, group, k, out_dtype=torch.float32)
    want = x.double() @ dense.double().T + bias.double()
    if m <= 64:  # weights enter unrounded: the fp32 result, rounded once
        assert within_one_ulp_16(out, want.float().cpu().numpy())
    else:        # weights rounded once to the activation type
        error = (out.double() - want).norm() / want.norm()
        assert error <= (4e-3 if act == torch.bfloat16 else 5e-4)
    again = torch.empty_like(out)
    lib.dq_gemm_shards(x.data_ptr(), tag, m, ctypes.byref(w), 1, bias.data_ptr(), again.data_ptr(), rows, tag, stream)
    assert torch.equal(out, again)


@pytest.mark.parametrize("m", [2, 7, 12, 40, 130])
def test_shards_of_mixed_widths_in_one_launch(m):
    from dynquant_b200 import ops
    from dynquant_b200.plugin import DynQuantLinearMethod, ShardSpec

    k, sizes, widths = 1408, (300, 128, 77), (8, 2, 3)  # 11 steps of 64-value groups: the tcgen05 kernel at any row count
    method, layer = DynQuantLinearMethod(None, [ShardSpec(str(i), b, 64, n) for i, (n, b) in enumerate(zip(sizes, widths))]), torch.nn.Module()
    method.create_weights(layer, k, list(sizes), k, sum(sizes), torch.bfloat16, device="cuda")
    shards = [random_qt(n, k, b, group=64, meta=torch.bfloat16, seed=b) for n, b in zip(sizes, widths)]
    for i, qt in enumerate(shards):
        method.load_shard(layer, i, qt)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()
    bias = torch.randn(sum(sizes)).to(torch.bfloat16).cuda()
    before = ops.launch_count()
    got = method.apply(layer, x, bias)
    assert ops.launch_count() - before == 1 and ops.last_kernel() == "gemm_umma_kernel"
    want = torch.cat([torch.from_numpy(oracle_gemv(x, qt)) for qt in shards], dim=1) + bias.float().cpu()
    error = (got.float().cpu() - want).norm() / want.norm()
    assert error <= 4e-3


@pytest.mark.parametrize(("m", "k", "sizes", "widths", "group"), [
    (9, 4096, (19000,), (3,), 128),               # 149 row tiles, the last one ragged: a whole wave and one tile
    (64, 4096, (12000, 7101, 300), (4, 2, 8), 64),  # the cut falls into the second shard
    (200, 4096, (12001, 7000), (4, 4), 128),      # an odd row count before the cut: output columns that start anywhere
])
def test_a_last_wave_of_few_tiles_is_a_launch_of_its_own(m, k, sizes, widths, group):
    from dynquant_b200 import ops
    from dynquant_b200.plugin import DynQuantLinearMethod, ShardSpec

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are chosen for 148 SMs")
    method, layer = DynQuantLinearMethod(None, [ShardSpec(str(i), b, group, n) for i, (n, b) in enumerate(zip(sizes, widths))]), torch.nn.Module()
    method.create_weights(layer, k, list(sizes), k, sum(sizes), torch.bfloat16, device="cuda")
    shards = [random_qt(n, k, b, group=group, meta=torch.bfloat16, seed=b) for n, b in zip(sizes, widths)]
    for i, qt in enumerate(shards):
        method.load_shard(layer, i, qt)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()
    bias = torch.randn(sum(sizes), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    before = ops.launch_count()
    got = method.apply(layer, x, bias)
    assert ops.launch_count() - before == 2 and ops.last_kernel() == "gemm_umma_kernel"
    dense = torch.cat([ops.dequant(q.packed, q.scales, q.offsets, q.bits, group, k, out_dtype=torch.float32) for q in shards])
    want = x.double() @ dense.double().T + bias.double()
    if m <= 64:
        assert within_one_ulp_16(got, want.float().cpu().numpy())
    else:
        assert (got.double() - want).norm() / want.norm() <= 4e-3
    assert torch.equal(got, method.apply(layer, x, bias))


@pytest.mark.parametrize("m", [40, 200])
def test_a_shard_that_the_kernel_does_not_take_behind_a_whole_wave(m):
    """148 row tiles that could be a launch of their own, and behind them a matrix of a group size that is no power of
    two: another path computes all of it."""
    from dynquant_b200 import ops
    from dynquant_b200.plugin import DynQuantLinearMethod, ShardSpec

    k, sizes, groups = 6144, (148 * 128, 300), (128, 96)
    method, layer = DynQuantLinearMethod(None, [ShardSpec(str(i), 4, g, n) for i, (n, g) in enumerate(zip(sizes, groups))]), torch.nn.Module()
    method.create_weights(layer, k, list(sizes), k, sum(sizes), torch.bfloat16, device="cuda")
    shards = [random_qt(n, k, 4, group=g, meta=torch.bfloat16, seed=n) for n, g in zip(sizes, groups)]
    for i, qt in enumerate(shards):
        method.load_shard(layer, i, qt)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()
    dense = torch.cat([ops.dequant(q.packed, q.scales, q.offsets, q.bits, g, k, out_dtype=torch.float32) for q, g in zip(shards, groups)])
    want = x.double() @ dense.double().T
    # bf16 outputs, and above 64 rows bf16 weights: 2 ** -9 each at most
    assert (method.apply(layer, x, None).double() - want).norm() / want.norm() <= 4e-3


@pytest.mark.parametrize(("tokens", "experts", "topk", "hidden", "inter", "widths", "act", "meta"), [
    (1, 8, 2, 256, 192, (4, 3), torch.bfloat16, torch.float16),      # one token; 64-row blocks that end inside a tile
    (64, 4, 2, 512, 128, (2, 8), torch.float16, torch.float16),      # tiles of 64 columns and fewer
    (130, 2, 2, 384, 320, (8, 2), torch.bfloat16, torch.bfloat16),   # every expert has every token: 128 + 2 columns
    (700, 16, 4, 1024, 512, (3, 4), torch.bfloat16, torch.float16),  # several tiles per block, small and large in turn
])
def test_an_expert_layer_over_many_tokens_matches_its_small_calls(tokens, experts, topk, hidden, inter, widths, act, meta):
    import ctypes

    from dynquant_b200 import _lib, ops
    from dynquant_b200.workloads import random_quant_tensor, seeded_routing

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    gate_up = random_quant_tensor(experts * 2 * inter, hidden, widths[0], meta_dtype=meta, device="cuda", generator=gen)
    down = random_quant_tensor(experts * hidden, inter, widths[1], meta_dtype=meta, device="cuda", generator=gen)
    ids, weights = seeded_routing(tokens, experts, topk, seed=tokens, device="cuda")
    ids[0, 0] = -1  # an assignment that belongs to nobody here
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(act)
    want = torch.cat([ops.moe_gemv(x[i:i + 64].contiguous(), ids[i:i + 64].contiguous(), weights[i:i + 64].contiguous(), gate_up, down,
                                   num_experts=experts, out_dtype=torch.float32) for i in range(0, tokens, 64)])
    lib, tag, need = _lib.load(), _lib.DQ_BF16 if act == torch.bfloat16 else _lib.DQ_F16, ctypes.c_int64()
    _lib.check(lib.dq_moe_gemm_scratch_bytes(tokens, topk, hidden, inter, experts, tag, ctypes.byref(need)))
    scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    banks = [ops.weight_descriptor("moe", q.packed, q.scales, q.offsets, q.bits, 128, q.in_features) for q in (gate_up, down)]
    outs = []
    for _ in range(2):
        y = torch.full((tokens + 2, hidden), 7.0, device="cuda")
        _lib.check(lib.dq_moe_gemm(x.data_ptr(), tag, tokens, ids.data_ptr(), weights.data_ptr(), topk, 0, experts, ctypes.byref(banks[0]),
                                   ctypes.byref(banks[1]), hidden, inter, y[1:-1].data_ptr(), _lib.DQ_F32, scratch.data_ptr(), need.value, stream))
        outs.append(y)
    assert ops.last_kernel() == "moe_umma_kernel" and lib.dq_gemm_status(stream) == _lib.DQ_OK
    assert torch.equal(outs[0], outs[1]) and bool((outs[0][0] == 7.0).all()) and bool((outs[0][-1] == 7.0).all())
    # the intermediate is rounded on both sides: flips of its last bit are what differs
    assert (outs[0][1:-1] - want).norm() / want.norm() <= (1e-3 if act == torch.bfloat16 else 2e-4)


def gemm(x, qt):
    """``dq_gemm_shards`` of one matrix."""
    import ctypes

    from dynquant_b200 import _lib, ops

    lib, tag = _lib.load(), _lib.DQ_BF16 if x.dtype == torch.bfloat16 else _lib.DQ_F16
    w = ops.weight_descriptor("gemm", qt.packed, qt.scales, qt.offsets, qt.bits, qt.geometry.effective_group, qt.in_features)
    out = torch.empty(x.shape[0], qt.num_rows, dtype=x.dtype, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.dq_gemm_shards(x.data_ptr(), tag, x.shape[0], ctypes.byref(w), 1, None, out.data_ptr(), qt.num_rows, tag, stream))
    return out


def moe_gemm(x, ids, weights, gate_up, down, experts, *, first_expert=0):
    """``dq_moe_gemm`` with fp32 results."""
    import ctypes

    from dynquant_b200 import _lib, ops

    lib, tag, need = _lib.load(), _lib.DQ_BF16 if x.dtype == torch.bfloat16 else _lib.DQ_F16, ctypes.c_int64()
    (tokens, hidden), topk, inter = x.shape, ids.shape[1], down.in_features
    _lib.check(lib.dq_moe_gemm_scratch_bytes(tokens, topk, hidden, inter, experts, tag, ctypes.byref(need)))
    scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    banks = [ops.weight_descriptor("moe", q.packed, q.scales, q.offsets, q.bits, 128, q.in_features) for q in (gate_up, down)]
    y = torch.empty(tokens, hidden, device="cuda")
    _lib.check(lib.dq_moe_gemm(x.data_ptr(), tag, tokens, ids.data_ptr(), weights.data_ptr(), topk, first_expert, experts, ctypes.byref(banks[0]),
                               ctypes.byref(banks[1]), hidden, inter, y.data_ptr(), _lib.DQ_F32, scratch.data_ptr(), need.value, stream))
    return y


def test_an_expert_layer_over_more_tokens_than_a_grid_has_rows():
    from dynquant_b200.workloads import random_quant_tensor, seeded_routing

    tokens, experts, hidden, inter = 70000, 8, 256, 128  # a grid's y axis ends at 65535
    gen = torch.Generator(device="cuda").manual_seed(1)
    gate_up = random_quant_tensor(experts * 2 * inter, hidden, 4, meta_dtype=torch.float16, device="cuda", generator=gen)
    down = random_quant_tensor(experts * hidden, inter, 3, meta_dtype=torch.float16, device="cuda", generator=gen)
    ids, weights = seeded_routing(tokens, experts, 2, seed=1, device="cuda")
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    whole = moe_gemm(x, ids, weights, gate_up, down, experts)
    parts = [moe_gemm(x[i:i + 30000], ids[i:i + 30000], weights[i:i + 30000], gate_up, down, experts) for i in range(0, tokens, 30000)]
    assert torch.equal(whole, torch.cat(parts))


def test_a_block_that_gives_up_reports_it_and_leaves_the_device_usable():
    from dynquant_b200 import _lib, ops
    from dynquant_b200.workloads import random_quant_tensor, seeded_routing

    lib, gen = _lib.load(), torch.Generator(device="cuda").manual_seed(1)
    for m, rows, k in ((24, 1000, 4096), (40, 20000, 512), (300, 1000, 2048), (4096, 4096, 512)):  # sliced and not, split and not
        qt = random_quant_tensor(rows, k, 4, meta_dtype=torch.float16, device="cuda", generator=gen)
        x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
        want = gemm(x, qt)
        for _ in range(3):
            lib.dq_gemm_fail_next(1)
            gemm(x, qt)
        with pytest.raises(RuntimeError, match="ran out"):
            ops.check_status()
        ops.check_status()  # once
        assert torch.equal(gemm(x, qt), want)
    bank = [random_quant_tensor(n, k, 3, meta_dtype=torch.float16, device="cuda", generator=gen) for n, k in ((8 * 512, 512), (8 * 512, 256))]
    ids, weights = seeded_routing(200, 8, 2, seed=1, device="cuda")
    x = torch.randn(200, 512, device="cuda", generator=gen).to(torch.bfloat16)
    want = moe_gemm(x, ids, weights, *bank, 8)
    lib.dq_gemm_fail_next(1)
    moe_gemm(x, ids, weights, *bank, 8)
    torch.cuda.synchronize()
    assert lib.dq_poll_status(0) == _lib.DQ_ERR_DEVICE and lib.dq_poll_status(0) == _lib.DQ_OK
    assert torch.equal(moe_gemm(x, ids, weights, *bank, 8), want)


def test_a_module_raises_what_its_last_call_reported():
    from dynquant_b200 import _lib
    from dynquant_b200.runtime import DynQuantLinear

    layer = DynQuantLinear(random_qt(512, 1024, 3, meta=torch.bfloat16, seed=1))
    x = torch.randn(100, 1024, device="cuda").to(torch.bfloat16)
    want = layer(x)
    _lib.load().dq_gemm_fail_next(1)
    layer(x)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="ran out"):
        layer(x)
    assert torch.equal(layer(x), want)


def scaled_rows(qt, exponents):
    """Row i times 2^exponents[i % len]."""
    factor = 2.0 ** torch.tensor(exponents, dtype=torch.float32, device="cuda").repeat(-(-qt.num_rows // len(exponents)))[:qt.num_rows, None]
    qt.scales, qt.offsets = ((t.float() * factor).to(t.dtype) for t in (qt.scales, qt.offsets))
    return qt


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize(("m", "rows", "k", "group", "meta", "x_exponent", "exponents"), [
    (24, 300, 4224, 64, torch.bfloat16, 4, range(-18, 2)),      # sliced; weights down to where fp16 has none
    (24, 300, 4096, 128, torch.bfloat16, -13, range(0, 22)),    # ... and past 65504
    (64, 20000, 512, 128, torch.float16, 4, range(-12, 6)),     # several tiles per block
    (17, 129, 12288, 128, torch.float16, -6, range(-3, 12)),    # more groups than a warp has lanes
])
def test_fp16_weights_of_any_size_enter_unrounded(bits, m, rows, k, group, meta, x_exponent, exponents):
    from dynquant_b200 import ops

    exponents = list(exponents)
    qt = scaled_rows(random_qt(rows, k, bits, group=group, meta=meta, seed=bits), exponents)
    x = (torch.randn(m, k, generator=torch.Generator().manual_seed(m)) * 2.0 ** x_exponent).to(torch.float16).cuda()
    got = gemm(x, qt)
    assert ops.last_kernel() == "gemm_umma_kernel"
    want = x.double() @ ops.dequant(qt.packed, qt.scales, qt.offsets, bits, group, k, out_dtype=torch.float32).double().T
    for i in range(len(exponents)):  # each size against its own largest result
        part = want[:, i::len(exponents)]
        assert float(part.abs().max()) < 65504
        assert within_one_ulp_16(got[:, i::len(exponents)], part.float().cpu().numpy())


@pytest.mark.parametrize("meta", [torch.float16, torch.bfloat16])
def test_fp16_expert_weights_of_any_size_enter_unrounded(meta):
    from dynquant_b200 import ops
    from dynquant_b200.workloads import random_quant_tensor, seeded_routing

    tokens, experts, topk, hidden, inter = 300, 8, 2, 1024, 384
    gen = torch.Generator(device="cuda").manual_seed(3)
    gate_up = random_quant_tensor(experts * 2 * inter, hidden, 3, meta_dtype=meta, device="cuda", generator=gen)
    down = random_quant_tensor(experts * hidden, inter, 4, meta_dtype=meta, device="cuda", generator=gen)
    small = -14 if meta == torch.bfloat16 else -6
    exponents = list(range(-16, 16)) if meta == torch.bfloat16 else list(range(-6, 10))
    gate_up, down = scaled_rows(gate_up, [small]), scaled_rows(down, exponents)
    ids, weights = seeded_routing(tokens, experts, topk, seed=1, device="cuda")
    x = (torch.randn(tokens, hidden, device="cuda", generator=gen) * 2.0 ** -small).clamp(-65504, 65504).to(torch.float16)
    got = moe_gemm(x, ids, weights, gate_up, down, experts)
    want = torch.cat([ops.moe_gemv(x[i:i + 64].contiguous(), ids[i:i + 64].contiguous(), weights[i:i + 64].contiguous(), gate_up, down,
                                   num_experts=experts, out_dtype=torch.float32) for i in range(0, tokens, 64)])
    for i in range(len(exponents)):  # (flips of the rounded intermediate's last bit are what differs)
        a, b = got[:, i::len(exponents)], want[:, i::len(exponents)]
        assert (a - b).norm() <= 2e-4 * b.norm()


def small_moe(experts, hidden, inter, seed=1):
    from dynquant_b200.workloads import random_quant_tensor

    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (random_quant_tensor(experts * 2 * inter, hidden, 3, meta_dtype=torch.bfloat16, device="cuda", generator=gen),
            random_quant_tensor(experts * hidden, inter, 4, meta_dtype=torch.bfloat16, device="cuda", generator=gen), gen)


@pytest.mark.parametrize("first_expert", [0, 24])
def test_skewed_routing_over_a_rank_of_experts(first_expert):
    """A few experts take nearly all tokens, many take one or none; a rank's ids carry global numbers."""
    from dynquant_b200 import ops

    tokens, experts, hidden, inter = 600, 40, 512, 256
    gate_up, down, gen = small_moe(experts, hidden, inter)
    hot = torch.tensor([[0, 1], [1, 2], [2, 0]], device="cuda").repeat(tokens // 3, 1)  # 400 tokens each: four tiles
    ids = hot.to(torch.int32)
    ids[:20, 0] = torch.arange(10, 30, device="cuda", dtype=torch.int32)                # twenty experts with one token
    ids[::7, 1] = 60                                                                    # nobody's
    ids = (ids + first_expert).contiguous()
    weights = torch.rand(tokens, 2, device="cuda", generator=gen)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    got = moe_gemm(x, ids, weights, gate_up, down, experts, first_expert=first_expert)
    want = torch.cat([ops.moe_gemv(x[i:i + 60].contiguous(), ids[i:i + 60].contiguous(), weights[i:i + 60].contiguous(), gate_up, down,
                                   num_experts=experts, first_expert=first_expert, out_dtype=torch.float32) for i in range(0, tokens, 60)])
    assert (got - want).norm() <= 1e-3 * want.norm()  # flips of the rounded intermediate's last bit
    for token in (0, 19, 21, 599):  # one-token experts and hot ones alike, row by row
        assert (got[token] - want[token]).norm() <= 4e-3 * want[token].norm()


@pytest.mark.parametrize("tokens", [200, 4097, 9000])
def test_plugin_expert_layer_over_many_tokens(tokens):
    """Through the plugin's method: the tcgen05 kernels, 4096 tokens a call at most."""
    from dynquant_b200 import ops
    from dynquant_b200.plugin import DynQuantMoEMethod
    from dynquant_b200.workloads import seeded_routing

    experts, hidden, inter = 8, 256, 128
    gate_up, down, gen = small_moe(experts, hidden, inter)
    method, layer = DynQuantMoEMethod(None, bits_gate_up=3, bits_down=4), torch.nn.Module()
    method.create_weights(layer, experts, hidden, inter, torch.bfloat16, device="cuda")
    method.load_banks(layer, gate_up, down)
    ids, weights = seeded_routing(tokens, experts, 2, seed=2, device="cuda")
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    got = method.apply(layer, x, weights, ids)
    assert ops.last_kernel() == "moe_umma_kernel"
    assert torch.equal(got, moe_gemm(x, ids, weights, gate_up, down, experts).to(torch.bfloat16))
    assert torch.equal(method.apply(layer, x, weights, ids.long()), got)
    want = torch.cat([ops.moe_gemv(x[i:i + 64].contiguous(), ids[i:i + 64].contiguous(), weights[i:i + 64].contiguous(), gate_up, down,
                                   num_experts=experts, out_dtype=torch.float32) for i in range(0, min(tokens, 4160), 64)])
    # one rounding of the output (2^-9) and flips of the intermediate's last bit
    assert (got[:len(want)].float() - want).norm() <= 4e-3 * want.norm()


@pytest.mark.parametrize(("m", "rows", "k", "bits", "kernel"), [
    (1, (1536,), 14336, 4, "gemv_mma_tile_kernel"),          # sliced eight ways: not few slices
    (1, (1536,), 13824, 3, "gemv_mma_stream_sliced_kernel"),  # a long axis of more than 1280 rows
    (1, (1152,), 13824, 4, "gemm_umma_kernel"),
    (6, (512,), 14336, 4, "gemm_umma_kernel"),
    (9, (2048,), 8192, 4, "gemv_rows_kernel"),
    (1, (8192,), 2560, 3, "gemv_mma_tile_kernel"),           # 20 M values on a short axis
    (1, (5120,), 5120, 3, "gemv_mma_stream_sliced_kernel"),
    (2, (11008, 11008), 4096, 3, "gemv_mma_tile_kernel"),    # 172 CTAs of 296
    (2, (14336, 14336), 4096, 3, "gemv_mma_stream_sliced_multi_kernel"),  # 224
])
def test_lines_between_the_kernels(m, rows, k, bits, kernel):
    from dynquant_b200 import ops

    shards = [random_qt(n, k, bits, meta=torch.bfloat16, seed=i) for i, n in enumerate(rows)]
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()
    got = ops.quantized_matmul(x, shards[0]) if len(shards) == 1 else ops.gemv_shards(x, shards)
    assert ops.last_kernel() == kernel
    dense = torch.cat([ops.dequant(q.packed, q.scales, q.offsets, bits, 128, k, out_dtype=torch.float32) for q in shards])
    assert within_one_ulp_16(got, (x.double() @ dense.double().T).float().cpu().numpy())


@pytest.mark.parametrize("m", [2, 40])
def test_fp16_shards_whose_metadata_start_anywhere(m):
    """Eleven or 22 groups a row and odd row counts: rows of scales that start on no 16-byte boundary, the last
    ones at the end of the buffer."""
    from dynquant_b200 import ops
    from dynquant_b200.plugin import DynQuantLinearMethod, ShardSpec

    k, sizes, widths = 1408, (301, 127, 77), (8, 2, 4)
    method, layer = DynQuantLinearMethod(None, [ShardSpec(str(i), b, 64, n) for i, (n, b) in enumerate(zip(sizes, widths))]), torch.nn.Module()
    method.create_weights(layer, k, list(sizes), k, sum(sizes), torch.float16, device="cuda")
    shards = [scaled_rows(random_qt(n, k, b, group=64, seed=b), list(range(-9, 3))) for n, b in zip(sizes, widths)]
    for i, qt in enumerate(shards):
        method.load_shard(layer, i, qt)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.float16).cuda()
    got = method.apply(layer, x)
    assert ops.last_kernel() == "gemm_umma_kernel"
    start = 0
    for qt in shards:
        dense = ops.dequant(qt.packed, qt.scales, qt.offsets, qt.bits, 64, k, out_dtype=torch.float32)
        part, want = got[:, start:start + qt.num_rows], x.double() @ dense.double().T
        start += qt.num_rows
        for i in range(12):
            assert within_one_ulp_16(part[:, i::12], want[:, i::12].float().cpu().numpy())
