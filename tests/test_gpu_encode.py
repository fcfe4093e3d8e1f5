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
