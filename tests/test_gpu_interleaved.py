"""Interleaved gate/up rows (row 2j = gate j, row 2j + 1 = up j) read where they lie: bit for bit the result of the same
call on de-interleaved weights, scales and biases, in every kernel that reads w13 (one-SM, two-SM with one and with four
boxes per stage, W8A16's widening kernel) and with channel counts that end inside a 16-, 64- and 128-channel block.
bf16 biases equal the same biases given as fp32."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["bf16", "w8a16_fixed", "w8a16_bf16"])
@pytest.mark.parametrize("tokens,hidden,inter,tile", [(5, 64, 16, 0), (37, 144, 80, 0), (70, 128, 144, 0), (300, 128, 192, 0), (300, 144, 272, 512)])
def test_interleaved_rows_equal_deinterleaved(cuda_device, kind, tokens, hidden, inter, tile):
    generator = torch.Generator().manual_seed(tokens + inter)
    experts, top_k = 3, 2
    ids = torch.stack([torch.randperm(experts, generator=generator)[:top_k] for _ in range(tokens)]).to(cuda_device)
    x = torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16).to(cuda_device)
    weights = torch.rand((tokens, top_k), generator=generator).to(cuda_device)
    bias13 = bias2 = s13 = s2 = None
    options = {}
    if kind == "bf16":
        w13 = (torch.randn((experts, 2 * inter, hidden), generator=generator) * 0.1).to(torch.bfloat16)
        w2 = (torch.randn((experts, hidden, inter), generator=generator) * 0.1).to(torch.bfloat16)
        bias13 = torch.randn((experts, 2 * inter), generator=generator).to(torch.bfloat16)
        bias2 = torch.randn((experts, hidden), generator=generator).to(torch.bfloat16)
    else:
        w13 = torch.randint(-127, 128, (experts, 2 * inter, hidden), generator=generator, dtype=torch.int8)
        w2 = torch.randint(-127, 128, (experts, hidden, inter), generator=generator, dtype=torch.int8)
        s13 = torch.rand((experts, 2 * inter), generator=generator) * 1e-3
        s2 = torch.rand((experts, hidden), generator=generator) * 1e-3
        options = {"w8a16": True, "w8a16_form": _lib.W8A16_FIXED_POINT if kind == "w8a16_fixed" else _lib.W8A16_BF16_ACTIVATIONS}

    def run(activation, w13, s13, bias13, bias2):
        on_gpu = [None if t is None else t.to(cuda_device) for t in (w13, s13, bias13, bias2)]
        result = _lib.moe_forward(x, on_gpu[0], w2.to(cuda_device), weights, ids, s13=on_gpu[1], s2=None if s2 is None else s2.to(cuda_device),
                                  activation=activation, w13_bias=on_gpu[2], w2_bias=on_gpu[3], gate_up_tile=tile, down_tile=tile, **options)
        result.raise_for_status()
        return result.out

    got = run(_lib.ACTIVATION_SWIGLUOAI | _lib.W13_INTERLEAVED, w13, s13, bias13, bias2)

    def straight(t):
        return None if t is None else cases.gate_then_up(t)

    fp32 = [None if b is None else b.float() for b in (straight(bias13), bias2)]
    expected = run(_lib.ACTIVATION_SWIGLUOAI, straight(w13), straight(s13), *fp32)
    assert torch.isfinite(got.float()).all() and float(got.float().abs().max()) > 0
    assert torch.equal(got, expected)
