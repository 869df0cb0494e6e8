"""Two-SM work items around the sizes where they change shape: one MMA (up to 256 token rows) or two over the ring of
accumulator blocks (up to 320), one item or several per expert, accumulators that wrap and that share blocks with the one
before them (several units per SM pair).  Against the one-SM kernel on the same rows: the integer paths bit for bit, bf16
to the rounding of sums taken in another order (a flipped bf16 of the intermediate moves an output by about 2^-9 of it)."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu

# Routes per expert, in an order that puts small units behind large ones and the other way round.
MIXED = [288, 320, 65, 257, 640, 33, 256, 319, 641, 1, 321, 300]
EVEN = [320] * 12
ODD = [289] * 10


@pytest.mark.parametrize("rows", [MIXED, EVEN, ODD], ids=["mixed", "even", "odd"])
@pytest.mark.parametrize("kind", ["w8a8", "w8a16", "bf16"])
def test_against_one_sm_kernel(cuda_device, kind, rows):
    hidden, inter, experts = 4096, 2048, len(rows)
    if kind == "w8a16":
        rows = [(r + 1) // 2 for r in rows]  # two token rows per route
    generator = torch.Generator(device=cuda_device).manual_seed(sum(rows))
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(rows))
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].reshape(-1, 1).to(cuda_device)
    tokens = ids.shape[0]
    x = torch.randn((tokens, hidden), generator=generator, device=cuda_device).to(torch.bfloat16)
    weights = torch.rand((tokens, 1), generator=generator, device=cuda_device)
    options = {}
    if kind == "bf16":
        w13 = (torch.randn((experts, 2 * inter, hidden), generator=generator, device=cuda_device) * 0.02).to(torch.bfloat16)
        w2 = (torch.randn((experts, hidden, inter), generator=generator, device=cuda_device) * 0.02).to(torch.bfloat16)
    else:
        w13 = torch.randint(-127, 128, (experts, 2 * inter, hidden), generator=generator, device=cuda_device, dtype=torch.int8)
        w2 = torch.randint(-127, 128, (experts, hidden, inter), generator=generator, device=cuda_device, dtype=torch.int8)
        options = {"s13": torch.rand((experts, 2 * inter), generator=generator, device=cuda_device) * 1e-3,
                   "s2": torch.rand((experts, hidden), generator=generator, device=cuda_device) * 1e-3, "w8a16": kind == "w8a16"}
    expected = _lib.moe_forward(x, w13, w2, weights, ids, gate_up_tile=128, down_tile=128, **options)
    expected.raise_for_status()
    reference = expected.out.clone()
    result = _lib.moe_forward(x, w13, w2, weights, ids, gate_up_tile=512, down_tile=512, **options)
    result.raise_for_status()
    if kind == "bf16":
        error = (result.out.float() - reference.float()).norm() / reference.float().norm()
        assert float(error) <= 4e-3
    else:
        assert torch.equal(result.out.view(torch.int16), reference.view(torch.int16))


def test_ends_without_an_epilogue(cuda_device, monkeypatch):
    """The diagnostic library's switch for an epilogue that reads nothing: units still hand their accumulators on."""
    hidden, inter, experts = 4096, 2048, len(MIXED)
    ids = torch.repeat_interleave(torch.arange(experts, device=cuda_device), torch.tensor(MIXED, device=cuda_device)).reshape(-1, 1)
    x = torch.zeros((ids.shape[0], hidden), dtype=torch.bfloat16, device=cuda_device)
    w13 = torch.zeros((experts, 2 * inter, hidden), dtype=torch.int8, device=cuda_device)
    w2 = torch.zeros((experts, hidden, inter), dtype=torch.int8, device=cuda_device)
    monkeypatch.setenv("FUSED_CPP_MOE_GEMM_DIAG", "1")
    result = _lib.moe_forward(x, w13, w2, torch.ones(ids.shape, device=cuda_device), ids, gate_up_tile=512, down_tile=512, diagnostic=True,
                              s13=torch.ones((experts, 2 * inter), device=cuda_device), s2=torch.ones((experts, hidden), device=cuda_device))
    assert result.status() == (_lib.OK, 0)
