"""The kernels of a forward overlap their neighbours (programmatic dependent launches): calls issued back to back on one
workspace, with other inputs each time, and calls replayed from a CUDA graph give the bits of calls that are waited for one
by one.  Token counts on both sides of the split between the one-SM and the two-SM kernel, with thin experts, fat experts
and both; integer paths are exact, and bf16 runs the same kernels on the same rows."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu

HIDDEN, INTER, EXPERTS, TOP_K = 512, 256, 8, 2


def _inputs(kind, tokens, fat_share, device):
    generator = torch.Generator(device=device).manual_seed(tokens)
    shape13, shape2 = (EXPERTS, 2 * INTER, HIDDEN), (EXPERTS, HIDDEN, INTER)
    options = {}
    if kind == "bf16":
        w13 = (torch.randn(shape13, generator=generator, device=device) * 0.05).to(torch.bfloat16)
        w2 = (torch.randn(shape2, generator=generator, device=device) * 0.05).to(torch.bfloat16)
    else:
        w13 = torch.randint(-127, 128, shape13, generator=generator, device=device, dtype=torch.int8)
        w2 = torch.randint(-127, 128, shape2, generator=generator, device=device, dtype=torch.int8)
        options = {"s13": torch.rand(shape13[:2], generator=generator, device=device) * 1e-3,
                   "s2": torch.rand(shape2[:2], generator=generator, device=device) * 1e-3, "w8a16": kind == "w8a16"}
    calls = []
    for _ in range(6):
        scores = torch.rand((tokens, EXPERTS), generator=generator, device=device)
        scores[:, :2] += fat_share
        ids = torch.topk(scores, TOP_K, dim=1).indices
        calls.append((torch.randn((tokens, HIDDEN), generator=generator, device=device).to(torch.bfloat16),
                      torch.rand((tokens, TOP_K), generator=generator, device=device), ids))
    return w13, w2, options, calls


@pytest.mark.parametrize("tokens,fat_share", [(1, 0.0), (64, 0.0), (65, 0.0), (200, 0.9), (700, 0.6), (2000, 2.0)])
@pytest.mark.parametrize("kind", ["w8a8", "w8a16", "bf16"])
def test_back_to_back_equals_one_by_one(cuda_device, kind, tokens, fat_share):
    w13, w2, options, calls = _inputs(kind, tokens, fat_share, cuda_device)

    def run(call, out=None):
        return _lib.moe_forward(call[0], w13, w2, call[1], call[2], out=out, **options)

    expected = []
    for call in calls:
        result = run(call)
        result.raise_for_status()
        expected.append(result.out.clone())
    for _ in range(5):
        results = [run(call) for call in calls]
        results[-1].raise_for_status()
        for result, reference in zip(results, expected):
            assert torch.equal(result.out.view(torch.int16), reference.view(torch.int16))
    outs = [torch.empty_like(call[0]) for call in calls]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for call, out in zip(calls, outs):
            run(call, out)
    for _ in range(8):  # replays leave no host gaps between the calls
        for out in outs:
            out.zero_()
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        for out, reference in zip(outs, expected):
            assert torch.equal(out.view(torch.int16), reference.view(torch.int16))
