"""The one-launch route build at the sizes where it changes shape: one CTA to eight (1024 routes each before a warp takes
a second round), a run that ends inside a warp, 32 histogram rows up to 1024 experts and fewer above.  Lists against the
oracle's counting sort, work items against the rule (experts with at most 64 rows in one list, the others in the other)."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu

SPLIT_ROWS, BIG_ROWS = 64, 320


def _covered_rows(items: torch.Tensor, rows_most: int) -> dict:
    """expert -> sorted positions its items cover, in order."""
    covered: dict = {}
    for expert, first, rows, _ in items.tolist():
        assert 0 < rows <= rows_most
        covered.setdefault(expert, []).extend(range(first, first + rows))
    return covered


@pytest.mark.parametrize("tokens,experts,top_k", [
    (1, 1, 1), (1024, 16, 1), (1025, 16, 1), (683, 40, 3), (4097, 33, 2), (9001, 7, 1), (700, 1024, 12), (700, 1025, 12), (300, 2048, 32),
    # several CTAs with a number of experts that leaves lanes of the last warp out of the loops in front of the cluster barriers
    (1100, 31, 1), (2100, 257, 4), (16384, 257, 9),
])
def test_lists_and_items(cuda_device, tokens, experts, top_k):
    generator = torch.Generator().manual_seed(tokens + experts)
    ids = torch.randint(0, experts, (tokens, top_k), generator=generator, dtype=torch.int64)
    ids[: tokens // 3] %= max(1, experts // 3)  # some experts with many rows
    routes, inter = tokens * top_k, 16
    w13 = torch.zeros((experts, 2 * inter, 16), dtype=torch.int8, device=cuda_device)
    w2 = torch.zeros((experts, 16, inter), dtype=torch.int8, device=cuda_device)
    result = _lib.moe_forward(torch.ones((tokens, 16), dtype=torch.bfloat16, device=cuda_device), w13, w2,
                              torch.ones((tokens, top_k), device=cuda_device), ids.to(cuda_device),
                              s13=torch.ones((experts, 2 * inter), device=cuda_device), s2=torch.ones((experts, 16), device=cuda_device))
    result.raise_for_status()
    counts, offsets, order = oracle.route_build(ids, experts)
    assert torch.equal(result.region("counts", torch.int32, (experts,)).cpu(), counts)
    assert torch.equal(result.region("offsets", torch.int32, (experts + 1,)).cpu(), offsets)
    assert torch.equal(result.region("sorted_routes", torch.int32, (routes,)).cpu(), order)
    assert torch.equal(result.region("row_expert", torch.int32, (routes,)).cpu().long(), ids.reshape(-1)[order.long()])
    positions = torch.empty(routes, dtype=torch.int32)
    positions[order.long()] = torch.arange(routes, dtype=torch.int32)
    assert torch.equal(result.region("route_pos", torch.int32, (routes,)).cpu(), positions)
    assert result.status_word(3) == int((counts > 0).sum())
    max_items = experts + routes // 8 + 1
    lists = result.region("items", torch.int32, (4, max_items, 4)).cpu()
    thin = _covered_rows(lists[0, : result.status_word(2)], SPLIT_ROWS)
    thick = _covered_rows(lists[2, : result.status_word(6)], BIG_ROWS) if tokens > SPLIT_ROWS else {}
    for expert in range(experts):
        rows = list(range(int(offsets[expert]), int(offsets[expert + 1])))
        where = thick if len(rows) > SPLIT_ROWS else thin
        assert where.pop(expert, []) == rows
    assert not thin and not thick
