"""fmoe_append_shared_route against the tensor operations it replaces: rows that end inside a block, one token, many."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top_k", [(1, 1), (37, 6), (64, 3), (2049, 8), (1, 31)])
def test_rows(cuda_device, tokens, top_k):
    generator = torch.Generator(device=cuda_device).manual_seed(tokens)
    weights = torch.rand((tokens, top_k), generator=generator, device=cuda_device)
    ids = torch.randint(0, 40, (tokens, top_k), generator=generator, device=cuda_device)
    # A transposed view of the ids: the call takes any strides.
    got_weights, got_ids = _lib.append_shared_route(weights, ids.t().contiguous().t(), 40, 2.5)
    assert torch.equal(got_weights, torch.cat((weights * 2.5, torch.ones((tokens, 1), device=cuda_device)), dim=1))
    assert torch.equal(got_ids, torch.cat((ids, torch.full((tokens, 1), 40, device=cuda_device)), dim=1))
