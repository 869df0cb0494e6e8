"""Route build and token rows of a small batch in one launch: routes, rows and scales against the two-launch form.

The limits of the one-launch form are 1024 routes, 512 experts and four tokens per SM; the sizes lie on either side of
them and of its 512-thread rounds (512 routes, 8192 columns)."""
import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu


def _rows(result, tokens, top_k, hidden, experts, dtype):
    """(sorted routes, route positions, rows, scales) of a finished call, from its workspace."""
    routes = tokens * top_k
    valid = int(result.region("offsets", torch.int32, (experts + 1,))[experts])
    return (result.region("sorted_routes", torch.int32, (routes,))[:valid].clone(), result.region("route_pos", torch.int32, (routes,)).clone(),
            result.region("a_rows", dtype, (routes, hidden))[:valid].clone(), result.region("a_scale", torch.float32, (routes,))[:valid].clone())


@pytest.mark.parametrize("tokens,top_k,experts,hidden", [(1, 1, 2, 16), (1, 8, 256, 7168), (3, 8, 5, 8208), (64, 8, 256, 2048), (65, 8, 512, 256),
                                                         (128, 8, 33, 1040), (129, 8, 33, 1040), (32, 32, 64, 256), (70, 6, 513, 256)])
@pytest.mark.parametrize("numerics", [_lib.NUMERICS_TORCHREF, _lib.NUMERICS_NATIVE])
def test_int8_rows_and_routes(tokens, top_k, experts, hidden, numerics):
    generator = torch.Generator().manual_seed(tokens * 131 + experts)
    x = torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(experts, generator=generator)[:top_k] if top_k <= experts else torch.randint(0, experts, (top_k,), generator=generator)
                       for _ in range(tokens)])
    if tokens > 2:
        ids[1, 0] = -1  # dropped routes: below and above the valid range
        ids[2, top_k - 1] = experts
    weights = torch.rand((tokens, top_k), generator=generator)
    inter = 16
    w13 = torch.zeros((experts, 2 * inter, hidden), dtype=torch.int8, device="cuda")
    w2 = torch.zeros((experts, hidden, inter), dtype=torch.int8, device="cuda")
    s13, s2 = torch.ones((experts, 2 * inter), device="cuda"), torch.ones((experts, hidden), device="cuda")
    result = _lib.moe_forward(x.cuda(), w13, w2, weights.cuda(), ids.cuda(), s13=s13, s2=s2, numerics=numerics)
    error, _ = result.status()
    assert (error != 0) == (tokens > 2)
    order, pos, rows, scales = _rows(result, tokens, top_k, hidden, experts, torch.int8)
    flat = ids.reshape(-1)
    valid = (flat >= 0) & (flat < experts)
    expected_order = torch.argsort(torch.where(valid, flat, experts), stable=True)[:int(valid.sum())]
    assert torch.equal(order.cpu().long(), expected_order)
    expected_pos = torch.full((tokens * top_k,), -1, dtype=torch.int64)
    expected_pos[expected_order] = torch.arange(expected_order.numel())
    assert torch.equal(pos.cpu().long(), expected_pos)
    q, scale = _lib.quantize_rows(x.cuda(), numerics=numerics)
    token_of = (expected_order // top_k).cuda()
    assert torch.equal(rows, q[token_of])
    assert torch.equal(scales, scale[token_of])


@pytest.mark.parametrize("tokens,top_k,experts,hidden", [(1, 2, 3, 32), (37, 4, 16, 2064), (128, 8, 20, 4096), (40, 3, 7, 8208)])
def test_bf16_rows(tokens, top_k, experts, hidden):
    generator = torch.Generator().manual_seed(7)
    x = torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(experts, generator=generator)[:top_k] for _ in range(tokens)])
    inter = 16
    w13 = torch.zeros((experts, 2 * inter, hidden), dtype=torch.bfloat16, device="cuda")
    w2 = torch.zeros((experts, hidden, inter), dtype=torch.bfloat16, device="cuda")
    result = _lib.moe_forward(x, w13, w2, torch.ones((tokens, top_k), device="cuda"), ids.cuda())
    result.raise_for_status()
    order, _, rows, _ = _rows(result, tokens, top_k, hidden, experts, torch.bfloat16)
    assert torch.equal(order.cpu().long(), torch.argsort(ids.reshape(-1), stable=True))
    assert torch.equal(rows, x[(order // top_k).long()])


@pytest.mark.parametrize("tokens,hidden", [(297, 256), (592, 1040), (593, 256)])  # a second wave of CTAs; four tokens per SM of 148 and one more
def test_many_tokens_of_one_route(tokens, hidden):
    test_int8_rows_and_routes(tokens, 1, 16, hidden, _lib.NUMERICS_TORCHREF)


@pytest.mark.parametrize("tokens,top_k,experts,hidden", [(1, 1, 2, 16), (3, 2, 2, 8208), (37, 4, 16, 272), (129, 8, 9, 144), (297, 3, 5, 48)])
def test_plane_rows(tokens, top_k, experts, hidden):
    """Two int8 rows per route: 256 * high + low is the row's value in units of its largest magnitude / 32512, ties to even."""
    generator = torch.Generator().manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16)
    x[tokens // 2] = 0
    ids = torch.stack([torch.randperm(experts, generator=generator)[:top_k] for _ in range(tokens)])
    inter = hidden + 16  # wider than the rows: the planes of the intermediate have a region of their own
    w13 = torch.zeros((experts, 2 * inter, hidden), dtype=torch.int8, device="cuda")
    w2 = torch.zeros((experts, hidden, inter), dtype=torch.int8, device="cuda")
    result = _lib.moe_forward(x.cuda(), w13, w2, torch.ones((tokens, top_k), device="cuda"), ids.cuda(), w8a16=True, w8a16_form=_lib.W8A16_FIXED_POINT,
                              s13=torch.ones((experts, 2 * inter), device="cuda"), s2=torch.ones((experts, hidden), device="cuda"))
    result.raise_for_status()
    order, _, planes, scales = _rows(result, tokens, top_k, 2 * hidden, experts, torch.int8)
    assert torch.equal(order.cpu().long(), torch.argsort(ids.reshape(-1), stable=True))
    rows = x.float()[(order.cpu() // top_k).long()]
    amax = rows.abs().amax(dim=1)
    scale = torch.where(amax > 0, amax / 32512.0, torch.ones(()))
    assert torch.equal(scales.cpu(), scale)
    high, low = planes.cpu().view(-1, 2, hidden).to(torch.int32).unbind(1)
    assert torch.equal((256 * high + low).float(), torch.round(rows / scale[:, None]).clamp(-32512, 32512))
