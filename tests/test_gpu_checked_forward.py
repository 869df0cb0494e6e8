"""fmoe_forward_checked: the status of the call itself, on every path, front form and thread; none left over for the next."""
import threading

import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu


def _call(path: str, tokens: int, bad_route: int | None, wait: bool):
    hidden, inter, experts, top_k = 64, 32, 4, 2
    generator = torch.Generator().manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16).cuda()
    ids = torch.randint(0, experts, (tokens, top_k), generator=generator)
    if bad_route is not None:
        ids.view(-1)[bad_route] = experts
    weights = torch.rand((tokens, top_k), generator=generator).cuda()
    kind = torch.bfloat16 if path == "bf16" else torch.int8
    w13 = torch.randint(-9, 10, (experts, 2 * inter, hidden), generator=generator).to(kind).cuda()
    w2 = torch.randint(-9, 10, (experts, hidden, inter), generator=generator).to(kind).cuda()
    scales = {} if path == "bf16" else {"s13": torch.full((experts, 2 * inter), 0.01).cuda(), "s2": torch.full((experts, hidden), 0.01).cuda()}
    workspace = torch.empty(1 << 22, dtype=torch.uint8, device="cuda")  # (the cached one belongs to one call at a time)
    return _lib.moe_forward(x, w13, w2, weights, ids.cuda(), w8a16=path == "w8a16", wait=wait, workspace=workspace, **scales)


@pytest.mark.parametrize("path", ["w8a8", "bf16", "w8a16"])
@pytest.mark.parametrize("tokens", [3, 700])  # route build beside the token rows, and by itself (a cluster)
def test_status_comes_with_the_call(path, tokens):
    bad = _call(path, tokens, 5, True)
    assert bad.checked == (_lib.ERR_EXPERT_ID_RANGE, 5)
    with pytest.raises(_lib.FusedMoEError, match="flat route 5"):
        bad.raise_for_status()
    good = _call(path, tokens, None, True)
    assert good.checked == (_lib.OK, 0)
    assert torch.equal(good.out, _call(path, tokens, None, False).out)
    assert _call(path, tokens, 5, False).status() == (_lib.ERR_EXPERT_ID_RANGE, 5)


def test_threads_see_their_own_status():
    results = {}

    def work(index):
        with torch.cuda.stream(torch.cuda.Stream()):
            results[index] = [_call("w8a8", 40, index if index % 2 else None, True).checked for _ in range(20)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for index in range(4):
        assert results[index] == [(_lib.ERR_EXPERT_ID_RANGE, index) if index % 2 else (_lib.OK, 0)] * 20
