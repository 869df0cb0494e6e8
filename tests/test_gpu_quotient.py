"""The branch-free quotient of the SwiGLU epilogues: the compiler's reciprocal and division bit for bit, and the plain statement
outside its ranges."""
import ctypes

import pytest
import torch

from fused_cpp_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_every_divisor_mantissa():
    lib = _lib.load_diag()
    lib.fmoe_diag_quotient_check.argtypes = [ctypes.c_uint32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
    mismatches = torch.zeros(1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.fmoe_diag_quotient_check(12345, 64, mismatches.data_ptr(), stream), lib)
    assert int(mismatches.item()) == 0


@pytest.mark.parametrize("tokens", [3, 40, 300])  # 16- and 64-row tile, two-SM kernel
def test_elements_outside_the_ranges(tokens):
    """Rows whose gates overflow the exponent's clamp, vanish, or are zero: route rows equal the oracle's bit for bit."""
    generator = torch.Generator().manual_seed(tokens)
    hidden, inter, experts, top_k = 64, 64, 1, 1
    x = torch.randn((tokens, hidden), generator=generator)
    x *= torch.tensor([1.0, 1e4, 1e-12, 0.0, 1e12, 1e-30]).repeat(tokens // 6 + 1)[:tokens, None]
    x = x.to(torch.bfloat16)
    w13 = torch.randint(-127, 128, (experts, 2 * inter, hidden), generator=generator, dtype=torch.int8)
    w2 = torch.randint(-127, 128, (experts, hidden, inter), generator=generator, dtype=torch.int8)
    s13 = torch.rand((experts, 2 * inter), generator=generator) * 1e-2
    s2 = torch.rand((experts, hidden), generator=generator) * 1e-2
    ids = torch.zeros((tokens, top_k), dtype=torch.int64)
    weights = torch.ones((tokens, top_k))
    expected = oracle.w8a8_forward(x, w13, s13, w2, s2, weights, ids)
    result = _lib.moe_forward(x.cuda(), w13.cuda(), w2.cuda(), weights.cuda(), ids.cuda(), s13=s13.cuda(), s2=s2.cuda())
    result.raise_for_status()
    assert torch.equal(result.out.cpu().view(torch.int16), expected.view(torch.int16))
