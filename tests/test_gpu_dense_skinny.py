"""Dense W8A8 linear at the sizes where its kernels change: row tiles of 16 to 128 rows and the two-SM kernel above, K
ranges of one 128-byte block up to several per part of the cluster split, K and N off every vector and tile width, rows
too long for the register-held quantiser (16384 columns), one and two weight matrices.  Bit for bit against the oracle."""
from __future__ import annotations

import pytest
import torch

from fused_cpp_b200 import i8gemm
from oracle import oracle

pytestmark = pytest.mark.gpu


def _weight(n, k, generator):
    return torch.randint(-127, 128, (n, k), dtype=torch.int8, generator=generator), torch.rand(n, generator=generator) * 0.01 + 1e-3


@pytest.mark.parametrize("rows,k,n,x_dtype,out_dtype,with_bias", [
    (1, 8, 1, torch.bfloat16, torch.float32, True), (16, 128, 128, torch.bfloat16, torch.bfloat16, False),
    (17, 264, 129, torch.float32, torch.bfloat16, True), (32, 2056, 520, torch.bfloat16, torch.float32, False),
    (33, 1000, 130, torch.float32, torch.float32, True), (64, 4096, 1536, torch.bfloat16, torch.bfloat16, True),
    (65, 777, 300, torch.bfloat16, torch.bfloat16, False), (128, 1536, 4000, torch.bfloat16, torch.bfloat16, True),
    (129, 1536, 300, torch.float32, torch.bfloat16, True), (3, 16384, 136, torch.bfloat16, torch.bfloat16, False),
    # Above 128 rows with a long K range: row tiles of the split kernel, the last one short, and its limits.
    (129, 5200, 300, torch.bfloat16, torch.bfloat16, True), (256, 5120, 130, torch.float32, torch.float32, True),
    (385, 5128, 257, torch.bfloat16, torch.float32, False), (300, 5112, 64, torch.bfloat16, torch.bfloat16, False),
    (1100, 5120, 1025, torch.bfloat16, torch.bfloat16, True), (1100, 5120, 1000, torch.bfloat16, torch.bfloat16, False),
    (592, 264, 130, torch.bfloat16, torch.bfloat16, False), (593, 264, 130, torch.bfloat16, torch.bfloat16, True),
    (5, 16400, 200, torch.bfloat16, torch.float32, True), (2, 16392, 64, torch.float32, torch.float32, False),
    # One CTA per channel block: whole and short batches of sixteen rows, channels off the block, either output type.
    (15, 100, 129, torch.bfloat16, torch.bfloat16, True), (31, 128, 257, torch.bfloat16, torch.float32, False),
    (64, 64, 64, torch.bfloat16, torch.bfloat16, True), (97, 96, 130, torch.float32, torch.float32, True),
    (127, 128, 200, torch.bfloat16, torch.bfloat16, False), (128, 64, 64, torch.bfloat16, torch.float32, True),
    # More channel blocks than resident CTAs: the two-SM kernel over 64 rows.
    (113, 512, 37000, torch.bfloat16, torch.bfloat16, True), (65, 264, 38017, torch.float32, torch.float32, True),
    (128, 128, 40000, torch.bfloat16, torch.bfloat16, False), (64, 128, 40000, torch.bfloat16, torch.bfloat16, True),
])
def test_product(cuda_device, rows, k, n, x_dtype, out_dtype, with_bias):
    generator = torch.Generator().manual_seed(rows + k + n)
    weight, scale = _weight(n, k, generator)
    x = torch.randn((rows, k), generator=generator).to(x_dtype)
    bias = torch.randn(n, generator=generator) if with_bias else None
    got = i8gemm.dynamic_scaled_mm(x.to(cuda_device), i8gemm.prepare(weight, scale), bias=None if bias is None else bias.to(cuda_device), out_dtype=out_dtype)
    torch.testing.assert_close(got.cpu(), oracle.i8gemm_dynamic(x, weight, scale, bias, out_dtype), atol=0, rtol=0)


@pytest.mark.parametrize("rows,k,first_n,second_n", [(1, 1536, 4000, 72), (40, 512, 130, 129), (128, 300, 64, 700), (100, 144, 30000, 9000), (200, 512, 300, 130), (200, 5136, 130, 260)])
def test_pair(cuda_device, rows, k, first_n, second_n):
    generator = torch.Generator().manual_seed(rows + k)
    first, second = _weight(first_n, k, generator), _weight(second_n, k, generator)
    x = torch.randn((rows, k), generator=generator).to(torch.bfloat16)
    got = i8gemm.dynamic_scaled_mm_pair(x.to(cuda_device), i8gemm.prepare(*first), i8gemm.prepare(*second))
    for out, (weight, scale) in zip(got, (first, second)):
        torch.testing.assert_close(out.cpu(), oracle.i8gemm_dynamic(x, weight, scale, None, torch.bfloat16, clamp_low=-127), atol=0, rtol=0)


@pytest.mark.parametrize("rows,k,n", [(5, 2048, 1536), (70, 1024, 136), (200, 5120, 512)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8])
def test_output_view_at_any_element(cuda_device, rows, k, n, out_dtype, offset):
    """The caller's output may start at any element of an allocation (a K split stores vectors only where that is aligned)."""
    generator = torch.Generator().manual_seed(rows + k)
    weight, scale = _weight(n, k, generator)
    x = torch.randn((rows, k), generator=generator).to(torch.bfloat16)
    packed = i8gemm.prepare(weight, scale)
    buffer = torch.full((offset + rows * n + 8,), 7.0, dtype=out_dtype, device=cuda_device)
    out = buffer[offset:offset + rows * n].view(rows, n)
    i8gemm.i8gemm_dynamic_scaled_mm(out, x.to(cuda_device), packed.packed_weight, packed.weight_scale, None, packed.k, packed.n,
                                    packed.k_padded, packed.n_padded)
    assert torch.equal(out.cpu(), oracle.i8gemm_dynamic(x, weight, scale, None, out_dtype))
    assert bool((buffer[:offset] == 7).all()) and bool((buffer[offset + rows * n:] == 7).all())
    if out_dtype is torch.bfloat16:
        other = torch.empty_like(out)
        i8gemm.i8gemm_dynamic_scaled_mm_pair(out, other, x.to(cuda_device), packed.packed_weight, packed.weight_scale, packed.k,
                                             packed.n, packed.k_padded, packed.n_padded, packed.packed_weight, packed.weight_scale,
                                             packed.n, packed.n_padded)
        assert torch.equal(out, other)
        assert torch.equal(other.cpu(), oracle.i8gemm_dynamic(x, weight, scale, None, out_dtype, clamp_low=-127))


@pytest.mark.parametrize("k", [64, 72, 77, 16392], ids=["held", "held_padded", "scalar", "long"])
@pytest.mark.parametrize("rows", [8, 600])
def test_rows_of_a_few_smallest_numbers(cuda_device, rows, k):
    """fp32 rows whose largest magnitude is a few units of the smallest fp32 number: amax / 127 is rounded to whole units, up to
    15938 units quotients can leave +-127.5, and both clamps bind (-128 below, for the single product)."""
    generator = torch.Generator().manual_seed(k)
    units = torch.tensor([190, 63, 254, 100, 64, 1000, 15938, 15939])[torch.arange(rows) % 8].unsqueeze(1)
    steps = torch.randint(-1000, 1001, (rows, k), generator=generator) * units // 1000
    steps[:, 0], steps[:, 1] = -units[:, 0], units[:, 0]
    x = torch.where(steps < 0, (-steps) | -(1 << 31), steps).to(torch.int32).view(torch.float32)
    assert torch.equal(x.abs().view(torch.int32).amax(dim=1), units[:, 0].to(torch.int32))
    weight = torch.randint(-127, 128, (40, k), dtype=torch.int8, generator=generator)
    scale = torch.full((40,), 1e30)
    got = i8gemm.dynamic_scaled_mm(x.to(cuda_device), i8gemm.prepare(weight, scale), out_dtype=torch.float32)
    expected = oracle.i8gemm_dynamic(x, weight, scale, None, torch.float32)
    assert torch.equal(got.cpu(), expected) and bool((expected != 0).any())


@pytest.mark.parametrize("rows,k,n", [(4, 256, 40000), (4, 2048, 1536), (96, 512, 12000), (700, 512, 1536), (128, 128, 40000)],
                         ids=["one_part", "split", "row_tile_128", "two_sm", "two_sm_wide"])
@pytest.mark.parametrize("graph", [False, True], ids=["eager", "graph"])
def test_buffers_rewritten_between_calls(cuda_device, rows, k, n, graph):
    """Rows and a weight that are streamed into fixed buffers: what a call read of them must not be found again by the next."""
    generator = torch.Generator().manual_seed(n)
    rounds = [(_weight(n, k, generator), torch.randn(n, generator=generator)) for _ in range(3)]
    rows_of = [torch.randn((rows, k), generator=generator).to(torch.bfloat16) for _ in rounds]
    packed = i8gemm.prepare(*rounds[0][0])
    bias = rounds[0][1].to(cuda_device)
    sources = [(i8gemm.prepare(*weight), values.to(cuda_device), x.to(cuda_device)) for (weight, values), x in zip(rounds, rows_of)]
    device_x = torch.empty_like(sources[0][2])

    def passes():
        outs = []
        for source, values, x in sources:
            device_x.copy_(x)
            packed.packed_weight.copy_(source.packed_weight)
            packed.weight_scale.copy_(source.weight_scale)
            bias.copy_(values)
            outs.append(i8gemm.dynamic_scaled_mm(device_x, packed, bias=bias, out_dtype=torch.float32))
        return outs

    expected = [oracle.i8gemm_dynamic(x, *weight, values, torch.float32).to(cuda_device)
                for (weight, values), x in zip(rounds, rows_of)]
    outs = passes()
    if graph:
        torch.cuda.synchronize()
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured):
            outs = passes()
    for _ in range(6):
        if graph:
            captured.replay()
            captured.replay()
        else:
            outs = passes()
        torch.cuda.synchronize()
        for out, reference in zip(outs, expected):
            assert torch.equal(out, reference)
