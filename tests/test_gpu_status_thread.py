"""A thread that has read a status block gives its page-locked words back when it ends: that may happen while another thread
captures a graph, and the capture stays valid."""
from __future__ import annotations

import threading
import time

import pytest
import torch

from fused_cpp_b200 import _lib

pytestmark = pytest.mark.gpu


def test_thread_ends_during_a_capture(cuda_device):
    generator = torch.Generator(device=cuda_device).manual_seed(5)
    x = torch.randn((4, 256), generator=generator, device=cuda_device).to(torch.bfloat16)
    w13 = (torch.randn((4, 128, 256), generator=generator, device=cuda_device) * 0.05).to(torch.bfloat16)
    w2 = (torch.randn((4, 256, 64), generator=generator, device=cuda_device) * 0.05).to(torch.bfloat16)
    weights = torch.rand((4, 2), generator=generator, device=cuda_device)
    ids = torch.randint(0, 4, (4, 2), generator=generator, device=cuda_device)
    result = _lib.moe_forward(x, w13, w2, weights, ids)
    result.raise_for_status()
    expected, out = result.out.clone(), torch.empty_like(x)
    torch.cuda.synchronize()
    read, leave = threading.Event(), threading.Event()

    def read_status():
        result.raise_for_status()
        read.set()
        leave.wait(60)

    thread = threading.Thread(target=read_status)
    thread.start()
    assert read.wait(60)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        _lib.moe_forward(x, w13, w2, weights, ids, out=out)
        leave.set()
        thread.join()
        time.sleep(0.5)  # join returns before the native thread has run its last destructors
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), expected.view(torch.int16))
