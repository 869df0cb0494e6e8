"""Rules that the host side and the kernels share, taken from the sources themselves (tests/host_rules.cpp, built with g++)."""
from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fused_cpp_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    target = str(tmp_path_factory.mktemp("host_rules") / "host_rules.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-I", os.path.join(cuda, "include"),
                    os.path.join(HERE, "host_rules.cpp"), "-o", target], check=True)
    lib = ctypes.CDLL(target)
    lib.dense_vector_store.argtypes = [ctypes.c_size_t, ctypes.c_int, ctypes.c_int]
    return lib


@pytest.mark.parametrize("bf16", [1, 0])
def test_dense_vector_store_is_aligned_in_every_row(rules, bf16):
    size = 2 if bf16 else 4
    for n in range(1, 20):
        for offset in range(0, 9):  # the view starts `offset` elements into an allocation
            out = (1 << 20) + offset * size
            aligned = all((out + (row * n + channel) * size) % (4 * size) == 0 and channel + 4 <= n
                          for row in range(4) for channel in range(0, n, 4))
            assert rules.dense_vector_store(out, n, bf16) == aligned
