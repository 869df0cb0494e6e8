"""Rules that the host side and the kernels share, taken from the sources themselves (tests/host_rules.cpp, built with g++)."""
from __future__ import annotations

import ctypes
import os
import random
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


@pytest.mark.parametrize("sizes", [(1, 320), (65, 256), (257, 320), (1, 32), (256, 256)], ids=str)
def test_accumulator_ring(rules, sizes):
    """A unit's MMAs lie on consecutive columns inside tensor memory, and what it takes over from the unit before it is that
    unit's leading blocks, as many as are counted.  (The unit before that one has been read by then.)"""
    rng = random.Random(sizes[0])
    count, ring, worst = 20000, 16, 0
    rows = [rng.randint(*sizes) for _ in range(count)]
    slots, shared = (ctypes.c_int * (3 * count))(), (ctypes.c_int * count)()
    rules.place_units((ctypes.c_int * count)(*rows), count, slots, shared)
    before: list = []
    for i, unit_rows in enumerate(rows):
        start, blocks, head = slots[3 * i:3 * i + 3]
        tail = blocks - head
        assert blocks == (unit_rows + 31) // 32 and 0 <= tail
        for first, length in ((start, head), (start + head, tail)):
            assert length <= 8 and first % ring + length <= ring
        assert tail == 0 or (head >= 2 and tail >= 2 and blocks > 8)
        taken = [block % ring for block in range(start, start + blocks)]
        assert len(set(taken)) == blocks
        overlap = [index for index, block in enumerate(before) if block in taken]
        assert overlap == list(range(shared[i]))
        worst = max(worst, shared[i])
        before = taken
    if sizes[1] <= 256:
        assert worst <= 7
    if sizes in ((1, 32), (256, 256)):
        assert worst == 0


@pytest.mark.parametrize("read", [True, False], ids=["read", "not read"])
def test_every_warp_hands_blocks_over_once(rules, read):
    """Also where the epilogue is switched off and a unit has no chunks to read."""
    for blocks in range(1, 11):
        for handed_over in range(0, blocks + 1):
            for first, step in ((0, 1), (0, 2), (1, 2)):
                early = ctypes.c_int(0)
                arrivals = rules.handover_arrivals(first, step, handed_over, blocks if read else 0, ctypes.byref(early))
                assert arrivals == (1 if handed_over else 0), (blocks, handed_over, first, step)
                assert early.value == 0
