"""The TORCHREF activation quantiser on the GPU replaces x / scale by x * (1 / scale) wherever that cannot change
the rounded integer, and keeps the division otherwise (quantize4_torchref_fast in csrc/common.cuh).  The float model of
that rule (test_quantiser_fused_model.py) against the exact statement clamp(rint(x / scale), +-127) of
tests/test_moe_w8a8.py:40-43 on millions of random values and on inputs placed on the rounding boundaries.  The device
code itself is compared with the oracle bit for bit in the GPU tests."""
from __future__ import annotations

import numpy as np

from tests.test_quantiser_fused_model import bf16, exact, fast


def test_fast_path_equals_division_on_random_rows():
    rng = np.random.default_rng(7)
    count = 2_000_000
    amax = np.maximum(np.abs(rng.standard_normal(count)).astype(np.float32) * np.float32(rng.uniform(1e-3, 50)), np.float32(1e-6))
    v = bf16(amax * rng.uniform(-1, 1, count).astype(np.float32))
    v = np.where(np.abs(v) > amax, amax, v)  # the rounding to bf16 may not leave the row's range
    scale = np.maximum((amax / np.float32(127.0)).astype(np.float32), np.float32(1e-30))
    got, slow = fast(v, scale)
    assert np.array_equal(got, exact(v, scale))
    assert slow.mean() < 4e-3  # the division is the rare case (it decides groups of four)


def test_fast_path_equals_division_on_rounding_boundaries():
    rng = np.random.default_rng(8)
    count = 2_000_000
    scale = (np.abs(rng.standard_normal(count)).astype(np.float32) * np.float32(0.05) + np.float32(1e-4)).astype(np.float32)
    half = rng.integers(-127, 127, count).astype(np.float32) + np.float32(0.5)
    for nudge in (0, 1, -1, 2, -2):
        v = (half * scale).astype(np.float32)
        v = (v.view(np.int32) + np.int32(nudge)).view(np.float32)  # the boundary value and its neighbours in float32
        got, _ = fast(v, scale)
        assert np.array_equal(got, exact(v, scale))


def test_fast_path_handles_zero_rows_and_overflow():
    scale = np.full(4, 1e-30, dtype=np.float32)  # the clamp of an all-zero row
    v = np.array([0.0, 1e-31, -1e-28, 3e-29], dtype=np.float32)
    got, _ = fast(v, scale)
    assert np.array_equal(got, exact(v, scale))
    big = np.array([1e30, -1e30, np.inf, np.nan], dtype=np.float32)  # the row's scale is infinite
    got, slow = fast(big, np.full(4, np.inf, dtype=np.float32))
    assert slow.all() and np.array_equal(got, np.array([0, 0, 127, 127], dtype=np.float32))
