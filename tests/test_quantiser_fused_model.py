"""The TORCHREF quantiser's fast path in its fused form (quantize4_torchref_fast in csrc/common.cuh): x * (1 / scale) is
rounded by one fused multiply-add with 1.5 * 2^23, a second one gives the distance to that integer, and the exact statement
clamp(rint(x / scale), +-127) decides a group of four when a distance is above 0.4999 or not a number.  A float64 model of
it (the product of two fp32 values is exact there, so rounding it once is the fused operation) against the exact statement:
random rows, values on the rounding boundaries, rows of infinities, NaN and magnitudes whose scale or reciprocal leaves the
fp32 range.  The scale is the row's own, as everywhere the device function is called: no quotient that leaves a byte may stay
outside the exact branch, for there is no clamp in front of the stored byte."""
from __future__ import annotations

import numpy as np
import pytest


def exact(values, scale, clamp_low=-127.0):
    with np.errstate(all="ignore"):
        rounded = np.rint((values / scale).astype(np.float32))
    return np.fmax(np.fmin(rounded, np.float32(127.0)), np.float32(clamp_low))  # fminf / fmaxf: NaN ends at +127


def fast(values, scale, clamp_low=-127.0):
    """What the device stores for consecutive groups of four values, and which values the exact statement decided."""
    with np.errstate(all="ignore"):
        inverse = (np.float32(1.0) / scale).astype(np.float32)
        product = values.astype(np.float64) * inverse.astype(np.float64)
        nearest = np.rint(product)
        distance = np.abs((product - nearest).astype(np.float32))
        slow = ~(distance <= np.float32(0.4999))
    groups = np.repeat(slow.reshape(-1, 4).any(axis=1), 4)
    # The sum's low byte, read as a signed one: an integer outside a byte would wrap, and the statement would then differ.
    byte = np.where(groups, 0, nearest).astype(np.int64).astype(np.uint8).view(np.int8).astype(np.float32)
    return np.where(groups, exact(values, scale, clamp_low), byte), groups


def bf16(values):
    bits = values.astype(np.float32).view(np.uint32)
    return ((bits + np.uint32(0x7FFF) + ((bits >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(np.float32)


@pytest.mark.parametrize("floor", [1e-30, 0.0], ids=["activation", "plain"])
@pytest.mark.parametrize("magnitude", [1.0, 3e-3, 50.0, 1e-29, 1e-37, 2e-38, 1e38])
def test_rows(magnitude, floor):
    rng = np.random.default_rng(11)
    rows, columns = 4000, 64
    with np.errstate(over="ignore"):
        values = bf16(rng.standard_normal((rows, columns)).astype(np.float32) * np.float32(magnitude))
    amax = np.abs(values).max(axis=1, keepdims=True)
    with np.errstate(all="ignore"):
        scale = np.maximum((amax / np.float32(127.0)).astype(np.float32), np.float32(floor))
    scale = np.broadcast_to(np.where(amax > 0, scale, np.float32(1.0)), values.shape)
    got, slow = fast(values.reshape(-1), scale.reshape(-1))
    assert np.array_equal(got, exact(values.reshape(-1), scale.reshape(-1)))
    if 1e-28 < magnitude < 1e30:
        assert slow.mean() < 5e-2  # the division is the rare case (bf16 rows have more exact ties than random reals)


def test_boundaries_and_non_finite_rows():
    halves = (np.arange(-127, 127) + 0.5).astype(np.float32)
    for step in (-2, -1, 0, 1, 2):
        for scale in (np.float32(1.0), np.float32(1.0 / 127.0), np.float32(0.0078125), np.float32(0.3)):
            values = (halves * scale).view(np.int32) + step
            values = np.concatenate([values.view(np.float32), np.full(2, 127.0, np.float32) * scale])
            scales = np.full(values.shape, scale, np.float32)
            got, _ = fast(values, scales)
            assert np.array_equal(got, exact(values, scales))
    odd = np.array([np.inf, -np.inf, np.nan, 1.0, np.nan, 0.0, -3.0, 2.0], np.float32)
    for scale in (np.float32(np.inf), np.float32(1.0), np.float32(3.0 / 127.0)):
        values = odd if np.isinf(scale) else np.where(np.isinf(odd), np.float32(0.5), odd)
        scales = np.full(values.shape, scale, np.float32)
        got, _ = fast(values, scales)
        assert np.array_equal(got, exact(values, scales))


@pytest.mark.parametrize("clamp_low", [-127.0, -128.0])
def test_scales_rounded_to_few_units(clamp_low):
    """fp32 rows whose scale has few significant bits: every magnitude up to 20000 units of the smallest fp32 number, then around
    the scales of 2^-130 .. 2^-125, where the reciprocal stops overflowing."""
    near = np.concatenate([np.round(127 * 2.0 ** (19 + step / 8)).astype(np.int64) + np.arange(-40, 41) for step in range(49)])
    units = np.concatenate([np.arange(1, 20001), near])
    amax = units.astype(np.int32).view(np.float32)
    scale = (amax / np.float32(127.0)).astype(np.float32)
    fractions = np.float32([1.0, 0.999, 0.5, 0.0, -1.0, -0.996, -0.25, 1e-3])
    values = (amax[:, None] * fractions).astype(np.float32)
    scales = np.broadcast_to(scale[:, None], values.shape).reshape(-1)
    got, slow = fast(values.reshape(-1), scales, clamp_low)
    assert np.array_equal(got, exact(values.reshape(-1), scales, clamp_low))
    assert got.min() == clamp_low and not slow.all()
