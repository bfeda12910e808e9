"""The activation and its division, against the oracle and against IEEE division, bit by bit."""

import ctypes

import numpy as np
import pytest
import torch

import device

pytestmark = pytest.mark.gpu


def _around(value: float, count: int = 1 << 16) -> np.ndarray:
    """`count` neighbours of a value on either side of it."""
    bits = int(np.float32(value).view(np.uint32))
    return np.arange(max(bits - count, bits & 0x80000000), bits + count, dtype=np.uint32).view(np.float32)


def _gates() -> np.ndarray:
    generator = np.random.default_rng(5)
    parts = [np.arange(1 << 16, dtype=np.uint32) << 16]  # every BF16 value
    parts += [_around(x).view(np.uint32) for x in (
        87.0, -87.0, 88.0, -88.0, 8.6736174e-19, -8.6736174e-19,  # where the forms change
        2.0 ** -23, -7.5e-8, -3.8e-8, 1e-38, -1e-38, 3.4e38, -3.4e38, 4.9, -4.9, 9.0, -9.0)]
    # Just below zero, where the divisor of the GELU form has a significand of ones only.
    parts.append(np.arange(0xB3000000, 0xB3800000, dtype=np.uint32))
    parts.append(np.arange(1 << 16, dtype=np.uint32) | 0x80000000)  # denormals
    parts.append(np.arange(1 << 16, dtype=np.uint32))
    parts.append(generator.integers(0, 1 << 32, 1 << 20, dtype=np.uint32))
    parts.append(generator.normal(0, 3, 1 << 20).astype(np.float32).view(np.uint32))
    return np.concatenate(parts).view(np.float32)


@pytest.mark.parametrize("activation", [0, 1])
def test_activation_gives_the_oracles_bits(oracle, activation):
    gates = _gates()
    x = torch.from_numpy(gates).cuda()
    out = torch.empty_like(x)
    device.call("check_activate", x, out, x.numel(), activation)
    want = np.empty_like(gates)
    oracle.load().oracle_activate(
        ctypes.c_void_p(gates.ctypes.data), ctypes.c_void_p(want.ctypes.data),
        ctypes.c_int64(gates.size), ctypes.c_int(activation))
    got = out.cpu().numpy()
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), gates[~same][:8]


@pytest.mark.parametrize("numerator", ["two", "any"])
@pytest.mark.parametrize("side", ["below", "above"])
def test_division_from_either_neighbour_of_the_reciprocal(numerator, side):
    """The approximate reciprocal is within one unit in its last place and no more is promised: every
    significand of the divisor, with the value just below and just above its true reciprocal."""
    divisor = (np.arange(1 << 23, dtype=np.uint32) + np.float32(1.0).view(np.uint32)).view(np.float32)
    x = np.full_like(divisor, 2.0)
    if numerator == "any":
        x = np.random.default_rng(7).uniform(-4.0, 4.0, divisor.size).astype(np.float32)
    true = 1.0 / divisor.astype(np.float64)
    near = true.astype(np.float32)
    away = np.float32(0.0 if side == "below" else 2.0)
    wrong_side = (near > true) if side == "below" else (near < true)
    exact = near == true  # powers of two: the neighbour itself is one unit away
    reciprocal = np.where(wrong_side | exact, np.nextafter(near, away), near).astype(np.float32)
    arrays = [torch.from_numpy(a).cuda() for a in (x, divisor, reciprocal)]
    out = torch.empty_like(arrays[0])
    device.call("check_divide", *arrays, out, out.numel())
    got, want = out.cpu().numpy(), x / divisor
    assert np.array_equal(got, want), divisor[got != want][:8]
