"""The fixed-point dot products of the slot layout, restated on the CPU.

The kernel turns k and q into integers ``rint(x * 2^(30 - e))``, ``2^e`` above the largest magnitude, cuts them into four
signed base-256 digits, lets the integer tensor cores sum codes times digits and rounds the total once.
"""

from __future__ import annotations

import numpy as np
import pytest


def _fix_scale(x):
    bits = np.abs(x).max().astype(np.float32).view(np.uint32)
    e = max(int(bits >> 23), 30)
    return np.uint32((283 - e) << 23).view(np.float32)


def _digits(fixed):
    d = ((fixed.astype(np.int64) + 0x00808080) & 0xFFFFFFFF).astype(np.uint32) ^ np.uint32(0x00808080)
    return np.stack([(d >> s).astype(np.uint8).view(np.int8) for s in (0, 8, 16, 24)])


def test_digits_add_up_at_the_ends_of_the_range():
    edge = np.array([0, 1, -1, 127, 128, -128, -129, 0x7F7F7F, 0x808080, -0x808080, -0x808081, 2**30, -2**30], np.int64)
    rng = np.random.default_rng(0)
    fixed = np.concatenate([edge, rng.integers(-2**30, 2**30 + 1, 4096)])
    d = _digits(fixed).astype(np.int64)
    assert np.array_equal(d[0] + 256 * d[1] + 65536 * d[2] + 2**24 * d[3], fixed)
    # 128 products of a code and a digit, two digits combined: within 32 bits
    assert 128 * 127 * 128 * 257 < 2**31


@pytest.mark.parametrize("bits", [8, 11, 24], ids=["bf16", "fp16", "fp32"])
def test_one_rounding_per_total(bits):
    """Against 64 bits, no further off than packed fp32 multiply-adds (two chains of 8 per lane, a tree over 8 lanes)."""
    rng = np.random.default_rng(bits)
    ours = chain = size = 0.0
    for _ in range(200):
        codes = np.clip(np.rint(42 * rng.standard_normal((16, 128))), -127, 127)
        x = rng.standard_normal(128).astype(np.float32)
        m, ex = np.frexp(x)
        x = np.ldexp(np.rint(m * 2**bits), ex - bits).astype(np.float32)
        exact = codes @ x.astype(np.float64)
        scale = _fix_scale(x)
        fixed = np.rint(x.astype(np.float64) * scale).astype(np.int64)
        assert np.abs(fixed).max() <= 2**30
        d = _digits(fixed).astype(np.int64)
        assert np.array_equal((d * np.array([1, 256, 65536, 2**24])[:, None]).sum(0), fixed)
        total = (codes.astype(np.int64) @ fixed).astype(np.float32) * (np.float32(1) / scale)
        # products of a code and a 24-bit number are rounded here, fused in the kernel that this replaced: allow for that below
        acc = np.zeros((16, 8, 2), np.float32)
        for c in range(16):
            term = codes[:, c::16] * x[c::16].astype(np.float64)
            acc[:, :, (c >> 1) & 1] = (acc[:, :, (c >> 1) & 1] + term).astype(np.float32)
        p = acc[:, :, 0] + acc[:, :, 1]
        p = ((p[:, 0] + p[:, 4]) + (p[:, 2] + p[:, 6])) + ((p[:, 1] + p[:, 5]) + (p[:, 3] + p[:, 7]))
        ours += ((total - exact) ** 2).sum(); chain += ((p - exact) ** 2).sum(); size += (exact ** 2).sum()
    assert np.sqrt(ours / size) <= np.sqrt(chain / size)
    assert np.sqrt(ours / size) < 2.0**-24                      # half a unit in the last place, rms well below it


def test_what_16_bit_types_lose_is_nothing():
    """bf16 down to 2^-23 of the largest element and fp16 down to its subnormals next to 64 are whole numbers after scaling."""
    top = np.float32(1.9921875)
    bf16 = np.ldexp(np.arange(128, 256), -7).astype(np.float32)
    for shift in (0, 8, 22):
        y = np.ldexp(bf16, -shift).astype(np.float64) * _fix_scale(np.array([top]))
        assert np.array_equal(y, np.rint(y)), shift
    y = np.ldexp(np.arange(1, 2048), -24).astype(np.float64) * _fix_scale(np.array([63.0], np.float32))
    assert np.array_equal(y, np.rint(y))
