"""recip64_normal (csrc/common.cuh) restated on the CPU: the integer conversions to and
from the FP32 reciprocal give what the conversions themselves give, for either
sign, at rounding ties and at significands that carry into the exponent."""
from __future__ import annotations

import numpy as np


def seed_by_bits(f: float) -> float:
    u = int(np.float64(f).view(np.uint64))
    top = u >> 32
    sign = top & 0x80000000
    assert not ((((top >> 20) & 0x7FF) - 923) & 0xFFFFFFFF) > 200
    dropped = u & 0x1FFFFFFF
    b = ((u >> 29) - (896 << 23)) & 0xFFFFFFFF
    assert b < 1 << 31
    b += 1 if dropped > 0x10000000 or (dropped == 0x10000000 and b & 1) else 0
    with np.errstate(all="ignore"):
        x = int((np.float32(1.0) / np.uint32(b).view(np.float32)).view(np.uint32))
    hi = ((x >> 3) + (896 << 20)) | sign
    return float(np.uint64((hi << 32) | ((x << 29) & 0xFFFFFFFF)).view(np.float64))


def seed_by_conversion(f: float) -> float:
    return float(np.float32(1.0) / np.float32(f))


def test_seeds_are_the_conversions():
    rng = np.random.default_rng(0)
    x = rng.uniform(1.0, 2.0, 4000) * 2.0 ** rng.integers(-99, 99, 4000)
    m = rng.integers(0, 1 << 23, 300)
    ties = (1.0 + (m * 2.0 ** 29 + 2.0 ** 28) * 2.0 ** -52) * 2.0 ** rng.integers(-5, 5, 300)
    carry = np.array([np.nextafter(2.0, 1.0), np.nextafter(4.0, 1.0), 2.0 ** -100, 2.0 ** 100, 1.0, 5.7, 99.0])
    for f in np.concatenate([x, ties, carry]):
        for s in (f, -f):
            assert seed_by_bits(s) == seed_by_conversion(s), s

