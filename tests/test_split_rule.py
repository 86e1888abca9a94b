"""Integer rules of the transfer kernel, restated here and checked over every
input they can meet: the division-free split of padded tile indices
(split_factor / SplitP) and the fixed-point scale (pow2_scale)."""

import struct

import numpy as np
import pytest

TILE, WIDE_TILE = 2304, 5632  # entries of the largest static tile, of a whole-segment kernel's
FACTOR_ULPS = 2  # documented error bound of the approximate division


def split_factors(d):
    """Every multiplier the device may compute for divisor d."""
    q = np.float32(4194304.0 / d)
    lo = hi = q
    for _ in range(FACTOR_ULPS):
        lo, hi = np.nextafter(lo, np.float32(0)), np.nextafter(hi, np.float32(np.inf))
    return range(int(np.float32(lo + np.float32(0.1))) + 1, int(np.float32(hi + np.float32(0.1))) + 2)


@pytest.mark.parametrize("first,step,last", [(4, 8, 68), (16, 32, TILE // 3)])
def test_split_is_exact_for_every_tile_stride(first, step, last):
    """y strides are 4 mod 8 (a box edge is at most 64), x strides 16 mod 32 and
    at most a third of the tile (a box has three x planes)."""
    t = np.arange(TILE, dtype=np.uint64)
    for d in range(first, last + 1, step):
        for m in split_factors(d):
            assert (t * np.uint64(m)).max() < 2**32
            assert np.array_equal((t * np.uint64(m)) >> np.uint64(22), t // np.uint64(d)), (d, m)


@pytest.mark.parametrize("first,step,last", [(4, 8, 68), (16, 32, WIDE_TILE // 3)])
def test_wide_split_is_exact_for_every_tile_stride(first, step, last):
    t = np.arange(WIDE_TILE, dtype=np.uint64)
    for d in range(first, last + 1, step):
        lo = hi = np.float32(4294967296.0 / d)
        for _ in range(FACTOR_ULPS):
            lo, hi = np.nextafter(lo, np.float32(0)), np.nextafter(hi, np.float32(np.inf))
        q = lo
        while q <= hi:
            m = int(np.float32(q * np.float32(1.0 + 4.76837158e-7))) + 1
            assert m < 2**32 and np.array_equal((t * np.uint64(m)) >> np.uint64(32), t // np.uint64(d)), (d, m)
            q = np.nextafter(q, np.float32(np.inf))


def bits(x):
    return struct.unpack("<i", struct.pack("<f", x))[0]


def pow2_scale(total):
    total = max(np.float32(total), np.float32(1e-30))
    k = (bits(float(total)) - 1) >> 23
    return struct.unpack("<f", struct.pack("<i", min(max(29 + 254 - k, 7), 247) << 23))[0]


def test_scale_is_the_largest_power_of_two_within_the_bound():
    rng = np.random.default_rng(0)
    totals = [np.float32(2.0**e) for e in range(-89, 99)]
    totals += [np.nextafter(t, np.float32(0)) for t in totals] + [np.nextafter(t, np.float32(np.inf)) for t in totals]
    totals += [np.float32(v) for v in np.exp(rng.uniform(np.log(1e-26), np.log(1e29), 4000))]
    for t in totals:
        s = pow2_scale(t)
        assert np.log2(s) == np.floor(np.log2(s)) and 2.0**-120 <= s <= 2.0**120
        if 2.0**-120 < s < 2.0**120:  # not clamped
            assert float(t) * s <= 2.0**30 < float(t) * s * 2, (t, s)
