"""The half-precision arithmetic of the warp-cooperative BC1 trials (qt_bc1_coop.cuh), on the CPU: palettes formed
from halves 1536 + v equal the interpolators' integers for every pair of channel values, and a palette row times a
texel column gives |c|^2 - 2 p.c exactly, in any order of summation."""

import numpy as np
import pytest

A, B = (v.astype(np.float64) for v in np.meshgrid(np.arange(256), np.arange(256), indexing="ij"))


def _half(x):
    """Round to the nearest half (ties to even), as one HFMA2 or HADD2 does with its exact result."""
    return x.astype(np.float16).astype(np.float64)


@pytest.mark.parametrize("name,sub,exact", [
    ("ideal", 1537.0, lambda a, b: (2 * a + b) // 3),
    ("round", 1536.0, lambda a, b: (2 * a + b + 1) // 3),
])
def test_interpolated_thirds(name, sub, exact):
    third = np.float64(np.uint16(0x3555).view(np.float16))
    a0 = _half((1536 + A) - 1536)
    b0 = _half((1536 + B) - sub)
    t = _half(2 * a0 + b0)
    q = _half(t * third + 1536)
    assert np.array_equal(q, 1536 + exact(A, B)), name
    assert q.max() < 2048 and q.min() >= 1536  # unit spacing: the low byte is the value


def test_packed_amd_and_halves():
    a, b = A.astype(np.uint32), B.astype(np.uint32)
    x, y = a | (b << 16), b | (a << 16)  # two channels a word, both orders
    amd = ((43 * x + 21 * y + 0x00200020) >> 6) & 0x00FF00FF
    assert np.array_equal(amd & 0xFFFF, (43 * a + 21 * b + 32) >> 6) and np.array_equal(amd >> 16, (43 * b + 21 * a + 32) >> 6)
    for bias in (0, 1):
        h = ((x + y + bias * 0x00010001) >> 1) & 0x00FF00FF
        assert np.array_equal(h & 0xFFFF, (a + b + bias) >> 1) and np.array_equal(h >> 16, (a + b + bias) >> 1)


def test_row_times_column_is_exact():
    rng = np.random.default_rng(0)
    c = np.concatenate([rng.integers(0, 256, (4000, 3)), [[0, 0, 0], [255, 255, 255], [255, 0, 0]]])
    p = np.concatenate([rng.integers(0, 256, (4000, 3)), [[255, 255, 255], [255, 255, 255], [0, 0, 0]]])
    n = (c * c).sum(1)
    row = np.stack([1536 + c[:, 0], 1536 + c[:, 1], 1536 + c[:, 2], 1536 + rng.integers(0, 256, len(c)), 1024 + (n & 255), 1024 + (n >> 8),
                    np.full(len(c), 3072), np.full(len(c), 1024)], 1).astype(np.float64)
    col = np.stack([-2 * p[:, 0], -2 * p[:, 1], -2 * p[:, 2], np.zeros(len(c)), np.ones(len(c)), np.full(len(c), 256), p.sum(1), np.full(len(c), -257)],
                   1).astype(np.float64)
    assert np.array_equal(_half(row), row) and np.array_equal(_half(col), col)  # every entry is a half
    terms = row * col
    assert np.array_equal(terms.sum(1), n - 2 * (p * c).sum(1))
    assert np.abs(terms).sum(1).max() < 2 ** 24  # so float32 sums are exact in any order
