"""The FP32 limiter's two forms pick the same value: with d = |den| and
q = num*sign(den), max(0, min(2d, max(q, min(2q, d)))) (the reference's, with
the division multiplied out) and max(0, min(2q, d), min(q, 2d)), the minima
taken on magnitudes with the product's sign as the GPU instruction does.
Every candidate is an input or its double, so the results are equal exactly,
in every region of r = num/den and on its edges."""
from __future__ import annotations

import numpy as np
import pytest


def clamp(den, num):
    s = np.where(np.signbit(den), np.float32(-1), np.float32(1))
    q, d = num * s, np.abs(den)
    return s * np.maximum(np.float32(0), np.minimum(d + d, np.maximum(q, np.minimum(q + q, d))))


def min_xorsign(a, b):
    m = np.minimum(np.abs(a), np.abs(b))
    return np.where(np.signbit(a) ^ np.signbit(b), -m, m)


def two_minima(den, num):
    b = np.maximum(np.maximum(min_xorsign(num + num, den), min_xorsign(num, den + den)), np.float32(0))
    return np.where(np.signbit(den), -b, b)


@pytest.mark.parametrize("scale", [1e-20, 1e-3, 1.0, 300.0, 1e20])
def test_same_value(scale):
    rng = np.random.default_rng(5)
    den = (scale * rng.standard_normal(4000)).astype(np.float32)
    r = np.concatenate([rng.uniform(-3, 3, 3900), np.tile([-0.0, 0.0, 0.5, 1.0, 2.0], 20)]).astype(np.float32)
    num = den * r
    den[::97] = 0.0
    num[::89] = 0.0
    assert np.array_equal(clamp(den, num), two_minima(den, num))
