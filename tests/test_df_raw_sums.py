"""Unnormalised float-float sums (df_add_raw, df_norm; fl_device.cuh) against exact
arithmetic, in f32 on the CPU: four products at a time with a normalisation after
them, and a tree of 32, lose no more than 2^-44 of the sum of the terms."""
from fractions import Fraction

import numpy as np
import pytest

F = np.float32


def add_raw(a, b):
    s = F(a[0] + b[0])
    bb = F(s - a[0])
    e = F(F(a[0] - F(s - bb)) + F(b[0] - bb))
    return s, F(F(a[1] + b[1]) + e)


def norm(a):
    hi = F(a[0] + a[1])
    return hi, F(a[1] - F(hi - a[0]))


def prod(x, y):
    p = F(x * y)
    return p, F(float(Fraction(float(x)) * Fraction(float(y)) - Fraction(float(p))))


@pytest.mark.parametrize("seed,same", [(1, True), (2, True), (3, False), (4, False)])
def test_chain_and_tree(seed, same):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal((32, 64)) * 10.0 ** rng.integers(-3, 4, (32, 64))).astype(F)
    y = x if same else rng.standard_normal((32, 64)).astype(F)
    lanes, exact, size = [], Fraction(0), Fraction(0)
    for i in range(32):
        a = (F(0), F(0))
        for j in range(64):
            a = add_raw(a, prod(x[i, j], y[i, j]))
            if j % 4 == 3:
                a = norm(a)
            t = Fraction(float(x[i, j])) * Fraction(float(y[i, j]))
            exact += t
            size += abs(t)
        lanes.append(a)
    while len(lanes) > 1:
        h = len(lanes) // 2
        lanes = [add_raw(lanes[k], lanes[k + h]) for k in range(h)]
    hi, lo = norm(lanes[0])
    assert abs(Fraction(float(hi)) + Fraction(float(lo)) - exact) <= size * Fraction(1, 2**44)
