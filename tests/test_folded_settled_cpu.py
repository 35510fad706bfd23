"""When the folded inverse transforms take a float as settled (FoldedSettled,
csrc/line_dct.cuh), the kernels' own code on the host: never with a tie between
floats within the bound, in particular next to powers of two, where the tie
below is half as far as the one above; and always with the ties clearly
further away."""

import ctypes
from fractions import Fraction

import numpy as np
import pytest

from tests.native_util import load


@pytest.fixture(scope="module")
def settled(tmp_path_factory):
    native = load("folded_passes", tmp_path_factory.mktemp("native"))

    def call(values, bound: float) -> bool:
        a = np.ascontiguousarray(values, np.float64)
        return bool(native.folded_settled(ctypes.c_void_p(a.ctypes.data), a.size,
                                          ctypes.c_double(bound)))

    return call


def to_float32(x: Fraction) -> Fraction:
    """x rounded to the nearest float, ties to even, in one rounding."""
    if x == 0:
        return x
    e = 0
    while abs(x) >= Fraction(2) ** (e + 1):
        e += 1
    while abs(x) < Fraction(2) ** e:
        e -= 1
    quantum = Fraction(2) ** (max(e, -126) - 23)
    return round(x / quantum) * quantum


def may_differ(v: float, bound: float) -> bool:
    f = to_float32(Fraction(v))
    return any(to_float32(Fraction(v) + s * Fraction(bound)) != f for s in (-1, 1))


EXPONENTS = [-130, -126, -60, -1, 0, 1, 40]
# Offsets from 2^e in units of 2^(e-25): up to the tie above, and below 2^e.
OFFSETS = [0.0, 2.0 ** -27, 2.0 ** -10, 0.5, 0.999, 1.0, 1.5, 2.0, 3.0, 4.0, -2.0 ** -27, -0.5, -1.0]
BOUNDS = [2.0 ** -28, 2.0 ** -12, 0.25, 0.499, 0.5, 0.51, 0.9, 0.999, 1.0, 1.001, 1.5, 1.8, 1.999,
          2.0, 2.5]


@pytest.mark.parametrize("e", EXPONENTS)
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_settled_only_where_the_float_cannot_differ(settled, e, sign):
    unit = 2.0 ** (e - 25)
    for offset in OFFSETS:
        for scaled in BOUNDS:
            v, bound = sign * (2.0 ** e + offset * unit), scaled * unit
            if settled([v], bound):
                assert not may_differ(v, bound), (offset, scaled)
            # In a column with values that are far from any tie.
            if settled([v, sign * 2.0 ** (e + 3), v], bound):
                assert not may_differ(v, bound), (offset, scaled)


def test_settled_over_random_values(settled):
    rng = np.random.default_rng(1)
    accepted = 0
    for _ in range(4000):
        e = int(rng.integers(-20, 20))
        v = float(np.float32(rng.uniform(1, 2) * 2.0 ** e)) + float(rng.uniform(-1, 1)) * 2.0 ** (e - 24)
        bound = 2.0 ** (e - float(rng.uniform(23, 50)))
        got = settled([v], bound)
        if got:
            assert not may_differ(v, bound)
            accepted += 1
        distance = abs(v - float(np.float32(v)))
        if bound < 0.99 * 2.0 ** (e - 25) and distance + bound < 0.99 * 2.0 ** (e - 24):
            assert got, (v, bound)
    assert accepted > 2000


@pytest.mark.parametrize("v", [0.0, float("nan"), float("inf")])
def test_zero_and_non_finite_values_are_not_settled(settled, v):
    assert not settled([1.0, v], 2.0 ** -60)
