"""The rounding bound of the folded inverse transforms (csrc/line_dct.cuh):
the committed half tables with their stated error, and |folded - sequential|
<= FoldBound * (sum of magnitudes), in exact arithmetic with every operation
rounded once, for the kernels' own operation order."""

import re
from fractions import Fraction

import numpy as np
import pytest

from tests.test_dct_basis_cpu import CSRC, committed_tables

SQRT2 = 1.41421356237309515
U = 2.0 ** -53


def half_error(n: int) -> float:
    text = (CSRC / "dct_basis.inc").read_text()
    return float.fromhex(re.search(rf"kDctInverseHalfError{n} = (\S+);", text).group(1))


def line_bound(n: int) -> float:
    return (n + n // 2 + 1) * U * SQRT2 + half_error(n)


@pytest.mark.parametrize("n", [8, 16, 32])
def test_half_tables_are_within_their_stated_error(n):
    tables = committed_tables()
    inverse = tables[f"Inverse{n}"].reshape(n, n)
    half = tables[f"InverseHalf{n}"].reshape(n, n // 2)
    sign = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)[:, None]
    mirrored = sign * half[:, ::-1]
    worst = max(abs(Fraction(a) - Fraction(b)) for a, b in
                zip(np.hstack([half, mirrored]).ravel(), inverse.ravel()))
    assert worst <= Fraction(half_error(n))
    assert np.abs(inverse).max() <= SQRT2 * (1 + 2 * U)


def fma(a: float, b: float, c: float) -> float:
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # one rounding


def folded(line, half, n):
    out = [0.0] * n
    for x in range(n // 2):
        even, odd = 0.0 + line[0], line[1] * half[1][x]
        for u in range(2, n, 2):
            even = fma(line[u], half[u][x], even)
            odd = fma(line[u + 1], half[u + 1][x], odd)
        out[x], out[n - 1 - x] = even + odd, even - odd
    return out


def sequential(line, inverse, n):
    out = []
    for x in range(n):
        acc = 0.0
        for u in range(n):
            acc += line[u] * inverse[u][x]
        out.append(acc)
    return out


def both_passes(block, w, h, tables, one_line, name):
    row_table = tables[f"{name}{w}"].reshape(w, -1).tolist()
    column_table = tables[f"{name}{h}"].reshape(h, -1).tolist()
    rows = [one_line(list(map(float, r)), row_table, w) for r in block]
    return np.array([one_line([r[x] for r in rows], column_table, h) for x in range(w)]).T


@pytest.mark.parametrize("w,h", [(8, 8), (16, 8), (8, 16), (16, 16), (32, 16), (16, 32),
                                 (32, 32)])
@pytest.mark.parametrize("kind", ["normal", "one", "spread", "cancel"])
def test_folded_and_sequential_sums_differ_within_the_bound(w, h, kind):
    rng = np.random.default_rng(w * 100 + h)
    block = rng.normal(0, 1, (h, w)).astype(np.float32)
    if kind == "one":
        block[:] = 0
        block[h - 1, w - 1] = np.float32(1) / np.float32(3)
    elif kind == "spread":
        block *= np.exp2(rng.integers(-40, 40, (h, w))).astype(np.float32)
    elif kind == "cancel":
        block[:, 1::2] = -block[:, ::2]
    tables = committed_tables()
    a = both_passes(block, w, h, tables, folded, "InverseHalf")
    b = both_passes(block, w, h, tables, sequential, "Inverse")
    bound = 1.001 * SQRT2 * (line_bound(w) + line_bound(h)) * float(
        np.abs(block.astype(np.float64)).sum())
    assert np.abs(a - b).max() <= bound
