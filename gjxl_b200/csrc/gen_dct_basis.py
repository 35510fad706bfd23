"""Writes dct_basis.inc: the double-precision DCT-II / DCT-III bases of
lengths 8, 16 and 32 (and the forward bases transposed) as exact
hexadecimal literals in constant memory, plus global-memory copies of the
two length-32 tables that the cost kernels stage into shared memory with
coalesced loads.

The values follow the reference's MakeBasis (src/codec/dct.cpp:21-41):
basis[f * N + s] = (scale * alpha) * cos((s + 0.5) * f * pi / N), with
scale = sqrt(2) / N (forward) or sqrt(2) (inverse) and alpha = 1 / sqrt(2)
for f = 0, evaluated left to right in IEEE double with the C library's cos
(Python's math.cos calls it), so every literal equals the reference's table.

Run: python gjxl_b200/csrc/gen_dct_basis.py > gjxl_b200/csrc/dct_basis.inc
"""

import math
import struct
import sys


def basis(n: int, forward: bool) -> list[float]:
    sqrt_two = math.sqrt(2.0)
    scale = sqrt_two / float(n) if forward else sqrt_two
    out = []
    for frequency in range(n):
        alpha = 1.0 / sqrt_two if frequency == 0 else 1.0
        for sample in range(n):
            angle = (float(sample) + 0.5) * float(frequency) * math.pi / float(n)
            out.append(scale * alpha * math.cos(angle))
    return out


def render() -> str:
    lines = [
        "// Generated by gen_dct_basis.py: DCT bases of the reference CPU transform",
        "// (src/codec/dct.cpp:21-41), basis[frequency * N + sample], exact doubles.",
        "#pragma once",
        "",
    ]
    tables = []
    for direction, forward in (("Forward", True), ("Inverse", False)):
        for n in (8, 16, 32):
            tables.append((f"kDct{direction}{n}", basis(n, forward)))
    # The forward bases transposed, [sample * N + frequency], for the
    # table-driven line passes.
    for n in (8, 16, 32):
        b = basis(n, True)
        tables.append((f"kDctForwardT{n}", [b[f * n + s] for s in range(n) for f in range(n)]))
    # The inverse bases' first halves for the folded passes, [frequency * N / 2
    # + sample]: the mean of the two table values that mirror one another, and
    # how far either is from it.
    folds = []
    for n in (8, 16, 32):
        b = basis(n, False)
        half, error = [], 0.0
        for u in range(n):
            for x in range(n // 2):
                near, far = b[u * n + x], b[u * n + n - 1 - x] * (-1.0 if u % 2 else 1.0)
                mean = 0.5 * (near + far)
                half.append(mean)
                error = max(error, abs(near - mean), abs(far - mean))
        tables.append((f"kDctInverseHalf{n}", half))
        folds.append((n, error))
    staged = [(f"kDctStaged{name[4:]}", values) for name, values in tables
              if name in ("kDctForwardT32", "kDctInverse32")]
    for index, (name, values) in enumerate(tables + staged):
        space = "__constant__" if index < len(tables) else "__device__ const __align__(16)"
        lines.append(f"static {space} double {name}[{len(values)}] = {{")
        for i in range(0, len(values), 4):
            lines.append("  " + ", ".join(v.hex() for v in values[i:i + 4]) + ",")
        lines.append("};")
        lines.append("")
    lines.append("// Largest distance between an inverse basis value and its half-table entry.")
    for n, error in folds:
        lines.append(f"constexpr double kDctInverseHalfError{n} = {error.hex()};")
    lines.append("")
    # Single-precision copies (each value rounded to nearest float) of the
    # lengths 8 and 16, for the FP32 transform passes of the fast cost mode.
    lines.append("// Rounded to float for the FP32 passes.")
    for name, values in tables:
        if not any(name == f"kDct{d}{n}" for d in ("Forward", "Inverse") for n in (8, 16)):
            continue
        rounded = [struct.unpack("<f", struct.pack("<f", v))[0] for v in values]
        lines.append(f"static __constant__ float {name}F[{len(values)}] = {{")
        for i in range(0, len(rounded), 4):
            lines.append("  " + ", ".join(v.hex() + "f" for v in rounded[i:i + 4]) + ",")
        lines.append("};")
        lines.append("")
    return "\n".join(lines)


if __name__ == "__main__":
    sys.stdout.write(render())
