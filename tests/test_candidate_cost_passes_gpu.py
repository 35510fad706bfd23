"""Candidate costs of every family against a restatement in NumPy of the
sequential double sums (EstimateAcStrategyCost, src/codec/ac_strategy.cpp:
880-994), for residuals that the folded inverse transforms settle, that they
have to transform again (magnitudes outside the settled range) and that are
zero: within one ulp of the eighth root, which the cost's last additions keep
within two ulp. A pixel's last bit rarely shows in a cost; the passes' pixels are
compared in test_folded_passes_gpu.py."""

import numpy as np
import pytest
import torch

from gjxl_b200 import _lib
from tests.gpu_util import host, to_device, zeros

pytestmark = pytest.mark.gpu
F = np.float32
FAMILIES = [(0, 8, 8), (6, 8, 16), (7, 16, 8), (4, 16, 16), (10, 16, 32), (11, 32, 16),
            (5, 32, 32)]
DESC = np.dtype([("block_x", "<u4"), ("block_y", "<u4"), ("quant_norm", "<f4"),
                 ("entropy_multiplier", "<f4"), ("cfl_x", "<f4"), ("cfl_b", "<f4")])


def bases(n):
    from tests.test_dct_basis_cpu import committed_tables
    t = committed_tables()
    return t[f"Forward{n}"].reshape(n, n), t[f"Inverse{n}"].reshape(n, n).T


def lines(x, basis):
    """out[..., k] = sum_s x[..., s] * basis[k][s], in order, each rounded."""
    acc = np.zeros(x.shape[:-1] + (basis.shape[0],))
    for s in range(basis.shape[1]):
        acc = acc + x[..., s:s + 1] * basis[:, s]
    return acc


def in_order(terms):
    return np.add.accumulate(np.concatenate([[F(0)], terms]).astype(F), dtype=F)[-1]


def ceil_log2(v):
    return 0 if v <= 1 else int(v - 1).bit_length()


def cost(pixels, mask, strategy, w, h, qn, cfl, entropy_multiplier):
    n = w * h
    fw, iw = bases(w)
    fh, ih = bases(h)
    rows = lines(pixels.astype(np.float64), fw)
    coef = lines(rows.swapaxes(-1, -2), fh).swapaxes(-1, -2).astype(F)
    entropy, loss = F(0), F(0)
    v, u = np.mgrid[0:h, 0:w]
    j = v * w + u if h < w else u * h + v  # coefficient_index
    offsets, multipliers = (12.0, 0.0, 4.0), (2.0441408586549744e7, 1.0, 1.266770081387616)
    for c in range(3):
        dq, inv = np.zeros(n, F), np.zeros(n, F)
        _lib.call("gjxl_b200_quant_matrix", strategy, c, dq.ctypes.data, inv.ctypes.data, n)
        decorrelated = coef[c] - coef[1] * F((cfl[0], 0.0, cfl[1])[c])
        scaled = decorrelated * inv[j] * F(qn)
        rounded = np.trunc(scaled)
        rounded = np.where(np.abs(scaled - rounded) >= F(0.5),
                           rounded + np.copysign(F(1), scaled), rounded).astype(F)
        residual = dq[j] * (scaled - rounded)
        roots = np.zeros(n, F)
        roots[j.ravel()] = np.sqrt(np.abs(rounded)).ravel()
        back = lines(residual.astype(np.float64), iw)
        back = lines(back.swapaxes(-1, -2), ih).swapaxes(-1, -2).astype(F)
        weighted = (mask + F(offsets[c])) * back
        for _ in range(3):
            weighted = weighted * weighted
        loss += in_order(weighted.ravel()) * F(multipliers[c])
        entropy += F(10.833273317067883) * in_order(roots)
        bits = ceil_log2(int((rounded != 0).sum()) + 1) + 1
        entropy += F(9.3089059022677905) * F(ceil_log2(bits + 17) + bits)
        if c == 0 and n > 64:
            weight = F(1) + min(F(3), F(n // 64) / F(8))
            entropy, loss = entropy * weight, loss * weight
    root = F(np.float64(loss / F(n)) ** 0.125)
    return entropy * F(entropy_multiplier) + F(1.2) * (root * F(n) / F(qn))


@pytest.mark.parametrize("strategy,w,h", FAMILIES)
@pytest.mark.parametrize("kind", ["random", "smooth", "flat", "zero", "tiny"])
def test_costs_match_the_sequential_sums(cuda, strategy, w, h, kind):
    rng = np.random.default_rng(strategy * 10 + 1)
    side = 72
    y, x = np.mgrid[0:side, 0:side]
    image = rng.normal(0, 1, (3, side, side)) * [[[0.02]], [[0.3]], [[0.3]]]
    if kind == "smooth":
        image = np.stack([0.01 * np.sin(x / 9), 0.4 + 0.2 * np.cos(y / 7), x * y / 9000.0])
    elif kind == "flat":
        image = np.ones((3, side, side)) * [[[0.01]], [[0.4]], [[0.3]]]
    elif kind == "zero":
        image = image * 0
    elif kind == "tiny":
        image = image * 1e-36
    image = image.astype(F)
    mask = (rng.random((side, side)) + 0.5).astype(F)
    desc = np.zeros(3, DESC)
    limit = side // 8 - np.array([w // 8, h // 8])
    desc["block_x"] = [0, limit[0], 1]
    desc["block_y"] = [0, limit[1], 2]
    desc["quant_norm"], desc["entropy_multiplier"] = [0.7, 0.2, 1.3], 1.1
    desc["cfl_x"], desc["cfl_b"] = [0.0, 0.05, -0.1], [1.0, 0.9, 1.05]
    out = zeros((3,))
    d_image, d_mask = to_device(image), to_device(mask)
    d_desc = torch.from_numpy(desc.view(np.uint8).copy()).cuda()
    _lib.call("gjxl_b200_ac_strategy_candidate_costs", strategy, d_image.data_ptr(), side,
              side * side, d_mask.data_ptr(), side, side, side, d_desc.data_ptr(), 3, None, None,
              None, None, 1.0, 0, out.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
    got = host(out)
    for d, g in zip(desc, got):
        x0, y0 = int(d["block_x"]) * 8, int(d["block_y"]) * 8
        want = cost(image[:, y0:y0 + h, x0:x0 + w], mask[y0:y0 + h, x0:x0 + w], strategy, w, h,
                    d["quant_norm"], (d["cfl_x"], d["cfl_b"]), d["entropy_multiplier"])
        ulp = abs(int(F(g).view(np.int32)) - int(F(want).view(np.int32)))
        assert ulp <= 2, (g, want)
