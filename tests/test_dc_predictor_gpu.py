"""The weighted DC predictor's wavefront (gjxl_b200_dc_tokenize, prediction 1)
against a sample-by-sample restatement in Python integers, at the row counts
where its layout changes (a warp owns 32 rows, a group is 256 blocks) and
with values that leave its 32-bit bounds in some rows only."""

import numpy as np
import pytest

from gjxl_b200 import stages
from tests.gpu_util import host, to_device

pytestmark = pytest.mark.gpu

RECIPROCAL = [(1 << 24) // (i + 1) for i in range(64)]


def predict_plane(q: np.ndarray) -> tuple[list, list]:
    """(property, residual) of every sample of one group's channel, raster
    order (src/codec/modular/prediction.h:59-150)."""
    h, w = q.shape
    err = np.zeros((h + 1, w + 2), object)          # signed errors, row -1 zero
    pe = [[[0] * 4 for _ in range(w + 1)] for _ in range(2)]  # rolling rows
    props, residuals = [], []
    for y in range(h):
        cur, prev = pe[y & 1], pe[(y & 1) ^ 1]
        for x in range(w):
            W = int(q[y, x - 1]) if x else int(q[y - 1, x]) if y else 0
            N = int(q[y - 1, x]) if y else W
            NW = int(q[y - 1, x - 1]) if x and y else W
            NE = int(q[y - 1, x + 1]) if y and x + 1 < w else N
            NN = int(q[y - 2, x]) if y > 1 else N
            e = lambda dx: err[y, min(max(x + dx, 0), w - 1)]
            en, enw, ene = e(0), e(-1), e(1)
            ew = err[y + 1, x - 1] if x else 0
            north, nw = prev[x], prev[x - 1] if x else prev[x]
            ne = prev[x + 1] if x + 1 < w else north
            weights = []
            for i in range(4):
                s = north[i] + nw[i] + ne[i]
                shift = max(0, (s + 1).bit_length() - 6)
                weights.append(4 + (((13, 12, 12, 12)[i] * RECIPROCAL[s >> shift]) >> shift))
            drop = sum(weights).bit_length() - 5
            weights = [v >> drop for v in weights]
            total = sum(weights)
            p = [(W + NE - N) * 8, N * 8 - (((en + ew + ene) * 16) >> 5),
                 W * 8 - (((en + ew + enw) * 10) >> 5),
                 N * 8 - ((enw * 7 + en * 7 + ene * 7) >> 5)]
            acc = (total >> 1) - 1 + sum(a * b for a, b in zip(p, weights))
            pred = (acc * RECIPROCAL[total - 1]) >> 24
            if ((en ^ ew) | (en ^ enw)) <= 0:
                lo, hi = min(W, NE, N) * 8, max(W, NE, N) * 8
                pred = min(max(pred, lo), hi)
            prop = ew
            for v in (en, enw, ene):
                if abs(v) > abs(prop):
                    prop = v
            value = int(q[y, x])
            props.append(prop)
            residuals.append(value - ((pred + 3) >> 3))
            err[y + 1, x] = pred - value * 8
            sub = [(abs(v - value * 8) + 3) >> 3 for v in p]
            cur[x] = sub
            prev[x + 1] = [a + b for a, b in zip(prev[x + 1], sub)]
        # The row above row 0 is the second rolling row: it holds only what
        # row 0 added to it.
        pe[(y & 1) ^ 1] = [[0] * 4 for _ in range(w + 1)]
    return props, residuals


def token(v: int) -> int:
    return 2 * v if v >= 0 else -2 * v - 1


@pytest.mark.parametrize("bx,by,wide", [(1, 1, 0), (1, 40, 0), (40, 1, 0), (2, 33, 0), (9, 64, 0),
                                        (33, 65, 0), (70, 32, 1), (20, 70, 1), (261, 9, 0),
                                        (7, 260, 1)])
def test_weighted_tokens_match_restatement(cuda, bx, by, wide):
    rng = np.random.default_rng(bx * 1000 + by)
    q = np.cumsum(rng.integers(-3, 4, (3, by, bx)), 2).astype(np.int32)
    q += rng.integers(-40, 41, (3, by, 1)).astype(np.int32)
    if wide:  # one row far outside the 32-bit bounds, one just at them
        q[1, by // 2] += 1 << 26
        q[0, by // 3] -= (1 << 21) - 3
        q[2, by - 1, bx // 2:] += 1 << 23
    cells = np.full((by, bx), 1, np.uint8)
    raw = np.full((by, bx), 5, np.int32)
    tiles = ((by + 7) // 8, (bx + 7) // 8)
    cfl = to_device(np.zeros(tiles, np.int8))
    got = stages.dc_tokenize(to_device(q), to_device(cells), to_device(raw), cfl, cfl,
                             prediction=1)
    values = host(got["dc"]).view(np.uint32)[:, 1]
    want = []
    for gy in range(0, by, 256):
        for gx in range(0, bx, 256):
            for c in (1, 0, 2):
                _, r = predict_plane(q[c, gy:gy + 256, gx:gx + 256])
                want += [token(v) for v in r]
    assert int(host(got["error"])[0]) == 0
    bad = np.nonzero(values != np.array(want, np.uint64).astype(np.uint32))[0]
    assert bad.size == 0, f"{bad.size} of {values.size} tokens differ, first at {bad[:5]}"
