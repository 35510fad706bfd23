"""Stages whose kernels share their work out by tile, strip or lane, against
restatements in NumPy, at extents with partial tiles and strips: the strategy
merge (SearchTile, src/codec/ac_strategy.cpp:591-773) on the kernel's own costs,
the initial chroma-from-luma maps (src/codec/chroma_from_luma.cpp:22-151), and
the coefficient orders (src/codestream/coefficient_order.cpp:568-830)."""

import numpy as np
import pytest
import torch

from gjxl_b200 import _lib, stages
from tests.gpu_util import STRATEGY_COVERED, host, to_device, zeros
from tests.test_dct_basis_cpu import committed_tables

pytestmark = pytest.mark.gpu
F = np.float32
FAMILIES = [0, 6, 7, 4, 10, 11, 5]  # strategy of each cost plane


class Tile:
    def __init__(self, costs, w, h, multiplier):
        self.costs, self.w, self.h = costs, w, h
        self.cell = {(x, y): (0, True) for x in range(w) for y in range(h)}
        self.cost = {(x, y): F(costs[0, y, x] * multiplier) for x in range(w) for y in range(h)}
        self.priority = dict.fromkeys(self.cell, 0)

    def of(self, strategy, x, y):
        return F(self.costs[FAMILIES.index(strategy), y, x])

    def area(self, strategy, x, y):
        cw, ch = STRATEGY_COVERED[strategy]
        return [(x + dx, y + dy) for dy in range(ch) for dx in range(cw)]

    def place(self, strategy, x, y, cost):
        for at in self.area(strategy, x, y):
            self.cell[at], self.cost[at] = (strategy, at == (x, y)), F(0)
        self.cost[x, y] = cost

    def crosses_row(self, x, y, end):
        if x >= self.w or y >= self.h or y % 8 == 0:
            return False
        while x != 0 and not self.cell[x, y][1]:
            x -= 1
        while x < min(end, self.w):
            strategy, anchor = self.cell[x, y]
            if not anchor:
                return True
            x += STRATEGY_COVERED[strategy][0]
        return False

    def crosses_column(self, x, y, end):
        if x >= self.w or y >= self.h or x % 8 == 0:
            return False
        while y != 0 and not self.cell[x, y][1]:
            y -= 1
        while y < min(end, self.h):
            strategy, anchor = self.cell[x, y]
            if not anchor:
                return True
            y += STRATEGY_COVERED[strategy][1]
        return False

    def try_merge(self, strategy, x, y, priority):
        current = F(0)
        for at in self.area(strategy, x, y):
            if self.priority[at] >= priority:
                return
            current = F(current + self.cost[at])
        candidate = self.of(strategy, x, y)
        if candidate < current:
            for at in self.area(strategy, x, y):
                self.priority[at] = priority
            self.place(strategy, x, y, candidate)

    def divide(self, n, x, y):
        if (self.crosses_row(x, y, x + n) or self.crosses_row(x, y + n, x + n) or
                self.crosses_column(x, y, y + n) or self.crosses_column(x + n, y, y + n)):
            return
        half = n // 2
        tall, wide, square = (6, 7, 4) if n == 2 else (10, 11, 5)
        columns = not self.crosses_column(x + half, y, y + n)
        rows = not self.crosses_row(x, y + half, x + n)
        q = [[F(0), F(0)], [F(0), F(0)]]
        for dy in range(n):
            for dx in range(n):
                q[dy // half][dx // half] = F(q[dy // half][dx // half] + self.cost[x + dx, y + dy])
        left, right = F(q[0][0] + q[1][0]), F(q[0][1] + q[1][1])
        top, bottom = F(q[0][0] + q[0][1]), F(q[1][0] + q[1][1])

        def price(strategy, allowed, at_x, at_y):
            if not allowed or self.cell[at_x, at_y][0] == strategy:
                return F(3.40282347e+38)
            return self.of(strategy, at_x, at_y)

        vl, vr = price(tall, columns, x, y), price(tall, columns, x + half, y)
        ht, hb = price(wide, rows, x, y), price(wide, rows, x, y + half)
        whole = self.of(square, x, y)
        vertical, horizontal = F(min(vl, left) + min(vr, right)), F(min(ht, top) + min(hb, bottom))
        if whole < vertical and whole < horizontal:
            self.place(square, x, y, whole)
        elif vertical < horizontal:
            if vl < left:
                self.place(tall, x, y, vl)
            if vr < right:
                self.place(tall, x + half, y, vr)
        else:
            if ht < top:
                self.place(wide, x, y, ht)
            if hb < bottom:
                self.place(wide, x, y + half, hb)

    def search(self, step):
        w, h = self.w, self.h
        for strategy, priority in ((6, 2), (7, 2), (11, 4), (10, 4)):
            cw, ch = STRATEGY_COVERED[strategy]
            for y in range(0, h - ch + 1, ch):
                for x in range(0, w - cw + 1, cw):
                    n = 4 if priority == 4 else 2
                    fits = y + n <= h and x + n <= w
                    if fits and strategy in (7, 11) and y % n == 0 and x % n == 0:
                        self.divide(n, x, y)
                    elif not fits and (y if strategy in (7, 11) else x) % n == 0:
                        self.try_merge(strategy, x, y, priority)
        for y in range(h - 1):
            for x in range(w - 1):
                if (y | x) % 2 != 0:
                    self.divide(2, x, y)
        for y in range(0, h - 3, step):
            for x in range(0, w - 3, step):
                if (y | x) % 4 != 0:
                    self.divide(4, x, y)
        return {at: s << 1 | anchor for at, (s, anchor) in self.cell.items()}


def opsin_planes(rng, bx, by):
    """Smooth content with textured and flat patches."""
    y, x = np.mgrid[0:by * 8, 0:bx * 8]
    busy = np.kron(rng.random((by, bx)) < 0.3 * (np.arange(bx) // 6 % 3), np.ones((8, 8)))
    noise = rng.normal(0, 1, (3, by * 8, bx * 8)) * busy * [[[0.004]], [[0.06]], [[0.05]]]
    base = np.stack([0.01 * np.sin(x / 7), 0.4 + 0.2 * np.cos(y / 11 + x / 29), 0.35 + x * 1e-3])
    return (base + noise).astype(F)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bx,by", [(1, 1), (2, 1), (1, 2), (3, 5), (7, 6), (6, 7), (5, 7), (7, 4),
                                   (4, 5), (8, 8), (9, 13), (20, 6), (24, 18)])
def test_strategy_merge(cuda, bx, by, dense):
    rng = np.random.default_rng(100 * bx + by)
    tx, ty = (bx + 7) // 8, (by + 7) // 8
    used = set()
    for target in (0.5, 2.0, 8.0):
        costs = zeros((7, by, bx))
        cells = torch.zeros((by, bx), dtype=torch.uint8, device="cuda")
        field = to_device((rng.random((by, bx)) * 0.3 / target + 0.3).astype(F))
        mask = to_device((rng.random((by * 8, bx * 8)) + 0.5).astype(F))
        maps = [to_device(rng.integers(-8, 9, (ty, tx)).astype(np.int8)) for _ in range(2)]
        stages.ac_strategy_search(to_device(opsin_planes(rng, bx, by)), field, mask, *maps, costs,
                                  cells, target=target, dense=dense)
        costs, cells = host(costs), host(cells)
        multiplier = F(1) + F(-0.4) / (F(target) + F(1.4))
        want = np.zeros_like(cells)
        for y0 in range(0, by, 8):
            for x0 in range(0, bx, 8):
                w, h = min(8, bx - x0), min(8, by - y0)
                tile = Tile(costs[:, y0:y0 + h, x0:x0 + w], w, h, multiplier)
                for (x, y), cell in tile.search(1 if dense else 2).items():
                    want[y0 + y, x0 + x] = cell
        assert np.array_equal(cells, want)
        used |= set((cells >> 1).ravel().tolist())
    if bx == 24:
        assert len(used) >= 6, used  # the content takes most strategies


def sum_in_order(terms):
    return np.add.accumulate(np.concatenate([[F(0)], terms]).astype(F), dtype=F)[-1]


def fma(a, b, c):
    return (a.astype(np.longdouble) * np.longdouble(b) + c.astype(np.longdouble)).astype(F)


def cfl_multiplier(a, b):
    """a, b: a tile's (luma / 84, base * luma - chroma) in element order."""
    x, n = F(0), F(a.size)
    for _ in range(20):
        center = fma(a, x, b)
        scale = np.where(np.abs(center) >= 100, F(0), F(2.0 / 3.0) * a)
        sums = []
        for at in (x, F(x + F(100)), F(x - F(100))):
            r = fma(a, at, b)
            d = scale * (np.abs(r) + F(1))
            d = np.where(r < 0, -d, d)
            lane = [sum_in_order(d[s::4]) for s in range(4)]
            sums.append(F(F(lane[0] + lane[1]) + F(lane[2] + lane[3])))
        regular = [F(F(F(2) * F(1e-9) * n) * at) for at in (x, F(x + F(100)), F(x - F(100)))]
        center, plus, minus = (F(r + s) for r, s in zip(regular, sums))
        step = F(center / F(F(F(plus - minus) / F(200)) + F(0.85)))
        x = F(x - np.clip(step, F(-20), F(20)))
        if abs(step) < F(3e-3):
            break
    x = x - F(2.6) if x >= F(2.6) else x + F(2.6) if x <= F(-2.6) else F(0)
    return int(np.clip(np.copysign(np.floor(abs(x) + F(0.5)), x), -128, 127))


@pytest.mark.parametrize("bx,by", [(1, 1), (1, 2), (2, 3), (5, 1), (3, 8), (8, 8), (9, 10), (19, 5)])
def test_initial_cfl(cuda, bx, by):
    """Tiles of one block (half a chunk of terms) up to 64 (32 chunks)."""
    rng = np.random.default_rng(10 * bx + by)
    planes = opsin_planes(rng, bx, by)
    texture = rng.normal(0, 0.05, planes.shape[1:])
    planes[1] += texture
    planes[0] += 0.03 * texture
    planes[2] += 1.2 * texture + rng.normal(0, 0.02, texture.shape)
    planes = planes.astype(F)
    tx, ty = (bx + 7) // 8, (by + 7) // 8
    maps = [torch.zeros((ty, tx), dtype=torch.int8, device="cuda") for _ in range(2)]
    stages.initial_cfl(to_device(planes), *maps)
    basis = committed_tables()["Forward8"].reshape(8, 8)
    inverse = []
    for c in (0, 2):
        dq, inv = np.zeros(64, F), np.zeros(64, F)
        _lib.call("gjxl_b200_quant_matrix", 0, c, dq.ctypes.data, inv.ctypes.data, 64)
        inverse.append(inv)
    blocks = planes.reshape(3, by, 8, bx, 8).transpose(0, 1, 3, 2, 4).astype(np.float64)
    rows, coef = np.zeros(blocks.shape), np.zeros(blocks.shape)
    for x in range(8):
        rows = rows + blocks[..., x:x + 1] * basis[:, x]
    for y in range(8):
        coef = coef + basis[:, y][:, None] * rows[..., y:y + 1, :]
    # Storage index u * 8 + v; the lowest frequency is left out.
    coef = coef.astype(F).swapaxes(-1, -2).reshape(3, by, bx, 64)
    coef[..., 0] = 0
    for k, (c, base) in enumerate(((0, F(0)), (2, F(1)))):
        luma, chroma = coef[1] * inverse[k], coef[c] * inverse[k]
        a, b = luma / F(84), base * luma - chroma
        want = np.array([[cfl_multiplier(a[y:y + 8, x:x + 8].ravel(), b[y:y + 8, x:x + 8].ravel())
                          for x in range(0, bx, 8)] for y in range(0, by, 8)])
        got = host(maps[k])
        assert np.array_equal(got, want), (got, want)
    if bx * by >= 64:
        assert host(maps[1]).any()  # the content gives the map something to say


ORDER_FAMILY = {0: 0, 4: 2, 5: 3, 6: 4, 7: 4, 10: 6, 11: 6}
FAMILY = {0: (0, 64, 1), 2: (64, 256, 4), 3: (320, 1024, 16), 4: (1344, 128, 2), 6: (1472, 512, 8)}


def random_cells(rng, bx, by, strategies):
    cells = np.zeros((by, bx), np.uint8)
    filled = np.zeros((by, bx), bool)
    for y in range(by):
        for x in range(bx):
            if filled[y, x]:
                continue
            fits = []
            for s in strategies:
                cw, ch = STRATEGY_COVERED[s]
                if (x % 32 + cw <= 32 and y % 32 + ch <= 32 and x + cw <= bx and y + ch <= by and
                        not filled[y:y + ch, x:x + cw].any()):
                    fits.append(s)
            s = int(rng.choice(fits))
            cw, ch = STRATEGY_COVERED[s]
            filled[y:y + ch, x:x + cw] = True
            cells[y:y + ch, x:x + cw] = s << 1
            cells[y, x] |= 1
    return cells


@pytest.mark.parametrize("bx,by,strategies", [
    (5, 1, [0]), (3, 4, list(STRATEGY_COVERED)), (33, 9, list(STRATEGY_COVERED)),
    (64, 35, list(STRATEGY_COVERED)), (40, 33, [0, 5]), (6, 31, [0, 6, 7])])
def test_coefficient_orders(cuda, bx, by, strategies):
    rng = np.random.default_rng(bx + by)
    cells = random_cells(rng, bx, by, strategies)
    qac = rng.integers(-2, 3, (3, by * 8, bx * 8)).astype(np.int32)
    qac *= rng.random(qac.shape) < 0.5
    raw = torch.full((by, bx), 5, dtype=torch.int32, device="cuda")
    context_map = stages.BlockContextMap.make((), bytes(3 * 13), 1)
    tokens = stages.AcTokens(bx, by)
    runs = [tokens.tokenize(to_device(cells), raw, to_device(qac), context_map, mode)
            for mode in (0, 1)]
    natural, got = (host(r["orders"]).view(np.uint32) for r in runs)
    counts = np.zeros((3, 1984), np.uint32)
    present = 0
    for y, x in np.argwhere(cells & 1):
        strategy = int(cells[y, x]) >> 1
        cw, ch = STRATEGY_COVERED[strategy]
        start, n, _ = FAMILY[ORDER_FAMILY[strategy]]
        present |= 1 << ORDER_FAMILY[strategy]
        block = qac[:, y * 8:(y + ch) * 8, x * 8:(x + cw) * 8].reshape(3, -1)
        counts[:, start:start + n] += block == 0
    assert np.array_equal(host(runs[1]["order_population"]).view(np.uint32)[:5952], counts.ravel())
    used = 0
    for family, (start, n, llf) in FAMILY.items():
        custom = natural[family, :, :n].copy()
        if present >> family & 1 and (bx >= 5 or by >= 5):
            for c in range(3):
                keys = (counts[c, start + custom[c]].astype(F) * (F(1) / np.sqrt(F(n))) +
                        F(0.1)).astype(np.uint64)
                custom[c, llf:] = custom[c, llf:][np.argsort(keys[llf:], kind="stable")]
        if (custom != natural[family, :, :n]).any():
            used |= 1 << family
        assert np.array_equal(got[family, :, :n], custom), family
    assert host(runs[1]["masks"]).view(np.uint32).tolist() == [present, used]
    tokens.close()
