"""A distance map's pixel depends on the image within the blurs' reach only, so
that the map of a crop equals the crop of the map away from the crop's
borders, bit for bit, wherever the crop puts the pixel in the kernels' 32 x 32
tiles and 8-row runs (crops start at even pixels: one scale is halved)."""

import numpy as np
import pytest
import torch

from gjxl_b200.stages import Butteraugli
from tests.gpu_util import assert_bitexact, host, to_device, zeros

pytestmark = pytest.mark.gpu

# Reach of one pixel in its own scale: blurs of radius 16 + 7 + 3, one of 5
# taps, the mask's (radius 6) and the Malta lines (4); the half scale doubles
# it, and its resampling adds two.
REACH = 2 * (16 + 7 + 3 + 2 + 6 + 4 + 2)


def distance_map(r, d):
    _, h, w = r.shape
    b = Butteraugli(w, h)
    b.prepare(to_device(r))
    dmap, score, err = zeros((h, w)), zeros((1,), torch.float64), zeros((1,), torch.int32)
    b.compare(to_device(d), dmap, score, err)
    out = host(dmap)
    assert int(host(err)[0]) == 0
    b.close()
    return out


@pytest.mark.parametrize("x0,y0,w,h", [(0, 0, 321, 300), (2, 6, 317, 289), (30, 34, 290, 257),
                                       (64, 32, 255, 225), (18, 14, 256, 256)])
def test_map_of_a_crop_is_the_crop_of_the_map(cuda, x0, y0, w, h):
    rng = np.random.default_rng(7)
    y, x = np.mgrid[0:310, 0:340]
    base = 0.3 + 0.2 * np.sin(x / 11.0) * np.cos(y / 7.0) + 0.1 * rng.random((3, 310, 340))
    r = base.astype(np.float32)
    d = np.clip(base + rng.normal(0, 0.02, base.shape), 0, 1).astype(np.float32)
    whole = distance_map(r, d)
    part = distance_map(r[:, y0:y0 + h, x0:x0 + w], d[:, y0:y0 + h, x0:x0 + w])
    inner = np.s_[REACH:-REACH, REACH:-REACH]
    left, top = REACH * (x0 > 0), REACH * (y0 > 0)  # shared borders keep their pixels
    assert_bitexact(part[top:-REACH, left:-REACH],
                    whole[y0:y0 + h, x0:x0 + w][top:-REACH, left:-REACH], "crop")
    assert part[inner].size > 0 and part[inner].max() > 0
