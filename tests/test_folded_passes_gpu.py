"""The folded inverse passes' pixels (csrc/line_dct.cuh) against the sequential
double sums in NumPy, bit for bit: random planes, planes of very small, very
large and non-finite values, and planes whose coefficients cancel at a pixel
until the sums' rounding errors decide its float - around zero, where the
folded sum gives another float and only the columns transformed again are
right, and around a tie between two floats."""

import ctypes

import numpy as np
import pytest
import torch

from tests.gpu_util import host, to_device
from tests.native_util import load
from tests.test_dct_basis_cpu import committed_tables

pytestmark = pytest.mark.gpu
F = np.float32
SIZES = [(8, 8), (16, 8), (8, 16), (16, 16), (32, 16), (16, 32), (32, 32)]


@pytest.fixture(scope="module")
def native(cuda, tmp_path_factory):
    return load("folded_passes", tmp_path_factory.mktemp("native"))


def lines(x, basis):
    """out[..., k] = sum_s x[..., s] * basis[s][k] in order, each rounded."""
    acc = np.zeros(x.shape[:-1] + (basis.shape[1],))
    for s in range(basis.shape[0]):
        acc = acc + x[..., s:s + 1] * basis[s]
    return acc


def sequential(planes, iw, ih):
    rows = lines(planes.astype(np.float64), iw)
    return lines(rows.swapaxes(-1, -2), ih).swapaxes(-1, -2).astype(F)


def cancel(rng, plane, iw, ih, at, target):
    """Sets four coefficients of `plane`, one after the other, so that the
    pixel `at` comes ever closer to `target`: each is the float that makes up
    the rest, so that the rest shrinks by about 2^-24 a time."""
    h, w = plane.shape
    weight = np.outer(ih[:, at[0]], iw[:, at[1]])
    free = [tuple(i) for i in np.argwhere(np.abs(weight) > 0.3)]
    chosen = [free[i] for i in rng.permutation(len(free))[:4]]
    for i in chosen:
        plane[i] = 0
    for i in chosen:
        rest = target - float((plane.astype(np.longdouble) * weight).sum())
        plane[i] = F(rest / weight[i])


def run(native, w, h, planes):
    per_batch = 3072 // (w * h)
    count = planes.shape[0]
    assert count % per_batch == 0
    d_in = to_device(planes)
    folded, pixels = torch.empty_like(d_in), torch.empty_like(d_in)
    listed = torch.zeros(count // per_batch, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    status = native.folded_passes(w, h, ctypes.c_void_p(d_in.data_ptr()), count // per_batch,
                                  ctypes.c_void_p(folded.data_ptr()),
                                  ctypes.c_void_p(pixels.data_ptr()),
                                  ctypes.c_void_p(listed.data_ptr()))
    assert status == 0
    return host(folded), host(pixels), host(listed)


def same_floats(a, b):
    """Equal bits; any NaN equals any other."""
    return (a.view(np.int32) == b.view(np.int32)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("kind", ["random", "sparse", "spread", "tiny", "huge", "non-finite",
                                  "zero", "around zero", "around a tie"])
def test_pixels_are_the_sequential_sums(native, w, h, kind):
    rng = np.random.default_rng(100 * w + h)
    tables = committed_tables()
    iw, ih = tables[f"Inverse{w}"].reshape(w, w), tables[f"Inverse{h}"].reshape(h, h)
    count = 2 * 3072 // (w * h)
    planes = rng.normal(0, 1, (count, h, w)).astype(F)
    if kind == "sparse":
        planes *= rng.random((count, h, w)) < 0.1
    elif kind == "spread":
        planes *= np.exp2(rng.integers(-30, 30, planes.shape)).astype(F)
    elif kind == "tiny":
        planes *= F(1e-38)
    elif kind == "huge":
        planes *= F(1e34)
    elif kind == "non-finite":
        planes[::2, h - 1, 3] = F(np.inf)
        planes[1::2, 0, 0] = F(np.nan)
    elif kind == "zero":
        planes[:] = 0
    elif kind.startswith("around"):
        for plane in planes:
            at = (int(rng.integers(h)), int(rng.integers(w)))
            target = 0.0
            if kind == "around a tie":
                f = F(rng.uniform(0.5, 1.0) * 2.0 ** -rng.integers(0, 8))
                target = 0.5 * (float(f) + float(np.nextafter(f, F(2))))
            cancel(rng, plane, iw, ih, at, target)
    with np.errstate(all="ignore"):
        want = sequential(planes, iw, ih)
    folded, pixels, listed = run(native, w, h, planes)
    assert same_floats(pixels, want).all()
    # Without a float that only the second transform gets right, the planes
    # around zero would test nothing.
    if kind == "around zero":
        assert not same_floats(folded, want).all()
    if kind == "zero":
        assert listed.sum() == 0
    if kind in ("tiny", "huge", "non-finite", "around zero"):
        assert listed.sum() > 0
