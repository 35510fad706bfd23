"""The quantizer's median and median absolute deviation at the field sizes
where the selection's cluster grows (4096, 8192 and 16384 values) and just past
them, from the session's published field: the global scale of
CreateQuantizerFromField (src/codec/quantizer.cpp)."""

import numpy as np
import pytest
import torch

from gjxl_b200.session import AnalysisSession
from gjxl_b200.synthetic import generate_srgb8

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("w,h", [(8, 8), (250, 9), (512, 512), (520, 512), (1024, 512),
                                 (1032, 512), (1024, 1024), (1032, 1024)])
def test_quantizer_from_the_final_field(cuda, w, h):
    s = AnalysisSession(w, h, butteraugli_target=1.0, effort=5)
    s.analyze_host(generate_srgb8(w, h, 40 + w, sensor_noise=True),
                   torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = s.host_results()
    field = got["final_quant"].astype(F).ravel()
    n = field.size
    median = np.sort(field)[n // 2]
    mad = np.sort(np.abs(field - median))[n // 2]
    scale = int(np.clip(F(65536) * (median - mad) / F(5), F(1), F(32768)))
    assert int(got["quantizer_params"][0]) == scale
    s.close()


# 640 x 640 = 409600 blocks are the most that the cluster's shared memory holds;
# above, the selections run as grid-wide kernels.
@pytest.mark.parametrize("w,h", [(5120, 5120), (5128, 5120)])
def test_quantizer_around_the_largest_cluster_field(cuda, w, h):
    tile = generate_srgb8(640, 512, 77, sensor_noise=True)
    img = np.tile(tile, (h // 512, -(-w // 640), 1))[:, :w].copy()
    # Each tile darker than the last, so that the field does not repeat.
    img[::2] //= np.linspace(1, 4, w).astype(np.uint8)[None, :, None]
    s = AnalysisSession(w, h, butteraugli_target=1.0, effort=5)
    s.analyze_host(img, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert s.host_error() == 0
    got = s.host_results()
    field = got["final_quant"].astype(F).ravel()
    assert field.size == (w // 8) * (h // 8)
    median = np.sort(field)[field.size // 2]
    mad = np.sort(np.abs(field - median))[field.size // 2]
    scale = int(np.clip(F(65536) * (median - mad) / F(5), F(1), F(32768)))
    assert int(got["quantizer_params"][0]) == scale
    s.close()
