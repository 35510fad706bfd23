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
