"""HEVC deblocking (csrc/hevc_deblock.cu) reads and writes a vertical edge's line
as words where the luma plane's base and stride allow it, sample by sample
elsewhere: the same picture in planes of every alignment gives the same samples,
and nothing beyond the width changes.
"""
import numpy as np
import pytest

import hevc_db_inputs as hdi
from test_gpu_hevc_deblock import _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bit_depth", [8, 10])
@pytest.mark.parametrize("width,height", [(8, 8), (40, 24), (264, 136)])
def test_every_stride_gives_the_same_samples(gpu, width, height, bit_depth):
    case = hdi.make_case(21, width, height, bit_depth=bit_depth, log2_ctb=4, slices=2 if width > 8 else 1,
                         tiles=2 if width > 32 else 1, lossless=0.1, qp_range=(20, 51))
    results = []
    for pad in (0, 1, 2, 4, 8):
        planes = []
        for c, p in enumerate(case["planes"]):
            w = width >> (1 if c else 0)
            q = np.full((p.shape[0], (w + 7) // 8 * 8 + pad), 3, p.dtype)
            q[:, :w] = p[:, :w]
            planes.append(q)
        got = _run_gpu(gpu, dict(case, planes=planes, strides=[q.shape[1] for q in planes]))
        for c, g in enumerate(got):
            assert (g[:, width >> (1 if c else 0):] == 3).all()
        results.append([g[:, :width >> (1 if c else 0)] for c, g in enumerate(got)])
    if width > 8:
        assert any((r != p[:, :r.shape[1]]).any() for r, p in zip(results[0], case["planes"]))
    for r in results[1:]:
        for a, b in zip(r, results[0]):
            np.testing.assert_array_equal(a, b)
