"""The full search with several threads per column (csrc/me.cu), which frames of
few macroblocks take, and with one, on either side of the line between them (8
macroblocks per SM at +-16, 16 at +-32): vectors and costs equal the CPU oracle's.
"""
import numpy as np
import pytest

from test_gpu_parity import _frames, _pad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,W,H", [(16, 16, 16), (16, 96, 80), (16, 592, 512), (16, 608, 512), (32, 16, 32), (32, 208, 160),
                                   (32, 592, 1024), (32, 608, 1024)])
@pytest.mark.parametrize("noise", [False, True])
def test_wide_search(gpu, oracle_mod, R, W, H, noise):
    import torch
    if noise:
        rs = np.random.Generator(np.random.PCG64(W + R))
        (y0, uv0), (y1, uv1) = [(rs.integers(0, 256, (H, W), dtype=np.uint8), np.zeros((H // 2, W), np.uint8)) for _ in range(2)]
    else:
        (y0, uv0), (y1, uv1) = _frames(W, H, 2, seed=W + R, pan=True, noise_patch=True)
    mv = torch.zeros(((W // 16) * (H // 16), 4), dtype=torch.int32, device="cuda")
    gpu.me_full_search(gpu.NV12.from_host(y1, uv1), gpu.NV12.from_host(y0, uv0), W, H, W, H, R, 5, 512, mv)
    torch.cuda.synchronize()
    ry, _ = _pad(y0, uv0, W, H)
    want = oracle_mod.me_frame(oracle_mod.frame(W, H, 26, coded_clamp=True), np.ascontiguousarray(y1),
                               np.ascontiguousarray(ry), R, 5, 512)
    np.testing.assert_array_equal(mv.cpu().numpy(), want)
