"""Uploads from page-locked host memory whose rows lie apart (csrc/upload.cu):
every alignment of the source, widths around the kernel's 16-byte units and
512-byte segments, source pitches of its own. The surface holds the frame's
bytes, and its bytes beyond the frame keep theirs.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,pad,off", [(2, 2, 0, 0), (16, 16, 1, 3), (30, 18, 0, 5), (176, 144, 0, 0), (498, 20, 3, 15),
                                         (512, 34, 16, 8), (514, 6, 0, 1), (1022, 50, 7, 2), (1040, 10, 0, 12)])
def test_upload_rows(gpu, W, H, pad, off):
    import torch
    rs = np.random.Generator(np.random.PCG64(W + off))
    P, W2, H2 = W + pad, W + 18, H + 4
    n = P * (H + H // 2)
    pinned = torch.zeros(n + 32, dtype=torch.uint8).pin_memory()
    host = pinned.numpy()
    host[:] = rs.integers(0, 256, n + 32, dtype=np.uint8)
    ctx = gpu.Context()
    img, mem = ctx.create_image(W2, H2)
    before_y, before_uv = rs.integers(0, 256, (H2, W2), dtype=np.uint8), rs.integers(0, 256, (H2 // 2, W2), dtype=np.uint8)
    ctx.upload(img, mem, before_y, before_uv)
    c = ctypes.byref(ctx.ctx)
    base = pinned.data_ptr() + off
    assert ctx.L.gpu_compute_upload_nv12(c, ctypes.byref(img), mem, ctypes.c_void_p(base), P,
                                         ctypes.c_void_p(base + P * H), P, W, H) == 0
    got_y, got_uv = np.zeros((H2, W2), np.uint8), np.zeros((H2 // 2, W2), np.uint8)
    assert ctx.L.gpu_compute_download_nv12(c, ctypes.byref(img), mem, ctypes.c_void_p(got_y.ctypes.data), W2,
                                           ctypes.c_void_p(got_uv.ctypes.data), W2, W2, H2) == 0
    want = host[off:off + n].reshape(-1, P)[:, :W]
    before_y[:H, :W] = want[:H]
    before_uv[:H // 2, :W] = want[H:]
    np.testing.assert_array_equal(got_y, before_y)
    np.testing.assert_array_equal(got_uv, before_uv)
