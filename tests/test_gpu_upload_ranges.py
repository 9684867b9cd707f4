"""Which host memory the row upload may read (csrc/upload.cu): only a range that lies
in one page-locked object from its first to its last byte. The decision alone is
checked for ranges that do not (nothing is launched on them), the upload for planes
registered apart and for surfaces it has to refuse.
"""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Range(ctypes.Structure):
    _fields_ = [("locked", ctypes.c_bool), ("dev", ctypes.c_void_p)]


def _pages(n):
    raw = np.zeros(n + 4096, np.uint8)
    off = -raw.ctypes.data % 4096
    return raw[off:off + n]


def _pin(gpu, a, lo, hi):
    assert gpu.lib().b200enc_pin_host(ctypes.c_void_p(a.ctypes.data + lo), ctypes.c_size_t(hi - lo)) == 0


def _unpin(gpu, a, lo):
    assert gpu.lib().b200enc_unpin_host(ctypes.c_void_p(a.ctypes.data + lo)) == 0


def test_range_decision(gpu):
    import torch
    torch.zeros(1, device="cuda")
    fn = gpu.lib().b200enc_host_range
    fn.restype, fn.argtypes = _Range, [ctypes.c_void_p, ctypes.c_size_t]
    a = _pages(16 * 4096)
    base = a.ctypes.data
    _pin(gpu, a, 100, 20000)
    _pin(gpu, a, 8 * 4096, 9 * 4096)

    def at(lo, hi):
        r = fn(base + lo, hi - lo)
        return r.locked, r.dev == base + lo if r.dev else None

    try:
        assert at(100, 20000) == (True, True)
        assert at(5000, 5001) == (True, True)
        assert at(100, 20001) == (True, None)  # a byte too many
        assert at(19999, 20002) == (True, None)
        assert at(5000, 8 * 4096 + 10) == (True, None)  # ends in another registration, a hole between
        assert at(8 * 4096, 9 * 4096) == (True, True)
        assert at(8 * 4096, 9 * 4096 + 1) == (True, None)
        assert at(0, 200) == (False, None)  # begins before it
        assert at(12 * 4096, 13 * 4096) == (False, None)  # pageable
    finally:
        _unpin(gpu, a, 100)
        _unpin(gpu, a, 8 * 4096)
    assert at(100, 20000) == (False, None)
    d = torch.zeros(64, dtype=torch.uint8, device="cuda")
    r = fn(d.data_ptr(), 64)
    assert not r.locked and not r.dev


def test_planes_registered_apart(gpu):
    W, H, P = 178, 146, 192
    rs = np.random.Generator(np.random.PCG64(9))
    a = _pages(24 * 4096)
    a[:] = rs.integers(0, 256, a.size, dtype=np.uint8)
    uv_at = 12 * 4096
    y_bytes, uv_bytes = (H - 1) * P + W, (H // 2 - 1) * P + W
    _pin(gpu, a, 0, y_bytes)
    _pin(gpu, a, uv_at, uv_at + uv_bytes)
    try:
        ctx = gpu.Context()
        img, mem = ctx.create_image(W, H)
        c, vp = ctypes.byref(ctx.ctx), ctypes.c_void_p
        assert ctx.L.gpu_compute_upload_nv12(c, ctypes.byref(img), mem, vp(a.ctypes.data), P,
                                             vp(a.ctypes.data + uv_at), P, W, H) == 0
        y, uv = np.zeros((H, W), np.uint8), np.zeros((H // 2, W), np.uint8)
        assert ctx.L.gpu_compute_download_nv12(c, ctypes.byref(img), mem, vp(y.ctypes.data), W, vp(uv.ctypes.data), W,
                                               W, H) == 0
        np.testing.assert_array_equal(y, np.lib.stride_tricks.as_strided(a, (H, W), (P, 1)))
        np.testing.assert_array_equal(uv, np.lib.stride_tricks.as_strided(a[uv_at:], (H // 2, W), (P, 1)))
        # a surface without a chroma plane, or with rows that overlap: refused, nothing read or written
        bad = type(img).from_buffer_copy(img)
        bad.uv_plane = None
        assert ctx.L.gpu_compute_upload_nv12(c, ctypes.byref(bad), mem, vp(a.ctypes.data), P,
                                             vp(a.ctypes.data + uv_at), P, W, H) != 0
        bad = type(img).from_buffer_copy(img)
        bad.pitch = W - 2
        assert ctx.L.gpu_compute_upload_nv12(c, ctypes.byref(bad), mem, vp(a.ctypes.data), P,
                                             vp(a.ctypes.data + uv_at), P, W, H) != 0
        # and the refusal is not the next upload's, here or in a thread that has made no call yet
        for where in ("here", "thread"):
            rc = []
            up = lambda: rc.append(ctx.L.gpu_compute_upload_nv12(  # noqa: E731
                c, ctypes.byref(img), mem, vp(a.ctypes.data), P, vp(a.ctypes.data + uv_at), P, W, H))
            a[:y_bytes] ^= 0x55
            if where == "thread":
                t = threading.Thread(target=up)
                t.start()
                t.join()
            else:
                up()
            assert rc == [0]
            assert ctx.L.gpu_compute_download_nv12(c, ctypes.byref(img), mem, vp(y.ctypes.data), W,
                                                   vp(uv.ctypes.data), W, W, H) == 0
            np.testing.assert_array_equal(y, np.lib.stride_tricks.as_strided(a, (H, W), (P, 1)))
    finally:
        _unpin(gpu, a, 0)
        _unpin(gpu, a, uv_at)
