"""The HEVC search planes (csrc/hevc.cu) against the eight-tap filters in NumPy,
at the edges of the kernel's 128x32 tiles and four-sample units: pictures of one
sample and up, every remainder of the width, unaligned pitches and margins.
All samples are whole numbers and equal; nothing outside the planes is written.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TAPS = np.array([-1, 4, -11, 40, 40, -11, 4, -1])


def _planes(ref, M, top):
    h, w = ref.shape
    y, x = np.arange(-M - 3, h + M + 4), np.arange(-M - 3, w + M + 4)
    e = ref[np.clip(y, 0, h - 1)][:, np.clip(x, 0, w - 1)].astype(np.int64)
    rows, cols = h + 2 * M, w + 2 * M
    t = sum(TAPS[k] * e[:, k:k + cols] for k in range(8))
    v = sum(TAPS[k] * e[k:k + rows, 3:3 + cols] for k in range(8))
    hv = sum(TAPS[k] * t[k:k + rows] for k in range(8))
    return [e[3:3 + rows, 3:3 + cols], np.clip((t[3:3 + rows] + 32) >> 6, 0, top), np.clip((v + 32) >> 6, 0, top),
            np.clip((hv + 2048) >> 12, 0, top)]


@pytest.mark.parametrize("bits", [8, 10])
@pytest.mark.parametrize("w,h,M,rpad,ppad", [(1, 1, 0, 0, 0), (2, 3, 10, 1, 3), (97, 33, 16, 2, 2), (96, 31, 16, 0, 0),
                                              (131, 65, 5, 1, 1), (258, 70, 16, 3, 2), (94, 40, 17, 2, 4)])
def test_planes(gpu, w, h, M, rpad, ppad, bits):
    import torch
    rs = np.random.Generator(np.random.PCG64(w * 31 + bits))
    top, dt, view = (255, np.uint8, np.uint8) if bits == 8 else (1023, np.uint16, np.int16)
    ref = np.full((h, w + rpad), top, dt)
    ref[:, :w] = np.where(rs.random((h, w)) < 0.3, rs.choice([0, top], (h, w)), rs.integers(0, top + 1, (h, w)))
    rows, cols = h + 2 * M, w + 2 * M
    planes = torch.full((4, rows, cols + ppad), 7, dtype=torch.uint8 if bits == 8 else torch.int16, device="cuda")
    gpu.hevc_build_hpel(torch.from_numpy(ref.view(view)).cuda(), w, h, M, planes)
    torch.cuda.synchronize()
    got = planes.cpu().numpy().astype(np.int64)
    for k, want in enumerate(_planes(ref[:, :w], M, top)):
        np.testing.assert_array_equal(got[k, :, :cols], want, err_msg="I H V HV".split()[k])
    assert (got[:, :, cols:] == 7).all()
