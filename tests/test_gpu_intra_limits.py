"""The intra wavefront with reconstruction limits (RW, RH) that end macroblocks
before the picture does (csrc/intra.cu): nothing outside the limits is written, in
particular not the bottom lines that one group of rows hands to the next, and the
macroblocks inside the limits are those of the whole picture. The sizes put the
limits before, at and behind a group's last row, and whole macroblocks outside.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,RW,RH", [(96, 112, 96, 50), (96, 112, 70, 112), (96, 192, 66, 62), (96, 192, 34, 130),
                                       (600, 160, 40, 20), (96, 112, 96, 112)])
@pytest.mark.parametrize("ctas", [0, 1])
def test_nothing_outside_the_limits(gpu, W, H, RW, RH, ctas):
    import torch
    rs = np.random.Generator(np.random.PCG64(W + H + RW + RH))
    base = rs.integers(40, 216, (H // 8 + 1, W // 8 + 1)).astype(np.float64)
    y = np.clip(np.kron(base, np.ones((8, 8)))[:H, :W] + rs.normal(0, 8, (H, W)), 0, 255).astype(np.uint8)
    uv = np.clip(128 + rs.normal(0, 30, (H // 2, W)), 0, 255).astype(np.uint8)
    cur = gpu.NV12.from_host(y, uv)
    mbw, mbh = (W + 15) // 16, H // 16
    got = {}
    for name, rw, rh in (("whole", W, H), ("limited", RW, RH)):
        out, rec, scr = gpu.Outputs(W, H), gpu.NV12(W, H), gpu.scratch(mbh)
        rec.buf.fill_(0xA5)
        gpu.i_frame(cur, W, H, rw, rh, 28, 1, out, rec, scr, ctas=ctas)
        torch.cuda.synchronize()
        assert gpu.wavefront_status(scr) == 0
        got[name] = (out.host(), rec.y.cpu().numpy(), rec.uv.cpu().numpy())
    (wo, wy, wuv), (lo, ly, luv) = got["whole"], got["limited"]
    assert (ly[RH:] == 0xA5).all() and (ly[:, RW:] == 0xA5).all()
    assert (luv[RH // 2:] == 0xA5).all() and (luv[:, RW // 2 * 2:] == 0xA5).all()
    iw, ih = RW // 16, RH // 16  # macroblocks wholly inside
    np.testing.assert_array_equal(ly[:16 * ih, :16 * iw], wy[:16 * ih, :16 * iw])
    np.testing.assert_array_equal(luv[:8 * ih, :16 * iw], wuv[:8 * ih, :16 * iw])
    for k in ("levels", "dc", "nz", "pred_mode"):
        a, b = lo[k].reshape(mbh, mbw, -1), wo[k].reshape(mbh, mbw, -1)
        np.testing.assert_array_equal(a[:ih, :iw], b[:ih, :iw], err_msg=k)
