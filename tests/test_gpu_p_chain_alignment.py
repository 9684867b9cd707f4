"""The fused P chain (csrc/pframe.cu) against the CPU oracle where its word and
vector accesses give way to bytes: source and reference pitches of every
alignment, widths with every remainder of a four-sample word, vectors at every
quarter sample and far outside the picture, extreme residuals and quantizers.
All outputs are whole numbers and equal.
"""
import numpy as np
import pytest

from test_gpu_parity import _cmp_out, _host_rec, _pad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,cpad,rpad,coded,qp", [(16, 16, 0, 0, True, 0), (18, 18, 1, 2, False, 51), (34, 20, 2, 6, True, 24),
                                                    (46, 34, 3, 14, False, 3), (62, 50, 4, 16, True, 37),
                                                    (96, 32, 8, 0, False, 12)])
def test_p_chain_alignment(gpu, oracle_mod, W, H, cpad, rpad, coded, qp):
    import torch
    rs = np.random.Generator(np.random.PCG64(W + qp))
    CW, CH = gpu.coded(W, H)
    RW, RH = (CW, CH) if coded else (W, H)

    def frame():  # extremes and noise: the residual reaches +-255
        y = np.where(rs.random((H, W)) < 0.5, rs.choice([0, 255], (H, W)), rs.integers(0, 256, (H, W))).astype(np.uint8)
        return y, rs.integers(0, 256, (H // 2, W)).astype(np.uint8)

    (y0, uv0), (y1, uv1) = frame(), frame()
    ry, ruv = _pad(y0, uv0, CW, CH)
    ref = gpu.NV12.from_host(np.ascontiguousarray(ry), np.ascontiguousarray(ruv), pitch=CW + rpad)
    cur = gpu.NV12.from_host(y1, uv1, pitch=W + cpad)
    mbs = (CW // 16) * (CH // 16)
    mvh = np.zeros((mbs, 4), np.int32)
    mvh[:, :2] = np.where(rs.random((mbs, 2)) < 0.2, rs.integers(-400, 401, (mbs, 2)), rs.integers(-70, 71, (mbs, 2)))
    out, rec = gpu.Outputs(W, H), gpu.NV12(W, H)
    gpu.p_frame(cur, ref, W, H, RW, RH, qp, torch.from_numpy(mvh).cuda(), out, rec)
    torch.cuda.synchronize()
    rec_y, rec_uv = np.zeros((CH, CW), np.uint8), np.zeros((CH // 2, CW), np.uint8)
    want = oracle_mod.p_frame(oracle_mod.frame(W, H, qp, coded_clamp=coded), np.ascontiguousarray(y1),
                              np.ascontiguousarray(uv1), ry, ruv, mvh, rec_y, rec_uv)
    _cmp_out(out.host(), want, f"P {W}x{H} qp{qp}", check_mv=False)
    gy, guv = _host_rec(rec, CW, CH)
    np.testing.assert_array_equal(gy[:RH, :RW], rec_y[:RH, :RW])
    np.testing.assert_array_equal(guv[:RH // 2, :RW], rec_uv[:RH // 2, :RW])
