"""The 8x8 HEVC transform kernels (csrc/hevc.cu) against the same integer
arithmetic in NumPy (matrix, rounding, int16 saturation of both passes,
quantiser and dequantiser): batches around a warp's four blocks and a CTA's 32,
zero blocks, saturating extremes, every rounding class. All results are equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D = np.array([[64] * 8, [89, 75, 50, 18, -18, -50, -75, -89], [83, 36, -36, -83, -83, -36, 36, 83],
              [75, -18, -89, -50, 50, 89, 18, -75], [64, -64, -64, 64, 64, -64, -64, 64],
              [50, -89, 18, 75, -75, -18, 89, -50], [36, -83, 83, -36, -36, 83, -83, 36],
              [18, -50, 75, -89, 89, -75, 50, -18]], np.int64)
LS = [40, 45, 51, 57, 64, 72]


def _sat(x):
    return np.clip(x, -32768, 32767)


def _forward(x, qp, bits, round_q12):
    s1 = bits - 6
    t = _sat((D @ x + (1 << (s1 - 1))) >> s1)
    c = _sat((t @ D.T + 256) >> 9)
    d, p = LS[qp % 6], qp // 6 + 4
    mag = ((np.abs(c) << (bits - 2)) + ((d << p) * round_q12) // 12) >> p
    level = np.minimum(mag // d, 32767)
    level = np.where(c < 0, -level, level)
    return np.where((x == 0).all(axis=(1, 2), keepdims=True), 0, level)


def _inverse(c, qp, bits):
    a, bd = qp // 6 + 4, bits - 2
    prod = c * LS[qp % 6]
    d = _sat(prod << (a - bd) if a >= bd else (prod + (1 << (bd - a - 1))) >> (bd - a))
    g = _sat((D.T @ d + 64) >> 7)
    s2 = 20 - bits
    return _sat((g @ D + (1 << (s2 - 1))) >> s2)


@pytest.mark.parametrize("bits", [8, 10])
@pytest.mark.parametrize("n,qp,round_q12", [(1, 0, 0), (3, 51, 2), (4, 30, 4), (31, 22, 12), (33, 37, 6), (1000, 27, 4)])
def test_dct8(gpu, n, qp, round_q12, bits):
    import torch
    rs = np.random.Generator(np.random.PCG64(n * 7 + bits))
    top = (1 << bits) - 1
    x = rs.integers(-top, top + 1, (n, 8, 8))
    x[::5] = 0
    x[1::7] = rs.choice([-32768, 32767, 0], x[1::7].shape)
    L, st = gpu.lib(), None
    src = torch.from_numpy(x.astype(np.int16)).cuda()
    out = torch.full((n + 1, 8, 8), 99, dtype=torch.int16, device="cuda")
    assert L.b200enc_hevc_transform_quant_8x8(gpu._p(src), gpu._p(out), n, qp, bits, round_q12, st) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out[:n].cpu().numpy(), _forward(x, qp, bits, round_q12))
    assert (out[n] == 99).all()
    c = (rs.integers(-300, 301, (n, 8, 8)) * (rs.random((n, 8, 8)) < 0.3)).astype(np.int64)
    c[1::7] = rs.choice([-32768, 32767, 1000], c[1::7].shape)
    lev = torch.from_numpy(c.astype(np.int16)).cuda()
    assert L.b200enc_hevc_dequant_itransform_8x8(gpu._p(lev), gpu._p(out), n, qp, bits, st) == 0
    torch.cuda.synchronize()
    want = c * LS[qp % 6]
    a, bd = qp // 6 + 4, bits - 2
    if a < bd or np.abs(want).max() << (a - bd) < 1 << 31:  # the kernel's product is 32-bit, as the reference's
        np.testing.assert_array_equal(out[:n].cpu().numpy(), _inverse(c, qp, bits))
    else:
        ok = (np.abs(want) << (a - bd) < 1 << 31).all(axis=(1, 2))
        np.testing.assert_array_equal(out[:n].cpu().numpy()[ok], _inverse(c, qp, bits)[ok])
    assert (out[n] == 99).all()
