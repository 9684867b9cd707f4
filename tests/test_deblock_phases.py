"""The tile deblocking's phases (csrc/deblock_tile.cuh), run on the CPU.

The kernel filters a tile in seven phases of independent lines; the same
functions, compiled for the host, must give the oracle's whole-picture
raster-order deblocking (clause 8.7) for every tile of a picture, whatever
order the lines of a phase run in: tiles from 1x1 to 16x8 macroblocks on
pictures they divide and pictures they do not, intra and inter, QPs whose
filters are off, weak and strong, 4x4 and 8x8 transforms. The margin samples
the tile may not depend on are filled with noise.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_deblock_tiles import _content

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include <cstring>
#include <vector>
#include "deblock_tile.cuh"
using namespace b200enc;
extern "C" int dt_sizes(int tw, int th, int* out) {
  out[0] = kDtTop + 16 * th + kDtBottom; out[1] = kDtTopC + 8 * th + kDtBottomC; out[2] = 16 * (tw + 1) + 4;
  return 0;
}
extern "C" unsigned dt_bs(int dir, int e, unsigned mq, unsigned mp, int mvd, int edge0, int intra, int t8) {
  return dt_strengths(dir, e, mq, mp, mvd, edge0, intra, t8);
}
extern "C" unsigned dt_t8(unsigned m) { return dt_mask_t8(m); }
extern "C" void dt_run(unsigned char* ly, unsigned char* cy, const unsigned char* bs, int TW, int TH, int L, int R, int T,
                       int B, const int* qv, int order) {
  std::vector<uint8_t> save((size_t)(TW + 2) * (TH + 2) * 64, 0xee);
  DbQ q; memcpy(&q, qv, sizeof(q));
  DtTile t{ly, cy, 16 * (TW + 1) + 4, bs, save.data(), TW + 2, TW, TH, L, R, T, B};
  for (int ph = 1; ph <= 7; ++ph) {
    const int n = dt_luma_lines(t, ph), m = dt_chroma_lines(t, ph);
    for (int i = 0; i < n; ++i) if (q.al && q.be) dt_luma_line(t, ph, order ? n - 1 - i : i, q);
    for (int i = 0; i < m; ++i) if (q.alc && q.bec) dt_chroma_line(t, ph, order ? m - 1 - i : i, q);
  }
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("dt")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "bc250-vaapi_b200", "csrc"),
                    "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    L = ctypes.CDLL(str(d / "shim.so"))
    L.dt_bs.restype = L.dt_t8.restype = ctypes.c_uint
    return L


def _tables():
    src = open(os.path.join(ROOT, "bc250-vaapi_b200", "csrc", "deblock.cu")).read()

    def table(name):
        body = src.split(name, 1)[1].split("= {", 1)[1].split("};", 1)[0]
        return [int(v) for v in body.replace("{", " ").replace("}", " ").replace(",", " ").split()]

    return table("kAlpha[52]"), table("kBeta[52]"), np.array(table("kTc0[52][3]")).reshape(52, 3)


def _chroma_qp(qp):
    return qp if qp < 30 else [29, 30, 31, 32, 32, 33, 34, 34, 35, 35, 36, 36, 37, 37, 37, 38, 38, 38, 39, 39, 39,
                               39][qp - 30]


def _strengths(shim, nz, mv, t8, mbw, mbh, intra):
    mask = ((nz[:, :16] & 0xFFFF) != 0) @ (1 << np.arange(16))
    mask = [shim.dt_t8(int(m)) if t8 is not None and t8[i] else int(m) for i, m in enumerate(mask)]
    bs = np.zeros((mbh, mbw, 8), np.uint32)
    for y in range(mbh):
        for x in range(mbw):
            i = y * mbw + x
            for d in range(2):
                nb = i - 1 if d == 0 else i - mbw
                inside = x > 0 if d == 0 else y > 0
                far = inside and bool((np.abs(mv[i, :2] - mv[nb, :2]) >= 4).any())
                for e in range(4):
                    bs[y, x, 4 * d + e] = shim.dt_bs(d, e, mask[i], mask[nb] if inside else 0, far, inside,
                                                     int(intra), int(t8 is not None and t8[i]))
    return bs.view(np.uint8).reshape(mbh, mbw, 32)


@pytest.mark.parametrize("mbw,mbh,tw,th", [(1, 1, 8, 8), (5, 4, 1, 1), (7, 5, 2, 3), (9, 7, 4, 4), (11, 6, 8, 2),
                                           (18, 9, 16, 8), (6, 10, 3, 8)])
@pytest.mark.parametrize("intra", [0, 1])
def test_phases_equal_raster_order(oracle_mod, shim, mbw, mbh, tw, th, intra):
    rs = np.random.Generator(np.random.PCG64(mbw * 100 + mbh * 10 + tw + intra))
    al, be, tc = _tables()
    for kind, qp in ((0, 27), (1, 38), (2, 33), (3, 51), (2, 20), (1, 10)):
        for use_t8 in (False, True):
            y, uv, nz, mv = _content(rs, mbw, mbh, kind)
            t8 = (rs.random(mbw * mbh) < 0.5).astype(np.uint8) if use_t8 else None
            wy, wuv = y.copy(), uv.copy()
            if use_t8:
                oracle_mod.deblock_t8(mbw, mbh, qp, intra, nz, t8, mv, wy, wuv)
            else:
                oracle_mod.deblock(mbw, mbh, qp, intra, nz, mv, wy, wuv)
            bs = _strengths(shim, nz, mv, t8, mbw, mbh, intra)
            qc = _chroma_qp(qp)
            qv = np.array([al[qp], be[qp], al[qc], be[qc], *tc[qp], *tc[qc], intra], np.int32)
            for x0 in range(0, mbw, tw):
                for y0 in range(0, mbh, th):
                    _tile(shim, rs, y, uv, bs, qv, mbw, mbh, x0, y0, min(tw, mbw - x0), min(th, mbh - y0), wy, wuv)


def _tile(shim, rs, y, uv, bs, qv, mbw, mbh, x0, y0, w, h, wy, wuv):
    rows, crows, sp = 10 + 16 * h + 7, 2 + 8 * h + 2, 16 * (w + 1) + 4
    Lm, R, T, B = int(x0 > 0), int(x0 + w < mbw), int(y0 > 0), int(y0 + h < mbh)
    ly = rs.integers(0, 256, (rows, sp)).astype(np.uint8)
    cy = rs.integers(0, 256, (crows, sp)).astype(np.uint8)
    # only the margin the kernel loads: 12 luma columns (8 chroma bytes) left, 4 right, 10 / 2 rows above, 7 / 2 below
    ra, rb, ca, cb = 16 * y0 - 10 * T, 16 * (y0 + h) + 7 * B, 16 * x0 - 12 * Lm, 16 * (x0 + w) + 4 * R
    ly[10 - 10 * T:10 + 16 * h + 7 * B, 16 - 12 * Lm:16 + 16 * w + 4 * R] = y[ra:rb, ca:cb]
    ra, rb, ca = 8 * y0 - 2 * T, 8 * (y0 + h) + 2 * B, 16 * x0 - 4 * Lm
    cy[2 - 2 * T:2 + 8 * h + 2 * B, 16 - 4 * Lm:16 + 16 * w + 4 * R] = uv[ra:rb, ca:cb]
    b = np.zeros((h + 2, w + 2, 32), np.uint8)
    b[1 - T:1 + h + B, 1 - Lm:1 + w + R] = bs[y0 - T:y0 + h + B, x0 - Lm:x0 + w + R]
    p = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    shim.dt_run(p(ly), p(cy), p(b), w, h, Lm, R, T, B, p(qv), int(rs.integers(0, 2)))
    np.testing.assert_array_equal(ly[10:10 + 16 * h, 16:16 + 16 * w], wy[16 * y0:16 * (y0 + h), 16 * x0:16 * (x0 + w)])
    np.testing.assert_array_equal(cy[2:2 + 8 * h, 16:16 + 16 * w], wuv[8 * y0:8 * (y0 + h), 16 * x0:16 * (x0 + w)])
