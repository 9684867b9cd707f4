"""GPU CAVLC (b200enc_cavlc_slices) against the serial writer of
oracle/cavlc_serial.cpp: identical slice bytes on synthetic outputs that reach
every table (dense and sparse blocks, trailing ones, level escapes up to the
36-bit ones, long zero runs, skip runs, all nC classes, every intra mode at
slice and picture edges), in 1 to 16 slices, with slice headers, with the
8x8 transform (all macroblocks, chosen per macroblock) and at quality levels
either side of the skip rule's change. On the CPU the serial writer is compared
with the reference's own where that is built."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_gpu_cavlc import _synthetic

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ZZ8 = np.array([0, 1, 8, 16, 9, 2, 3, 10, 17, 24, 32, 25, 18, 11, 4, 5, 12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6, 7,
                14, 21, 28, 35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39, 46,
                53, 60, 61, 54, 47, 55, 62, 63], np.uint8)


@pytest.fixture(scope="module")
def serial(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("cavlc") / "serial.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "bc250-vaapi_b200", "csrc"),
                    "-o", so, os.path.join(ROOT, "oracle", "cavlc_serial.cpp")], check=True)
    L = ctypes.CDLL(so)

    def run(mbw, mbh, qp, intra, ns, levels, dc, nz, pm, mv, headers=None, quality=4, t8=0, t8f=None):
        p = lambda x: None if x is None else ctypes.c_void_p(x.ctypes.data)  # noqa: E731
        hdr, hb = np.zeros((ns, 16), np.uint8), np.zeros(ns, np.int32)
        for k, (bits, n) in enumerate(headers or []):
            hb[k] = n
            hdr[k] = np.frombuffer(((bits << (128 - n)) if n else 0).to_bytes(16, "big"), np.uint8)
        out, nb = np.zeros(mbw * mbh * 3300 + 4096, np.uint8), np.zeros(ns, np.int64)
        L.orc_cavlc_slices(mbw, mbh, qp, int(intra), ns, quality, t8, p(levels), p(dc), p(nz), p(pm), p(mv), p(t8f),
                           p(ZZ8), p(hdr), p(hb), p(out), p(nb))
        ends = np.cumsum(nb)
        return [out[e - n:e].tobytes() for e, n in zip(ends, nb)]

    return run


def _gpu(gpu, mbw, mbh, qp, intra, ns, levels, dc, nz, pm, mv, headers=None, quality=4, t8=0, t8f=None):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (levels, dc, nz.view(np.int32), pm.view(np.int32), mv)]
    f = torch.from_numpy(t8f).cuda() if t8f is not None else None
    return gpu.cavlc_slices(mbw, mbh, qp, intra, ns, *[x.data_ptr() for x in t], headers=headers, quality_level=quality,
                            transform8x8=t8, t8_flags=f.data_ptr() if f is not None else 0)


def _masks(levels, t8f):
    """nz words as the P chain leaves them (8x8 macroblocks: by interleaved scan positions)."""
    mbs = levels.shape[0]
    nz = np.zeros((mbs, 24), np.uint32)
    for p in range(16):
        nz |= (levels[:, :, p] != 0).astype(np.uint32) << p
    for mb in np.flatnonzero(t8f) if t8f is not None else []:
        flat = levels[mb].reshape(-1)
        for b in range(16):
            q, i = b >> 2, b & 3
            x4, y4 = (b & 1) | ((b >> 1) & 2), ((b >> 1) & 1) | ((b >> 2) & 2)
            l16 = flat[64 * q + ZZ8[i::4].astype(int)]
            nz[mb, y4 * 4 + x4] = int(((l16 != 0) << np.arange(16)).sum())
    return nz


@pytest.mark.gpu
@pytest.mark.parametrize("intra", [1, 0])
@pytest.mark.parametrize("mbw,mbh,ns", [(1, 1, 1), (11, 9, 1), (11, 9, 3), (30, 17, 4), (7, 23, 16), (64, 40, 2)])
@pytest.mark.parametrize("qp", [12, 27, 45])
def test_slices_match_serial_writer(gpu, serial, intra, mbw, mbh, ns, qp):
    rs = np.random.Generator(np.random.PCG64(mbw * 131 + mbh * 7 + ns * 3 + qp + intra))
    args = list(_synthetic(rs, mbw, mbh, intra))
    args[0][0, 0] = np.array([32767, -32767] * 8, np.int16)  # the longest escapes
    if intra:
        args[0][:, :16, 0] = 0  # the chain leaves position 0 to the DC path
    args[2] = _masks(args[0], None)
    heads = [(int.from_bytes(rs.bytes(16), "big") >> (128 - n), n) for n in rs.integers(0, 129, ns).tolist()]
    got = _gpu(gpu, mbw, mbh, qp, intra, ns, *args, headers=heads)
    want = serial(mbw, mbh, qp, intra, ns, *args, headers=heads)
    for s, (g, w) in enumerate(zip(got, want)):
        assert g == w, f"slice {s}: {len(g)} vs {len(w)} bytes"


@pytest.mark.gpu
@pytest.mark.parametrize("choose", [0, 1])
@pytest.mark.parametrize("quality", [4, 5])
def test_transform8_and_quality_match_serial_writer(gpu, serial, choose, quality):
    rs = np.random.Generator(np.random.PCG64(17 + choose + 2 * quality))
    mbw, mbh, ns = 13, 8, 3
    levels, dc, nz, pm, mv = _synthetic(rs, mbw, mbh, 0)
    for mb in range(0, mbw * mbh, 3):  # no luma levels and tiny DC words: where the rule differs
        levels[mb, :16] = 0
        dc[mb] = rs.integers(-1, 2, 24)
        mv[mb, :2] = 0
    t8f = (rs.random(mbw * mbh) < 0.5).astype(np.uint8) if choose else np.ones(mbw * mbh, np.uint8)
    for t8 in (0, 1):
        nz = _masks(levels, t8f if t8 else None)
        a = (mbw, mbh, 30, 0, ns, levels, dc, nz, pm, mv)
        kw = dict(quality=quality, t8=t8, t8f=t8f if t8 and choose else None)
        assert _gpu(gpu, *a, **kw) == serial(*a, **kw)


def _nal(rbsp, ref_idc, kind):
    out, zeros = bytearray([0, 0, 0, 1, ref_idc << 5 | kind]), 0
    for b in rbsp:
        if zeros == 2 and b <= 3:
            out.append(3)
            zeros = 0
        out.append(b)
        zeros = zeros + 1 if b == 0 else 0
    return bytes(out)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,ns,qp", [(64, 48, 1, 30), (320, 192, 3, 14), (640, 480, 2, 38)])
def test_slice_nals_match_serial_writer(gpu, serial, W, H, ns, qp):
    """A context's NAL units: the serial writer's RBSP behind headers of 0 to
    128 bits (every bit offset of the data, headers full of zeros, so that
    emulation prevention acts), start codes, emulation prevention bytes."""
    from b200enc import synth
    seq = synth.Sequence(W, H, seed=W, pan=True)
    ctx = gpu.Context()
    ctx.configure(search_range=16, deblock=1)
    ctx.set_entropy(1)
    img, mem = ctx.create_image(W, H)
    out = np.zeros(W * H * 4 + 65536, np.uint8)
    try:
        for t, bits in enumerate((0, 1, 26, 27, 60, 95, 128)):
            y, uv = seq.frame(t)
            ctx.upload(img, mem, y // 64 * 64 if t == 3 else y, uv)
            slot = ctx.encode(img, W, H, qp, t % 4 == 0, ns)
            assert ctx.sync(slot) == 0
            g = {k: np.ascontiguousarray(v) for k, v in ctx.staging(slot).items()}
            hdr, hb = np.zeros((ns, 16), np.uint8), np.full(ns, bits, np.int32)
            hdr[:, 3] = 0x80
            n = ctx.slice_nals(slot, hdr, hb, 2, 1, out)
            heads = [(int.from_bytes(bytes(h), "big") >> (128 - bits), bits) for h in hdr]
            want = serial((W + 15) // 16, (H + 15) // 16, qp, int(t % 4 == 0), ns, g["levels"], g["dc"], g["nz"],
                          g["pred_mode"], g["mv"], headers=heads)
            assert out[:n].tobytes() == b"".join(_nal(w, 2, 1) for w in want), f"frame {t}"
    finally:
        ctx.destroy_image(img, mem)
        ctx.close()


@pytest.mark.parametrize("intra", [1, 0])
def test_serial_writer_matches_reference(oracle_mod, serial, intra):
    if not oracle_mod.cavlc_ref_available():
        pytest.skip("oracle/_ref/libcavlcref.so not built")
    rs = np.random.Generator(np.random.PCG64(3 + intra))
    mbw, mbh, ns = 12, 9, 2
    args = _synthetic(rs, mbw, mbh, intra)
    mbs = mbw * mbh
    want = [oracle_mod.ref_cavlc_slice_data(mbw, mbh, 27, intra, s * mbs // ns, (s + 1) * mbs // ns, *args, quality_level=4)
            for s in range(ns)]
    assert serial(mbw, mbh, 27, intra, ns, *args) == want
