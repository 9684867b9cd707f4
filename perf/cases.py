"""Performance cases of the encoder: the work its users have it do, through
its public entry points, over the range of sizes and options they use.

A case is a dict of plain values; `kind` says which entry points it goes
through:

  session   gpu_compute_* contexts (Context): whole GOPs of one or more
            concurrent streams, host frames or device surfaces in, slice NAL
            units, host staging or device outputs out - an encoder process;
  batch     b200enc_batch_* (Batch): many streams of uneven sizes a step;
  picture   the stage entry points on one P picture (search, P chain, tile
            deblocking; High-profile pictures add the 8x8 transform choice
            and CAVLC) - a host encoder that keeps its own loop;
  hevc      the HEVC encoder's per-picture primitives (half-sample planes,
            motion search, 8x8 transform and back, intra 4x4 modes);
  hevc_db   HEVC deblocking of one picture;
  train     one gradient of the motion-proposal network on one picture.

listed() are the measured cases, draw(rng) another one of the same ranges.
Video is synthetic, after the workloads' description: smooth gradients with
a sigma 8 texture under a quarter-pel global pan, six textured rectangles
moving on their own, a noise patch over 10 % of the frame.
"""
import ctypes
import math
import os
import random
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bc250-vaapi_b200"))
import b200enc  # noqa: E402
from b200enc import proposal as _proposal  # noqa: E402

ME_MODE = {"full": 0, "learned": 1, "learned_fp8": 3}
# frame sizes of the multi-stream mix (VGA, 720p, 1080p, 1440p), most of them small
BATCH_SIZES = [(640, 480), (640, 480), (640, 480), (1280, 720), (1280, 720), (1280, 720), (1920, 1080), (2560, 1440)]
HEVC_MARGIN = 16


def listed():
    return [
        # a video-call thumbnail: the smallest calls, latency and launches count
        dict(name="call_176x144", kind="session", w=176, h=144, streams=1, me="full", search=16, qp=26, slices=1,
             frames=5, gop=5, src="host", out="nals"),
        # VGA conference stream, the library's default search range, learned search, host frames to a bitstream
        dict(name="conference_640x480", kind="session", w=640, h=480, streams=1, me="learned", search=16, qp=30,
             slices=1, frames=12, gop=12, src="host", out="nals"),
        # the reference host encoder's own use: levels, DC, masks, modes and vectors staged for its entropy coder
        dict(name="staging_1080p", kind="session", w=1920, h=1080, streams=1, me="full", search=32, qp=27, slices=4,
             frames=8, gop=8, src="host", out="staging"),
        # a streaming server: eight 1080p streams, pinned host frames to Annex B slices (the headline workload)
        dict(name="server_1080p_x8", kind="session", w=1920, h=1080, streams=8, me="learned_fp8", search=32, qp=27,
             slices=4, frames=16, gop=16, src="host", out="nals"),
        # transcoding a decoder's 2160p surfaces, outputs kept on the device
        dict(name="surfaces_2160p", kind="session", w=3840, h=2160, streams=1, me="learned_fp8", search=32, qp=32,
             slices=4, frames=8, gop=8, src="device", out="device"),
        # an all-intra 720p contribution feed at a high rate
        dict(name="intra_720p", kind="session", w=1280, h=720, streams=1, me="full", search=16, qp=20, slices=4,
             frames=4, gop=1, src="host", out="nals"),
        # the multi-stream batch: eight streams of four sizes, one launch a stage, a captured graph a step
        dict(name="batch_mixed_x8", kind="batch", streams=8, me="learned_fp8", search=32, qp=28, steps=6, gop=6,
             graph=True, size_shift=0),
        # one P picture through the stage calls, a laptop camera's ragged size
        dict(name="picture_1366x766", kind="picture", w=1366, h=766, me="full", search=16, qp=24, t8=0, slices=1),
        # one High-profile P picture: 8x8 transform chosen per macroblock, CAVLC slices on the GPU
        dict(name="high_1080p", kind="picture", w=1920, h=1080, me="full", search=32, qp=22, t8=2, slices=4),
        # one 1080p picture of the HEVC encoder's primitives
        dict(name="hevc_1080p", kind="hevc", w=1920, h=1080, bits=8, qp=30),
        # a Main10 2160p picture through the HEVC deblocking filter
        dict(name="hevc_deblock_2160p10", kind="hevc_db", w=3840, h=2160, bits=10, qp=34),
        # one gradient of the proposal network on a 1080p picture's macroblocks
        dict(name="train_1080p", kind="train", w=1920, h=1080, search=32),
    ]


def _size(rng, lo, hi):
    """An even width between lo and hi, spread over its logarithm, and a
    height between 4:3 and 2:1 of it: mostly not whole macroblocks."""
    w = int(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2) * 2
    return w, max(32, int(w / rng.uniform(1.33, 2.0) / 2) * 2)


def draw(rng):
    kind = rng.choice(["session"] * 4 + ["batch"] + ["picture"] * 2 + ["hevc", "hevc_db", "train"])
    qp = rng.randint(18, 40)
    if kind == "session":
        w, h = _size(rng, 128, 2560)
        small = w * h <= 640 * 480
        frames = rng.randint(3, 10)
        out = rng.choice(["nals", "nals", "staging", "device"])
        return dict(kind=kind, w=w, h=h, streams=rng.choice([1, 1, 2, 4] if small else [1, 1, 2]),
                    me=rng.choice(list(ME_MODE)), search=rng.choice([16, 32]), qp=qp,
                    slices=rng.choice([1, 2, 4]) if h >= 128 else 1, frames=frames,
                    gop=rng.choice([1, frames, frames]), src="device" if out == "device" else "host", out=out)
    if kind == "batch":
        return dict(kind=kind, streams=rng.randint(2, 8), me=rng.choice(["full", "learned_fp8"]),
                    search=rng.choice([16, 32]), qp=qp, steps=rng.randint(2, 6), gop=6, graph=rng.random() < 0.5,
                    size_shift=rng.randint(0, 7))
    if kind == "picture":
        w, h = _size(rng, 64, 2560)
        return dict(kind=kind, w=w, h=h, me=rng.choice(["full", "learned_fp8"]), search=rng.choice([16, 32]), qp=qp,
                    t8=rng.choice([0, 0, 1, 2]), slices=rng.choice([1, 2, 4]) if h >= 128 else 1)
    if kind == "train":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, search=rng.choice([16, 32]))
    w, h = _size(rng, 128, 2560 if kind == "hevc" else 3840)
    return dict(kind=kind, w=w // 8 * 8, h=h // 8 * 8, bits=rng.choice([8, 10]), qp=qp)


# ---------------------------------------------------------------- inputs


def _bilinear(img, x0, y0, h, w):
    xi, yi = math.floor(x0), math.floor(y0)
    fx, fy = x0 - xi, y0 - yi
    b = img[yi:yi + h + 1, xi:xi + w + 1]
    top = b[:-1, :-1] * (1 - fx) + b[:-1, 1:] * fx
    bot = b[1:, :-1] * (1 - fx) + b[1:, 1:] * fx
    return top * (1 - fy) + bot * fy


def _video(w, h, n, seed):
    """n frames (y [h][w], uv [h/2][w]) of uint8 CUDA tensors, and the pan in
    quarter samples per frame."""
    r = random.Random(seed)
    g = torch.Generator("cuda").manual_seed(seed & 0x7FFFFFFF)
    m = 8 + 4 * n
    ch, cw = h + 2 * m + 2, w + 2 * m + 2
    yy = torch.arange(ch, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(cw, device="cuda", dtype=torch.float32)[None, :]
    luma = 128 + 60 * torch.sin(xx / (37 + 40 * r.random()) + 6 * r.random()) \
        + 40 * torch.cos(yy / (53 + 50 * r.random()) + 6 * r.random()) + 0.05 * (xx - cw / 2) * r.uniform(-1, 1)
    luma = luma + 8 * torch.randn((ch, cw), device="cuda", generator=g)
    pw = max(2, int(math.sqrt(0.15 * w * h)))
    ph = max(2, int(0.1 * w * h / pw))
    px, py = r.randint(m, max(m, m + w - pw)), r.randint(m, max(m, m + h - ph))
    luma[py:py + ph, px:px + pw] = 255 * torch.rand((ch, cw), device="cuda", generator=g)[py:py + ph, px:px + pw]
    luma = luma.clamp(0, 255)
    cy, cx = yy[: ch // 2], xx[:, : cw // 2]
    cb = (128 + 40 * torch.sin(cx / 23 + 6 * r.random()) + 20 * torch.cos(cy / 31)).clamp(0, 255)
    cr = (128 + 40 * torch.cos(cx / 29 + 6 * r.random()) - 20 * torch.sin(cy / 17)).clamp(0, 255)
    a, speed = r.uniform(0, 2 * math.pi), r.uniform(0, 4)
    vx, vy = round(4 * speed * math.cos(a)) / 4, round(4 * speed * math.sin(a)) / 4
    rects = []
    for _ in range(6):
        rw, rh = r.randint(max(8, w // 16), max(9, w // 4)), r.randint(max(8, h // 16), max(9, h // 4))
        tex = (r.uniform(40, 215) + 25 * torch.randn((rh + 2, rw + 2), device="cuda", generator=g)).clamp(0, 255)
        q = 1 if r.random() < 0.5 else 4
        rects.append((r.uniform(0, w - 8), r.uniform(0, h - 8), round(q * r.uniform(-8, 8)) / q,
                      round(q * r.uniform(-8, 8)) / q, tex, r.uniform(60, 196), r.uniform(60, 196)))
    out = []
    for t in range(n):
        ox, oy = m + vx * t, m + vy * t
        y = _bilinear(luma, ox, oy, h, w).clone()
        u = _bilinear(cb, ox / 2, oy / 2, h // 2, w // 2).clone()
        v = _bilinear(cr, ox / 2, oy / 2, h // 2, w // 2).clone()
        for x0, y0, dx, dy, tex, tu, tv in rects:
            rh, rw = tex.shape[0] - 2, tex.shape[1] - 2
            x, z = (x0 + dx * t) % (w + rw) - rw, (y0 + dy * t) % (h + rh) - rh
            xi, zi = math.floor(x), math.floor(z)
            b = _bilinear(tex, 1 - (x - xi), 1 - (z - zi), rh, rw)
            xa, xb, za, zb = max(0, xi), min(w, xi + rw), max(0, zi), min(h, zi + rh)
            if xa < xb and za < zb:
                y[za:zb, xa:xb] = b[za - zi:zb - zi, xa - xi:xb - xi]
                u[za // 2:(zb + 1) // 2, xa // 2:(xb + 1) // 2] = tu
                v[za // 2:(zb + 1) // 2, xa // 2:(xb + 1) // 2] = tv
        uv = torch.stack([u, v], dim=2).reshape(h // 2, w)
        out.append((y.round().clamp(0, 255).to(torch.uint8), uv.round().clamp(0, 255).to(torch.uint8)))
    return out, (round(4 * vx), round(4 * vy))


def _nv12(y, uv):
    """An NV12 surface at the coded size, edges replicated into its padding."""
    h, w = y.shape
    f = b200enc.NV12(w, h)
    for p, s in ((f.y, y), (f.uv, uv)):
        p[: s.shape[0], :w] = s
        if w < f.pitch:
            pad = s[:, -1:] if p is f.y else s[:, -2:].repeat(1, (f.pitch - w + 1) // 2)[:, : f.pitch - w]
            p[: s.shape[0], w:] = pad
        p[s.shape[0]:] = p[s.shape[0] - 1]
    return f


def _slice_headers(n):
    """n slice headers of a CAVLC stream's usual length: (uint8 [n][16], int32 [n])."""
    hdr, bits = np.zeros((n, 16), np.uint8), np.full(n, 27, np.int32)
    for k in range(n):
        hdr[k, :4] = (0x9A, 0x35 ^ k, 0x6C, 0x60)
    return hdr, bits


def _mbs(w, h):
    return ((w + 15) // 16) * ((h + 15) // 16)


# ---------------------------------------------------------------- sessions


class _Stream:
    pass


def _prepare_session(c, seed):
    S = _Stream()
    S.c, S.streams = c, []
    w, h = c["w"], c["h"]
    S.hdr, S.hdr_bits = _slice_headers(c["slices"])
    for s in range(c["streams"]):
        st = _Stream()
        frames, _ = _video(w, h, c["frames"], seed * 64 + s)
        st.ctx = b200enc.Context()
        st.ctx.configure(search_range=c["search"], deblock=1)
        if c["me"] != "full":
            st.ctx.set_me(ME_MODE[c["me"]])
        if c["out"] == "nals":
            st.ctx.set_entropy(2)
            # the pass's stream and each frame's bytes in it
            per_mb = int(40 * 2 ** ((36 - c["qp"]) / 6)) + 8
            st.nal = np.zeros(c["frames"] * (_mbs(w, h) * per_mb + 4096), np.uint8)
            st.sizes = np.zeros(c["frames"], np.int64)
        if c["src"] == "host":
            st.imgs = [st.ctx.create_image(w, h) for _ in range(2)]
            st.frames = []
            for y, uv in frames:
                p = torch.empty((h + h // 2, w), dtype=torch.uint8, pin_memory=True)
                p[:h].copy_(y)
                p[h:].copy_(uv)
                st.frames.append((p[:h].numpy(), p[h:].numpy()))
        else:
            st.frames = [_nv12(y, uv) for y, uv in frames]
        S.streams.append(st)
    if c["streams"] > 1:
        S.pool = ThreadPoolExecutor(c["streams"])
    return S


def _recon(ctx):
    y, uv, pitch = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_int()
    b200enc._check(ctx.L.b200enc_ctx_recon(ctypes.byref(ctx.ctx), ctypes.byref(y), ctypes.byref(uv),
                                           ctypes.byref(pitch)), "b200enc_ctx_recon")
    cw, ch = b200enc.coded(ctx.ctx.frame_width, ctx.ctx.frame_height)
    p = pitch.value
    return [b200enc.device_view(y.value, ch * p).view(ch, p)[:, :cw],
            b200enc.device_view(uv.value, ch // 2 * p).view(ch // 2, p)[:, :cw]]


def _device_outputs(ctx):
    p = [ctypes.c_void_p() for _ in range(5)]
    b200enc._check(ctx.L.b200enc_ctx_device_outputs(ctypes.byref(ctx.ctx), *[ctypes.byref(x) for x in p]),
                   "b200enc_ctx_device_outputs")
    n = _mbs(ctx.ctx.frame_width, ctx.ctx.frame_height)
    return [b200enc.device_view(x.value, n * b).view(t) for x, b, t in
            zip(p, (768, 96, 96, 4, 16), (torch.int16, torch.int32, torch.int32, torch.int32, torch.int32))]


def _encode_stream(S, st):
    """One pass of one stream: frame t is submitted while t - 1 is collected,
    as the boundary's two slots allow."""
    c, ctx = S.c, st.ctx
    w, h, at, staged, last = c["w"], c["h"], 0, {}, None

    def collect(t, slot, idr):
        nonlocal at
        if c["out"] == "nals":
            st.sizes[t] = ctx.slice_nals(slot, S.hdr, S.hdr_bits, 3 if idr else 2, 5 if idr else 1, st.nal[at:])
            at += int(st.sizes[t])
        else:
            if ctx.sync(slot) != 0:
                raise RuntimeError("gpu_compute_sync_slot failed")
            staged[slot] = ctx.staging(slot)

    for t in range(c["frames"]):
        f = st.frames[t]
        idr = t % c["gop"] == 0
        if c["src"] == "device":
            ctx.encode_device(f, w, h, c["qp"], idr, num_slices=c["slices"])
            continue
        img, mem = st.imgs[t & 1]
        ctx.upload(img, mem, f[0], f[1])
        slot = ctx.encode(img, w, h, c["qp"], idr, num_slices=c["slices"])
        if last is not None:
            collect(*last)
        last = (t, slot, idr)
    if last is not None:
        collect(*last)
    if c["out"] == "nals":
        out = [st.nal, st.sizes]
    elif c["out"] == "staging":
        out = [staged[k][n] for k in sorted(staged) for n in sorted(staged[k])]
    else:
        out = _device_outputs(ctx)
    return out + _recon(ctx)


def _run_session(S):
    if len(S.streams) == 1:
        return _encode_stream(S, S.streams[0])
    return list(S.pool.map(lambda st: _encode_stream(S, st), S.streams))


# ---------------------------------------------------------------- batches


def _prepare_batch(c, seed):
    S = _Stream()
    S.c = c
    S.sizes = [BATCH_SIZES[(k + c["size_shift"]) % len(BATCH_SIZES)] for k in range(c["streams"])]
    S.frames = [[_nv12(*f) for f in _video(w, h, c["steps"], seed * 64 + k)[0]] for k, (w, h) in enumerate(S.sizes)]
    S.qps = [c["qp"] + k % 5 - 2 for k in range(c["streams"])]
    S.batch = b200enc.Batch(S.sizes, search_range=c["search"], me_mode=ME_MODE[c["me"]], graph=c["graph"])
    return S


def _run_batch(S):
    n = len(S.sizes)
    for t in range(S.c["steps"]):
        S.batch.encode([f[t] for f in S.frames], S.qps, [t % S.c["gop"] == 0] * n)
    if S.batch.sync() != 0:
        raise RuntimeError("b200enc_batch_sync failed")
    out = []
    for s, (w, h) in enumerate(S.sizes):
        p, pitch = [ctypes.c_void_p() for _ in range(7)], ctypes.c_int()
        b200enc._check(S.batch.L.b200enc_batch_outputs(S.batch.h, s, *[ctypes.byref(x) for x in p],
                                                       ctypes.byref(pitch)), "b200enc_batch_outputs")
        cw, ch = b200enc.coded(w, h)
        mbs, q = _mbs(w, h), pitch.value
        out.append([b200enc.device_view(x.value, mbs * b).view(t) for x, b, t in
                    zip(p, (768, 96, 96, 4, 16),
                        (torch.int16, torch.int32, torch.int32, torch.int32, torch.int32))]
                   + [b200enc.device_view(p[5].value, ch * q).view(ch, q)[:, :cw],
                      b200enc.device_view(p[6].value, ch // 2 * q).view(ch // 2, q)[:, :cw]])
    return out


# ---------------------------------------------------------------- one picture


def _prepare_picture(c, seed):
    S = _Stream()
    S.c = c
    w, h = c["w"], c["h"]
    frames, pan = _video(w, h, 3, seed)
    S.ref, S.cur = _nv12(*frames[0]), _nv12(*frames[1])
    S.cw, S.ch = b200enc.coded(w, h)
    S.out = b200enc.Outputs(w, h)
    S.rec, S.dst = b200enc.NV12(w, h), b200enc.NV12(w, h)
    S.status = torch.zeros(4, dtype=torch.int32, device="cuda")
    mbs = _mbs(w, h)
    if c["me"] != "full":
        S.prop = _proposal.Proposal(mbs)
        S.prop.load(_proposal.DEFAULT_WEIGHTS)
        S.prev_mv = _prev_mv(w, h, pan, seed)
    S.t8 = torch.zeros(mbs, dtype=torch.uint8, device="cuda")
    if c["t8"]:
        L = b200enc.lib()
        S.cap = (mbs * 1400 // c["slices"] + 65536) // 4 * 4
        S.bits = torch.zeros(c["slices"] * S.cap, dtype=torch.uint8, device="cuda")
        S.nbytes = torch.zeros(c["slices"], dtype=torch.int32, device="cuda")
        n = L.b200enc_cavlc_scratch_bytes(S.cw // 16, S.ch // 16)
        S.scratch = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
        sp = (S.scratch.data_ptr() + 255) // 256 * 256
        S.hdr, S.hdr_bits = _slice_headers(c["slices"])
        vp, o = ctypes.c_void_p, S.out
        S.cavlc = b200enc.CavlcParams(
            S.cw // 16, S.ch // 16, c["qp"], 0, c["slices"], 4, vp(o.levels.data_ptr()), vp(o.dc.data_ptr()),
            vp(o.nz.data_ptr()), None, vp(o.mv.data_ptr()), vp(S.hdr.ctypes.data), vp(S.hdr_bits.ctypes.data),
            vp(S.bits.data_ptr()), S.cap, vp(S.nbytes.data_ptr()), None, vp(sp), n, 1, vp(S.t8.data_ptr()))
    return S


def _prev_mv(w, h, pan, seed):
    """The previous picture's field: the pan with a few vectors of their own."""
    mbs = _mbs(w, h)
    g = torch.Generator("cuda").manual_seed(seed + 7)
    mv = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    mv[:, 0], mv[:, 1] = pan
    own = torch.rand(mbs, device="cuda", generator=g) < 0.15
    mv[:, :2] += torch.randint(-24, 25, (mbs, 2), device="cuda", generator=g, dtype=torch.int32) * own[:, None]
    mv[:, 2] = torch.randint(600, 3000, (mbs,), device="cuda", generator=g, dtype=torch.int32)
    return mv


def _run_picture(S):
    c, o = S.c, S.out
    w, h, cw, ch = c["w"], c["h"], S.cw, S.ch
    if c["me"] == "full":
        b200enc.me_full_search(S.cur, S.ref, w, h, cw, ch, c["search"], 5, 512, o.mv)
    else:
        S.prop.me(S.cur, S.ref, w, h, cw, ch, S.prev_mv, c["search"], 5, 512, 0.9, o.mv, mode=ME_MODE[c["me"]])
    res = [o.levels, o.dc, o.nz, o.mv, S.dst.y[:, :cw], S.dst.uv[:, :cw]]
    if not c["t8"]:
        b200enc.p_frame(S.cur, S.ref, w, h, cw, ch, c["qp"], o.mv, o, S.rec)
        b200enc.deblock_tiles(cw // 16, ch // 16, c["qp"], 0, o.nz, o.mv, S.rec, S.dst, S.status)
        return res + [S.status]
    L, P, st = b200enc.lib(), b200enc._p, b200enc._stream(None)
    b200enc.p_frame_t8(S.cur, S.ref, w, h, cw, ch, c["qp"], o.mv, o, S.rec, c["t8"], S.t8)
    b200enc._check(L.b200enc_deblock_tiles_t8(cw // 16, ch // 16, c["qp"], 0, P(o.nz), P(S.t8), P(o.mv), S.rec.yp(),
                                              S.rec.uvp(), S.dst.yp(), S.dst.uvp(), S.rec.pitch, P(S.status), st),
                   "b200enc_deblock_tiles_t8")
    b200enc._check(L.b200enc_cavlc_slices(ctypes.byref(S.cavlc), st), "b200enc_cavlc_slices")
    return res + [S.status, S.t8, S.bits, S.nbytes]


# ---------------------------------------------------------------- HEVC


def _samples(t, bits):
    return t if bits == 8 else (t.to(torch.int16) * 4 + 1)


def _prepare_hevc(c, seed):
    S = _Stream()
    S.c = c
    w, h, bits, m = c["w"], c["h"], c["bits"], HEVC_MARGIN
    frames, pan = _video(w, h, 2, seed)
    S.ref, S.src = (_samples(f[0], bits).contiguous() for f in frames)
    S.planes = torch.zeros((4, h + 2 * m, (w + 2 * m + 127) // 128 * 128), dtype=S.ref.dtype, device="cuda")
    rs = np.random.Generator(np.random.PCG64(seed))
    ys, xs = np.mgrid[0:h - 7:8, 0:w - 7:8]
    n = xs.size
    jobs = np.zeros(n, b200enc.HEVC_ME_JOB)
    jobs["cu_x"], jobs["cu_y"] = xs.reshape(-1), ys.reshape(-1)
    pan = np.array(pan)
    jobs["mvp"] = pan + rs.integers(-4, 5, (n, 2, 2))
    jobs["starts"] = pan + rs.integers(-12, 13, (n, 16, 2))
    jobs["starts"][:, 0] = 0
    jobs["n_starts"] = rs.integers(2, 7, n)
    jobs["lambda_q8"] = int(256 * 0.57 * 2 ** ((c["qp"] - 12) / 6))
    S.jobs = torch.from_numpy(jobs.view(np.uint8)).cuda()
    S.res = torch.zeros(n * b200enc.HEVC_ME_RESULT.itemsize, dtype=torch.uint8, device="cuda")
    d = (S.src.to(torch.int16) - S.ref.to(torch.int16))[: h // 8 * 8, : w // 8 * 8]
    S.resid = d.reshape(h // 8, 8, w // 8, 8).permute(0, 2, 1, 3).reshape(-1, 64).contiguous()
    S.coeff, S.back = torch.zeros_like(S.resid), torch.zeros_like(S.resid)
    ys, xs = np.mgrid[0:h - 3:4, 0:w - 3:4]
    S.pus = torch.from_numpy(np.stack([xs, ys, np.zeros_like(xs)], axis=2).reshape(-1, 3).astype(np.int32)).cuda()
    S.modes = torch.zeros(S.pus.shape[0], dtype=torch.int32, device="cuda")
    S.preds = torch.zeros((S.pus.shape[0], 16), dtype=S.ref.dtype, device="cuda")
    return S


def _run_hevc(S):
    c = S.c
    w, h, bits = c["w"], c["h"], c["bits"]
    b200enc.hevc_build_hpel(S.ref, w, h, HEVC_MARGIN, S.planes)
    b200enc.hevc_motion_search(S.src, w, h, S.planes, HEVC_MARGIN, 1, S.jobs, S.res)
    b200enc.hevc_transform_quant_8x8(S.resid, S.coeff, c["qp"], 2, bits)
    b200enc.hevc_dequant_itransform_8x8(S.coeff, S.back, c["qp"], bits)
    b200enc.hevc_choose_luma_mode(S.src, S.ref, w, h, S.pus, S.modes, S.preds)
    return [S.planes, S.res, S.coeff, S.back, S.modes, S.preds]


def _prepare_hevc_db(c, seed):
    S = _Stream()
    w, h, bits = c["w"], c["h"], c["bits"]
    g = torch.Generator("cuda").manual_seed(seed)
    (y, uv), = _video(w, h, 1, seed)[0]
    maxv, k = (1 << bits) - 1, 1 << (bits - 8)

    def blocky(p, block):
        # a coded picture: every block with a small offset of its own
        hh, ww = p.shape
        o = 3 * torch.randn(((hh + block - 1) // block, (ww + block - 1) // block), device="cuda", generator=g)
        o = o.repeat_interleave(block, 0).repeat_interleave(block, 1)[:hh, :ww]
        v = ((p.float() + o) * k).round().clamp(0, maxv)
        return v.to(torch.uint8 if bits == 8 else torch.int16).contiguous()

    S.src = [blocky(y, 8), blocky(uv[:, 0::2], 4), blocky(uv[:, 1::2], 4)]
    S.out = [p.clone() for p in S.src]

    def rand(*shape):
        return torch.rand(shape, device="cuda", generator=g)

    ew, eh, pw, ph = w // 8, h // 8, w // 4, h // 4
    # coding blocks of 8 to 32: an edge on each 16x16 boundary and on some of the 8x8 ones, most of them transform edges
    yy, xx = torch.arange(eh, device="cuda")[:, None], torch.arange(ew, device="cuda")[None, :]
    e0 = (xx % 2 == 0) | (rand(eh, ew) < 0.4)
    e1 = (yy % 2 == 0) | (rand(eh, ew) < 0.4)
    S.edges = (e0.int() + 2 * e1.int() + 4 * (rand(eh, ew) < 0.7).int() + 8 * (rand(eh, ew) < 0.7).int()).to(torch.uint8)
    mvf = np.zeros((ph, pw), b200enc.HEVC_MVF)
    rs = np.random.Generator(np.random.PCG64(seed))
    up = lambda a, s: np.kron(a, np.ones((s, s), a.dtype))[:ph, :pw]  # noqa: E731
    bh, bw = (ph + 3) // 4, (pw + 3) // 4
    for li in range(2):
        for d in range(2):
            mvf["mv"][..., li, d] = up(rs.integers(-6, 7, (bh, bw)).astype(np.int16), 4)
    mvf["pred_flag"] = up(rs.choice([0, 1, 2, 3], (bh, bw), p=[0.1, 0.5, 0.1, 0.3]).astype(np.uint8), 4)
    mvf["ref_poc"][..., 1] = 4
    S.mvf = torch.from_numpy(mvf.view(np.uint8).reshape(-1)).cuda()
    S.cbf = (rand(ph, pw) < 0.4).to(torch.uint8)
    S.qp_y = (c["qp"] + torch.randint(-3, 4, (eh, ew), device="cuda", generator=g)).to(torch.int8)
    sf = np.zeros(1, b200enc.HEVC_SLICE_FILTER)
    S.sf = torch.from_numpy(sf.view(np.uint8)).cuda()
    S.params = b200enc.hevc_deblock_params(lambda t: t.data_ptr(), S.out, [p.stride(0) for p in S.out], w, h, bits,
                                           bits, 6, 3, S.edges, ew, S.qp_y, mvf=S.mvf, cbf=S.cbf, min_pu_width=pw,
                                           slice_filter=S.sf, n_slice_filter=1)
    return S


def _run_hevc_db(S):
    for d, s in zip(S.out, S.src):  # the next decoded picture arrives in the filter's planes
        d.copy_(s)
    b200enc.hevc_deblock(S.params)
    return S.out


# ---------------------------------------------------------------- training


def _train_inputs(c, seed):
    """Current and reference luma, the previous field, the search's logged
    winners and the nz words of one training picture (plain CUDA tensors)."""
    w, h, R = c["w"], c["h"], c["search"]
    frames, pan = _video(w, h, 2, seed)
    mbs = _mbs(w, h)
    prev = _prev_mv(w, h, pan, seed)
    g = torch.Generator("cuda").manual_seed(seed + 11)
    near = ((prev[:, :2] + 2) >> 2) + torch.randint(-3, 4, (mbs, 2), device="cuda", generator=g, dtype=torch.int32)
    near = near.clamp(-R, R)
    logged = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    logged[:, :2] = near * 4
    logged[:, 2] = prev[:, 2]
    logged[:, 3] = -(1 << 31) + (near[:, 1] + 128) * 256 + near[:, 0] + 128
    nz = torch.randint(0, 65536, (mbs, 24), device="cuda", generator=g, dtype=torch.int32)
    nz *= (torch.rand((mbs, 1), device="cuda", generator=g) < 0.5)
    return frames[1], frames[0], prev, logged, nz


def _train_params(seed):
    """He-uniform weights and small biases, layer by layer W [out][in] then b [out]."""
    rs = np.random.Generator(np.random.PCG64(seed))
    parts = []
    for i, n in _LAYERS:
        parts += [rs.uniform(-1, 1, n * i) * math.sqrt(6 / i) * (0.3 if n == 16 else 1.0), rs.uniform(-0.1, 0.1, n)]
    return np.concatenate(parts).astype(np.float32)


_LAYERS = [(8, 32), (128, 32), (128, 32), (128, 32), (96, 64), (64, 16)]


def _prepare_train(c, seed):
    S = _Stream()
    S.c, S.mbs = c, _mbs(c["w"], c["h"])
    cur, ref, S.prev, S.logged, S.nz = _train_inputs(c, seed)
    S.cur, S.ref = _nv12(*cur), _nv12(*ref)
    S.net = _proposal.Proposal(S.mbs, _train_params(seed))
    return S


def _run_train(S):
    c, P = S.c, S.net
    w, h = c["w"], c["h"]
    cw, ch = b200enc.coded(w, h)
    P.prepare(S.cur, S.ref, w, h, cw, ch, S.prev, c["search"], 512)
    P.labels(S.mbs, S.logged, S.nz)
    P.forward(S.mbs)
    P.backward(S.mbs)
    return [P.tensor(_proposal.T_LOGITS, torch.float32, (S.mbs, 16)),
            P.tensor(_proposal.T_GRADS, torch.float32, (_proposal.NUM_PARAMS,))]


def _exact_train(c, seed):
    """Logits and parameter gradients in 64 bits, no rounding anywhere."""
    (cur, _), (ref, _), prev, logged, nz = _train_inputs(c, seed)
    w, h, R = c["w"], c["h"], c["search"]
    mbw, mbh = (w + 15) // 16, (h + 15) // 16
    mbs, dev = mbw * mbh, cur.device
    # the coded-size planes: edges replicated
    iy, ix = torch.arange(mbh * 16, device=dev).clamp(max=h - 1), torch.arange(mbw * 16, device=dev).clamp(max=w - 1)
    cur, ref = cur[iy][:, ix].long(), ref[iy][:, ix].long()
    mb = torch.arange(mbs, device=dev)
    mx, my = mb % mbw, mb // mbw
    k16 = torch.arange(16, device=dev)
    rows, cols = my[:, None] * 16 + k16, mx[:, None] * 16 + k16
    cb = cur[rows[:, :, None], cols[:, None, :]]

    def block(dx, dy):
        yy, xx = (rows + dy[:, None]).clamp(0, mbh * 16 - 1), (cols + dx[:, None]).clamp(0, mbw * 16 - 1)
        return ref[yy[:, :, None], xx[:, None, :]]

    near = [(0, 0), (-1, -1), (0, -1), (1, -1), (-1, 0), (1, 0), (-1, 1), (0, 1), (1, 1)]
    cand, sad, sprev = [], [], []
    for dx, dy in near:
        m = prev[(my + dy).clamp(0, mbh - 1) * mbw + (mx + dx).clamp(0, mbw - 1)].long()
        cand.append(((m[:, :2] + 2) >> 2).clamp(-(R - 2), R - 2))
        sprev.append(m[:, 2])
    cand.append(torch.zeros_like(cand[0]))
    for v in cand:
        sad.append((cb - block(v[:, 0], v[:, 1])).abs().sum(dim=(1, 2)))
    cand, sad, sprev = torch.stack(cand, 1), torch.stack(sad, 1), torch.stack(sprev, 1)
    dup = torch.zeros((mbs, 10), dtype=torch.bool, device=dev)
    for a in range(10):
        for b in range(a):
            dup[:, a] |= (cand[:, a] == cand[:, b]).all(dim=1)
    # network input: 2x2 pels x (luma, residual at candidate 0), rows in Morton order
    res = cb - block(cand[:, 0, 0], cand[:, 0, 1])
    x = torch.stack([cb - 128, res], dim=3).double() / 64
    x = x.view(mbs, 8, 2, 8, 2, 2).permute(0, 1, 3, 2, 4, 5).reshape(mbs, 8, 8, 8)
    m64 = torch.arange(64, device=dev)
    mxy = (m64 & 1) | ((m64 >> 1) & 2) | ((m64 >> 2) & 4), ((m64 >> 1) & 1) | ((m64 >> 2) & 2) | ((m64 >> 3) & 4)
    x = x[:, mxy[1], mxy[0]].reshape(mbs * 64, 8)
    cap = lambda v: v.clamp(max=32767).double() / 4096  # noqa: E731
    c0 = cand[:, 0]
    side = torch.cat([cap(sad), cap(sad - sad.min(dim=1, keepdim=True)[0]), (cand[..., 0] - c0[:, :1]).double() / 8,
                      (cand[..., 1] - c0[:, 1:]).double() / 8, dup.double(), cap(sprev), c0.abs().double() / 32,
                      cb.diff(dim=2).abs().sum(dim=(1, 2))[:, None].double() / 7680,
                      cb.diff(dim=1).abs().sum(dim=(1, 2))[:, None].double() / 7680,
                      torch.zeros((mbs, 1), dtype=torch.float64, device=dev)], dim=1)
    p = torch.from_numpy(_train_params(seed)).to(dev).double().requires_grad_(True)
    Ws, o = [], 0
    for i, n in _LAYERS:
        Ws.append((p[o:o + n * i].view(n, i), p[o + n * i:o + n * i + n]))
        o += n * i + n
    a = x
    for li in range(4):
        a = torch.relu(a @ Ws[li][0].T + Ws[li][1])
        a = a.reshape(-1, 128) if li < 3 else a
    a = torch.relu(torch.cat([a, side], dim=1) @ Ws[4][0].T + Ws[4][1])
    z = a @ Ws[5][0].T + Ws[5][1]
    # -log of the probability of the candidates whose +-2 window holds the winner (or "none"), + 0.5 BCE no-residual
    dx, dy = (logged[:, 3] & 255) - 128, ((logged[:, 3] >> 8) & 255) - 128
    inside = ((dx[:, None] - cand[..., 0]).abs() <= 2) & ((dy[:, None] - cand[..., 1]).abs() <= 2) & ~dup
    target = torch.cat([inside, ~inside.any(dim=1, keepdim=True)], dim=1)
    valid = torch.cat([~dup, torch.ones((mbs, 1), dtype=torch.bool, device=dev)], dim=1)
    weight = (sad[:, 9] > 512).double()
    lp = z[:, :11].masked_fill(~valid, -math.inf).log_softmax(dim=1)
    ce = -lp.masked_fill(~target, -math.inf).logsumexp(dim=1)
    bce = torch.nn.functional.binary_cross_entropy_with_logits(z[:, 11], (nz == 0).all(dim=1).double(), reduction="none")
    loss = (weight * (ce + 0.5 * bce)).sum() / weight.sum().clamp(min=1)
    grad, = torch.autograd.grad(loss, p)
    return [z.detach(), grad]


# ---------------------------------------------------------------- the cases


def prepare(case, seed):
    return {"session": _prepare_session, "batch": _prepare_batch, "picture": _prepare_picture, "hevc": _prepare_hevc,
            "hevc_db": _prepare_hevc_db, "train": _prepare_train}[case["kind"]](case, seed)


class _Outputs(list):
    """A pass's outputs. Some are views of memory that the state's handles
    own, so they hold the state."""

    def __init__(self, values, state):
        super().__init__(values)
        self.state = state


def run(state):
    if hasattr(state, "net"):
        out = _run_train(state)
    else:
        out = {"session": _run_session, "batch": _run_batch, "picture": _run_picture, "hevc": _run_hevc}.get(
            getattr(state, "c", {}).get("kind"), _run_hevc_db)(state)
    return _Outputs(out, state)


def exact(case, seed):
    """Only the training case computes rounded numbers; every other output is
    whole samples, levels, vectors and bits."""
    return _exact_train(case, seed) if case["kind"] == "train" else None


NET_FLOPS = 2 * (64 * 8 * 32 + (16 + 4 + 1) * 128 * 32 + 96 * 64 + 64 * 16)  # the proposal network, per macroblock


def work(case):
    """Bytes: each picture, field and parameter read once, each output written
    once. Flops: the proposal network's (the rest is integer work)."""
    k = case["kind"]
    if k == "session":
        mbs, n = _mbs(case["w"], case["h"]), case["frames"] * case["streams"]
        intra = -(-case["frames"] // case["gop"]) * case["streams"]
        # source, reference in, reconstruction out; levels, DC, masks, modes, vectors out
        b = n * mbs * (384 + 384 + 768 + 96 + 96 + 4 + 16) + (n - intra) * mbs * 384
        return {"bytes": b, "flops": (n - intra) * mbs * NET_FLOPS if case["me"] != "full" else 0}
    if k == "batch":
        mbs = sum(_mbs(*BATCH_SIZES[(s + case["size_shift"]) % len(BATCH_SIZES)]) for s in range(case["streams"]))
        n, intra = case["steps"], -(-case["steps"] // case["gop"])
        return {"bytes": n * mbs * 1748 + (n - intra) * mbs * 384,
                "flops": (n - intra) * mbs * NET_FLOPS if case["me"] != "full" else 0}
    mbs = _mbs(case["w"], case["h"])
    if k == "picture":
        return {"bytes": mbs * (384 * 3 + 768 + 96 + 96 + 4 + 16) + (mbs * 120 if case["t8"] else 0),
                "flops": mbs * NET_FLOPS if case["me"] != "full" else 0}
    s = 1 if case.get("bits", 8) == 8 else 2
    px = case["w"] * case["h"]
    if k == "hevc":
        # reference in, four planes out; source and planes searched; residual to levels and back; modes and predictions
        return {"bytes": px * s * 5 + px * s * 5 + px // 64 * (88 + 32) + px * 2 * 4 + px * s * 3 + px // 16 * 16,
                "flops": 0}
    if k == "hevc_db":
        return {"bytes": int(px * 1.5 * s * 2) + px // 16 * 21 + px // 64 * 2, "flops": 0}
    return {"bytes": mbs * (256 * 2 + 16 * 2 + 96 + 64 * 8 * 2 + 64 * 2 + 64) + 4 * 2 * _proposal.NUM_PARAMS,
            "flops": 3 * mbs * NET_FLOPS}
