"""Kernels launched early on the stream (launch_early in csrc/common.cuh) wait for the
one before them, beyond the search and the P chain of test_gpu_launch_chain.py: tile
deblocking into the next reference and the three kernels of slice coding, the staging
of vectors and status with the entropy coder off, beside and instead of the level
staging, a training step's layers, and the HEVC primitives. Each chain over changing
inputs leaves what it leaves when the host waits after every call, with buffers of
its own per picture and with the same ones reused, and when it is captured.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sequence(gpu, W, H, n):
    from b200enc import synth
    seq = synth.Sequence(W, H, seed=11, pan=True, noise_patch=True)
    return [seq.frame(t) for t in range(n)]


def _same(a, b):
    assert len(a) == len(b)
    for i, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg=f"output {i}")


class _Coder:
    """b200enc_cavlc_slices into buffers of its own."""

    def __init__(self, gpu, W, H, ns, out):
        import torch
        CW, CH = gpu.coded(W, H)
        mbs = CW * CH // 256
        self.gpu, self.cap, self.ns = gpu, (mbs * 2560 // ns + 4096) // 4 * 4, ns
        self.bits = torch.zeros(ns * self.cap, dtype=torch.uint8, device="cuda")
        self.nbytes = torch.zeros(ns, dtype=torch.int32, device="cuda")
        n = gpu.lib().b200enc_cavlc_scratch_bytes(CW // 16, CH // 16)
        self.scratch = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
        vp, sp = ctypes.c_void_p, (self.scratch.data_ptr() + 255) // 256 * 256
        self.prm = gpu.CavlcParams(CW // 16, CH // 16, 30, 0, ns, 4, vp(out.levels.data_ptr()), vp(out.dc.data_ptr()),
                                   vp(out.nz.data_ptr()), None, vp(out.mv.data_ptr()), None, None,
                                   vp(self.bits.data_ptr()), self.cap, vp(self.nbytes.data_ptr()), None, vp(sp), n, 0, None)

    def __call__(self, stream):
        self.gpu._check(self.gpu.lib().b200enc_cavlc_slices(ctypes.byref(self.prm), self.gpu._stream(stream)), "cavlc")

    def slices(self):
        n, b = self.nbytes.cpu().numpy(), self.bits.cpu().numpy()
        return [b[k * self.cap:k * self.cap + n[k]] for k in range(self.ns)]


@pytest.mark.parametrize("W,H", [(64, 48), (640, 480)])
@pytest.mark.parametrize("reuse", [False, True])
def test_deblocking_and_slice_coding(gpu, W, H, reuse):
    import torch
    n, ns = 6, 2
    frames = [gpu.NV12.from_host(*f) for f in _sequence(gpu, W, H, n)]
    CW, CH = gpu.coded(W, H)

    def make():
        # reused: one set of outputs, two references; else a set per picture
        sets = 1 if reuse else n
        outs = [gpu.Outputs(W, H) for _ in range(sets)]
        recs = [gpu.NV12(W, H) for _ in range(sets)]
        refs = [gpu.NV12(W, H) for _ in range(2 if reuse else n)]
        sts = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(sets)]
        return outs, recs, refs, sts, [_Coder(gpu, W, H, ns, o) for o in outs]

    def run(bufs, each=lambda: None, stream=None):
        outs, recs, refs, sts, coders = bufs
        refs[0].buf.copy_(frames[0].buf)
        for t in range(1, n):
            k = t % len(outs)
            ref, dst, o, rec = refs[(t - 1) % len(refs)], refs[t % len(refs)], outs[k], recs[k]
            gpu.me_full_search(frames[t], ref, W, H, CW, CH, 16, 5, 512, o.mv, stream=stream)
            each()
            gpu.p_frame(frames[t], ref, W, H, CW, CH, 30, o.mv, o, rec, stream=stream)
            each()
            gpu.deblock_tiles(CW // 16, CH // 16, 30, 0, o.nz, o.mv, rec, dst, sts[k], stream=stream)
            each()
            coders[k](stream)
            each()

    def left(bufs):
        torch.cuda.synchronize()
        outs, recs, refs, sts, coders = bufs
        res = [x.cpu().numpy() for o in outs for x in (o.mv, o.levels, o.dc, o.nz, o.pred_mode)]
        res += [x.buf.cpu().numpy() for x in recs + refs] + [s.cpu().numpy() for s in sts]
        for c in coders:
            res += c.slices()
        return res

    bufs = make()
    run(bufs, torch.cuda.synchronize)
    want = left(bufs)
    for _ in range(10):
        bufs = make()
        torch.cuda.synchronize()
        run(bufs)
        _same(left(bufs), want)
    s, g, bufs = torch.cuda.Stream(), torch.cuda.CUDAGraph(), make()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        run(bufs, stream=s)
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            run(bufs, stream=s)
    for _ in range(2):
        g.replay()
    _same(left(bufs), want)


@pytest.mark.parametrize("W,H", [(80, 64), (640, 480)])
@pytest.mark.parametrize("entropy", [0, 1, 2])
@pytest.mark.parametrize("deblock", [0, 1])
def test_staged_outputs(gpu, W, H, entropy, deblock):
    import torch
    n, ns = 6, 2
    src = _sequence(gpu, W, H, n)
    hdr, hb = np.zeros((ns, 16), np.uint8), np.full(ns, 27, np.int32)
    hdr[:, 0] = 0x9A

    def run(wait):
        ctx = gpu.Context()
        ctx.configure(search_range=16, deblock=deblock)
        if entropy:
            ctx.set_entropy(entropy)
        imgs = [ctx.create_image(W, H) for _ in range(2)]
        nal, res, last = np.zeros(W * H * 4 + 65536, np.uint8), [], None

        def collect(t, slot):
            assert ctx.sync(slot) == 0
            got = ctx.staging(slot)
            res.extend(got[k].copy() for k in (("mv",) if entropy == 2 else ("mv", "levels", "dc", "nz", "pred_mode")))
            if entropy:
                m = ctx.slice_nals(slot, hdr, hb, 2, 1, nal)
                res.append(nal[:m].copy())

        for t in range(n):
            img, mem = imgs[t & 1]
            ctx.upload(img, mem, *src[t])
            if wait:
                torch.cuda.synchronize()
            slot = ctx.encode(img, W, H, 30, t % 4 == 0, ns)
            if wait:
                torch.cuda.synchronize()
            if last is not None:
                collect(*last)
            last = (t, slot)
        collect(*last)
        y, uv = ctx.recon_host()
        res += [y.copy(), uv.copy()]
        for img, mem in imgs:
            ctx.destroy_image(img, mem)
        ctx.close()
        return res

    want = run(True)
    for _ in range(3):
        _same(run(False), want)


def test_training_step(gpu):
    """Activations are equal; gradients are sums of FP32 atomics, whose order is free:
    at most 296 shares added in any order are within 296 x 2^-24 of the sum of their
    magnitudes, under 1e-3 of the layer's norm for cancellation up to fiftyfold."""
    import torch
    from b200enc import proposal as pp
    W, H = 640, 480
    CW, CH = gpu.coded(W, H)
    mbs = CW * CH // 256
    a, b = [gpu.NV12.from_host(*f) for f in _sequence(gpu, W, H, 2)]
    rs = np.random.Generator(np.random.PCG64(5))
    prev = np.zeros((mbs, 4), np.int32)
    prev[:, :2] = rs.integers(-40, 41, (mbs, 2))
    prev = torch.from_numpy(prev).cuda()
    logged = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    gpu.me_full_search_ex(b, a, W, H, CW, CH, 16, 5, 512, logged, flags=gpu.ME_LOG_INTEGER)
    nz = torch.from_numpy(rs.integers(0, 2, (mbs, 24)).astype(np.int32)).cuda()

    def run(each):
        P = pp.Proposal(mbs, pp.init_params(3))
        torch.cuda.synchronize()
        for call in (lambda: P.prepare(b, a, W, H, CW, CH, prev, 16, 512), lambda: P.labels(mbs, logged, nz),
                     lambda: P.forward(mbs), lambda: P.backward(mbs)):
            call()
            each()
        torch.cuda.synchronize()
        acts = [P.tensor(k, torch.int16, (mbs, w)).cpu().numpy() for k, w in ((2, 512), (3, 2048), (4, 512), (5, 128), (6, 96), (7, 64))]
        acts.append(P.tensor(pp.T_LOGITS, torch.int32, (mbs, 16)).cpu().numpy())
        return acts, P.tensor(pp.T_GRADS, torch.float32, (pp.NUM_PARAMS,)).cpu().numpy().astype(np.float64)

    want, want_g = run(torch.cuda.synchronize)
    for _ in range(5):
        acts, g = run(lambda: None)
        _same(acts, want)
        for wo, bo, i, o in pp.layer_offsets():
            for lo, hi in ((wo, bo), (bo, bo + o)):
                assert np.linalg.norm(g[lo:hi] - want_g[lo:hi]) <= 1e-3 * np.linalg.norm(want_g[lo:hi])


@pytest.mark.parametrize("bits", [8, 10])
def test_hevc_primitives(gpu, bits):
    import torch
    import hevc_db_inputs as hdi
    W, H, M, n = 208, 136, 16, 4
    dt = torch.uint8 if bits == 8 else torch.int16
    pics = [torch.from_numpy((f[0].astype(np.int16) << (bits - 8))).to(dt).cuda().contiguous()
            for f in _sequence(gpu, W, H, n + 1)]
    ys, xs = np.mgrid[0:H - 7:8, 0:W - 7:8]
    jobs = np.zeros(xs.size, gpu.HEVC_ME_JOB)
    jobs["cu_x"], jobs["cu_y"], jobs["n_starts"], jobs["lambda_q8"] = xs.reshape(-1), ys.reshape(-1), 2, 900
    jobs["starts"][:, 1] = 9
    jobs = torch.from_numpy(jobs.view(np.uint8)).cuda()
    resid = [torch.randint(-200, 201, (xs.size, 64), dtype=torch.int16, device="cuda",
                           generator=torch.Generator("cuda").manual_seed(t)) for t in range(n)]
    case = hdi.make_case(3, 416, 240, bit_depth=bits, log2_ctb=5)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()  # noqa: E731
    maps = {k: dev(case[k]) for k in ("edges", "mvf", "cbf", "qp_y", "no_filter", "slice_of_ctb", "tile_of_ctb")
            if case[k] is not None}
    sf = dev(case["slice_filter"])
    planes0 = [dev(p) for p in case["planes"]]

    def make():
        hp = torch.zeros((4, H + 2 * M, 256), dtype=dt, device="cuda")
        res = torch.zeros(xs.size * gpu.HEVC_ME_RESULT.itemsize, dtype=torch.uint8, device="cuda")
        return hp, res, torch.zeros_like(resid[0]), torch.zeros_like(resid[0]), [p.clone() for p in planes0]

    def run(bufs, each=lambda: None):
        hp, res, coeff, back, planes = bufs
        q = hdi.params(gpu, dict(case, **maps), lambda t: t.data_ptr(), planes=planes, slice_filter=None)
        q.slice_filter, q.n_slice_filter = sf.data_ptr(), len(case["slice_filter"])
        for t in range(n):
            for call in (lambda: gpu.hevc_build_hpel(pics[t], W, H, M, hp),
                         lambda: gpu.hevc_motion_search(pics[t + 1], W, H, hp, M, 1, jobs, res),
                         lambda: gpu.hevc_transform_quant_8x8(resid[t], coeff, 30, 2, bits),
                         lambda: gpu.hevc_dequant_itransform_8x8(coeff, back, 30, bits),
                         lambda: gpu.hevc_transform_quant_4x4(back.view(-1, 16), coeff.view(-1, 16), 30, 1, 2, bits),
                         lambda: gpu.hevc_dequant_itransform_4x4(coeff.view(-1, 16), back.view(-1, 16), 30, 1, bits),
                         lambda: gpu.hevc_deblock(q)):
                call()
                each()

    def left(bufs):
        torch.cuda.synchronize()
        hp, res, coeff, back, planes = bufs
        return [x.cpu().numpy() for x in [hp, res, coeff, back] + planes]

    bufs = make()
    run(bufs, torch.cuda.synchronize)
    want = left(bufs)
    for _ in range(10):
        bufs = make()
        torch.cuda.synchronize()
        run(bufs)
        _same(left(bufs), want)
