"""A kernel launched early (launch_early in csrc/common.cuh) waits for everything in
front of it on its stream, not only for the kernel: an event of another stream, and a
copy from page-locked memory. The input arrives some milliseconds late; the result is
that of the input's new contents.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("late", ["event", "copy"])
@pytest.mark.parametrize("what", ["p_frame", "deblock_tiles", "prepare", "hevc_build_hpel"])
def test_waits_for_what_is_in_front(gpu, late, what):
    import torch
    from b200enc import proposal, synth
    W, H = 320, 192
    mbw, mbh = W // 16, H // 16
    mbs = mbw * mbh
    seq = synth.Sequence(W, H, seed=3, pan=True)
    old, new = (gpu.NV12.from_host(*seq.frame(t)) for t in (0, 5))
    ref = gpu.NV12.from_host(*seq.frame(4))
    mv = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    out, dst = gpu.Outputs(W, H), gpu.NV12(W, H)
    out.nz.fill_(3)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    planes = torch.zeros((4, H + 32, 384), dtype=torch.uint8, device="cuda")
    P = proposal.Proposal(mbs, proposal.init_params(1))

    def call(cur, stream):
        if what == "p_frame":
            gpu.p_frame(cur, ref, W, H, W, H, 30, mv, out, dst, stream=stream)
        elif what == "deblock_tiles":
            gpu.deblock_tiles(mbw, mbh, 40, 0, out.nz, mv, cur, dst, status, stream=stream)
        elif what == "prepare":
            P.prepare(cur, ref, W, H, W, H, mv, 16, 512, stream=stream)
        else:
            gpu.hevc_build_hpel(cur.y[:, :W], W, H, 16, planes, stream=stream)

    def result():
        torch.cuda.synchronize()
        return [x.cpu().numpy().copy() for x in (out.levels, out.nz, dst.buf, planes, P.tensor(2, torch.int16, (mbs, 512)))]

    call(new, torch.cuda.current_stream())
    want = result()
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    host = new.buf.cpu().pin_memory()
    for _ in range(5):
        cur = gpu.NV12(W, H)
        cur.buf.copy_(old.buf)
        for x in (out.levels, dst.buf, planes):
            x.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            call(cur, s)  # a kernel in front, of the old contents
        if late == "event":
            with torch.cuda.stream(side):
                torch.cuda._sleep(4_000_000)
                cur.buf.copy_(new.buf)
            s.wait_stream(side)
        else:
            with torch.cuda.stream(s):
                torch.cuda._sleep(4_000_000)
                cur.buf.copy_(host, non_blocking=True)
        with torch.cuda.stream(s):
            call(cur, s)
        for a, b in zip(result(), want):
            np.testing.assert_array_equal(a, b)
