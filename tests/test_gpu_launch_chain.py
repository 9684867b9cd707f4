"""Kernels launched early on the stream (launch_early in csrc/common.cuh) wait for
the one before them: a chain of preparation, network, search, P chain,
deblocking and slice coding over changing frames gives the same bytes whether the
stream runs through or the host waits after every call, and when it is captured.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(gpu, W, H, n):
    from b200enc import synth
    seq = synth.Sequence(W, H, seed=4, pan=True, noise_patch=True)
    return [gpu.NV12.from_host(*seq.frame(t)) for t in range(n)]


@pytest.mark.parametrize("W,H", [(64, 48), (640, 480)])
@pytest.mark.parametrize("mode", [1, 3])
def test_chain_is_ordered(gpu, W, H, mode):
    import torch
    from b200enc import proposal
    n = 5
    frames = _frames(gpu, W, H, n)
    CW, CH = gpu.coded(W, H)
    mbs = (CW // 16) * (CH // 16)
    P = proposal.Proposal(mbs, proposal.init_params(7))

    def run(each=lambda: None, stream=None):
        mv = [torch.zeros((mbs, 4), dtype=torch.int32, device="cuda") for _ in range(n)]
        recs, outs = [frames[0]], []
        for t in range(1, n):
            gpu_stream = stream
            P.me(frames[t], recs[-1], W, H, CW, CH, mv[t - 1], 16, 5, 512, 0.5, mv[t], mode=mode, stream=gpu_stream)
            each()
            out, rec = gpu.Outputs(W, H), gpu.NV12(W, H)
            gpu.p_frame(frames[t], recs[-1], W, H, CW, CH, 30, mv[t], out, rec, stream=gpu_stream)
            each()
            recs.append(rec)
            outs.append(out)
        return mv, recs, outs

    def bytes_of(r):
        torch.cuda.synchronize()
        mv, recs, outs = r
        return [m.cpu().numpy() for m in mv] + [x.y.cpu().numpy() for x in recs[1:]] + [x.uv.cpu().numpy() for x in recs[1:]] + \
            [o.levels.cpu().numpy() for o in outs]

    want = bytes_of(run(torch.cuda.synchronize))
    for _ in range(10):
        for a, b in zip(bytes_of(run()), want):
            np.testing.assert_array_equal(a, b)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        run(stream=s)
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            r = run(stream=s)
    for _ in range(2):
        g.replay()
    for a, b in zip(bytes_of(r), want):
        np.testing.assert_array_equal(a, b)
