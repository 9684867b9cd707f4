"""The layer kernels of the proposal network's training (csrc/lp_train.cu) at
the edges of their 128-row tiles and 64-row chunks: one macroblock, a few, just
over one tile or chunk of a layer, and enough for every CTA to walk several.

Tolerances as in test_gpu_proposal.py, set before the first run: a forward
output within one BF16 rounding of the exact value plus 1e-5 x sum|a w|;
weight and bias gradients within 2e-2 relative L2 error of the oracle's
backward on the same activations (BF16 rounding of the inner gradients).
"""
import numpy as np
import pytest

from test_gpu_proposal import _acts, _prepared, _random_params, pr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mbw,mbh", [(1, 1), (3, 1), (13, 5), (43, 3), (100, 30)])
def test_layers_at_tile_edges(gpu, mbw, mbh):
    import torch
    from b200enc import proposal as pp
    W, H = mbw * 16, mbh * 16
    P, want, mbs, (cur, ref, RW, RH, *_rest) = _prepared(gpu, W, H, 32, "near", True, seed=20 + mbw)
    params = _random_params(6)
    P.set_params(params)
    logged = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    gpu.me_full_search_ex(cur, ref, W, H, RW, RH, 32, 5, 512, logged, flags=gpu.ME_LOG_INTEGER)
    nz = torch.zeros((mbs, 24), dtype=torch.int32, device="cuda")
    P.labels(mbs, logged, nz)
    P.forward(mbs)
    P.backward(mbs)
    torch.cuda.synchronize()
    a = _acts(P, mbs)
    ins = [a["a0"], a["y0"].reshape(-1, 128), a["y1"].reshape(-1, 128), a["y2"].reshape(-1, 128), a["f"], a["h"]]
    outs = [a["y0"], a["y1"], a["y2"], a["y3"], a["h"], a["logits"]]
    for l, (Wl, bl) in enumerate(pr.unpack(params)):
        A, Wb = ins[l].astype(np.float64), pr.bf16(Wl).astype(np.float64)
        z = A @ Wb.T + bl
        tol = 1e-5 * (np.abs(A) @ np.abs(Wb).T + np.abs(bl)) + 1e-6
        if l < 5:
            z = np.maximum(z, 0)
            tol += 2.0 ** -8 * z
        assert (np.abs(outs[l] - z) <= tol).all(), l
    state = want["state"]
    lab, norez, w = pr.labels(state, want["cand"], logged.cpu().numpy()[:, 3], nz.cpu().numpy())
    _, g5 = pr.loss_and_grad(a["logits"], lab, norez, w, (state >> 8) & 0x3FF)
    want_g = pr.backward(params, a, g5.astype(np.float32))
    got_g = P.tensor(pp.T_GRADS, torch.float32, (pp.NUM_PARAMS,)).cpu().numpy().astype(np.float64)
    for l, (wo, bo, i, n) in enumerate(pp.layer_offsets()):
        for lo, hi, what in ((wo, bo, "W"), (bo, bo + n, "b")):
            d = np.linalg.norm(got_g[lo:hi] - want_g[lo:hi])
            assert d <= 2e-2 * np.linalg.norm(want_g[lo:hi]), (l, what, d)
