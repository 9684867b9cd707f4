"""The intra wavefront's row groups (csrc/intra.cu) at their edges: rows longer
than the 32-macroblock line ring, pictures of less than, exactly and more than
a group's four rows, slices that start anywhere in a row, pictures that end
inside a macroblock with either clamp, both corner rules, and fewer CTAs than
groups (one CTA doing all luma, then all chroma). Equal to the oracle's
raster-order frame."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(16, 16), (40, 64), (520, 80), (1064, 40), (200, 216)])
@pytest.mark.parametrize("slices,corner", [(1, 1), (3, 1), (3, 0), (7, 1)])
@pytest.mark.parametrize("coded", [True, False])
@pytest.mark.parametrize("ctas", [0, 1, 3])
def test_row_groups_match_oracle(gpu, oracle_mod, W, H, slices, corner, coded, ctas):
    import torch
    mbw, mbh = (W + 15) // 16, (H + 15) // 16
    slices = min(slices, mbw * mbh)
    rs = np.random.Generator(np.random.PCG64(W * 7 + H + slices + corner))
    base = rs.integers(40, 216, (H // 8 + 2, W // 8 + 2)).astype(np.float64)
    y = np.clip(np.kron(base, np.ones((8, 8)))[:H, :W] + rs.normal(0, 8, (H, W)), 0, 255).astype(np.uint8)
    y[:, : W // 2] = np.clip(np.arange(H)[:, None] * 2 + np.arange(W // 2) * 3 - 100, 0, 255).astype(np.uint8)  # Plane
    uv = np.clip(128 + rs.normal(0, 30, (H // 2, W)), 0, 255).astype(np.uint8)
    cur = gpu.NV12.from_host(y, uv)
    CW, CH = gpu.coded(W, H)
    RW, RH = (CW, CH) if coded else (W, H)
    for qp in (3, 24, 41):
        out, rec, scr = gpu.Outputs(W, H), gpu.NV12(W, H), gpu.scratch(mbh)
        gpu.i_frame(cur, W, H, RW, RH, qp, slices, out, rec, scr, ctas=ctas, flags=corner)
        torch.cuda.synchronize()
        assert gpu.wavefront_status(scr) == 0
        f = oracle_mod.frame(W, H, qp, coded_clamp=coded, num_slices=slices, corner_check=bool(corner))
        ry, ruv = np.zeros((CH, CW), np.uint8), np.zeros((CH // 2, CW), np.uint8)
        want = oracle_mod.i_frame(f, y, uv, ry, ruv)
        got = out.host()
        for k in ("levels", "dc", "nz", "pred_mode", "mv"):
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} qp {qp}")
        np.testing.assert_array_equal(rec.y.cpu().numpy()[:RH, :RW], ry[:RH, :RW])
        np.testing.assert_array_equal(rec.uv.cpu().numpy()[: RH // 2, : RW // 2 * 2], ruv[: RH // 2, : RW // 2 * 2])
