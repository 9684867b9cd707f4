"""The full search's elimination (csrc/me.cu) on content that drives it to its
edges: pictures where every candidate's bound survives (uniform noise, flat
pictures whose candidates all tie), where almost none does (steep ramps),
where bounds equal costs (8x8 tiles of one value: the winner must still be
the first in raster order), and saturated checkerboards. Vectors and SADs
equal the oracle's exhaustive search, grid and list form, both ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _picture(rs, kind, W, H, shift):
    yy, xx = np.mgrid[0:H, 0:W]
    if kind == "noise":
        return rs.integers(0, 256, (H, W)).astype(np.uint8)
    if kind == "flat":
        return np.full((H, W), 90 + 2 * shift, np.uint8)
    if kind == "ramp":
        return np.clip(4 * (xx + 3 * shift) + 3 * (yy - shift) - 200 + rs.integers(0, 3, (H, W)), 0, 255).astype(np.uint8)
    if kind == "tiles":
        return ((((xx + 3 * shift) // 8 + (yy + 2 * shift) // 8) % 5) * 50).astype(np.uint8)
    return ((((xx + yy + shift) & 1) * 255)).astype(np.uint8)


@pytest.mark.parametrize("kind", ["noise", "flat", "ramp", "tiles", "checker"])
@pytest.mark.parametrize("W,H", [(16, 16), (80, 48), (150, 134)])
@pytest.mark.parametrize("rng,lam", [(16, 0), (16, 5), (32, 5), (32, 1023)])
def test_elimination_is_exhaustive(gpu, oracle_mod, kind, W, H, rng, lam):
    import torch
    rs = np.random.Generator(np.random.PCG64(W * 10 + rng + lam))
    ry, cy = _picture(rs, kind, W, H, 0), _picture(rs, kind, W, H, 1)
    uv = np.full((H // 2, W), 128, np.uint8)
    ref, cur = gpu.NV12.from_host(ry, uv), gpu.NV12.from_host(cy, uv)
    mbs = ((W + 15) // 16) * ((H + 15) // 16)
    f = oracle_mod.frame(W, H, 26, coded_clamp=False)
    for zt in (512, -1):
        want = oracle_mod.me_frame(f, np.ascontiguousarray(cy), np.ascontiguousarray(ry), rng, lam, zt)
        mv = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
        gpu.me_full_search(cur, ref, W, H, W, H, rng, lam, zt, mv)
        lst = torch.arange(mbs - 1, -1, -1, dtype=torch.int32, device="cuda")
        cnt = torch.tensor([mbs], dtype=torch.int32, device="cuda")
        mv2 = torch.zeros_like(mv)
        gpu.me_full_search_ex(cur, ref, W, H, W, H, rng, lam, zt, mv2, lst, cnt, mbs)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(mv.cpu().numpy(), want, err_msg=f"grid zt {zt}")
        np.testing.assert_array_equal(mv2.cpu().numpy(), want, err_msg=f"list zt {zt}")
