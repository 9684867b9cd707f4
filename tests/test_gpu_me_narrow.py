"""The full search with one thread per column (csrc/me.cu), which frames of many
macroblocks and long lists take: the content that drives the elimination to its
edges (test_gpu_me_elimination.py, whose pictures take the wide form) on frames
above the line between the forms, lambda at both ends, ragged right and bottom
macroblocks, as a grid and as a list, whose line lies at a capacity of 100
macroblocks per SM. Vectors and SADs equal the oracle's exhaustive search.
"""
import numpy as np
import pytest

from test_gpu_me_elimination import _picture

pytestmark = pytest.mark.gpu

KINDS = ["noise", "flat", "ramp", "tiles", "checker"]


def _pair(gpu, kind, W, H, seed):
    rs = np.random.Generator(np.random.PCG64(seed))
    ry, cy = _picture(rs, kind, W, H, 0), _picture(rs, kind, W, H, 1)
    uv = np.full((H // 2, W), 128, np.uint8)
    return cy, ry, gpu.NV12.from_host(cy, uv), gpu.NV12.from_host(ry, uv)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rng,lam,W,H", [(16, 0, 598, 522), (16, 1023, 598, 522), (32, 0, 790, 790), (32, 1023, 790, 790)])
def test_grid(gpu, oracle_mod, kind, rng, lam, W, H):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mbs = ((W + 15) // 16) * ((H + 15) // 16)
    assert mbs > (8 if rng == 16 else 16) * sms
    cy, ry, cur, ref = _pair(gpu, kind, W, H, rng + lam)
    mv = torch.zeros((mbs, 4), dtype=torch.int32, device="cuda")
    gpu.me_full_search(cur, ref, W, H, W, H, rng, lam, -1, mv)
    torch.cuda.synchronize()
    f = oracle_mod.frame(W, H, 26, coded_clamp=False)
    want = oracle_mod.me_frame(f, np.ascontiguousarray(cy), np.ascontiguousarray(ry), rng, lam, -1)
    np.testing.assert_array_equal(mv.cpu().numpy(), want)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rng,lam", [(16, 5), (32, 1023)])
def test_list(gpu, oracle_mod, kind, rng, lam):
    import torch
    W, H = 2554, 1530
    mbw, mbh = 160, 96
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert mbw * mbh > 100 * sms
    cy, ry, cur, ref = _pair(gpu, kind, W, H, 3 * rng)
    pick = [0, mbw - 1, mbw * mbh - 1, mbw * (mbh - 1), 50 * mbw + 77, 2 * mbw + 3, 95 * mbw + 80, 40 * mbw + 159]
    lst = torch.full((mbw * mbh,), 7, dtype=torch.int32, device="cuda")
    lst[:len(pick)] = torch.tensor(pick, dtype=torch.int32, device="cuda")
    cnt = torch.tensor([len(pick)], dtype=torch.int32, device="cuda")
    mv = torch.full((mbw * mbh, 4), -9, dtype=torch.int32, device="cuda")
    gpu.me_full_search_ex(cur, ref, W, H, W, H, rng, lam, -1, mv, lst, cnt, mbw * mbh)
    torch.cuda.synchronize()
    got = mv.cpu().numpy()
    f = oracle_mod.frame(W, H, 26, coded_clamp=False)
    cy, ry = np.ascontiguousarray(cy), np.ascontiguousarray(ry)
    for mb in pick:
        mby, mbx = divmod(mb, mbw)
        key = oracle_mod.me_rect_key(f, cy, ry, rng, lam, mbx, mby, -rng, -rng, rng, rng)
        my, mx = divmod(key & 0x3FFF, 2 * rng + 1)
        mx, my = mx - rng, my - rng
        want = oracle_mod.me_refine(f, cy, ry, mbx, mby, mx, my, (key >> 14) - lam * (abs(mx) + abs(my)))
        np.testing.assert_array_equal(got[mb], want, err_msg=f"mb {mb}")
    rest = np.ones(mbw * mbh, bool)
    rest[pick] = False
    assert (got[rest] == -9).all()
