"""HEVC deblocking on either side of the line between eight and 32 segments a warp
(csrc/hevc_deblock.cu): a picture stacked on itself until it is over the line, with no
edge along the seams, filters to the picture's own result, copy by copy; pictures
just under and just over the line; every option of the maps, planes whose rows are not
aligned for whole words, and the buffers' padding left alone.
"""
import numpy as np
import pytest

import hevc_db_inputs as hdi

pytestmark = pytest.mark.gpu
FEW = 110000


def _dev(a):
    import torch
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def _filter(gpu, case):
    import torch
    planes = [_dev(p) for p in case["planes"]]
    bufs = {k: _dev(case[k]) for k in ("edges", "mvf", "cbf", "qp_y", "no_filter", "slice_of_ctb", "tile_of_ctb")}
    sf = _dev(case["slice_filter"])
    q = hdi.params(gpu, dict(case, **bufs), lambda t: t.data_ptr(), planes=planes, slice_filter=None)
    q.slice_filter, q.n_slice_filter = sf.data_ptr(), len(case["slice_filter"])
    gpu.hevc_deblock(q)
    torch.cuda.synchronize()
    return [t.cpu().numpy().view(p.dtype).reshape(p.shape) for t, p in zip(planes, case["planes"])]


def _stack(case, n):
    """n copies of the case's picture, one under the other."""
    H, cs, cb = case["height"], 1 << case["log2_ctb"], 1 << case["log2_min_cb"]
    assert H % cs == 0
    rows = {"edges": H // 8, "mvf": H // 4, "cbf": H // 4, "qp_y": H // cb, "no_filter": H // cb}
    big = dict(case, height=H * n)
    big["planes"] = [np.concatenate([p] * n) for p in case["planes"]]
    for k, r in rows.items():
        if case[k] is not None:
            big[k] = np.concatenate([case[k][:r]] * n)
    big["edges"] = big["edges"].copy()
    big["edges"][::H // 8] &= ~np.uint8(2)
    for k in ("slice_of_ctb", "tile_of_ctb"):
        if case[k] is not None:
            big[k] = np.concatenate([case[k]] * n)
    return big


@pytest.mark.parametrize("bit_depth", [8, 10])
@pytest.mark.parametrize("kw,pad", [(dict(), 32), (dict(slices=3, tiles=2, lossless=0.1, cb_qp_offset=-5, cr_qp_offset=7,
                                                        qp_range=(-12, 51)), 30), (dict(intra=True), 32),
                                    (dict(slices=2, tiles=3, across_tiles=True, qp_range=(40, 51)), 33)])
def test_stacked_picture(gpu, bit_depth, kw, pad):
    case = hdi.make_case(21 + bit_depth + pad, 416, 256, bit_depth=bit_depth, log2_ctb=6, log2_min_cb=3, pad=pad, **kw)
    case["edges"] = case["edges"].copy()
    n = FEW // ((416 // 8) * (256 // 4)) + 1
    small, big = _filter(gpu, case), _filter(gpu, _stack(case, n))
    for c in range(3):
        h = small[c].shape[0]
        assert (small[c] != case["planes"][c]).any()
        for k in range(n):
            np.testing.assert_array_equal(big[c][k * h:(k + 1) * h], small[c], err_msg=f"plane {c}, copy {k}")


@pytest.mark.parametrize("extra", [0, 1])
def test_at_the_line(gpu, extra):
    """64 samples wide: the last picture under the line and the first over it, equal
    where they overlap (the taller one's last rows aside)."""
    h = FEW // 8 * 4 // 64 * 64
    case = hdi.make_case(5, 64, 256, log2_ctb=6, slices=1)
    n = h // 256 + extra
    assert (64 // 8 * (n * 256 // 4) > FEW) == bool(extra)
    small, big = _filter(gpu, case), _filter(gpu, _stack(case, n))
    for c in range(3):
        hh = small[c].shape[0]
        for k in (0, 1, n // 2, n - 1):
            np.testing.assert_array_equal(big[c][k * hh:(k + 1) * hh], small[c])
