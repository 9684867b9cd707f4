"""Still pictures through the GPU slice coder: a few coded macroblocks between
skip runs of any length, at a slice's start, end and across its chunks of
macroblocks, whole slices skipped; identical bytes to the serial writer.
"""
import numpy as np
import pytest

from test_gpu_cavlc import _synthetic
from test_gpu_cavlc_serial import _gpu, _masks, serial  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mbw,mbh,ns", [(11, 9, 1), (120, 68, 1), (120, 68, 4), (50, 40, 16)])
@pytest.mark.parametrize("coded", ["none", "first", "last", "rare", "pairs", "half"])
def test_still_pictures(gpu, serial, mbw, mbh, ns, coded):  # noqa: F811
    rs = np.random.Generator(np.random.PCG64(mbw + ns + len(coded)))
    levels, dc, nz, pm, mv = _synthetic(rs, mbw, mbh, 0)
    n = mbw * mbh
    keep = np.zeros(n, bool)
    if coded == "first":
        keep[0] = True
    elif coded == "last":
        keep[-1] = True
    elif coded == "rare":
        keep[rs.integers(0, n, max(2, n // 400))] = True
    elif coded == "pairs":
        keep[5::97] = keep[6::97] = True
    elif coded == "half":
        keep[: n // 2] = rs.random(n // 2) < 0.5
    levels[~keep] = 0
    dc[~keep] = 0
    mv[:, :2] = 0
    nz = _masks(levels, None)
    heads = [(int.from_bytes(rs.bytes(16), "big") >> (128 - b), b) for b in rs.integers(0, 129, ns).tolist()]
    got = _gpu(gpu, mbw, mbh, 27, 0, ns, levels, dc, nz, pm, mv, headers=heads)
    want = serial(mbw, mbh, 27, 0, ns, levels, dc, nz, pm, mv, headers=heads)
    for s, (g, w) in enumerate(zip(got, want)):
        assert g == w, f"slice {s}: {len(g)} vs {len(w)} bytes"
