"""Threads that deblock pictures of different tile shapes at once: the kernel's
shared-memory limit is the process's, and no thread's launch may fail for
another's. Results equal a single thread's.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tile_shapes_in_threads(gpu):
    import torch
    cases = [(5, 4, 0), (120, 68, 0), (120, 68, 1), (64, 40, 0), (100, 90, 1), (11, 9, 1)]
    rs = np.random.Generator(np.random.PCG64(8))

    def make(mbw, mbh):
        W, H = 16 * mbw, 16 * mbh
        src = gpu.NV12.from_host(rs.integers(0, 256, (H, W), dtype=np.uint8), rs.integers(0, 256, (H // 2, W), dtype=np.uint8))
        nz = torch.from_numpy(rs.integers(0, 2, (mbw * mbh, 24), dtype=np.int32)).cuda()
        mv = torch.from_numpy(rs.integers(-9, 10, (mbw * mbh, 4), dtype=np.int32)).cuda()
        return src, nz, mv, torch.zeros(4, dtype=torch.int32, device="cuda")

    def run(case, inputs, n):
        mbw, mbh, intra = case
        src, nz, mv, status = inputs
        dst = gpu.NV12(16 * mbw, 16 * mbh)
        stream = torch.cuda.Stream()
        for _ in range(n):
            gpu.deblock_tiles(mbw, mbh, 30, intra, nz, mv, src, dst, status, stream=stream)
        stream.synchronize()
        return dst.buf.cpu().numpy()

    inputs = [make(w, h) for w, h, _ in cases]
    torch.cuda.synchronize()
    want = [run(c, i, 1) for c, i in zip(cases, inputs)]
    with ThreadPoolExecutor(len(cases)) as pool:
        for got, w in zip(pool.map(lambda a: run(*a, 400), zip(cases, inputs)), want):
            np.testing.assert_array_equal(got, w)
