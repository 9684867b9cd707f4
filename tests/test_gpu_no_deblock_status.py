"""A frame without the deblocking pass reports success whatever the pass's
status word holds: the device memory a context gets is filled first, so an
unwritten word would read as an error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("intra_first", [True, False])
def test_status_without_deblocking(gpu, intra_first):
    import torch
    W, H = 320, 200
    rs = np.random.Generator(np.random.PCG64(3))
    junk = [torch.full((1 << k,), 0xA5, dtype=torch.uint8, device="cuda") for k in range(9, 24)]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()  # back to the driver: the context's allocations may reuse it
    ctx = gpu.Context()
    ctx.configure(search_range=16, coded_clamp=True, deblock=0)
    img, mem = ctx.create_image(W, H)
    for t in range(3):
        ctx.upload(img, mem, rs.integers(0, 256, (H, W), dtype=np.uint8), rs.integers(0, 256, (H // 2, W), dtype=np.uint8))
        slot = ctx.encode(img, W, H, 27, intra_first and t == 0)
        assert ctx.sync(slot) == 0
