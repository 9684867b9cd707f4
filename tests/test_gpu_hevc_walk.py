"""The HEVC motion search (csrc/hevc.cu) against a one-candidate-at-a-time walk
in Python, from the contract in include/b200enc.h: pitches and addresses of
every alignment, both sample types, no starting point, repeated and far ones,
CUs at every edge. All results are whole numbers and equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 11


def _mvd_bits(d):
    a = abs(int(d))
    return 1 if a == 0 else 3 if a == 1 else 5 + 2 * (((a - 2) // 2 + 1).bit_length() - 1)


def _walk(src, planes, w, h, qpel, shift, job):
    cx, cy = int(job["cu_x"]), int(job["cu_y"])
    cu = src[cy:cy + 8, cx:cx + 8].astype(np.int64)

    def block(x, y):
        p = planes[(x >> 1 & 1) + 2 * (y >> 1 & 1)]
        return p[(y >> 2) + M:(y >> 2) + M + 8, (x >> 2) + M:(x >> 2) + M + 8].astype(np.int64)

    def sad(x, y):
        x = min(max(cx * 4 + x, -(M - 2) * 4), (w - 8 + M - 2) * 4)
        y = min(max(cy * 4 + y, -(M - 2) * 4), (h - 8 + M - 2) * 4)
        b = block(x - x % 2, y - y % 2)
        if x % 2 or y % 2:
            b = (b + block(x + x % 2, y + y % 2) + 1) >> 1
        return int(np.abs(cu - b).sum()) >> shift

    def bits(p, x, y):
        return _mvd_bits(x - int(p[0])) + _mvd_bits(y - int(p[1]))

    best = [None, 0, 0, 0]  # cost, x, y, sad

    def score(x, y):
        s = sad(x, y)
        c = s * 256 + int(job["lambda_q8"]) * min(bits(p, x, y) for p in job["mvp"])
        if best[0] is None or c < best[0]:
            best[:] = [c, x, y, s]
            return True
        return False

    lim = (-cx - 8, w - cx, -cy - 8, h - cy)
    for sx, sy in job["starts"][:max(0, int(job["n_starts"]))].astype(int):
        score(min(max((sx + 2) >> 2, lim[0]), lim[1]) * 4, min(max((sy + 2) >> 2, lim[2]), lim[3]) * 4)
    x0, y0 = best[1] // 4, best[2] // 4
    bx, by, back = x0, y0, -1
    for _ in range(32):
        won = -1
        for k, (dx, dy) in enumerate(((-1, 0), (1, 0), (0, -1), (0, 1))):
            x, y = bx + dx, by + dy
            if k == back or not (lim[0] <= x <= lim[1] and lim[2] <= y <= lim[3]) or max(abs(x - x0), abs(y - y0)) > 64:
                continue
            if score(x * 4, y * 4):
                won = k
        if won < 0:
            break
        bx, by = best[1] // 4, best[2] // 4
        back = won ^ 1
    mx, my = bx * 4, by * 4
    for st in ((2, 1) if qpel else (2,)):
        c0x, c0y = mx, my
        for dx, dy in ((-1, -1), (0, -1), (1, -1), (-1, 0), (1, 0), (-1, 1), (0, 1), (1, 1)):
            if score(c0x + dx * st, c0y + dy * st):
                mx, my = best[1], best[2]
    idx = int(bits(job["mvp"][1], mx, my) < bits(job["mvp"][0], mx, my))
    return (mx, my), idx, best[0], best[3]


@pytest.mark.parametrize("bits", [8, 10])
@pytest.mark.parametrize("w,h,pad,qpel", [(8, 8, 0, 1), (24, 16, 1, 1), (72, 40, 2, 0), (75, 43, 3, 1)])
def test_walk(gpu, w, h, pad, qpel, bits):
    import torch
    rs = np.random.Generator(np.random.PCG64(w + pad + bits))
    top, dt = 1 << bits, np.uint8 if bits == 8 else np.uint16
    yy, xx = np.mgrid[0:h + 2 * M, 0:w + 2 * M]
    base = np.clip(top * (0.5 + 0.4 * np.sin(xx / 5) * np.cos(yy / 7)), 0, top - 1)
    planes = np.zeros((4, h + 2 * M, w + 2 * M + pad), dt)
    for k in range(4):  # any samples will do: the search only reads the planes
        planes[k, :, :w + 2 * M] = np.clip(base + rs.integers(-9, 10, base.shape), 0, top - 1)
    planes[:, :4] = rs.integers(0, top, planes[:, :4].shape)
    src = np.zeros((h, w + pad), dt)
    src[:, :w] = np.clip(base[M + 1:M + 1 + h, M + 2:M + 2 + w] + rs.integers(-9, 10, (h, w)), 0, top - 1)
    cus = [(x, y) for y in sorted({*range(0, h - 7, 8), h - 8}) for x in sorted({*range(0, w - 7, 8), w - 8})]
    jobs = np.zeros(len(cus), gpu.HEVC_ME_JOB)
    for j, (x, y) in enumerate(cus):
        jobs[j]["cu_x"], jobs[j]["cu_y"] = x, y
        jobs[j]["mvp"] = rs.integers(-30, 31, (2, 2))
        st = rs.integers(-30, 31, (16, 2))
        st[3:6] = st[0]
        st[::5] = rs.choice([-32768, -700, 900, 32767], st[::5].shape)
        jobs[j]["starts"] = st
        jobs[j]["n_starts"] = (0, 1, 16, 5, 4, 9, 20)[j % 7]
        jobs[j]["lambda_q8"] = int(rs.integers(0, 4000))
    view = np.uint8 if bits == 8 else np.int16
    src_d = torch.from_numpy(src.view(view)).cuda()
    planes_d = torch.from_numpy(planes.view(view)).cuda()
    res_d = torch.zeros(len(jobs) * gpu.HEVC_ME_RESULT.itemsize, dtype=torch.uint8, device="cuda")
    gpu.hevc_motion_search(src_d, w, h, planes_d, M, qpel, torch.from_numpy(jobs.view(np.uint8)).cuda(), res_d)
    torch.cuda.synchronize()
    got = res_d.cpu().numpy().view(gpu.HEVC_ME_RESULT)
    for j, job in enumerate(jobs):
        g = got[j]
        assert (tuple(map(int, g["mv"])), int(g["mvp_idx"]), int(g["cost_q8"]), int(g["sad"])) == \
            _walk(src, planes, w, h, qpel, 0 if bits == 8 else 2, job), cus[j]
