"""Kernels placed while the one before them drains still see all of its writes: chains of scans whose input is the last
one's output, with other kernels between them, on a side stream and in a captured graph; and frames one after another
into the same buffers."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _chain(scan, torch, x, out, n, steps):
    s = torch.cuda.current_stream().cuda_stream
    for k in range(steps):
        scan(x.data_ptr(), out.data_ptr(), n, s)
        if k % 2:
            torch.remainder(out[1:], 1009, out=x)     # another library's kernel reads and writes between
        else:
            scan(out.data_ptr(), out.data_ptr(), n, s)   # in place, straight after
            x.copy_(out[1:]).bitwise_and_(0xFFFF)


def _want(a, steps):
    x = a.astype(np.int64)
    for k in range(steps):
        out = np.concatenate([[0], np.cumsum(x)]).astype(np.int32)
        if k % 2:
            x = np.remainder(out[1:], 1009).astype(np.int64)
        else:
            out = np.concatenate([[0], np.cumsum(out[:-1].astype(np.int64))]).astype(np.int32)
            x = (out[1:] & 0xFFFF).astype(np.int64)
    return x.astype(np.int32), out


@pytest.mark.parametrize("n", [1, 1000, 32768, 32769, 700001])
def test_chained_scans(gpu, n):
    import torch
    steps = 9
    a = np.random.default_rng(n).integers(0, 5000, size=n, dtype=np.int32)
    want_x, want_out = _want(a, steps)
    for scan in (gpu.exclusive_scan_i32, gpu.exclusive_scan_i32_noalloc):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            x, out = torch.from_numpy(a).cuda(), torch.zeros(n + 1, dtype=torch.int32, device="cuda")
            _chain(scan, torch, x, out, n, steps)
        st.synchronize()
        assert np.array_equal(x.cpu().numpy(), want_x) and np.array_equal(out.cpu().numpy(), want_out)
    x0 = torch.from_numpy(a).cuda()
    x, out = x0.clone(), torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.copy_(x0)
        _chain(gpu.exclusive_scan_i32_noalloc, torch, x, out, n, steps)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy(), want_x) and np.array_equal(out.cpu().numpy(), want_out)


def test_frames_in_a_row(gpu, oracle_lib):
    # two scenes in turn on one stream without a wait: each frame's kernels reuse the last one's buffers
    import torch
    rng = np.random.default_rng(11)
    imgs, rs, outs = [], [], []
    for k in range(2):
        b = scenes.Builder(400, 300)
        for i in range(60 + 200 * k):
            b.path(rule=i % 2, rgba=(i % 251, 60 * k, 200, 90 + i % 160))
            x, y, s = rng.uniform(-20, 380), rng.uniform(-20, 280), rng.uniform(3, 90)
            b.polygon([(x, y), (x + s, y + 0.3 * s), (x + 0.4 * s, y + s)])
        d = b.arrays()
        imgs.append(oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))
        r = gpu.ScanlineVGRasterizer(mode=1)
        r.initialize(None, 400, 300)
        r.loadVG(scenes.to_container(d))
        rs.append(r)
        outs.append(torch.zeros((300, 400, 4), dtype=torch.uint8, device="cuda"))
    for _ in range(6):
        for r, out in zip(rs, outs):
            out.zero_()
            torch.cuda.synchronize()
            r.render_device(out.data_ptr())
            r.render_device(out.data_ptr())
    torch.cuda.synchronize()
    for img, out, r in zip(imgs, outs, rs):
        assert np.array_equal(out.cpu().numpy(), img)
        r.close()
