"""The standalone scans at the sizes where their launch shape changes, at addresses that are not 16-byte aligned, in
place, with several streams at once, and in a captured graph."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 127, 16383, 16384, 16385, 32767, 32768, 32769, 4096 * 9 - 1, 608 * 4096 - 1, 608 * 4096,
         608 * 4096 + 1, 1217 * 4096 + 77]


def _ref(a):
    out = np.zeros(a.size + 1, np.int64)
    np.cumsum(a.astype(np.int64), out=out[1:])
    return out.astype(np.int32)   # wraps like the device scan


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (1, 0), (0, 3), (2, 1)])
def test_sizes_and_alignments(gpu, n, off_in, off_out):
    import torch
    a = np.random.default_rng(n).integers(-(1 << 30), 1 << 30, size=n, dtype=np.int32)
    d_in = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    d_in[off_in:off_in + n] = torch.from_numpy(a).cuda()
    for scan in (gpu.exclusive_scan_i32, gpu.exclusive_scan_i32_noalloc):
        d_out = torch.full((n + 8,), -7, dtype=torch.int32, device="cuda")
        scan(d_in.data_ptr() + 4 * off_in, d_out.data_ptr() + 4 * off_out, n)
        got = d_out.cpu().numpy()
        assert np.array_equal(got[off_out:off_out + n + 1], _ref(a))
        assert np.all(got[:off_out] == -7) and np.all(got[off_out + n + 1:] == -7)


@pytest.mark.parametrize("n", [16385, 32769, 608 * 4096 + 1])
def test_in_place(gpu, n):
    import torch
    a = np.random.default_rng(n).integers(0, 40, size=n, dtype=np.int32)
    for scan in (gpu.exclusive_scan_i32, gpu.exclusive_scan_i32_noalloc):
        buf = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        buf[:n] = torch.from_numpy(a).cuda()
        scan(buf.data_ptr(), buf.data_ptr(), n)
        assert np.array_equal(buf.cpu().numpy(), _ref(a))


def test_several_streams_and_a_captured_graph(gpu):
    import torch
    n = 300001
    ins = [torch.randint(0, 40, (n,), dtype=torch.int32, device="cuda") for _ in range(4)]
    outs = [torch.zeros(n + 1, dtype=torch.int32, device="cuda") for _ in range(4)]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, i, o in zip(streams, ins, outs):
            gpu.exclusive_scan_i32(i.data_ptr(), o.data_ptr(), n, ctypes.c_void_p(s.cuda_stream))
    torch.cuda.synchronize()
    for i, o in zip(ins, outs):
        assert np.array_equal(o.cpu().numpy(), _ref(i.cpu().numpy()))
    g = torch.cuda.CUDAGraph()
    o = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    with torch.cuda.graph(g):
        gpu.exclusive_scan_i32(ins[0].data_ptr(), o.data_ptr(), n,
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    ins[0].copy_(ins[1])
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(o.cpu().numpy(), _ref(ins[1].cpu().numpy()))
    gpu.scan_status()
