"""Where a frame's pixels go: device memory that kernels write themselves, at any 4-byte offset and at offsets that are
not, and page-locked host memory."""
import ctypes

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _frame(w, h):
    rng = np.random.default_rng(w)
    b = scenes.Builder(w, h)
    for i in range(25):
        b.path(rule=i % 2, rgba=(i * 9, 70, 210, 60 + 7 * i))
        x, y, s = rng.uniform(-9, w), rng.uniform(-9, h), rng.uniform(2, 60)
        b.polygon([(x, y), (x + s, y + 0.3 * s), (x + 0.4 * s, y + s)])
    return b.arrays()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (258, 130)])
def test_device_offsets(gpu, oracle_lib, w, h, mode):
    import torch
    d = _frame(w, h)
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=mode).get("image").reshape(-1)
    r = gpu.ScanlineVGRasterizer(mode=mode)
    r.initialize(None, w, h)
    r.loadVG(scenes.to_container(d))
    b = gpu.SceneBatch(mode=mode)
    b.add_scene(scenes.to_container(d))
    b.render()
    for off in (0, 4, 8, 16, 1, 6):
        for put in (lambda at: r.render_device(at), lambda at: gpu._check(gpu.lib().sr_batch_get_image(b._h, 0, at, 1, None))):
            buf = torch.full((w * h * 4 + 64,), 7, dtype=torch.uint8, device="cuda")
            put(buf.data_ptr() + off)
            torch.cuda.synchronize()
            got = buf.cpu().numpy()
            assert np.array_equal(got[off:off + want.size], want)
            assert np.all(got[:off] == 7) and np.all(got[off + want.size:] == 7)
    assert np.array_equal(r.dump("image").reshape(-1), want)   # the frame stays with the context too
    if mode == 1:
        host = r.render_aa(4)
        dev = torch.zeros(host.size, dtype=torch.uint8, device="cuda")
        gpu._check(gpu.lib().sr_render_aa(r._ctx, 4, dev.data_ptr(), 1, None))
        assert np.array_equal(dev.cpu().numpy(), host.reshape(-1))
    b.close()
    r.close()


def test_other_memory(gpu, oracle_lib):
    d = _frame(90, 60)
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image").reshape(-1)
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, 90, 60)
    r.loadVG(scenes.to_container(d))
    pin = gpu.PinnedBuffer(want.size)
    for is_device in (0, 1):   # page-locked host memory, also where the call says device memory
        ctypes.memset(pin.ptr, 7, want.size)
        gpu._check(gpu.lib().sr_render(r._ctx, pin.ptr, is_device, None))
        assert np.array_equal(np.ctypeslib.as_array(ctypes.cast(pin.ptr, ctypes.POINTER(ctypes.c_uint8)), (want.size,)), want)
    r.close()
