"""Predictions for so many paths that their inputs, and then their outputs, are more than 2^32 values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [715827883, (1 << 31) + 3])
def test_predict_many_paths(gpu, n):
    # the same 1,000 rows over and over (equal rows give equal predictions), compared with a call of their own
    import torch
    need = 32 * n + (8 << 30)
    if torch.cuda.mem_get_info()[0] < need:
        pytest.skip("needs %.0f GB of device memory" % (need / 1e9))
    rng = np.random.default_rng(5)
    rows = np.abs(rng.normal(2.0, 1.0, (1000, 6))).astype(np.float32)
    sz = gpu.Sizer(seed=3)
    sz.set_norm(gpu.sizer_norm(rows, rows[:, :2]))
    want = torch.from_numpy(sz.predict(gpu.DeviceArray.from_numpy(rows)).numpy()).cuda()
    base = torch.from_numpy(rows).cuda()
    reps, rest = divmod(n, 1000)
    x = torch.empty((n, 6), dtype=torch.float32, device="cuda")
    x[:reps * 1000].view(reps, 1000, 6).copy_(base.expand(reps, 1000, 6))
    x[reps * 1000:].copy_(base[:rest])
    y = torch.full((n + 8, 2), 7.5, dtype=torch.float32, device="cuda")
    st = torch.cuda.current_stream()
    assert gpu.lib().sr_sizer_predict(sz._h, x.data_ptr(), n, y.data_ptr(), st.cuda_stream) == 0
    for r0 in range(0, reps, 100000):   # (in parts: a comparison of the whole would hold as much again)
        part = y[r0 * 1000:min(r0 + 100000, reps) * 1000].view(-1, 1000, 2)
        assert bool((part == want).all())
    assert torch.equal(y[reps * 1000:n], want[:rest])
    assert bool((y[n:] == 7.5).all())
    sz.close()
    del x, y, part
    torch.cuda.empty_cache()
