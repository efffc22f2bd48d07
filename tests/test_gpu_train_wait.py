"""Training whose shuffle's sort gives up (one poll a wait): SR_ERR_TIMEOUT, no access to a row that there is not, and the
sizer trains on from a state that is set again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(1 << 20, 4096), (700001, 100000), (2000, 512)])
def test_shuffle_gives_up(gpu, n, batch):
    rng = np.random.default_rng(n)
    xh = np.abs(rng.normal(2.0, 1.0, (n, 6))).astype(np.float32)
    x, t = gpu.DeviceArray.from_numpy(xh), gpu.DeviceArray.from_numpy(np.ascontiguousarray(xh[:, :2]))
    sz = gpu.Sizer(seed=1)
    sz.set_norm(gpu.sizer_norm(xh[:500], xh[:500, :2]))
    start = sz.state()
    gave_up = 0
    for turn in range(6):
        gpu.set_spin_limit(1)
        try:
            sz.train(x, t, epochs=2, batch=batch, seed=turn)
        except gpu.SRError as e:
            assert e.code == 4
            gave_up += 1
        finally:
            gpu.set_spin_limit(0)
        sz.load_state(start)
    assert gave_up or n < 10000   # (one tile has nothing to wait for)
    losses = [sz.train(x, t, epochs=1, batch=batch, seed=turn) for turn in range(2)]
    assert np.isfinite(losses).all() and losses[1] < losses[0]
    sz.close()
