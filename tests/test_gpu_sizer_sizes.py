"""The sizing network's kernels at the sizes where a warp's eight paths and a CTA's 32 samples are not full, against the
float64 restatement.  Tolerances as in test_gpu_sizer.py (predictions and loss 1e-4 relative, gradients 2e-3 of the
largest entry): the sums are FP32 in another order."""
import numpy as np
import pytest

from oracle import mlp_ref as M

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    x = np.abs(rng.normal(2.0, 1.0, (n, 6))).astype(np.float32)
    return x, (x[:, :2] + 0.1 * rng.normal(size=(n, 2))).astype(np.float32)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 63, 65, 1000, 40001])
def test_predict_and_gradient_sizes(gpu, n):
    xh, th = _rows(n, n)
    sz = gpu.Sizer(seed=n)
    norm = gpu.sizer_norm(*_rows(500, 1))
    sz.set_norm(norm)
    params = sz.state()["params"]
    x, t = gpu.DeviceArray.from_numpy(xh), gpu.DeviceArray.from_numpy(th)
    guard = gpu.DeviceArray.from_numpy(np.full((n + 8, 2), 7.5, np.float32))
    sz.predict(x, out=guard)
    y = guard.numpy()
    assert np.allclose(y[:n], M.forward(params, norm, xh), rtol=1e-4, atol=1e-4)
    assert np.all(y[n:] == 7.5)
    loss, g = sz.loss_grad(x, t)
    want_loss, want_g = M.loss_grad(params, norm, xh, th)
    assert loss == pytest.approx(want_loss, rel=1e-4)
    assert np.abs(g - want_g).max() <= 2e-3 * np.abs(want_g).max()
    sz.close()


@pytest.mark.parametrize("n,batch", [(33, 32), (100, 64), (129, 1000)])
def test_steps_match_the_restatement(gpu, n, batch):
    """Adam by the step's last CTA, over several steps in row order; parameters whose gradient is not tiny agree to
    4e-6 a step (a step moves a parameter by at most 1e-3)."""
    xh, th = _rows(n, 3 * n)
    sz = gpu.Sizer(seed=2)
    norm = gpu.sizer_norm(*_rows(500, 1))
    sz.set_norm(norm)
    p = sz.state()["params"].astype(np.float64)
    m, v, steps = np.zeros_like(p), np.zeros_like(p), 0
    strong = np.ones(p.size, bool)
    for at in range(0, n, batch):
        _, g = M.loss_grad(p.astype(np.float32), norm, xh[at:at + batch], th[at:at + batch])
        steps += 1
        strong &= np.abs(g) > 1e-2 * np.abs(g).max()
        p, m, v = M.adam_step(p, m, v, g, steps, lr=1e-3)
    x, t = gpu.DeviceArray.from_numpy(xh), gpu.DeviceArray.from_numpy(th)
    sz.train(x, t, epochs=1, batch=batch, shuffle=False, lr=1e-3)
    st = sz.state()
    assert st["step"] == steps
    assert np.allclose(st["params"][strong], p[strong], rtol=0, atol=4e-6 * steps)
    sz.close()
