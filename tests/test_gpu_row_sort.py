"""The row order of paint runs in one pass, at the row counts where its digits widen and where it gives way to digit
passes, with one tile of runs and with many, in reference mode (two pixel rows a row) too."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _scene(h, n, seed):
    rng = np.random.default_rng(seed)
    b = scenes.Builder(96, h)
    for i in range(n):
        b.path(rule=i % 2, rgba=(int(rng.integers(256)), 90, i % 256, 60 + i % 190))
        x, y = rng.uniform(-10, 90), rng.uniform(-0.1 * h, h)
        b.polygon([(x, y), (x + rng.uniform(1, 60), y + rng.uniform(0, 0.3) * h), (x - 5, y + rng.uniform(0, 0.6) * h)])
    return b.arrays()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", [256, 257, 512, 513, 1024, 1025, 2048])
@pytest.mark.parametrize("n", [3, 150])
def test_rows(gpu, oracle_lib, h, n, mode):
    d = _scene(h, n, h + n)
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=mode).get("image")
    r = gpu.ScanlineVGRasterizer(mode=mode)
    r.initialize(None, 96, h)
    r.loadVG(scenes.to_container(d))
    for _ in range(2):   # exact, then pre-sized (tiles launched for more runs than there are)
        assert np.array_equal(r.render(), want)
    r.close()
