"""Crossing chains split by how many there are: stretches of 8, 16 and 64 roots on either side of the totals where the
length changes (2,432 and 24,320 warps' shares on 152 SMs)."""
import numpy as np
import pytest

import scenes
from test_gpu_segsort import _render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 2300, 2600, 25000])
def test_many_long_chains(gpu, oracle_lib, n):
    # a cubic of 256 to 500 crossings in x and in y a path, monotonic and not, and the line that closes it: about a
    # share a path at 16 roots a lane
    rng = np.random.default_rng(n)
    w, h = 640, 600
    b = scenes.Builder(w, h)
    for i in range(n):
        b.path(rule=i % 2, rgba=(i % 251, 90, 200, 20 + i % 100))
        x0, y0 = rng.uniform(0, 60, 2)
        x1, y1 = x0 + rng.uniform(270, 500), y0 + rng.uniform(270, 480)
        bend = rng.uniform(-0.3, 1.3, 4) if i % 3 else rng.uniform(0, 1, 4)
        p = [(x0, y0), (x0 + bend[0] * (x1 - x0), y0 + bend[1] * (y1 - y0)),
             (x0 + bend[2] * (x1 - x0), y0 + bend[3] * (y1 - y0)), (x1, y1)]
        b.curve(scenes.CUBIC, p)
        b.curve(scenes.LINE, [p[3], p[0]])
    d = b.arrays()
    img, _ = _render(gpu, d)
    assert np.array_equal(img, oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))
