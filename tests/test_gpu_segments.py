"""The pixels a warp of the resolve paints (64, 128 or 256), on either side of the frame sizes where that changes (6,080
and 30,400 segments of 256 pixels on 152 SMs), at widths that leave part of a segment, solid and gradient."""
import numpy as np
import pytest

import scenes
from test_gpu_segsort import _render

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (63, 6079), (65, 6080), (255, 6079), (257, 3041), (257, 15199), (257, 15201)]


@pytest.mark.parametrize("w,h", SIZES)
def test_solid(gpu, oracle_lib, w, h):
    # layers over whole rows (one of them opaque), over parts of a row, and a pixel wide
    rng = np.random.default_rng(w + h)
    b = scenes.Builder(w, h)
    for i in range(160):
        b.path(rule=i % 2, rgba=(int(rng.integers(256)), int(rng.integers(256)), 77 + i, 255 if i == 70 else 40 + i))
        if i % 4 == 0:
            x0, x1 = -5.0, w + 5.0
        else:
            x0 = rng.uniform(-0.2, 1.0) * w
            x1 = x0 + (0.9 if i % 4 == 1 else rng.uniform(0.1, 0.9) * w)
        y0 = rng.uniform(-0.2, 0.8) * h
        y1 = y0 + rng.uniform(0.05, 0.6) * h
        b.polygon([(x0, y0), (x1, y0 + 0.3), (x1 + 0.2, y1), (x0 + 0.4, y1 + 1.1)])
    d = b.arrays()
    img, _ = _render(gpu, d)
    assert np.array_equal(img, oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))


@pytest.mark.parametrize("w,h", SIZES)
def test_gradient(gpu, oracle_lib, w, h):
    d = scenes.gradients(w, h)
    img, _ = _render(gpu, d)
    assert np.array_equal(img, oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))
