"""The resolve in reference mode (a pixel takes the latest record over it) with 64 and with 256 pixels a warp, at canvas
edges that leave part of a segment or of a cell row: covered, half covered and empty rows, rows of more than 32 records,
solid colours of every alpha and gradients."""
import numpy as np
import pytest

import scenes
from test_gpu_segments import SIZES

pytestmark = pytest.mark.gpu


def _check(gpu, oracle_lib, d):
    r = gpu.ScanlineVGRasterizer(mode=0)
    r.initialize(None, d["width"], d["height"])
    r.loadVG(scenes.to_container(d))
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=0).get("image")
    for _ in range(2):
        assert np.array_equal(r.render(), want)
    r.close()


@pytest.mark.parametrize("w,h", SIZES + [(511, 15201), (16001, 63)])
def test_solid(gpu, oracle_lib, w, h):
    rng = np.random.default_rng(w + h)
    b = scenes.Builder(w, h)
    for i in range(120):
        b.path(rule=i % 2, rgba=(int(rng.integers(256)), int(rng.integers(256)), 77 + i, int(rng.integers(1, 256))))
        x0 = -5.0 if i % 7 == 0 else rng.uniform(-0.2, 1.0) * w
        x1 = w + 5.0 if i % 7 == 0 else x0 + (0.9 if i % 4 == 1 else rng.uniform(0.1, 0.9) * w)
        y0 = rng.uniform(-0.2, 0.8) * h
        y1 = y0 + rng.uniform(0.02, 0.4) * h
        b.polygon([(x0, y0), (x1, y0 + 0.3), (x1 + 0.2, y1), (x0 + 0.4, y1 + 1.1)])
    _check(gpu, oracle_lib, b.arrays())


@pytest.mark.parametrize("w,h", [(1, 1), (63, 6079), (257, 3041), (511, 15201)])
def test_gradient(gpu, oracle_lib, w, h):
    _check(gpu, oracle_lib, scenes.gradients(w, h))
