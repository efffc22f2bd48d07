"""The tables of the per-path sort built beside the fragments (frames of up to 4,096 paths) and by a launch of their own,
at the edges of the CTAs that build them."""
import numpy as np
import pytest

import scenes
from test_gpu_tables import _sparse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_paths", [127, 128, 129, 4095, 4096, 4097])
def test_paths(gpu, oracle_lib, n_paths):
    d = _sparse(n_paths, n_paths)
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image")
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, d["width"], d["height"])
    r.loadVG(scenes.to_container(d))
    for _ in range(2):   # exact, then pre-sized
        assert np.array_equal(r.render(), want)
        assert r.sort_tiles()[0] > 0
    r.close()
