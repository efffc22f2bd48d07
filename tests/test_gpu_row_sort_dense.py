"""The row order on both sides of the draw capacity from which canvases of 513 to 1,024 rows take digit passes: with few
runs in much room, and with rows of thousands of runs."""
import numpy as np
import pytest

import scenes
from test_gpu_row_sort import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", [512, 513, 1024])
def test_draw_capacities(gpu, oracle_lib, mode, h):
    h *= 2 - mode   # rows of two pixels
    d = _scene(h, 60, h)
    want = oracle_lib.Frame(scenes.to_oracle(d), mode=mode).get("image")
    b = gpu.SceneBatch(mode=mode)
    b.add_scene(scenes.to_container(d))
    for draws in (3499999, 3500000, 3500001, 6000000):
        b.render(capacity=200000, draw_capacity=draws, refit=False)
        assert np.array_equal(b.image(0), want)
    b.close()


@pytest.mark.parametrize("n", [3000, 4400])   # 2.5 and 3.7 million draw records
def test_dense_rows(gpu, oracle_lib, n):
    s = oracle_lib.synth(0, 1, width=1024, height=1024, n_paths=n)
    want = oracle_lib.Frame(s, mode=1).get("image")
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, 1024, 1024)
    r.loadVG(gpu.VGContainer.from_arrays(1024, 1024, s.position, s.pos_path_idx, s.curve_pos_map, s.curve_type,
                                         s.curve_path_idx, s.fill_rule, s.fill_info))
    for _ in range(3):
        assert np.array_equal(r.render(), want)
    r.close()
