"""Scenes of more records than a frame takes (2^30): refused at every total, also where it passes 2^31 or 2^32, by a
first frame and by one that was sized from a small frame of as many curves and paths; the context goes on."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

SIDE = 16384


def _diagonals(n, scale):
    i = np.arange(n, dtype=np.float64)
    p = np.stack([0.3 + 1e-5 * i, np.full(n, 0.2), np.full(n, SIDE - 0.4), SIDE - 0.3 - 1e-5 * i], 1) * scale
    paths = (n + 99) // 100
    return dict(width=SIDE, height=SIDE, position=p.astype(np.float32).reshape(-1),
                pos_path_idx=np.repeat(np.arange(n, dtype=np.uint32) // 100, 2),
                curve_pos_map=np.arange(0, 2 * n, 2, dtype=np.uint32), curve_type=np.full(n, scenes.LINE, np.uint32),
                curve_path_idx=np.arange(n, dtype=np.uint32) // 100, fill_rule=np.zeros(paths, np.uint32),
                fill_info=np.full(paths, 0xFF102030, np.uint32))


@pytest.mark.parametrize("n", [33000, 66000, 98500, 131100])   # 1.08, 2.16, 3.23 and 4.2956 (2^32 + 666,000) x 10^9
def test_too_many_records(gpu, oracle_lib, n):
    dot, full = (scenes.to_container(_diagonals(n, s)) for s in (1e-3, 1.0))
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, SIDE, SIDE)
    r.loadVG(full)
    for _ in range(2):
        with pytest.raises(gpu.SRError) as e:   # exact
            r.render_device()
        assert e.value.code == 3 and "out of range" in str(e.value)
    for _ in range(2):
        r.loadVG(dot)
        r.render_device()
        first = r.dump("draw_list")
        r.render_device()
        assert r.stats()["n_intersections"] < 1 << 26
        assert np.array_equal(r.dump("draw_list"), first)
        r.loadVG(full)
        with pytest.raises(gpu.SRError) as e:   # pre-sized, then exact
            r.render_device()
        assert e.value.code == 3 and "out of range" in str(e.value)
    r.close()


def test_batch_capacity(gpu):
    b = gpu.SceneBatch(mode=1)
    b.add_scene(scenes.to_container(_diagonals(66000, 1.0)))
    for refit in (False, True):
        with pytest.raises(gpu.SRError) as e:
            b.render(capacity=100000, refit=refit)
        assert e.value.code == 3
    b.close()
