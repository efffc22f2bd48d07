"""Long rows of paths without curves: before the first curve, between curves and after the last, around the length from
which a warp fills them in, in scenes of few curves (eight lanes a curve) and of many, alone and in a batch."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

W, H = 150, 110


def _scene(gaps, filler, seed):
    """A triangle, then gaps[i] paths without curves, for each i (0: none before); filler triangles in the last path."""
    rng = np.random.default_rng(seed)
    b = scenes.Builder(W, H)
    for i, gap in enumerate(gaps):
        for _ in range(gap):
            b.path(rgba=(9, 9, 9, 255))
        if i + 1 == len(gaps):
            break
        b.path(rule=i % 2, rgba=(60 * i % 251, 120, 200, 90 + 20 * (i % 8)))
        for _ in range(filler if i + 2 == len(gaps) else 1):
            x, y, s = rng.uniform(-5, W), rng.uniform(-5, H), rng.uniform(2, 30)
            b.polygon([(x, y), (x + s, y + 0.3 * s), (x + 0.4 * s, y + s)])
    return b.arrays()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("filler", [1, 6000])   # 18,000 curves: a thread a curve
@pytest.mark.parametrize("gaps", [(0, 30, 31, 32, 33, 0), (31, 32, 33, 34, 35, 36, 37, 38), (129, 1, 130, 131, 132, 133),
                                  (0, 0, 100003), (100001, 0, 0), (50002, 0, 33, 50003, 50001)])
def test_gaps(gpu, oracle_lib, gaps, filler, mode):
    d = _scene(gaps, filler, len(gaps))
    of = oracle_lib.Frame(scenes.to_oracle(d), mode=mode)
    r = gpu.ScanlineVGRasterizer(mode=mode)
    r.initialize(None, W, H)
    r.loadVG(scenes.to_container(d))
    for _ in range(2):
        assert np.array_equal(r.render(), of.get("image"))
        assert r.stats()["n_draw_records"] == of.n_draw
    r.close()


def test_batch(gpu, oracle_lib):
    ds = [_scene(g, 1, 7) for g in [(40, 0, 41), (0, 0), (1000, 50, 2000), (33, 33, 33, 33)]]
    b = gpu.SceneBatch(mode=1)
    for d in ds:
        b.add_scene(scenes.to_container(d))
    for cap in (-1, 20000):
        b.render(capacity=cap, refit=False)
        for i, d in enumerate(ds):
            assert np.array_equal(b.image(i), oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))
    b.close()
