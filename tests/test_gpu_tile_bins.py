"""The bins of the per-path tile sort where they can go wrong: cells and rows crowded up to and past a bin's limit (the
tile then takes digit passes), runs of off-canvas records of several paths in a tile, row 0 (ranked last), and as many
paths in a tile as bins allow, fewer and more."""
import numpy as np
import pytest

import scenes
from test_gpu_segsort import _render

pytestmark = pytest.mark.gpu


def _check(gpu, oracle_lib, b):
    d = b.arrays()
    img, _ = _render(gpu, d)
    assert np.array_equal(img, oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))


@pytest.mark.parametrize("crowd", [60, 63, 64, 65, 300])
def test_crowded_cell(gpu, oracle_lib, crowd):
    # hexagons inside one cell, six records each (360, 378, 384, 390, 1800), among records all over the canvas
    rng = np.random.default_rng(crowd)
    b = scenes.Builder(900, 700)
    b.path(rule=1, rgba=(40, 200, 90, 130))
    b.polygon([(3.2, 2.1), (880.7, 340.3), (12.9, 690.4), (400.1, 5.0)])
    for i in range(crowd):
        x, y = 500.1 + 0.5 * rng.uniform(), 300.1 + 0.5 * rng.uniform()
        b.polygon([(x, y), (x + 0.2, y + 0.05), (x + 0.3, y + 0.2), (x + 0.2, y + 0.3), (x + 0.05, y + 0.25),
                   (x + 0.01, y + 0.1)])
    _check(gpu, oracle_lib, b)


@pytest.mark.parametrize("lines", [1, 7, 40])
def test_crowded_rows(gpu, oracle_lib, lines):
    # long flat strips in row 0 and two more rows of a wide canvas
    b = scenes.Builder(1300, 40)
    b.path(rule=1, rgba=(200, 30, 90, 150))
    for i in range(lines):
        for y in (0.2, 7.1, 33.3):
            b.polygon([(1.5 * i, y), (1290.0 - i, y + 0.01 * i), (1200.0 - 3 * i, y + 0.4)])
    _check(gpu, oracle_lib, b)


@pytest.mark.parametrize("w,h", [(33, 1), (64, 31), (257, 129)])
def test_off_canvas_runs(gpu, oracle_lib, w, h):
    # paths mostly outside the canvas on every side, many of them in a tile
    rng = np.random.default_rng(w)
    b = scenes.Builder(w, h)
    for i in range(90):
        b.path(rule=i % 2, rgba=(i % 251, 60, 200, 90 + i % 160))
        for _ in range(1 + i % 3):
            x, y = rng.uniform(-0.8 * w, 1.6 * w), rng.uniform(-1.5 * h - 20, 2.0 * h + 20)
            s = rng.uniform(0.5, 0.9) * (w + h)
            b.polygon([(x, y), (x + s, y + 0.7 * s), (x - 0.4 * s, y + s)])
    _check(gpu, oracle_lib, b)


@pytest.mark.parametrize("n_paths", [600, 1364, 1366, 3000])
def test_small_paths_of_a_tile(gpu, oracle_lib, n_paths):
    # slivers of a record or two, in a canvas few enough bins can hold the rows of
    b = scenes.Builder(50, 45)
    for i in range(n_paths):
        b.path(rule=i % 2, rgba=(i % 251, 120, 30, 100 + i % 150))
        x, y = (7 * i) % 49 + 0.1, (11 * i) % 46 - 0.8
        b.polygon([(x, y), (x + 0.7, y + 0.2), (x + 0.3, y + 0.6)])
    _check(gpu, oracle_lib, b)
