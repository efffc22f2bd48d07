"""Lines whose crossings are not numbers (0 * inf): their records are the sequential merge's, in one place each.  Such a
line starts on a grid line and ends within a denormal of it; another kind has a point that the matrix sends to infinity.
Images and record counts are the oracle's exactly, in a first (exact) and a pre-sized frame, alone and in a batch, after
frames that left other records in the buffers."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

TINY = -1e-40   # a float32 denormal: 1 / TINY overflows


def _line(kind, a, b):
    return {"x": [(0.0, a), (TINY, b)],          # x root NaN, y roots in order
            "x_only": [(0.0, a), (TINY, a + 0.2)],   # no y root beside it (a within a row)
            "y": [(a, 0.0), (b, TINY)],          # y root NaN
            "y_only": [(a, 0.0), (a + 0.2, TINY)],
            "both": [(0.0, 0.0), (TINY, TINY)]}[kind]


def _scene(kinds, length, n, w, h):
    """n triangles whose first side is such a line of about `length` crossings, between ordinary ones."""
    rng = np.random.default_rng(n * length)
    b = scenes.Builder(w, h)
    for i in range(n):
        b.path(rule=i % 2, rgba=(i * 37 % 251, 200, i % 7 * 30, 90 + i % 160))
        p, q = _line(kinds[i % len(kinds)], 0.25 + 0.125 * (i % 5), length + 0.5 - 0.25 * (i % 3))
        if i % 2:
            p, q = (p, q) if i % 4 == 1 else (q, p)   # (backwards they end on the grid line: the root is a number)
        b.polygon([p, q, (rng.uniform(2, w), rng.uniform(2, h))])
        b.path(rule=0, rgba=(20, i % 251, 90, 200))
        x, y = rng.uniform(0, w), rng.uniform(0, h)
        b.polygon([(x, y), (x + 9.3, y + 2.1), (x + 3.2, y + 14.6)])
    return b.arrays()


def _check(gpu, oracle, d, mode, mvp=None):
    of = oracle.Frame(scenes.to_oracle(d), mode=mode, mvp=mvp)
    r = gpu.ScanlineVGRasterizer(mode=mode)
    r.initialize(None, d["width"], d["height"])
    other = scenes.Builder(d["width"], d["height"])   # leaves records of curves that the next scene does not have
    for i in range(300):
        other.path(rgba=(1, 2, 3, 255)).polygon([(3, 1 + i % 9), (11.5, 4), (5, 3 + i % 20)])
    r.loadVG(scenes.to_container(other.arrays()))
    r.render()
    r.loadVG(scenes.to_container(d))
    if mvp is not None:
        r.setMVP(mvp)
    for _ in range(2):
        assert np.array_equal(r.render(), of.get("image"))
        st = r.stats()
        assert st["n_intersections"] == of.n_intersections and st["n_draw_records"] == of.n_draw
    rec, want = r.dump("intersection"), of.get("intersection").reshape(-1, 2)
    t, tw = rec[:, 1].copy().view(np.float32), want[:, 1].copy().view(np.float32)
    assert np.array_equal(rec[:, 0], want[:, 0])
    assert np.all((rec[:, 1] == want[:, 1]) | (np.isnan(t) & np.isnan(tw)))
    r.close()
    return of


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kinds", [("x",), ("x_only",), ("y",), ("y_only",), ("both",),
                                   ("x", "y", "both", "x_only", "y_only")])
@pytest.mark.parametrize("length,n", [(1, 3), (20, 1), (20, 24), (70, 5), (300, 9)])
def test_denormal_extents(gpu, oracle_lib, mode, kinds, length, n):
    of = _check(gpu, oracle_lib, _scene(kinds, length, n, length + 33, length + 40), mode)
    t = of.get("intersection").reshape(-1, 2)[:, 1].copy().view(np.float32)
    assert np.any(np.isnan(t) | (t >= 2))


@pytest.mark.parametrize("mode", [0, 1])
def test_in_a_batch(gpu, oracle_lib, mode):
    ds = [_scene(("x", "y", "both", "x_only", "y_only"), k, 7, k + 33, k + 21) for k in (3, 20, 130)]
    b = gpu.SceneBatch(mode=mode)
    for d in ds:
        b.add_scene(scenes.to_container(d))
    for cap in (-1, 40000):
        b.render(capacity=cap, refit=False)
        for i, d in enumerate(ds):
            assert np.array_equal(b.image(i), oracle_lib.Frame(scenes.to_oracle(d), mode=mode).get("image"))
    b.close()


@pytest.mark.parametrize("row3", [(1, 0, -8), (0, 1, -6), (1, 1, -14)])
def test_points_at_infinity(gpu, oracle_lib, row3):
    # (pixel mode: the reference's two passes count the lines of a two-pixel grid up to infinity differently)
    # w = 0 on the lines x = 8, y = 6 and x + y = 14: vertices there go to infinity, or to NaN from the origin of a row
    mvp = np.array([1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, row3[0], row3[1], 0, row3[2]], np.float32)
    b = scenes.Builder(64, 48)
    for i, pts in enumerate([[(8, 6), (30, 2), (12, 40)], [(2, 3), (8, 20), (40, 30)], [(8, 2), (8, 11), (9, 30)],
                             [(8, 0), (20, 9), (3, 20)], [(0, 6), (14, 0), (22, 33)], [(10, 9), (20, 30), (40, 12)]]):
        b.path(rule=i % 2, rgba=(40 * i, 90, 30, 120 + 20 * i)).polygon(pts)
    _check(gpu, oracle_lib, b.arrays(), 1, mvp)
