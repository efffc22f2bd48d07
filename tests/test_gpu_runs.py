"""Paint runs (a path's touching draw records of a row painted as one) where they begin, break and are cut: rows with more
records than a warp's 256 or a tile's 2,048, even-odd holes one cell wide, cells without a gap between them, spans
from the canvas's edges; and the reference's draw list, which a read-back still gives."""
import numpy as np
import pytest

import scenes
from parity_util import compare_all, render_both

pytestmark = pytest.mark.gpu


def _comb(w, h, teeth, step, rule):
    """One path with `teeth` teeth, each `step` pixels from the next: a row holds two crossings a tooth."""
    b = scenes.Builder(w, h)
    b.path(rule, (200, 40, 90, 150))
    x0 = 0.3
    pts = []
    for i in range(teeth):
        x = x0 + i * step
        pts += [(x, 1.2), (x + 0.5 * step, h - 1.4), (x + 0.55 * step, h - 1.4)]
    pts += [(x0 + teeth * step, 1.2), (x0 + teeth * step, 0.1), (x0, 0.1)]
    b.polygon(pts)
    b.path(rule, (10, 200, 90, 255))
    b.polygon([(x - 7.5, h - y) for x, y in pts])
    return b.arrays()


def _nested(w, h, rule):
    """Rectangles inside one another, at distances of a fraction of a cell to a few cells: an even-odd path is holes
    and walls of that width."""
    b = scenes.Builder(w, h)
    b.path(rule, (20, 90, 220, 120))
    x0, y0, x1, y1 = -3.0, -2.0, w + 4.0, h + 1.0
    for d in (0.4, 0.9, 1.0, 1.1, 2.0, 0.2, 3.7, 1.0, 5.0, 0.6, 1.0):
        if x1 - x0 < 2 or y1 - y0 < 2:
            break
        b.polygon([(x0, y0), (x1, y0), (x1, y1), (x0, y1)])
        x0, y0, x1, y1 = x0 + d, y0 + d, x1 - d, y1 - d
    b.path(rule, (250, 20, 20, 255))
    b.polygon([(-20, 3.5), (w + 20, 3.5), (w + 20, 4.5), (-20, 4.5)])
    return b.arrays()


CASES = {
    "comb-90": lambda rule: _comb(300, 40, 90, 3.1, rule),
    "comb-200": lambda rule: _comb(600, 24, 200, 2.9, rule),
    "comb-1100": lambda rule: _comb(4400, 12, 1100, 3.7, rule),
    "nested": lambda rule: _nested(61, 37, rule),
    "nested-odd": lambda rule: _nested(300, 41, rule),
}


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_runs(gpu, oracle_lib, name, rule, mode):
    d = CASES[name](rule)
    of, r, img = render_both(gpu, oracle_lib, d, mode)
    compare_all(of, r, img, mode)
    r.close()
    for wind_items in (4, 8):   # without kept stages: the per-path sort, both tile sizes, exact and pre-sized
        r = gpu.ScanlineVGRasterizer(mode=mode)
        r.initialize(None, d["width"], d["height"])
        r.set_tuning(wind_items=wind_items)
        r.loadVG(scenes.to_container(d))
        for _ in range(2):
            assert np.array_equal(r.render(), of.get("image"))
        assert np.array_equal(r.dump("draw_list"), of.get("draw_list"))
        assert np.array_equal(r.dump("intersection"), of.get("intersection"))
        r.close()


def test_draw_list_read_back_after_other_calls(gpu, oracle_lib):
    """The last frame's draw list and records stay readable after a new scene is loaded (twice), and the frame after
    them is right; a rendered draw list is read back as given."""
    a, b = CASES["comb-90"](0), CASES["nested-odd"](1)
    fa = oracle_lib.Frame(scenes.to_oracle(a), width=300, height=41, mode=1)
    fb = oracle_lib.Frame(scenes.to_oracle(b), width=300, height=41, mode=1)
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, 300, 41)
    r.loadVG(scenes.to_container(a))
    r.render()
    r.loadVG(scenes.to_container(b))
    r.loadVG(scenes.to_container(b))
    assert np.array_equal(r.dump("draw_list"), fa.get("draw_list"))
    assert np.array_equal(r.dump("draw_list"), fa.get("draw_list"))
    assert np.array_equal(r.dump("intersection"), fa.get("intersection"))
    assert np.array_equal(r.render(), fb.get("image"))
    assert np.array_equal(r.dump("draw_list"), fb.get("draw_list"))
    assert np.array_equal(r.render(), fb.get("image"))
    rec = np.array([[(5 << 16) | 3, 7, -1, 0], [(6 << 16) | 100, 200, 0x7F0000FF, 0]], np.int32)
    r.render_draw_list(rec)
    assert np.array_equal(r.dump("draw_list"), rec)
    assert np.array_equal(r.render(), fb.get("image"))
    r.close()
