"""Crossing chains at the lengths where their split over lanes changes, and chains whose crossings all lie at small t,
where neighbouring stretches settle last: every stage against the oracle, bit for bit."""
import pytest

import scenes
from parity_util import compare_all, render_both

pytestmark = pytest.mark.gpu

LENGTHS = [1, 15, 16, 17, 31, 32, 33, 47, 63, 64, 127, 128, 129, 255, 256, 511, 512, 513, 1023, 1024, 1025, 2047]


def lengths_scene(ctype):
    """Paths of one curve each, with about n rows crossed for every n of LENGTHS (upwards and downwards)."""
    b = scenes.Builder(700, 2100)
    for i, n in enumerate(LENGTHS):
        for up in (False, True):
            x = 12.0 * (2 * i + up) + 3.3
            y0, y1 = 7.37, 7.37 + n
            if up:
                y0, y1 = y1, y0
            b.path(rgba=(40, 10 * i, 200, 180))
            h = y1 - y0
            if ctype == scenes.CUBIC:
                pts = [(x, y0), (x + 7.1, y0 + 0.21 * h), (x + 2.3, y0 + 0.7 * h), (x + 9.7, y1)]
            elif ctype == scenes.QUADRIC:
                pts = [(x, y0), (x + 8.7, y0 + 0.4 * h), (x + 3.9, y1)]
            elif ctype == scenes.ARC:
                w = 0.8
                pts = [(x, y0), (w * (x + 9.1), w * (y0 + 0.45 * h)), (x + 5.2, y1), (w, w)]
            else:
                pts = [(x, y0), (x + 6.6, y1)]
            b.curve(ctype, pts)
    return b.arrays()


def small_t_scene(ctype):
    """Curves that leave the canvas far behind: their crossings lie in the first 1/8 to 1/16384 of the piece, or, run
    the other way, in the last."""
    b = scenes.Builder(400, 1100)
    for i, far in enumerate([8.0, 64.0, 1024.0, 16384.0]):
        for back in (False, True):
            x, y1 = 40.0 * (2 * i + back) + 5.5, 1100.0 * far
            if ctype == scenes.CUBIC:
                pts = [(x, -3.7), (x + 9.0, 0.3 * y1), (x + 4.0, 0.66 * y1), (x + 12.0, y1)]
            else:
                pts = [(x, -3.7), (x + 9.0, 0.45 * y1), (x + 12.0, y1)]
            b.path(rgba=(200, 30 * i, 10, 160))
            b.curve(ctype, pts[::-1] if back else pts)
    return b.arrays()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("build,ctype", [
    (lengths_scene, scenes.LINE), (lengths_scene, scenes.QUADRIC), (lengths_scene, scenes.CUBIC),
    (lengths_scene, scenes.ARC), (small_t_scene, scenes.QUADRIC), (small_t_scene, scenes.CUBIC)])
def test_split_chains(gpu, oracle_lib, build, ctype, mode):
    of, r, img = render_both(gpu, oracle_lib, build(ctype), mode)
    compare_all(of, r, img, mode)
    r.close()
