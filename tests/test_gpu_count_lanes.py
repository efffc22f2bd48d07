"""The count pass with eight lanes a curve (up to 16,384 curves) and with one, at the edges of its CTAs and on either side
of that number: lines, quadrics, cubics of up to five pieces, on and off the canvas, every stage against the
oracle."""
import numpy as np
import pytest

import scenes
from parity_util import compare_all, render_both

pytestmark = pytest.mark.gpu


def _scene(n):
    rng = np.random.default_rng(n)
    b = scenes.Builder(120, 90)
    k = 0
    while k < n:
        b.path(rule=k % 2, rgba=(k % 251, 40, 200, 30 + k % 200))
        m = min(5, n - k)
        p0 = start = rng.uniform(-30, 140, 2)
        for i in range(m):
            p3 = start if i == m - 1 and m > 1 else p0 + rng.uniform(-14, 14, 2)
            c1, c2 = p0 + rng.uniform(-25, 25, 2), p3 + rng.uniform(-25, 25, 2)
            kind = (k + i) % 4
            if kind == 0:
                b.curve(scenes.CUBIC, [p0, c1, c2, p3])
            elif kind == 1:
                b.curve(scenes.QUADRIC, [p0, c1, p3])
            elif kind == 2:
                b.curve(scenes.LINE, [p0, p3])
            else:
                b.curve(scenes.CUBIC, [p0, p0 + (40, 0), p0 + (-40, 8), p3])   # turns in x and y
            p0 = p3
        k += m
    return b.arrays()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 16383, 16384, 16385])
def test_counts(gpu, oracle_lib, n, mode):
    of, r, img = render_both(gpu, oracle_lib, _scene(n), mode)
    compare_all(of, r, img, mode)
    r.close()
