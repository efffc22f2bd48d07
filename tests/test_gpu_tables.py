"""The tables a frame builds on the device (record offsets, paths' sort segments and tiles, row starts) at the edges of
the CTAs that build them, paths without curves among them, and a pre-sized frame that meets its first sort tile of
64-bit items."""
import numpy as np
import pytest

import scenes
from parity_util import compare_all, render_both
from test_gpu_segsort import _scattered

pytestmark = pytest.mark.gpu


def _sparse(n_paths, seed, w=160, h=130):
    """n_paths paths of which about a third have no curves, the first and last ones among them."""
    rng = np.random.default_rng(seed)
    b = scenes.Builder(w, h)
    for i in range(n_paths):
        b.path(rule=i % 2, rgba=(i % 251, 90, 200, 80 + i % 170))
        if n_paths > 2 and (i < 2 or i >= n_paths - 2 or rng.uniform() < 0.3):
            continue
        x, y, s = rng.uniform(-5, w), rng.uniform(-5, h), rng.uniform(0.5, 12)
        b.polygon([(x, y), (x + s, y + 0.3 * s), (x + 0.4 * s, y + s)])
    return b.arrays()


@pytest.mark.parametrize("n_paths", [1, 2, 255, 256, 257, 511, 513, 1024, 1500])
def test_paths_without_curves(gpu, oracle_lib, n_paths):
    d = _sparse(n_paths, n_paths)
    of, r, img = render_both(gpu, oracle_lib, d, 1)
    compare_all(of, r, img, 1)
    r.close()
    r = gpu.ScanlineVGRasterizer(mode=1)   # the per-path sort (kept stages use the radix sort); exact, then pre-sized
    r.initialize(None, d["width"], d["height"])
    r.loadVG(scenes.to_container(d))
    for _ in range(2):
        assert np.array_equal(r.render(), of.get("image"))
    r.close()


@pytest.mark.parametrize("curves", [1023, 1024, 1025, 2049])
def test_offset_scan_tiles(gpu, oracle_lib, curves):
    b = scenes.Builder(90, 70)
    for i in range(curves):
        if i % 7 == 0:
            b.path(rule=i % 2, rgba=(i % 251, 10, 20, 120))
        x, y = 1.37 * (i % 61), 1.91 * (i % 37)
        b.curve(scenes.LINE, [(x, y), (x + 2.5, y + 1.2 + 0.01 * (i % 11))])
    of, r, img = render_both(gpu, oracle_lib, b.arrays(), 1)
    compare_all(of, r, img, 1)
    r.close()


@pytest.mark.parametrize("h", [1, 1023, 1024, 1025, 3000])
def test_row_starts(gpu, oracle_lib, h):
    d = _sparse(400, h, w=64, h=h)
    of, r, img = render_both(gpu, oracle_lib, d, 1)
    compare_all(of, r, img, 1)
    r.close()


def test_presized_frame_with_its_first_wide_tile(gpu, oracle_lib):
    """The tile sort of a pre-sized frame launches no 64-bit pass when the last frame needed none; a frame that does
    is run again.  Same curve and path counts throughout, so that the second frame is pre-sized."""
    n = 3000
    wide = _scattered(4096, 4096, n, 6)
    fifth, dot = (dict(wide, position=(wide["position"] * np.float32(f)).astype(np.float32)) for f in (0.2, 0.01))
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, 4096, 4096)
    # (a fifth of the canvas still needs them; a hundredth, 41 pixels, does not)
    for d, is_wide in ((dot, False), (dot, False), (wide, True), (wide, True), (fifth, True), (dot, False)):
        r.loadVG(scenes.to_container(d))
        img = r.render()
        assert (r.sort_tiles()[1] > 0) == is_wide
        assert np.array_equal(img, oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image"))
    r.close()
