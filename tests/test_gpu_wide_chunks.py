"""A pre-sized frame whose first tiles of 64-bit items are chunks of a large path (one path of more than 4,096 records
over a canvas of 16,384 x 8,500 pixels): no kernel of that frame has sorted them when it merges the chunks, and it is run
again.  The images are the oracle's."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

W, H = 16384, 8500


def _scene(spread, n, seed):
    """n small triangles of one path, in no order: over the whole canvas and both side edges, or in a corner of it (by
    whole pixels apart, so that both have about as many records)."""
    rng = np.random.default_rng(seed)
    b = scenes.Builder(W, H).path(rule=0, rgba=(30, 90, 200, 180))
    for i in range(n):
        x, y = int(rng.integers(0, 16300)), int(rng.integers(0, 8480))
        x = -3 if i % 16 == 3 else W - 4 if i % 16 == 9 else x
        if not spread:
            x, y = x % 512 if 0 <= x < 16300 else 77, y % 512
        fx, fy, s = rng.uniform(0, 1), rng.uniform(0, 1), rng.uniform(4, 9)
        b.polygon([(x + fx, y + fy), (x + fx + s, y + fy + 0.3 * s), (x + fx + 0.4 * s, y + fy + s)])
    return b.arrays()


@pytest.mark.parametrize("n", [200, 900, 2600])
def test_first_wide_chunks(gpu, oracle_lib, n):
    near, far = _scene(False, n, 3), _scene(True, n, 3)
    want = [oracle_lib.Frame(scenes.to_oracle(d), mode=1).get("image") for d in (near, far)]
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, W, H)
    out = np.empty((H, W, 4), np.uint8)
    for d, img, wide in ((near, 0, False), (near, 0, False), (far, 1, True), (far, 1, True), (near, 0, False)):
        r.loadVG(scenes.to_container(d))
        assert np.array_equal(r.render(out), want[img])
        tiles = r.sort_tiles()
        assert (tiles[1] > 0) == wide and tiles[0] > 0
    assert r.stats()["reruns"] == 1 and r.stats()["n_intersections"] > 4096
    r.close()
